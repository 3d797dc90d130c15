"""Device weights read in place off a 16-byte boundary: at an 8-byte boundary
commitments, claims and proofs are the oracle's, also where padding runs hold
whole 16-byte units (a 300 x 1000 matrix has a bucket of width 128 with 104
real columns), and nonzero padding is still found; anything less aligned is
refused on the host.  Needs a B200."""
import numpy as np
import pytest
import torch

import oracle
import parcomm_b200 as qf
from parcomm_b200 import layout

pytestmark = pytest.mark.gpu

FIELDS = {"f65521": (qf.FIELD_F65521, np.int8), "koalabear": (qf.FIELD_KOALABEAR, np.int16)}
SHAPES = [(300, 1000), (129, 65), (1, 21), (300, 700)]


def shifted(bva, entries):
    """`bva` on the GPU, `entries` past an aligned address."""
    t = torch.zeros(bva.size + entries, dtype=torch.from_numpy(bva).dtype, device="cuda")
    t[entries:].copy_(torch.from_numpy(bva))
    return t[entries:]


@pytest.mark.parametrize("field", FIELDS)
@pytest.mark.parametrize("chunk_log, packed_log", [(16, 4), (14, 6), (16, 1)])
def test_weights_at_an_8_byte_boundary(field, chunk_log, packed_log):
    number, dtype = FIELDS[field]
    rng = np.random.default_rng(chunk_log + packed_log)
    mats = [rng.integers(-100, 100, s, dtype=dtype) for s in SHAPES]
    p = qf.Parameters(SHAPES, qf.Config(chunk_log=chunk_log, packed_log=packed_log), field=number)
    bva = layout.encode(p.shapes, mats)
    o_roots, o_claims, o_proof, _ = oracle.prove(p.shapes, chunk_log, packed_log, bva, field=field)
    weights = shifted(bva, 8 // bva.itemsize)
    assert weights.data_ptr() % 16 == 8
    c = p.commit_recomputed(weights)
    assert b"".join(c.roots) == o_roots
    claims = p.evaluate_claims(c, p.benchmark_points(c.roots))
    assert qf.claims_to_bytes(claims) == o_claims
    proof, _ = p.prove(c, claims)
    assert proof.to_bytes() == o_proof
    c.close()
    # One nonzero entry at each end and inside of the first padding run.
    for at in (104, 115, 127):
        bad = bva.copy()
        wide = next(b for b in layout.buckets(p.shapes)[0] if b.physical_cols == 104)
        bad[wide.offset + at] = 1
        with pytest.raises(qf.QfError, match="nonzero boundary padding"):
            p.commit_recomputed(shifted(bad, 8 // bva.itemsize))


@pytest.mark.parametrize("field", FIELDS)
def test_less_aligned_weights_are_refused(field):
    number, dtype = FIELDS[field]
    p = qf.Parameters(SHAPES, qf.Config(chunk_log=14, packed_log=4), field=number)
    bva = np.zeros(p.active, dtype=dtype)
    for entries in (1, 2, 3, 4, 7) if bva.itemsize == 1 else (1, 2, 3):
        weights = shifted(bva, entries)
        with pytest.raises(qf.QfError, match="8-byte boundary"):
            p.commit_recomputed(weights)
        if field == "f65521":
            root = torch.zeros(32, dtype=torch.uint8, device="cuda")
            with pytest.raises(qf.QfError, match="8-byte boundary"):
                p.block_root_noalloc(weights, 0, root, torch.cuda.current_stream().cuda_stream)
            torch.cuda.synchronize()
    c = p.commit(shifted(bva, 1), on_device=True)  # copied: any address
    c.close()

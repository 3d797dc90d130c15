"""Blocks of 2^7 to 2^14 packed elements, around the sizes up to which one tile
takes the whole Mobius transform (2^11, KoalaBear 2^12): roots, claims and proofs against the
oracle, and the root of each block without allocation.  Needs a B200."""
import numpy as np
import pytest
import torch

import oracle
import parcomm_b200 as qf
from parcomm_b200 import layout

pytestmark = pytest.mark.gpu

FIELDS = {"f65521": (qf.FIELD_F65521, np.int8, 3), "koalabear": (qf.FIELD_KOALABEAR, np.int16, 2)}


@pytest.mark.parametrize("field, log_elements", [("f65521", n) for n in range(7, 15)] + [("koalabear", n) for n in range(8, 15)])
def test_small_blocks(field, log_elements):
    number, dtype, lane_log = FIELDS[field]
    chunk_log = log_elements + lane_log
    rng = np.random.default_rng(log_elements)
    shapes = [(3 << (chunk_log - 8), 256), (1, 300)]
    mats = [rng.integers(-128, 128, s, dtype=dtype) for s in shapes]
    p = qf.Parameters(shapes, qf.Config(chunk_log=chunk_log, packed_log=4), field=number)
    bva = layout.encode(p.shapes, mats)
    o_roots, o_claims, o_proof, _ = oracle.prove(p.shapes, chunk_log, 4, bva, field=field)
    c = p.commit(bva)
    assert b"".join(c.roots) == o_roots
    if field == "f65521":
        weights = torch.from_numpy(bva).cuda()
        root = torch.zeros(32, dtype=torch.uint8, device="cuda")
        for b in range(p.blocks):
            p.block_root_noalloc(weights, b, root, torch.cuda.current_stream().cuda_stream)
            assert bytes(root.cpu().numpy()) == c.roots[b]
    claims = p.evaluate_claims(c, p.benchmark_points(c.roots))
    assert qf.claims_to_bytes(claims) == o_claims
    proof, _ = p.prove(c, claims)
    assert proof.to_bytes() == o_proof
    c.close()

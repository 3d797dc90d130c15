"""Claims and proofs whose lane projections meet the edges of the tensor-core
kernel (groups of eight tiles of 4096 rows, 32 rows per step): one row, rows
around 32 and 256, one tile, eight and nine tiles, each against the oracle; and
claims on weights at an 8-byte boundary, which keep the dp4a kernel (a proof
needs 16-byte rows).  Needs a B200."""
import numpy as np
import pytest
import torch

import oracle
import parcomm_b200 as qf
from parcomm_b200 import layout

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shapes", [
    [(1, 16), (31, 16), (33, 16), (5, 3)],
    [(255, 16), (257, 16), (64, 64)],
    [(4096, 16), (4097, 16)],
    [(32768, 16), (1, 1)],
    [(36864, 16), (300, 700)],
])
def test_projections_at_group_edges(shapes):
    rng = np.random.default_rng(len(shapes) + shapes[0][0])
    mats = [rng.integers(-128, 128, s, dtype=np.int8) for s in shapes]
    mats[0][:] = -128
    p = qf.Parameters(shapes, qf.Config(chunk_log=16, packed_log=4))
    bva = layout.encode(p.shapes, mats)
    o_roots, o_claims, o_proof, _ = oracle.prove(p.shapes, 16, 4, bva)
    odd = torch.zeros(p.active + 8, dtype=torch.int8, device="cuda")
    odd[8:].copy_(torch.from_numpy(bva))
    handles = [(p.commit(bva), True)]
    if p.blocks > 1:
        handles += [(p.commit_recomputed(bva), True), (p.commit_recomputed(odd[8:]), False)]
    for c, prove in handles:
        assert b"".join(c.roots) == o_roots
        claims = p.evaluate_claims(c, p.benchmark_points(c.roots))
        assert qf.claims_to_bytes(claims) == o_claims
        if prove:
            proof, _ = p.prove(c, claims)
            assert proof.to_bytes() == o_proof
        c.close()

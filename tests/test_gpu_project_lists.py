"""Claims and proofs over lists of more terms than the tensor-core projection has
CTAs, so that each CTA looks its first list entry up: many small matrices of one
size, and ragged ones whose terms run from one row to several tiles, resident and
streamed block by block, each against the oracle.  Needs a B200."""
import numpy as np
import pytest

import oracle
import parcomm_b200 as qf
from parcomm_b200 import layout

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shapes, chunk_log", [
    ([(16, 16)] * 149, 14),
    ([(16, 16)] * 700 + [(1, 16)] * 9, 16),
    ([(64, 64)] * 300 + [(37, 50)] * 40, 17),
    ([(500, 1000)] * 3 + [(90, 72)] * 60 + [(5, 3)] * 20, 18),
    ([(1100, 1024)] + [(16, 48)] * 150, 17),
    ([(16, 16)] * 3 + [(5000, 1024)], 20),
])
def test_lists_of_many_terms(shapes, chunk_log):
    rng = np.random.default_rng(len(shapes))
    mats = [rng.integers(-128, 128, s, dtype=np.int8) for s in shapes]
    p = qf.Parameters(shapes, qf.Config(chunk_log=chunk_log, packed_log=4))
    bva = layout.encode(p.shapes, mats)
    o_roots, o_claims, o_proof, _ = oracle.prove(p.shapes, chunk_log, 4, bva)
    handles = [p.commit(bva)] + ([p.commit_recomputed(bva)] if p.blocks > 1 else [])
    for c in handles:
        assert b"".join(c.roots) == o_roots
        claims = p.evaluate_claims(c, p.benchmark_points(c.roots))
        assert qf.claims_to_bytes(claims) == o_claims
        proof, _ = p.prove(c, claims)
        assert proof.to_bytes() == o_proof
        c.close()

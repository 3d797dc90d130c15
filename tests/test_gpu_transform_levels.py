"""The tensor-core transform passes at every number of strided levels: roots of
blocks of 2^28 and 2^29 weights (seven and eight levels), half live, and proofs
over two blocks of 2^26 and 2^27 (five and six), whose folded codeword starts
from an element vector, each against the oracle.  (Nine levels: the chunk-30
parity tests.)  Needs a B200."""
import numpy as np
import pytest
import torch

import oracle
import parcomm_b200 as qf

pytestmark = pytest.mark.gpu


def weights(p, seed):
    rng = np.random.default_rng(seed)
    bva = rng.integers(-128, 128, p.active, dtype=np.int8)
    bva[:4096] = -128
    return bva


@pytest.mark.parametrize("chunk_log", [28, 29])
def test_roots_at_seven_and_eight_levels(chunk_log):
    p = qf.Parameters([((1 << (chunk_log - 13)) + 1, 4096)], qf.Config(chunk_log=chunk_log, packed_log=4))
    assert p.blocks == 1
    bva = weights(p, chunk_log)
    c = p.commit(bva)
    assert b"".join(c.roots) == oracle.commit_roots(p.shapes, chunk_log, 4, bva)[:32]
    c.close()


@pytest.mark.parametrize("chunk_log", [26, 27])
def test_folded_codewords_at_five_and_six_levels(chunk_log):
    p = qf.Parameters([(1 << (chunk_log - 12), 4096), (1, 8192)], qf.Config(chunk_log=chunk_log, packed_log=4))
    assert p.blocks == 2
    bva = weights(p, chunk_log)
    o_roots, o_claims, o_proof, _ = oracle.prove(p.shapes, chunk_log, 4, bva)
    c = p.commit(torch.from_numpy(bva).cuda(), on_device=True)
    assert b"".join(c.roots) == o_roots
    claims = p.evaluate_claims(c, p.benchmark_points(c.roots))
    assert qf.claims_to_bytes(claims) == o_claims
    proof, _ = p.prove(c, claims)
    assert proof.to_bytes() == o_proof
    c.close()

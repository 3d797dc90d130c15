"""Block roots where the tensor-core transform passes begin and change form:
the largest block of the butterfly passes (chunk 25), the smallest of the
tensor-core ones (chunk 26: five strided levels, one stage), six strided levels
(chunk 27: two stages), each against the oracle.  The last block is partly
live, with a ragged end, and in the recompute mode the weights are read in
place at an 8-byte boundary that is no 16-byte one.  Needs a B200."""
import numpy as np
import pytest
import torch

import oracle
import parcomm_b200 as qf

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("chunk_log", [25, 26, 27])
def test_roots_at_the_edges_of_the_tensor_core_passes(chunk_log):
    shapes = [(1 << (chunk_log - 12), 4096), (1 << (chunk_log - 15), 4096), (1, 21)]
    p = qf.Parameters(shapes, qf.Config(chunk_log=chunk_log, packed_log=4))
    rng = np.random.default_rng(chunk_log)
    bva = rng.integers(-128, 128, p.active, dtype=np.int8)
    bva[:4096] = -128
    want = oracle.commit_roots(p.shapes, chunk_log, 4, bva)[: 32 * p.blocks]
    c = p.commit(bva)
    assert b"".join(c.roots) == want
    c.close()
    odd = torch.zeros(p.active + 8, dtype=torch.int8, device="cuda")
    odd[8:].copy_(torch.from_numpy(bva))
    assert odd[8:].data_ptr() % 16 == 8
    c = p.commit_recomputed(odd[8:])
    assert b"".join(c.roots) == want
    c.close()

"""Long runs of the tensor-core projections, past what the oracle takes in a
test: every CTA reads the equality projection's sums four times (2^24 elements,
221 or 222 stages of 512 in reads of 64, both TMEM buffers taken again) and adds
the last block's ragged end, and takes six or seven groups of the term
projection.  The other kernels of the same sums are the reference: one block per
launch for the equality projection, weights at an 8-byte boundary for the
claims; and the proof verifies.  Needs a B200."""
import numpy as np
import pytest
import torch

import parcomm_b200 as qf
from parcomm_b200 import layout

pytestmark = pytest.mark.gpu

FIELDS = {"f65521": (qf.FIELD_F65521, np.int8, 27), "koalabear": (qf.FIELD_KOALABEAR, np.int16, 26)}


@pytest.mark.parametrize("field", FIELDS)
def test_many_groups_per_cta(field):
    number, dtype, chunk_log = FIELDS[field]
    low = np.iinfo(dtype).min
    shapes = [(4 << (chunk_log - 12), 4096), (1, 70001)]
    p = qf.Parameters(shapes, qf.Config(chunk_log=chunk_log, packed_log=4), field=number)
    g = torch.Generator(device="cuda")
    g.manual_seed(chunk_log)
    step = 8 // np.dtype(dtype).itemsize
    store = torch.zeros(p.active + step, dtype=torch.from_numpy(np.zeros(1, dtype)).dtype, device="cuda")
    weights = store[step:]
    n = shapes[0][0] * shapes[0][1]
    weights[:n].random_(low, -low, generator=g)
    weights[: n // 8] = low
    row = next(b for b in layout.buckets(p.shapes)[0] if b.matrix == 1)
    weights[row.offset: row.offset + row.physical_cols].random_(low, -low, generator=g)
    c = p.commit(weights, on_device=True)
    points = p.benchmark_points(c.roots)
    claims = p.evaluate_claims(c, points)
    proof, _ = p.open(c, claims)
    p.verify(c.roots, claims, proof)
    qf.kernel_option("per_matrix", 1)
    try:
        alone, _ = p.open(c, claims)
    finally:
        qf.kernel_option("per_matrix", 0)
    assert alone.to_bytes() == proof.to_bytes()
    roots = c.roots
    c.close()
    assert weights.data_ptr() % 16 == 8
    r = p.commit_recomputed(weights)
    assert r.roots == roots
    assert qf.claims_to_bytes(p.evaluate_claims(r, points)) == qf.claims_to_bytes(claims)
    r.close()

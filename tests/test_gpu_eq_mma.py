"""Proofs whose equality projections meet the edges of the tensor-core kernel
(four blocks and more; 2^9 to 2^14 packed elements, or 2^20 and more, in stages
of 512 elements, eight blocks a launch): the sizes around each line, three,
four, eight and nine blocks, and last blocks whose live part ends inside a
16-byte unit, in a stage and before one, each against the oracle.  2^20 elements
are 14 stages for each CTA and its five buffers.  Needs a B200."""
import numpy as np
import pytest

import oracle
import parcomm_b200 as qf
from parcomm_b200 import layout

pytestmark = pytest.mark.gpu

FIELDS = {"f65521": (qf.FIELD_F65521, np.int8, 3), "koalabear": (qf.FIELD_KOALABEAR, np.int16, 2)}


@pytest.mark.parametrize("field", FIELDS)
@pytest.mark.parametrize("log_elements, blocks, live", [
    (8, 4, 77),       # of the last block: entries live
    (9, 4, 1003),
    (12, 3, 5),
    (12, 4, 4096),
    (12, 8, 4099),
    (12, 9, 8191),
    (14, 12, 19),
    (15, 4, 70001),
    (20, 4, 1234567),
])
def test_projections_at_stage_and_block_edges(field, log_elements, blocks, live):
    number, dtype, lane_log = FIELDS[field]
    chunk_log = log_elements + lane_log
    low = np.iinfo(dtype).min
    rng = np.random.default_rng(1000 * log_elements + blocks)
    shapes = [((blocks - 1) << (chunk_log - 8), 256)] if blocks > 1 else []
    shapes.append((1, live))
    mats = [rng.integers(low, -low, s, dtype=dtype) for s in shapes]
    mats[0][: max(1, mats[0].shape[0] // 2)] = low
    p = qf.Parameters(shapes, qf.Config(chunk_log=chunk_log, packed_log=4), field=number)
    bva = layout.encode(p.shapes, mats)
    o_roots, o_claims, o_proof, _ = oracle.prove(p.shapes, chunk_log, 4, bva, field=field)
    c = p.commit(bva)
    assert b"".join(c.roots) == o_roots
    claims = p.evaluate_claims(c, p.benchmark_points(c.roots))
    assert qf.claims_to_bytes(claims) == o_claims
    proof, _ = p.prove(c, claims)
    assert proof.to_bytes() == o_proof
    c.close()

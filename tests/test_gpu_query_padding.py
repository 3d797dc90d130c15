"""Proofs of matrices whose width is no power of two and whose padding is cut
into several column rectangles over the same rows, more rows than one CTA of
the query fold takes, each against the oracle.  Needs a B200."""
import numpy as np
import pytest

import oracle
import parcomm_b200 as qf
from parcomm_b200 import layout

pytestmark = pytest.mark.gpu

FIELDS = {"f65521": (qf.FIELD_F65521, np.int8), "koalabear": (qf.FIELD_KOALABEAR, np.int16)}


@pytest.mark.parametrize("field", FIELDS)
@pytest.mark.parametrize("shapes, chunk_log, packed_log", [
    ([(10, 4884), (6, 8192), (15, 3489), (1397, 38), (829, 64), (51, 1024)], 17, 6),
    ([(7, 5002), (2012, 18), (2, 16384), (18, 1911), (2, 16384), (26, 1378)], 14, 6),
    ([(126, 1024), (1566, 83), (78, 1650), (94, 1381), (252, 514), (7, 16384)], 15, 4),
    ([(6497, 949)], 20, 4),
])
def test_proofs_with_several_padding_rectangles(field, shapes, chunk_log, packed_log):
    number, dtype = FIELDS[field]
    rng = np.random.default_rng(chunk_log)
    mats = [rng.integers(-100, 100, s, dtype=dtype) for s in shapes]
    p = qf.Parameters(shapes, qf.Config(chunk_log=chunk_log, packed_log=packed_log), field=number)
    bva = layout.encode(p.shapes, mats)
    o_roots, o_claims, o_proof, _ = oracle.prove(p.shapes, chunk_log, packed_log, bva, field=field)
    c = p.commit(bva)
    assert b"".join(c.roots) == o_roots
    claims = p.evaluate_claims(c, p.benchmark_points(c.roots))
    assert qf.claims_to_bytes(claims) == o_claims
    proof, _ = p.prove(c, claims)
    assert proof.to_bytes() == o_proof
    c.close()

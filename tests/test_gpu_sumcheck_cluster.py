"""Sumchecks of a cluster of CTAs (vectors of 2^9 to 2^15 elements whose last
round leaves at least one element a CTA) and of one CTA (smaller ones): whole
proofs whose sumchecks meet the edges of both, against the oracle."""
import numpy as np
import pytest

from whirplonk_b200 import ProtocolParameters, prove_once, sample_goldilocks
from whirplonk_b200.whir import ENGINE_ID_BLAKE3, FIELD_GOLDILOCKS1

pytestmark = pytest.mark.gpu


# the rounds' vectors have 2^(n - k), 2^(n - 2k), ... elements, folded k times
@pytest.mark.parametrize("n,k,rho", [
    (19, 4, 1),  # 2^15 (the largest), 2^11, one CTA at 2^7
    (14, 5, 2),  # 2^9: the smallest of a cluster
    (15, 6, 1),  # 2^9 folded to 2^3: an element a CTA
    (15, 3, 1),  # 2^12, 2^9 folded to 2^6
    (17, 1, 1),  # single rounds of 2^16 (a launch each) down to the final vector
])
def test_proofs_match_oracle(gpu_ctx, oracle, n, k, rho):
    params = ProtocolParameters.cli(folding_factor=k, log_inv_rate=rho)
    coeffs = sample_goldilocks(710 + n + k, 1 << n)
    pts = sample_goldilocks(720 + n, 3 * n).reshape(1, n, 3)
    ev = np.array(gpu_ctx.mle_evaluate(coeffs, pts), dtype=np.uint64).reshape(1, 3)
    got = prove_once(n, params, coeffs, pts, ev, ctx=gpu_ctx)[:2]
    assert got == oracle.prove(n, k, rho, 100, 20, pts, coeffs, ev)


def test_base_field_target(gpu_ctx, oracle):
    n, k, rho = 17, 4, 1
    params = ProtocolParameters(False, rho, k, k, 32, 0, 1, ENGINE_ID_BLAKE3)
    coeffs = sample_goldilocks(741, 1 << n)
    pts = sample_goldilocks(742, 3 * n).reshape(1, n, 3)
    pts[:, :, 1:] = 0
    ev = np.array(gpu_ctx.mle_evaluate(coeffs, pts), dtype=np.uint64).reshape(1, 3)
    got = prove_once(n, params, coeffs, pts, ev, ctx=gpu_ctx, target_field=FIELD_GOLDILOCKS1)[:2]
    assert got == oracle.prove_forms(n, k, rho, 32, 0, [("mle", pts[0])], coeffs, ev, field1=True)

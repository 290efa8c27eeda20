"""The STIR covector update as an 8-bit contraction (vectors of 2^14 elements and
more): whole proofs whose rounds meet it at its smallest size, at odd splits,
for all three target fields' shapes of points, against the oracle."""
import numpy as np
import pytest

from whirplonk_b200 import ProtocolParameters, prove_once, sample_goldilocks
from whirplonk_b200.whir import ENGINE_ID_BLAKE3, FIELD_GOLDILOCKS1

pytestmark = pytest.mark.gpu


# folding k: the rounds' vectors have 2^(n - k), 2^(n - 2k), ... elements
@pytest.mark.parametrize("n,k,rho", [(18, 4, 1), (17, 3, 1), (17, 2, 2), (16, 1, 1)])
def test_proofs_match_oracle(gpu_ctx, oracle, n, k, rho):
    params = ProtocolParameters.cli(folding_factor=k, log_inv_rate=rho)
    coeffs = sample_goldilocks(610 + n + k, 1 << n)
    pts = sample_goldilocks(620 + n, 3 * n).reshape(1, n, 3)
    ev = np.array(gpu_ctx.mle_evaluate(coeffs, pts), dtype=np.uint64).reshape(1, 3)
    got = prove_once(n, params, coeffs, pts, ev, ctx=gpu_ctx)[:2]
    assert got == oracle.prove(n, k, rho, 100, 20, pts, coeffs, ev)


def test_no_out_of_domain_points(gpu_ctx, oracle):
    """Unique decoding: in-domain points only."""
    n, k, rho = 17, 3, 2
    params = ProtocolParameters(True, rho, k, k, 100, 20, 1, ENGINE_ID_BLAKE3)
    coeffs = sample_goldilocks(631, 1 << n)
    pts = sample_goldilocks(632, 3 * n).reshape(1, n, 3)
    ev = np.array(gpu_ctx.mle_evaluate(coeffs, pts), dtype=np.uint64).reshape(1, 3)
    got = prove_once(n, params, coeffs, pts, ev, ctx=gpu_ctx)[:2]
    assert got == oracle.prove_forms(n, k, rho, 100, 20, [("mle", pts[0])], coeffs, ev, unique=True)


def test_base_field_target(gpu_ctx, oracle):
    n, k, rho = 17, 3, 1
    params = ProtocolParameters(False, rho, k, k, 32, 0, 1, ENGINE_ID_BLAKE3)
    coeffs = sample_goldilocks(641, 1 << n)
    pts = sample_goldilocks(642, 3 * n).reshape(1, n, 3)
    pts[:, :, 1:] = 0
    ev = np.array(gpu_ctx.mle_evaluate(coeffs, pts), dtype=np.uint64).reshape(1, 3)
    got = prove_once(n, params, coeffs, pts, ev, ctx=gpu_ctx, target_field=FIELD_GOLDILOCKS1)[:2]
    assert got == oracle.prove_forms(n, k, rho, 32, 0, [("mle", pts[0])], coeffs, ev, field1=True)


# the single-launch form: vectors of 2^13 elements and fewer
@pytest.mark.parametrize("n,k,rho", [
    (17, 4, 1),  # 2^13 (the largest), 2^9, 2^5 (half a CTA's elements)
    (14, 1, 1),  # 2^13, 2^12, ... down to one element
    (12, 3, 3),  # few points: fewer than the warps
])
def test_small_vectors(gpu_ctx, oracle, n, k, rho):
    params = ProtocolParameters.cli(folding_factor=k, log_inv_rate=rho)
    coeffs = sample_goldilocks(650 + n + k, 1 << n)
    pts = sample_goldilocks(660 + n, 3 * n).reshape(1, n, 3)
    ev = np.array(gpu_ctx.mle_evaluate(coeffs, pts), dtype=np.uint64).reshape(1, 3)
    got = prove_once(n, params, coeffs, pts, ev, ctx=gpu_ctx)[:2]
    assert got == oracle.prove(n, k, rho, 100, 20, pts, coeffs, ev)

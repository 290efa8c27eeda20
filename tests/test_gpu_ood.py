"""Out-of-domain value of one vector at one point in one launch: whole proofs
whose vectors are smaller than a part, meet each part length, and take several
parts a warp, against the oracle."""
import numpy as np
import pytest

from whirplonk_b200 import ProtocolParameters, prove_once, sample_goldilocks

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,k,rho", [
    (7, 1, 1),   # 2^7 (one part of the smallest length), 2^6, 2^5, ...
    (20, 2, 1),  # 2^20: parts of 2^8; 2^18, 2^16, ...: parts of 2^7
    (21, 4, 1),  # parts of 2^9
    (23, 4, 1),  # parts of 2^10, up to two a warp
])
def test_proofs_match_oracle(gpu_ctx, oracle, n, k, rho):
    params = ProtocolParameters.cli(folding_factor=k, log_inv_rate=rho)
    coeffs = sample_goldilocks(810 + n + k, 1 << n)
    pts = sample_goldilocks(820 + n, 3 * n).reshape(1, n, 3)
    ev = np.array(gpu_ctx.mle_evaluate(coeffs, pts), dtype=np.uint64).reshape(1, 3)
    got = prove_once(n, params, coeffs, pts, ev, ctx=gpu_ctx)[:2]
    assert got == oracle.prove(n, k, rho, 100, 20, pts, coeffs, ev)

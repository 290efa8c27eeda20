"""Sumchecks that fold their whole vector: the final sumcheck of a configuration
with a long final vector (2^8 to 2^13 elements down to one), against the oracle;
up to 2^12 elements the rounds are one launch."""
import numpy as np
import pytest

from whirplonk_b200 import Config, MultilinearExtension, ProverState, _lib, sample_goldilocks
from whirplonk_b200.whir import ENGINE_ID_BLAKE3, FIELD_GOLDILOCKS1, FIELD_GOLDILOCKS3, DomainSeparator

pytestmark = pytest.mark.gpu
DS = bytes(range(96))


def config(n, k0, field):
    """No rounds: 2^n coefficients folded k0 times, then the final vector to one element."""
    size, m = 1 << n, 1 << (n - k0)
    c = _lib.WhirConfig()
    c.field = field
    c.batch_size = 1
    for i, b in enumerate(ENGINE_ID_BLAKE3):
        c.hash_id[i] = b
    c.initial_committer = _lib.IrsConfig(size, 2 * m, 1 << k0, 5, 1)
    c.initial_sumcheck = _lib.SumcheckConfig(k0, _lib.NO_POW)
    c.initial_skip_pow = _lib.NO_POW
    c.num_rounds = 0
    c.final_sumcheck = _lib.SumcheckConfig(n - k0, _lib.NO_POW)
    c.final_pow = _lib.NO_POW
    words = [size, 2 * m, 1 << k0, 5, 1, k0, _lib.NO_POW, _lib.NO_POW, 0, n - k0, _lib.NO_POW, _lib.NO_POW]
    return Config.custom(c), words


def prove(gpu_ctx, n, k0, field):
    """((narg, hints), oracle's inputs, kernels launched by the prove call)."""
    cfg, words = config(n, k0, field)
    coeffs = sample_goldilocks(9100 + 20 * n + k0, 1 << n)
    pt = sample_goldilocks(9200 + n, 3 * n).reshape(n, 3)
    if field == FIELD_GOLDILOCKS1:
        pt[:, 1:] = 0
    ev = np.array(gpu_ctx.mle_evaluate(coeffs, pt), dtype=np.uint64).reshape(1, 3)
    ps = ProverState.from_ds(DomainSeparator(DS[:64], DS[64:]), b"", gpu_ctx)
    w = cfg.commit(ps, coeffs)
    before = gpu_ctx.launch_count()
    cfg.prove(ps, coeffs, [w], [MultilinearExtension(pt)], [tuple(ev[0])])
    launched = gpu_ctx.launch_count() - before
    return ps.proof(), (words, [("mle", pt)], coeffs, ev), launched


@pytest.mark.parametrize("field", [FIELD_GOLDILOCKS3, FIELD_GOLDILOCKS1])
@pytest.mark.parametrize("n,k0", [(8, 0), (9, 0), (12, 0), (13, 4), (16, 4), (13, 1), (13, 0)])
def test_proofs_match_oracle(gpu_ctx, oracle, n, k0, field):
    got, (words, forms, coeffs, ev), _ = prove(gpu_ctx, n, k0, field)
    want = oracle.prove_config(words, DS, forms, coeffs, ev, deg=3 if field == FIELD_GOLDILOCKS3 else 1)
    assert got == want[:2]


def test_one_launch(gpu_ctx):
    launched = {n: prove(gpu_ctx, n, 0, FIELD_GOLDILOCKS3)[2] for n in (8, 9, 10, 11, 12)}
    assert len(set(launched.values())) == 1, launched

"""A zero-knowledge witness in a recycled device block: whatever the block held
before, the proof is the reference's.  Every ticket and counter that a kernel of
the two inner proofs counts on starts at zero by the commit's own doing."""
import ctypes
import hashlib
import json
import os

import pytest

from tests.zk_cases import case_config, case_params, case_seed, case_statement
from whirplonk_b200 import Context, _lib
from whirplonk_b200.zk import prove_zk_once

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))
ZK = json.load(open(os.path.join(HERE, "golden", "reference_proofs.json")))["zk"]


def check_proof(ctx, case):
    polys, forms, evals = case_statement(case)
    narg, hints = prove_zk_once(case["n"], case_params(case), polys, forms, evals, case_seed(case), ctx=ctx,
                                config=case_config(case))
    assert hashlib.sha256(narg).hexdigest() == case["narg_sha256"]
    assert hashlib.sha256(hints).hexdigest() == case["hints_sha256"]


@pytest.mark.parametrize("byte", [0xFF, 0x03])
@pytest.mark.parametrize("case", ZK, ids=lambda c: f"n{c['n']}_s{c['seed']}")
def test_recycled_block(case, byte):
    ctx = Context(0)
    try:
        check_proof(ctx, case)
        blocks = ctypes.c_size_t()
        _lib.check(_lib.load().whirgpu_debug_fill_zk_pool(ctx.handle, byte, ctypes.byref(blocks)), ctx.handle)
        assert blocks.value == 1  # the first proof's, taken again by the second
        check_proof(ctx, case)
    finally:
        ctx.close()

"""A bounded wait that runs out inside an encode's or a commitment's kernels is
reported by the call it belongs to, once, and by no other."""
import numpy as np
import pytest

from whirplonk_b200 import Context, _lib, sample_goldilocks
from whirplonk_b200._lib import E_DEVICE, WhirGpuError
from whirplonk_b200.rs import rs_commit_batch, rs_encode, rs_encode_status

pytestmark = pytest.mark.gpu
LOG_LEN, LOG_EXP, LOG_DEPTH = 12, 2, 4


@pytest.fixture
def ctx():
    c = Context(0)
    yield c
    c.close()


def expire(ctx, commit):
    _lib.check(_lib.load().whirgpu_debug_expire_wait(ctx.handle, commit), ctx.handle)


def encode(ctx, v):
    import torch

    dv = torch.from_numpy(v.view(np.int64)).cuda()
    tmp = torch.empty(v.size << LOG_EXP, dtype=torch.int64, device="cuda")
    out = torch.empty_like(tmp)
    torch.cuda.synchronize()
    try:
        rs_encode(ctx, dv.data_ptr(), 1, LOG_LEN, LOG_EXP, LOG_DEPTH, tmp.data_ptr(), out.data_ptr())
    finally:
        torch.cuda.synchronize()
    return out.cpu().numpy().view(np.uint64).reshape(1 << LOG_DEPTH, -1)


def test_encode_reports_once(ctx, oracle):
    v = sample_goldilocks(3301, 1 << LOG_LEN)
    N = (v.size >> LOG_DEPTH) << LOG_EXP
    rs_encode_status(ctx)  # nothing to report
    expire(ctx, 0)
    assert rs_commit_batch(ctx, v, LOG_EXP, LOG_DEPTH)[0] == oracle.rs_commit_root(v, N, 1 << LOG_DEPTH)  # not its own
    with pytest.raises(WhirGpuError) as e:
        rs_encode_status(ctx)
    assert e.value.status == E_DEVICE
    rs_encode_status(ctx)
    expire(ctx, 0)
    with pytest.raises(WhirGpuError) as e:  # the next encode reports it, too
        encode(ctx, v)
    assert e.value.status == E_DEVICE
    assert np.array_equal(encode(ctx, v), oracle.rs_encode_base(v, N, 1 << LOG_DEPTH).T)
    rs_encode_status(ctx)


def test_commitment_reports_once(ctx, oracle):
    v = sample_goldilocks(3302, 1 << LOG_LEN)
    root = oracle.rs_commit_root(v, (v.size >> LOG_DEPTH) << LOG_EXP, 1 << LOG_DEPTH)
    expire(ctx, 1)
    rs_encode_status(ctx)  # not its own
    with pytest.raises(WhirGpuError) as e:
        rs_commit_batch(ctx, v, LOG_EXP, LOG_DEPTH)
    assert e.value.status == E_DEVICE
    assert rs_commit_batch(ctx, v, LOG_EXP, LOG_DEPTH)[0] == root

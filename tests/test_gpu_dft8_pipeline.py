"""The encoder's contraction passes where a CTA takes many tiles of one coset (the
two buffers handed over and over, odd and even tile counts), where tiles of
several cosets meet in a CTA, short messages with many cosets, and buffers that
start between 16-byte boundaries (which take the butterfly passes): word for word
against the oracle's codewords."""
import numpy as np
import pytest

from whirplonk_b200 import sample_goldilocks
from whirplonk_b200.rs import rs_encode

pytestmark = pytest.mark.gpu


def codewords(gpu_ctx, v, count, lm, lx, ld, skew=(0, 0)):
    """skew: words by which the message and the scratch start off a 16-byte boundary."""
    import torch

    words = (count << (lm + ld)) << lx
    dv = torch.zeros(v.size + 1, dtype=torch.int64, device="cuda")
    dv[skew[0]:skew[0] + v.size] = torch.from_numpy(v.view(np.int64)).cuda()
    tmp = torch.empty(words + 1, dtype=torch.int64, device="cuda")
    out = torch.full((words,), -1, dtype=torch.int64, device="cuda")
    torch.cuda.synchronize()
    rs_encode(gpu_ctx, dv.data_ptr() + 8 * skew[0], count, lm + ld, lx, ld, tmp.data_ptr() + 8 * skew[1], out.data_ptr())
    torch.cuda.synchronize()
    return out.cpu().numpy().view(np.uint64).reshape(count, 1 << ld, 1 << (lm + lx))


def check(gpu_ctx, oracle, lm, lx, ld, count, skew=(0, 0)):
    v = sample_goldilocks(5500 + 100 * lm + 10 * lx + ld + count, count << (lm + ld))
    got = codewords(gpu_ctx, v, count, lm, lx, ld, skew)
    for k in range(count):
        rows = oracle.rs_encode_base(v[k << (lm + ld):(k + 1) << (lm + ld)], 1 << (lm + lx), 1 << ld)
        assert np.array_equal(got[k], rows.T), k


# (log message words per block, log expansion, log depth, vectors): 5 to 14 tiles a
# CTA and coset in both passes on 148 CTAs
@pytest.mark.parametrize("lm,lx,ld,count", [
    (8, 0, 6, 256), (9, 0, 6, 190), (10, 0, 6, 64), (11, 0, 6, 64), (12, 0, 6, 32), (12, 0, 2, 375), (13, 0, 6, 16),
    (14, 0, 6, 8), (14, 1, 6, 8), (15, 0, 5, 8), (16, 0, 6, 2), (16, 1, 4, 7), (17, 0, 5, 2), (18, 0, 5, 1), (19, 0, 4, 1),
    (20, 1, 3, 1), (20, 0, 0, 5)])
def test_many_tiles_a_cta(gpu_ctx, oracle, lm, lx, ld, count):
    check(gpu_ctx, oracle, lm, lx, ld, count)


# short messages with many cosets, from the size on at which they contract
@pytest.mark.parametrize("lm,lx,ld,count", [(8, 8, 4, 1), (8, 9, 4, 1), (8, 7, 4, 3), (9, 8, 4, 1), (9, 6, 4, 3), (10, 7, 4, 1)])
def test_short_messages(gpu_ctx, oracle, lm, lx, ld, count):
    check(gpu_ctx, oracle, lm, lx, ld, count)


@pytest.mark.parametrize("skew", [(1, 0), (0, 1), (1, 1)])
@pytest.mark.parametrize("lm,lx,ld,count", [(13, 3, 4, 1), (16, 1, 4, 1), (18, 1, 2, 1)])
def test_buffers_between_16_byte_boundaries(gpu_ctx, oracle, lm, lx, ld, count, skew):
    check(gpu_ctx, oracle, lm, lx, ld, count, skew)

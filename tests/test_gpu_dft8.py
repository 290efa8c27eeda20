"""The encoder's 8-bit contraction passes: every split of the message bits
(one- and two-round passes of radix 16, 32 and 64), several cosets, tiles that
span planes, and the shapes around the size from which they are used, word for
word against the oracle's codewords."""
import numpy as np
import pytest

from whirplonk_b200 import sample_goldilocks
from whirplonk_b200.rs import rs_encode

pytestmark = pytest.mark.gpu
P = 0xFFFFFFFF00000001
EDGE = np.array([0, 1, P - 1, P - 2, 0xFFFFFFFF, 0x100000000, 0xFEFFFFFFFFFFFFFF, 0x00FF00FF00FF00FF], dtype=np.uint64)

# (log message words per block, log expansion, log depth, vectors)
SHAPES = [(8, 8, 4, 1), (9, 7, 4, 1), (10, 6, 4, 1), (11, 5, 4, 1), (12, 4, 4, 1), (13, 3, 4, 1), (14, 2, 4, 1),
          (15, 1, 4, 1), (16, 0, 4, 1), (17, 1, 2, 1), (18, 2, 1, 1), (19, 1, 0, 1), (20, 1, 0, 1),
          (17, 1, 0, 5), (10, 8, 0, 8), (13, 5, 0, 5), (12, 4, 3, 3),  # odd plane counts
          (14, 1, 4, 1), (21, 1, 0, 1), (7, 9, 4, 1), (16, 4, 0, 1)]  # below the size, outside the range, one plane


def codewords(gpu_ctx, v, count, lm, lx, ld):
    import torch

    dv = torch.from_numpy(v.view(np.int64)).cuda()
    tmp = torch.empty((count << (lm + ld)) << lx, dtype=torch.int64, device="cuda")
    out = torch.full_like(tmp, -1)
    torch.cuda.synchronize()
    rs_encode(gpu_ctx, dv.data_ptr(), count, lm + ld, lx, ld, tmp.data_ptr(), out.data_ptr())
    torch.cuda.synchronize()
    return out.cpu().numpy().view(np.uint64).reshape(count, 1 << ld, 1 << (lm + lx))


@pytest.mark.parametrize("lm,lx,ld,count", SHAPES)
def test_codewords_match_oracle(gpu_ctx, oracle, lm, lx, ld, count):
    v = sample_goldilocks(4400 + 100 * lm + 10 * lx + ld, count << (lm + ld)).copy()
    v[:EDGE.size] = EDGE
    got = codewords(gpu_ctx, v, count, lm, lx, ld)
    for k in range(count):
        rows = oracle.rs_encode_base(v[k << (lm + ld):(k + 1) << (lm + ld)], 1 << (lm + lx), 1 << ld)
        assert np.array_equal(got[k], rows.T), k


@pytest.mark.parametrize("word", [P - 1, 0xFEFFFFFFFFFFFFFF, 0])
def test_constant_messages(gpu_ctx, oracle, word):
    """Byte sums at their largest: words of 0xFF bytes throughout."""
    lm, lx, ld = 12, 5, 4
    got = codewords(gpu_ctx, np.full(1 << (lm + ld), word, dtype=np.uint64), 1, lm, lx, ld)
    rows = oracle.rs_encode_base(np.full(1 << (lm + ld), word, dtype=np.uint64), 1 << (lm + lx), 1 << ld)
    assert np.array_equal(got[0], rows.T)

"""Commitments of several contexts at once, their encoder and leaf-ring CTAs
sharing SMs: every root equals the oracle's, and no worker ends early."""
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import pytest

from whirplonk_b200 import Context, sample_goldilocks
from whirplonk_b200.rs import rs_commit_batch

pytestmark = pytest.mark.gpu
SHAPES = [(22, 2, 4), (21, 3, 4), (20, 4, 3), (22, 1, 5), (20, 3, 2), (21, 2, 4)]  # log length, log expansion, log depth
PASSES = 15


def test_roots_match_oracle(gpu_ctx, oracle):
    import torch

    hosts = [sample_goldilocks(7300 + i, 1 << ll) for i, (ll, _, _) in enumerate(SHAPES)]
    want = [oracle.rs_commit_root(v, (v.size >> ld) << lx, 1 << ld) for v, (_, lx, ld) in zip(hosts, SHAPES)]
    dev = [torch.from_numpy(v.view(np.int64)).cuda() for v in hosts]
    torch.cuda.synchronize()

    def work(i):
        ll, lx, ld = SHAPES[i]
        ctx = Context(0)
        try:
            return [rs_commit_batch(ctx, None, lx, ld, on_device_ptr=dev[i].data_ptr(), count=1, log_len=ll)[0]
                    for _ in range(PASSES)]
        finally:
            ctx.close()

    with ThreadPoolExecutor(len(SHAPES)) as pool:
        for i, roots in enumerate(pool.map(work, range(len(SHAPES)))):  # re-raises a worker's exception
            assert roots == [want[i]] * PASSES, SHAPES[i]

"""MO transforms of several contexts in turn and on several threads, whose kept
workspaces come to more than the bound that idle contexts keep together."""
import threading

import numpy as np
import pytest
import torch

from hartreefock_b200 import engine as E
from hartreefock_b200 import molecules

pytestmark = pytest.mark.gpu


def test_contexts_take_turns_and_threads():
    Z, xyz = molecules.water_cluster(4, seed=2)
    C = torch.from_numpy(np.linalg.qr(np.random.default_rng(1).normal(size=(76, 76)))[0]).cuda()
    engines = [E.Engine(Z, xyz, "6-31g*") for _ in range(4)]  # 450 MB of workspace each
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    want = engines[0].mo_eri_ovov_tensor(C, 0, 20, 20, 56).clone()
    out = [[] for _ in engines]

    def work(k):
        stream = torch.cuda.Stream()
        with torch.cuda.stream(stream):
            for _ in range(6):
                out[k].append(engines[k].mo_eri_ovov_tensor(C, 0, 20, 20, 56).clone())
        stream.synchronize()

    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(engines))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    # the same sums; another order at most within a GEMM: 76 terms below 1 each
    for results in out:
        assert len(results) == 6
        assert all((x - want).abs().max().item() < 1e-12 for x in results)
    del out, results
    torch.cuda.empty_cache()
    kept = free - torch.cuda.mem_get_info()[0]
    assert kept < (1 << 30) + (512 << 20)  # the bound, the handles' own memory and torch's tensors
    for e in engines:
        e.close()

"""The device-pointer diffusion from several threads at once, each on a stream of its
own: the workspaces come from one pool, and the small grids' cooperative launches meet."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GRIDS = [(37, 21, 13), (32, 20, 17), (48, 48, 40), (23, 9, 40), (64, 40, 33), (16, 16, 3)]


def test_threads_and_streams(marl, oracle_mod):
    import torch

    p = marl.default_params()
    work = []
    for i, dims in enumerate(GRIDS):
        rng = np.random.default_rng(i)
        field = rng.random((*dims[::-1], 12), dtype=np.float32)
        occ = (rng.random(dims[::-1]) < 0.15).astype(np.uint8)
        cpu = field.copy()
        oracle_mod.diffuse(cpu, occ, dims, p, 7)
        work.append((dims, torch.from_numpy(field).cuda(), torch.from_numpy(occ).cuda(), cpu))
    torch.cuda.synchronize()
    wrong = []

    def call(dims, field, occ, want):
        stream = torch.cuda.Stream()
        with torch.cuda.stream(stream):
            f, s = torch.empty_like(field), torch.empty_like(field)
            for k in range(40):
                f.copy_(field)
                marl.diffuse_device(f.data_ptr(), s.data_ptr(), occ.data_ptr(), dims, p, 7, stream.cuda_stream)
                if not np.array_equal(f.cpu().numpy(), want):
                    wrong.append((dims, k))

    threads = [threading.Thread(target=call, args=w) for w in work]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong, wrong[:5]

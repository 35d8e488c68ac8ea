"""The stateless counting sort at the sizes where its passes change: digit
widths (1, 9, 10, 18, 19 and 28 bits of cells: one to four passes), counts around the block of 4096
keys, all keys equal, keys already sorted, and perm written over the keys.
The permutation equals numpy's stable argsort, exactly."""
import ctypes

import numpy as np
import pytest

from pbpic_b200 import _lib as L

pytestmark = pytest.mark.gpu


def run(keys, ncells, static, overlap):
    import torch
    n = len(keys)
    k = torch.from_numpy(keys).cuda()
    perm = k if overlap else torch.full((max(n, 1),), -1, dtype=torch.int32, device="cuda")
    counts = torch.full((ncells,), -1, dtype=torch.int32, device="cuda")
    lib = L.lib()
    fn = lib.pbpic_counting_sort_keys_static if static else lib.pbpic_counting_sort_keys
    L.check(fn(ctypes.c_void_p(k.data_ptr()), n, ncells, ctypes.c_void_p(perm.data_ptr()),
               ctypes.c_void_p(counts.data_ptr()), None))
    return perm.cpu().numpy()[:n], counts.cpu().numpy()


@pytest.mark.parametrize("static", [False, True])
@pytest.mark.parametrize("n,ncells", [(n, c) for n in (1, 4095, 4096, 4097, 70001)
                                      for c in (1, 2, 511, 512, 513, 1 << 18, (1 << 18) + 1)] + [(4097, (1 << 27) + 5)])
def test_sort(gpu_lib, static, n, ncells):
    rng = np.random.default_rng(n + ncells)
    for keys in (rng.integers(0, ncells, n), np.full(n, ncells - 1), np.sort(rng.integers(0, ncells, n))):
        keys = keys.astype(np.int32)
        for overlap in (False, True):
            perm, counts = run(keys.copy(), ncells, static, overlap)
            assert np.array_equal(perm, np.argsort(keys, kind="stable"))
            assert np.array_equal(counts, np.bincount(keys, minlength=ncells))


def test_calls_on_two_streams(gpu_lib):
    """Calls from two threads on two streams share the scratch pool."""
    import threading
    import torch
    from pbpic_b200.sim import counting_sort_keys
    rng = np.random.default_rng(4)
    jobs, errors = [], []
    for _ in range(2):
        keys = rng.integers(0, 5000, 300_000).astype(np.int32)
        jobs.append((keys, torch.from_numpy(keys).cuda(), torch.zeros(len(keys), dtype=torch.int32, device="cuda"),
                     torch.zeros(5000, dtype=torch.int32, device="cuda"), torch.cuda.Stream()))
    torch.cuda.synchronize()

    def work(job):
        try:
            for _ in range(20):
                counting_sort_keys(job[1].data_ptr(), len(job[0]), 5000, job[2].data_ptr(), job[3].data_ptr(),
                                   job[4].cuda_stream)
        except Exception as e:
            errors.append(e)
    threads = [threading.Thread(target=work, args=(j,)) for j in jobs]
    [t.start() for t in threads]
    [t.join() for t in threads]
    assert not errors
    for keys, _, perm, counts, _ in jobs:
        assert np.array_equal(perm.cpu().numpy(), np.argsort(keys, kind="stable"))
        assert np.array_equal(counts.cpu().numpy(), np.bincount(keys, minlength=5000))

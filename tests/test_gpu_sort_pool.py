"""The stand-alone sort's scratch: under stream capture (the graph's own
allocations), from several streams and threads at once, and across the
destruction of an engine, which gives the pool's memory back, the keys and the
permutation are those of a stable sort."""
import threading

import numpy as np
import pytest

from parity import morton_reference, stable_sort_reference

pytestmark = pytest.mark.gpu


def _arrays(n, seed):
    import torch
    rng = np.random.default_rng(seed)
    pos = (rng.random((3, n)) * 100).astype(np.float32)
    return pos, torch.tensor(pos, device="cuda"), *(torch.full((n,), -7, dtype=torch.int32, device="cuda") for _ in range(2))


def _sort(mpm, p, keys, perm, stream):
    mpm.sort_particles_device(p[0].data_ptr(), p[1].data_ptr(), p[2].data_ptr(), p.shape[1], keys.data_ptr(), perm.data_ptr(), stream)


def _check(pos, keys, perm):
    want = morton_reference(pos)
    assert np.array_equal(keys.cpu().numpy(), want)
    assert np.array_equal(perm.cpu().numpy(), stable_sort_reference(want))


@pytest.mark.parametrize("n", [1, 2049, 70000])
def test_captured(gpu_ok, mpm, n):
    import torch
    pos, p, keys, perm = _arrays(n, 5)
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        _sort(mpm, p, keys, perm, stream.cuda_stream)
    for seed in (6, 7):  # the graph sorts what the arrays hold when it runs
        pos = (np.random.default_rng(seed).random((3, n)) * 60).astype(np.float32)
        p.copy_(torch.tensor(pos))
        graph.replay()
        torch.cuda.synchronize()
        _check(pos, keys, perm)
    other = _arrays(n, 8)
    _sort(mpm, *other[1:], torch.cuda.current_stream().cuda_stream)  # outside the graph: the pool
    graph.replay()
    torch.cuda.synchronize()
    _check(other[0], *other[2:])
    _check(pos, keys, perm)


def test_streams_and_threads(gpu_ok, mpm):
    import torch
    from mpm_b200 import scenes
    sets = [_arrays(n, 20 + k) for k, n in enumerate((50000, 3000, 120000, 77777))]
    torch.cuda.synchronize()
    failed = []

    def work(k):
        try:
            torch.cuda.set_device(0)
            pos, p, keys, perm = sets[k]
            stream = torch.cuda.Stream()
            for _ in range(20):
                keys.fill_(-7)
                torch.cuda.current_stream().synchronize()
                _sort(mpm, p, keys, perm, stream.cuda_stream)
                stream.synchronize()
                _check(pos, keys, perm)
        except BaseException as err:  # noqa: BLE001 - reported below
            failed.append(err)

    def engines():
        for _ in range(10):
            mpm.Engine(scenes._cfg((16, 16, 16))).close()

    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(sets))] + [threading.Thread(target=engines)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed, failed

"""Threads that call one entry point with work of different sizes at the same time: the
kernels' shared memory is sized by the work, and no call may fail or differ because of
another thread's."""
import ctypes as C
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def dense_job(stream, W, H, D, seed):
    from doubleeye_b200 import _lib, dense
    rng = np.random.default_rng(seed)
    L, R = (torch.from_numpy(rng.integers(0, 256, (H, W), dtype=np.uint8)).cuda() for _ in "LR")
    cfg = dense.Cfg(dmax=D, iters=1)
    m = dense.DenseMatcher(cfg)
    out = m.new_outputs(H, W)
    arr, shapes = m._pairs([(L, R, 0, out)])
    need = m.workspace_bytes(shapes)
    args = (C.byref(cfg), arr, 1, m._workspace(need).data_ptr(), need, stream.cuda_stream)
    fn = _lib.lib().de_dense_dev
    return lambda: fn(*args), lambda: out["margin"].cpu().numpy().tobytes(), (m, L, R, cfg)


def detect_job(stream, W, H, cell, seed):
    from doubleeye_b200 import _lib, sparse
    img = torch.from_numpy(np.random.default_rng(seed).integers(0, 256, (H, W), dtype=np.uint8)).cuda()
    cfg, need = sparse.DetCfg(cell=cell, per_cell=2), C.c_size_t()
    _lib.check(_lib.lib().de_detect_workspace_bytes(W, H, C.byref(cfg), C.byref(need)))
    ws = torch.empty(need.value, dtype=torch.uint8, device="cuda")
    out = torch.zeros((512, 4), device="cuda")
    n = torch.zeros(1, dtype=torch.int32, device="cuda")
    args = (img.data_ptr(), W, H, C.byref(cfg), out.data_ptr(), 512, n.data_ptr(), ws.data_ptr(),
            need.value, stream.cuda_stream)
    fn = _lib.lib().de_detect_fast_dev
    return (lambda: fn(*args), lambda: (int(n.item()), out.cpu().numpy().tobytes()),
            (img, cfg, ws))


def edges_job(stream, E, m, n, seed):
    from doubleeye_b200 import _lib
    rng = np.random.default_rng(seed)
    ei, ej = (torch.from_numpy(rng.integers(0, k, E)).cuda() for k in (m, n))
    se, need = torch.from_numpy(rng.uniform(-0.5, 1.0, E)).cuda(), C.c_size_t()
    _lib.check(_lib.lib().de_masda_edges_workspace_bytes(E, m, n, C.byref(need)))
    ws = torch.empty(need.value, dtype=torch.uint8, device="cuda")
    assign = torch.empty(m, dtype=torch.int64, device="cuda")
    hist, nh = torch.empty(1, dtype=torch.float64, device="cuda"), torch.empty(1, dtype=torch.int32, device="cuda")
    args = (ei.data_ptr(), ej.data_ptr(), se.data_ptr(), E, m, n, -0.1, -0.1, 1, 0.4, 0.0,
            assign.data_ptr(), hist.data_ptr(), nh.data_ptr(), None, ws.data_ptr(), need.value,
            stream.cuda_stream)
    fn = _lib.lib().de_masda_edges_dev
    return (lambda: fn(*args), lambda: (assign.cpu().numpy().tobytes(), float(hist.item())),
            (ei, ej, se, ws, nh))


@pytest.mark.parametrize("make,sizes,reps", [
    (dense_job, [(40, 12, 16), (1000, 24, 16), (60, 600, 16)], 3000),
    (dense_job, [(150, 12, 100), (1020, 16, 100), (150, 700, 100)], 3000),
    (detect_job, [(64, 48, 8), (64, 48, 128)], 8000),
    (edges_job, [(20, 9, 9), (4000, 300, 400)], 4000)], ids=["d16", "d100", "detect", "edges"])
def test_sizes_side_by_side(make, sizes, reps):
    streams = [torch.cuda.Stream() for _ in sizes]
    jobs = [make(st, *s, seed) for seed, (s, st) in enumerate(zip(sizes, streams))]
    torch.cuda.synchronize()             # (the jobs run on streams of their own)
    want = []
    for run, result, _ in jobs:
        assert run() == 0
        torch.cuda.synchronize()
        want.append(result())
    failed = [0] * len(jobs)

    def loop(i):
        for _ in range(reps):
            failed[i] += jobs[i][0]() != 0
    threads = [threading.Thread(target=loop, args=(i,)) for i in range(len(jobs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert failed == [0] * len(jobs)
    assert [result() for _, result, _ in jobs] == want

"""Which column kernel runs: small work by itself takes the tensor-memory kernel, and any
column knob means the streaming kernel in the shape that the knob asks for.  The choice is
read from the kernel nodes of a captured graph.  The streaming shapes' write-back for the
reverse match is checked against the oracle bit for bit."""
import ctypes as C

import numpy as np
import pytest

from oracle.oracle import Oracle, default_cfg

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

KNOBS = [{}, dict(cols_kt=4), dict(cols_kt=8), dict(cols_kt=16), dict(cols_pf=4), dict(cols_pf=8),
         dict(cols_pf=16), dict(cols_cta=128), dict(cols_cta=256), dict(cols_async=0)]


@pytest.fixture
def knobs():
    from doubleeye_b200 import _lib
    names = ("cols_kt", "cols_pf", "cols_cta", "cols_async")
    saved = {n: _lib.get_param(n) for n in names}

    def put(kw):
        for n, v in kw.items():
            _lib.set_param(n, v)
    yield put
    put(saved)


def captured_kernels(run):
    """The (mangled) names of the kernels that run() launches on the current stream."""
    cu = C.CDLL("libcuda.so.1")
    run()                                # (module loading and first-use set-up)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(g, capture_error_mode="thread_local"):
        keep = run()
    graph, n = C.c_void_p(int(g.raw_cuda_graph())), C.c_size_t(0)
    assert cu.cuGraphGetNodes(graph, None, C.byref(n)) == 0
    nodes = (C.c_void_p * n.value)()
    assert cu.cuGraphGetNodes(graph, nodes, C.byref(n)) == 0
    names = []
    for node in nodes:
        kind = C.c_int()
        assert cu.cuGraphNodeGetType(C.c_void_p(node), C.byref(kind)) == 0
        if kind.value != 0:              # CU_GRAPH_NODE_TYPE_KERNEL
            continue
        params, name = (C.c_void_p * 32)(), C.c_char_p()   # CUDA_KERNEL_NODE_PARAMS: func first
        assert cu.cuGraphKernelNodeGetParams_v2(C.c_void_p(node), params) == 0
        assert cu.cuFuncGetName(C.byref(name), C.c_void_p(params[0])) == 0
        names.append(name.value.decode())
    del keep
    return " ".join(names)


@pytest.mark.parametrize("kw", KNOBS, ids=lambda k: "-".join(f"{n}{v}" for n, v in k.items()) or "none")
@pytest.mark.parametrize("W,H,D", [(97, 9, 16), (300, 40, 256), (848, 480, 128)])
def test_which_kernel(W, H, D, kw, knobs):
    from doubleeye_b200 import dense
    img = torch.zeros((H, W), dtype=torch.uint8, device="cuda")
    knobs(kw)
    names = captured_kernels(lambda: dense.cost_top2(img, img, dense.Cfg(dmax=D)))
    assert "k_rows" in names
    assert ("k_cols_tm" in names) == (not kw)
    assert ("6k_cols" in names) == bool(kw)


@pytest.mark.parametrize("kt,pf,cta,ring", [(4, 4, 128, 1), (4, 8, 256, 1), (4, 16, 128, 1),
                                            (8, 4, 256, 1), (8, 8, 128, 1), (8, 8, 256, 0),
                                            (16, 4, 128, 1)])
@pytest.mark.parametrize("W,H,D", [(97, 9, 16), (260, 133, 100), (300, 40, 192), (420, 60, 256)])
def test_reverse_match_of_streaming_shapes(W, H, D, kt, pf, cta, ring, knobs):
    from doubleeye_b200 import dense
    rng = np.random.default_rng(W + D)
    L = rng.integers(0, 256, (H, W), dtype=np.uint8)
    R = np.roll(L, -min(D, 7), 1) ^ rng.integers(0, 8, (H, W), dtype=np.uint8)
    kw = dict(dmin=1, dmax=D, iters=1, lrc=1)
    knobs(dict(cols_kt=kt, cols_pf=pf, cols_cta=cta, cols_async=ring))
    got = dense.run_dense(L, R, dense.Cfg(**kw))
    _, margin, cand = Oracle().dense(default_cfg(**kw), L, R)
    for a, b in ((got.margin, margin), (got.cand, cand)):
        assert ((a.view(np.uint32) == b.view(np.uint32)) | (np.isnan(a) & np.isnan(b))).all()

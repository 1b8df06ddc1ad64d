"""An edge list that names a node out of range is refused, and the call leaves its outputs
as they were: on both sides of the sizes that the one-CTA solve takes."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("E", [1, 600, 4096, 4097])
@pytest.mark.parametrize("where,value", [("left", 40), ("left", -1), ("right", 50),
                                         ("right", 1 << 40)])
def test_outputs_untouched(E, where, value):
    from doubleeye_b200 import _lib
    m, n, iters = 40, 50, 3
    e = torch.arange(E, device="cuda")
    ei, ej = e % m, (e * 7) % n
    (ei if where == "left" else ej)[E - 1] = value
    se = torch.linspace(-0.5, 1.0, E, dtype=torch.float64, device="cuda")
    need = C.c_size_t()
    _lib.check(_lib.lib().de_masda_edges_workspace_bytes(E, m, n, C.byref(need)))
    ws = torch.empty(need.value, dtype=torch.uint8, device="cuda")
    outs = [torch.full((m,), 12345, dtype=torch.int64, device="cuda"),
            torch.full((iters,), 12345.0, dtype=torch.float64, device="cuda"),
            torch.full((1,), 12345, dtype=torch.int32, device="cuda"),
            torch.full((E,), 12345.0, dtype=torch.float64, device="cuda")]
    with pytest.raises(_lib.DeError):
        _lib.check(_lib.lib().de_masda_edges_dev(
            ei.data_ptr(), ej.data_ptr(), se.data_ptr(), E, m, n, -0.1, -0.1, iters, 0.4, 1e-5,
            *(t.data_ptr() for t in outs), ws.data_ptr(), need.value,
            torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()
    for t in outs:
        assert bool((t == 12345).all())

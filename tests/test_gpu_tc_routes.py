"""Which calls of the plain f32 and c32 path leave the tensor-core families, and for what:
operands off their natural alignment, host operands under a workspace cap."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch_cuda():
    import torch

    assert torch.cuda.is_available(), "the -m gpu tests need a CUDA device"
    return torch


def column_major(tp, dtype, m, n, k):
    h = tp.Handle()
    infos = [tp.TensorInfo(dtype, [m, k], [1, m]), tp.TensorInfo(dtype, [k, n], [1, k]), tp.TensorInfo(dtype, [m, n], [1, m])]
    p = tp.TensorProduct.create(h, (0, infos[0], [0, 2]), (0, infos[1], [2, 1]), (0, infos[2], [0, 1]), (0, infos[2], [0, 1]))
    p._keep = (h, infos)
    return p


@pytest.mark.parametrize("autotune", [False, True])
@pytest.mark.parametrize("off", ["A", "B", "D"])
@pytest.mark.parametrize("m,n,k,splits", [(1000, 900, 600, False), (300, 260, 5000, True)])
def test_c32_operands_off_eight_bytes(tp, torch_cuda, m, n, k, splits, off, autotune):
    """They take what the choice without the tensor-core families takes (packed panels,
    split K for few tiles), and the report names it; an aligned call of the same plan
    is back on the tensor cores. D may lie off as before."""
    torch = torch_cuda
    gen = torch.Generator(device="cuda").manual_seed(4)
    real = lambda count: torch.randn(2 * count + 1, device="cuda", generator=gen)
    buf = {"A": real(m * k), "B": real(k * n), "D": torch.zeros(2 * m * n + 1, device="cuda")}
    ptr = {x: t.data_ptr() + (4 if x == off else 0) for x, t in buf.items()}
    view = {x: torch.complex(*t[(1 if x == off else 0):][: t.numel() - 1].double().view(-1, 2).unbind(1)) for x, t in buf.items()
            if x != "D"}
    want = (view["B"].view(n, k) @ view["A"].view(k, m)).reshape(-1)
    ex = tp.Executor()
    p = column_major(tp, tp.C32, m, n, k)
    p.set_autotune(autotune)
    model = p.report()
    for turn in range(2):  # measured, then from the cache
        buf["D"].zero_()
        tp.check(p.execute(ex, 1.0, ptr["A"], ptr["B"], 0.0, None, ptr["D"]))
        got = torch.complex(*buf["D"][(1 if off == "D" else 0):][: 2 * m * n].double().view(-1, 2).unbind(1))
        assert float((got - want).norm() / want.norm()) <= 1e-6
        rep = p.report()
        if off == "D":
            assert autotune or rep["family"] == model["family"]
        else:
            assert ".tcgen05." not in rep["family"]
            assert autotune or (".tma." in rep["family"] and (rep["split_k"] > 1) == splits), rep
    if not autotune and ".tcgen05." in model["family"]:
        aligned = {x: t.data_ptr() for x, t in buf.items()}
        tp.check(p.execute(ex, 1.0, aligned["A"], aligned["B"], 0.0, None, aligned["D"]))
        assert p.report()["family"] == model["family"]
    ex.close()

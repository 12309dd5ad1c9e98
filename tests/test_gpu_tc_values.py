"""Values that the BF16 planes of the plain f32 and c32 tensor-core kernels cannot carry
(csrc/k_tcstream.cu, csrc/k_split.cu), against the direct FFMA tile, on a B200."""
import numpy as np
import pytest

from test_gpu_parity import Op, make_product
from test_gpu_tc_stream import DIRECT, execute

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch_cuda():
    import torch

    assert torch.cuda.is_available(), "the -m gpu tests need a CUDA device"
    return torch


@pytest.fixture(scope="module")
def ex(tp, torch_cuda):
    e = tp.Executor()
    yield e
    e.close()


def matrix_pair(dt, m, n, k):
    """A as [k, m] and B as [n, k] views of column-major operands, all ones."""
    a, b = np.ones(m * k, dtype=dt), np.ones(k * n, dtype=dt)
    ops = Op(a, [m, k], [1, m], [0, 2]), Op(b, [k, n], [1, k], [2, 1])
    return ops, a.reshape(k, m), b.reshape(n, k)


def model_and_direct(tp, ex, torch, dt, A, B, m, n, family):
    D = Op(np.zeros(m * n, dtype=dt), [m, n], [1, m], [0, 1])
    p = make_product(tp, dt, A, B, None, D)
    assert family in p.report()["family"], p.report()["family"]
    out = []
    for kernel in (0, DIRECT[dt]):
        p.set_kernel(kernel)
        status, td = execute(torch, p, ex, dt, A, B, None, D, 1.0, 0.0)
        assert status == 0, tp.last_error()
        torch.cuda.synchronize()
        out.append(td.cpu().numpy())
    return out


# (m, n, k, family): split in flight, and planes packed first.
SHAPES = [(4000, 390, 40, ".stream."), (2200, 1300, 2500, ".split.")]


@pytest.mark.parametrize("side", ["A", "B"])
@pytest.mark.parametrize("what", ["one value", "one row", "all"])
@pytest.mark.parametrize("shape", SHAPES, ids=["in flight", "packed"])
@pytest.mark.parametrize("dt", sorted(DIRECT))
def test_elements_below_every_plane(tp, ex, torch_cuda, dt, shape, what, side):
    """Elements of 2^-135 round to zero in all three planes, but their products with
    elements of 2^99 are ordinary numbers. The other depths of those rows (or
    columns) are zero, the other rows ordinary."""
    m, n, k, family = shape
    (A, B), a, b = matrix_pair(dt, m, n, k)
    tiny, big = (a, b) if side == "A" else (b.T, a.T)  # tiny: [k, rows], big: [cols, k]
    rows = {"one value": [7], "one row": [133], "all": slice(None)}[what]
    depths = {"one value": slice(3, 4), "one row": slice(0, 9), "all": slice(None)}[what]
    tiny[:, rows] = 0
    tiny[depths, rows] = np.float32(2.0 ** -135)
    if what != "all":
        tiny[depths, :] = np.where(tiny[depths, :] == 1, 0, tiny[depths, :])
    big[:, depths] = np.float32(2.0 ** 99)
    x, y = model_and_direct(tp, ex, torch_cuda, dt, A, B, m, n, family)
    # Sums of at most k equal powers of two, and of ones: exact to f32 rounding.
    lim = 2.0 ** -20 * np.abs(y.astype("complex128"))
    assert np.all(np.abs(y) > 0)
    assert np.all(np.abs(x.astype("complex128") - y) <= lim)

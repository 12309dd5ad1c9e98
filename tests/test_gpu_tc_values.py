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


def tiny_block_case(dt, m, n, k, rng):
    """Ordinary values, but three quarters of the rows and half of the columns are zero,
    a few rows hold 1e-33 and others an infinity: outputs of every kind side by side."""
    (A, B), a, b = matrix_pair(dt, m, n, k)
    for x in (a, b):
        x[...] = rng.uniform(-1, 1, x.shape)
    a[:, ::4] = 0
    a[:, 1::4] *= np.float32(1e-33)
    b[::2] = 0
    a[min(5, k - 1), 1000:1003] = np.inf
    return A, B


@pytest.mark.parametrize("cmode", [None, "own", "in place"])
@pytest.mark.parametrize("shape", SHAPES + [(1100, 2600, 1100, ".split.")], ids=["in flight", "packed", "packed, few tiles"])
@pytest.mark.parametrize("dt", sorted(DIRECT))
def test_parts_computed_again(tp, ex, torch_cuda, dt, shape, cmode):
    """Tiles that are computed again in part, or left out first and computed whole
    (alpha and beta), give what the direct tile gives."""
    m, n, k, family = shape
    rng = np.random.default_rng(m)
    A, B = tiny_block_case(dt, m, n, k, rng)
    d0 = rng.uniform(-1, 1, m * n).astype(dt) if cmode else np.zeros(m * n, dtype=dt)
    D = Op(d0, [m, n], [1, m], [0, 1])
    C = None if cmode is None else D if cmode == "in place" else Op(rng.uniform(-1, 1, m * n).astype(dt), [m, n], [n, 1], [0, 1])
    p = make_product(tp, dt, A, B, C, D)
    assert family in p.report()["family"], p.report()["family"]
    out = []
    for kernel in (0, DIRECT[dt]):
        p.set_kernel(kernel)
        status, td = execute(torch_cuda, p, ex, dt, A, B, C, D, 1.0 if cmode is None else 1.5, 0.0 if cmode is None else -0.5)
        assert status == 0, tp.last_error()
        torch_cuda.cuda.synchronize()
        out.append(td.cpu().numpy().view("float32").reshape(n, -1))
    x, y = out
    assert np.array_equal(np.isfinite(x), np.isfinite(y)) and np.array_equal(np.isnan(x), np.isnan(y))
    # Each output within 60 roundings of its products' magnitudes, and of C's.
    a, b = np.abs(A.buf.reshape(k, m)).astype("float64"), np.abs(B.buf.reshape(n, k)).astype("float64")
    mag = np.repeat(b @ np.where(np.isfinite(a), a, 0), x.shape[1] // m, axis=1)
    lim = 60 * (2.0 ** -24 * 2 * mag + 2.0 ** -149) + (0 if cmode is None else 2.0 ** -22)
    ok = np.isfinite(y)
    assert np.all(np.abs(x[ok].astype("float64") - y[ok]) <= lim[ok])


@pytest.mark.parametrize("what", ["one NaN", "2^55"])
@pytest.mark.parametrize("m,n,k", [(2048, 2048, 256), (2048, 2048, 2048)])
@pytest.mark.parametrize("dt", sorted(DIRECT))
def test_values_outside_the_planes_take_no_cliff(tp, torch_cuda, dt, m, n, k, what):
    """At most twice the time of the FFMA tiles (and some for two small launches)."""
    torch = torch_cuda
    A = (torch.rand(k, m, device="cuda", dtype=getattr(torch, dt)) - 0.5).t()
    B = (torch.rand(n, k, device="cuda", dtype=getattr(torch, dt)) - 0.5).t()
    if what == "one NaN":
        A[7, 3] = float("nan")
    else:
        A.mul_(2.0 ** 55)
        B.mul_(2.0 ** 55)
    D = torch.zeros(n, m, device="cuda", dtype=A.dtype).t()
    e = tp.Executor(device=0, stream=torch.cuda.current_stream().cuda_stream, sync=False)
    lay = lambda t: tp.OperandSpec(tp.LayoutSpec(list(t.shape), list(t.stride())))
    prob = tp.Problem.from_labels({"float32": tp.F32, "complex64": tp.C32}[dt], lay(A), lay(B), lay(D), [0, 2], [2, 1], [0, 1])
    ms = []
    for kernel in (0, {"float32": 10, "complex64": 15}[dt]):
        plan = tp.Plan(prob, tp.PlanConfig(kernel=kernel))
        for _ in range(2):
            plan.execute_into(e, 1.0, A, B, D)
        t = [torch.cuda.Event(enable_timing=True) for _ in range(6)]
        for ev in t:
            ev.record()
            plan.execute_into(e, 1.0, A, B, D)
        torch.cuda.synchronize()
        ms.append(min(u.elapsed_time(v) for u, v in zip(t, t[1:])))
    e.close()
    assert ms[0] <= 2 * ms[1] + 0.05, ms


@pytest.mark.parametrize("dt,m,n,k", [("f32", 4000, 1000, 40), ("c32", 3000, 900, 30), ("f32", 2048, 2048, 1024),
                                      ("c32", 2048, 1024, 600)])
def test_a_captured_call_marks_its_tiles_anew(tp, dt, m, n, k):
    """Replays of one captured call: values that the planes carry, then an infinity and an
    element below 2^-100, then the first again."""
    import torch

    kind, wide = {"f32": (torch.float32, torch.float64), "c32": (torch.complex64, torch.complex128)}[dt]
    side = torch.cuda.Stream()
    ex = tp.Executor(device=0, stream=side.cuda_stream, sync=False)
    with torch.cuda.stream(side):
        make = lambda r, c: torch.randn(r * c, device="cuda", dtype=kind).as_strided([r, c], [1, r])
        A, B, D = make(m, k), make(k, n), make(m, n)
        first = A.clone()
    lay = lambda x: tp.OperandSpec(tp.LayoutSpec.col_major(x))
    plan = tp.Plan(tp.Problem.from_labels({"f32": tp.F32, "c32": tp.C32}[dt], lay([m, k]), lay([k, n]), lay([m, n]),
                                          [0, 2], [2, 1], [0, 1]))
    assert ".tcgen05." in plan.report()["family"]
    with torch.cuda.stream(side):
        plan.execute_into(ex, 1.0, A, B, D)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=side):
        plan.execute_into(ex, 1.0, A, B, D)
    finite = lambda t: torch.isfinite(torch.view_as_real(t).sum(-1) if t.is_complex() else t)
    for extreme in (False, True, False):
        with torch.cuda.stream(side):
            A.copy_(first)
            if extreme:
                A[5, 1], A[7, 2] = float("inf"), 2.0 ** -120
            D.zero_()
            graph.replay()
        torch.cuda.synchronize()
        want = A.to(wide) @ B.to(wide)
        ok = finite(want)
        assert bool((finite(D) == ok).all()) and bool(ok.all()) != extreme
        assert float((D.to(wide) - want)[ok].norm() / want[ok].norm()) <= 1e-6
    del graph
    ex.close()

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


def host_call(tp, torch, dtype, m, n, k, a_lead, limit=None, streaming=True):
    """D = A B of host operands, A with leading stride `a_lead`; returns the status, D's
    error against 64 bits, the family and the launches of the call."""
    gen = torch.Generator().manual_seed(m + n)
    make = lambda count: torch.randn(count, generator=gen, dtype=torch.complex64 if dtype == tp.C32 else torch.float32)
    a, b = make(a_lead * m * k).pin_memory(), make(k * n).pin_memory()
    d = torch.zeros(m * n, dtype=a.dtype).pin_memory()
    h = tp.Handle()
    infos = [tp.TensorInfo(dtype, [m, k], [a_lead, a_lead * m]), tp.TensorInfo(dtype, [k, n], [1, k]),
             tp.TensorInfo(dtype, [m, n], [1, m])]
    p = tp.TensorProduct.create(h, (0, infos[0], [0, 2]), (0, infos[1], [2, 1]), (0, infos[2], [0, 1]), (0, infos[2], [0, 1]))
    ex = tp.Executor()
    ex.set_profiling(True)
    ex.set_streaming(streaming)
    if limit:
        ex.set_workspace_limit(limit)
    status = p.execute(ex, 1.0, a.data_ptr(), b.data_ptr(), 0.0, None, d.data_ptr())
    wide = torch.complex128 if dtype == tp.C32 else torch.float64
    da, db = a.cuda().view(k, m, a_lead)[:, :, 0].to(wide), b.cuda().view(n, k).to(wide)
    want = db @ da
    err = float((d.cuda().view(n, m).to(wide) - want).norm() / want.norm())
    times = ex.kernel_times()
    ex.close()
    return status, err, p.report()["family"], times


@pytest.mark.parametrize("dtype", ["F32", "C32"])
@pytest.mark.parametrize("m,n,k,a_lead,what", [(9000, 1000, 64, 1, ".stream."),    # chunks on 16-byte groups
                                                (9006, 1000, 64, 1, ".stream."),    # and off them (4503 rows first)
                                                (8194, 1100, 60, 2, ".stream."),    # A through panels
                                                (6006, 3000, 2000, 1, ".split.")])   # planes packed first
def test_host_operands_streamed_to_the_tensor_cores(tp, torch_cuda, dtype, m, n, k, a_lead, what):
    status, err, family, times = host_call(tp, torch_cuda, getattr(tp, dtype), m, n, k, a_lead)
    assert status == 0, tp.last_error()
    assert what in family and times[family]["launches"] >= 2, (family, times)
    assert err <= 1e-6


@pytest.mark.parametrize("dtype", ["F32", "C32"])
def test_host_operands_streamed_under_a_workspace_cap(tp, torch_cuda, dtype):
    """Room for the operands and for packed panels of a chunk, not for planes: the call
    runs streamed on the packed family."""
    m, n, k = (8192, 5120, 960) if dtype == "F32" else (8192, 4096, 512)
    item = 4 if dtype == "F32" else 8
    spans = item * (m * k + k * n + m * n)
    # The first chunk (half the rows): panels of A' and B' (c32: 4 and 2 reals an element).
    panels = 4 * (4096 * k + k * n) if dtype == "F32" else 4 * (4 * 4096 * k + 2 * k * n)
    status, err, family, times = host_call(tp, torch_cuda, getattr(tp, dtype), m, n, k, 1, limit=spans + panels + (1 << 20))
    assert status == 0, tp.last_error()
    assert ".tcgen05." not in family and times[family]["launches"] >= 2, (family, times)
    assert err <= 1e-6
    status, err, family, _ = host_call(tp, torch_cuda, getattr(tp, dtype), m, n, k, 1)
    assert status == 0 and ".tcgen05." in family and err <= 1e-6


def test_a_cached_choice_beyond_the_cap_is_reported_as_the_models(tp, torch_cuda):
    torch = torch_cuda
    m, n, k = 2000, 2000, 40
    a, b = torch.randn(m * k, device="cuda"), torch.randn(k * n, device="cuda")
    d = torch.zeros(m * n, device="cuda")
    p = column_major(tp, tp.F32, m, n, k)
    p.set_autotune(True)
    ex = tp.Executor()
    call = lambda: tp.check(p.execute(ex, 1.0, a.data_ptr(), b.data_ptr(), 0.0, None, d.data_ptr()))
    call()
    tuned = p.report()
    assert tuned["choice"] == "autotuned" and ".tcgen05." in tuned["family"]
    call()
    assert p.report()["choice"] == "tuning-cache"
    ex.set_workspace_limit(64)
    call()
    rep = p.report()
    assert ".tcgen05." not in rep["family"] and rep["choice"] == "model"
    ex.close()


def labelled_call(tp, torch, dtype, spec, ext, beta, limits):
    """Runs the column-major contraction under each workspace limit (None: none) and yields
    (status, family, error against 64 bits)."""
    gen = torch.Generator(device="cuda").manual_seed(11)
    lhs, out = spec.split("->")
    la, lb = lhs.split(",")
    kind = torch.complex64 if dtype == tp.C32 else torch.float32

    def make(labels):
        shape = [ext[x] for x in labels]
        t = torch.randn(int(np.prod(shape)), generator=gen, device="cuda", dtype=kind)
        st = np.cumprod([1] + shape[:-1]).tolist()
        return t.as_strided(shape, st), tp.TensorInfo(dtype, shape, st), [ord(x) for x in labels]

    (a, ia, na), (b, ib, nb), (d, idd, nd) = make(la), make(lb), make(out)
    c = d.clone()
    h = tp.Handle()
    p = tp.TensorProduct.create(h, (0, ia, na), (0, ib, nb), (0, idd, nd), (0, idd, nd))
    wide = torch.complex128 if dtype == tp.C32 else torch.float64
    want = torch.einsum(spec, a.to(wide), b.to(wide)) + beta * c.to(wide)
    for limit in limits:
        ex = tp.Executor()
        if limit:
            ex.set_workspace_limit(limit)
        d.copy_(c)
        torch.cuda.synchronize()
        status = p.execute(ex, 1.0, a.data_ptr(), b.data_ptr(), beta, d.data_ptr() if beta else None, d.data_ptr())
        ex.close()
        yield status, p.report()["family"], float((d.to(wide) - want).norm() / want.norm())


# The cap leaves no room for what the tensor-core family lays out (a panel, planes of 6 bytes
# a real), but for what the general choice needs: nothing for a direct tile, packed panels
# of 4 bytes a real (tiles enough that it does not split K, which takes partials as well).
WITHIN = [
    ("ikmb,mjac->abcijk", dict(a=12, b=11, c=20, i=13, j=11, k=12, m=9), ".stream.", {"F32": 1 << 10, "C32": 1 << 10}),
    ("cbka,kj->abjc", dict(a=50, b=21, c=22, j=60, k=40), ".stream.", {"F32": 1 << 10, "C32": 1 << 10}),
    ("ka,kb->ab", dict(a=30000, b=32, k=24), ".stream.", {"F32": 1 << 10, "C32": 1 << 10}),
    ("mk,kn->mn", dict(m=2000, n=1900, k=700), ".split.", {"F32": 16 << 20, "C32": 40 << 20}),
    ("km,nk->mn", dict(m=2000, n=1900, k=600), ".split.", {"F32": 12 << 20, "C32": 36 << 20}),
]


@pytest.mark.parametrize("beta", [0.0, 0.5])
@pytest.mark.parametrize("spec,ext,family,limits", WITHIN)
@pytest.mark.parametrize("dtype", ["F32", "C32"])
def test_device_operands_under_a_workspace_cap(tp, torch_cuda, dtype, spec, ext, family, limits, beta):
    (s0, f0, e0), (s1, f1, e1) = labelled_call(tp, torch_cuda, getattr(tp, dtype), spec, ext, beta, (None, limits[dtype]))
    assert s0 == 0 and family in f0 and e0 <= 1e-6, (s0, f0, e0)
    assert s1 == 0 and ".tcgen05." not in f1 and e1 <= 1e-6, (s1, f1, e1, tp.last_error())

"""The gather-fed stream tiles on a B200, through the C ABI: persistent CTAs
whose producer warp gathers operand stages for the compute warps
(csrc/k_stream.cu), chosen by the model for contractions with at least a wave of
tiles whose gathers are coalesced.

Against the extended-precision label oracle at the plain bounds (relative
Frobenius f32 / c32 <= 1e-6, f64 / c64 <= 1e-13) over the forms the rule accepts:
either index fast in each operand, 16-byte groups or not (odd extents, odd
leading dimensions, an origin one element off), either output orientation, K
from 1 through the ends of a 16-deep stage, one row or column past a tile,
batches, negative strides, alpha / beta with C and in place; and against the
direct tile pinned on the same plan."""
import numpy as np
import pytest

from test_gpu_parity import Op, make_product, oracle_ref, plain_tol, rnd

pytestmark = pytest.mark.gpu

DIRECT = {"float64": 3}
DTYPES = list(DIRECT)


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


# (m, n, k, batch, A k-fast, B k-fast, D n-fast, leading pad, origin shift, beta, C: none / own / in place)
FORMS = [
    (1281, 577, 1, 1, False, True, False, 0, 0, 0.0, None),
    (1280, 641, 3, 1, True, False, False, 0, 0, 0.0, None),
    (1290, 578, 4, 1, True, True, False, 0, 0, 0.0, None),
    (1290, 578, 5, 1, False, False, True, 0, 0, 0.0, None),
    (1283, 600, 12, 1, True, True, True, 1, 0, 0.0, None),
    (1284, 600, 13, 1, False, True, False, 4, 0, -0.75, "own"),
    (1284, 600, 16, 1, False, True, False, 0, 1, 0.5, "in place"),
    (1284, 600, 17, 1, True, False, False, 4, 0, 0.0, None),
    (1281, 599, 50, 1, False, False, False, 3, 0, 0.0, None),
    (1281, 599, 66, 1, True, True, True, 0, 0, 0.5, "in place"),
    (30011, 31, 33, 1, False, True, False, 1, 0, 0.0, None),
    (29, 30000, 24, 1, True, True, False, 0, 0, 0.0, None),
    (20003, 45, 40, 1, True, True, False, 0, 0, 1.0, "own"),
    (20003, 72, 20, 1, True, False, False, 0, 0, 0.0, None),
    (130, 70, 100, 60, False, True, False, 2, 0, 0.0, None),
    (65, 129, 37, 70, True, False, True, 1, 0, -1.0, "own"),
]


def operand(rng, dt, rows, k, h, kfast, pad, shift, labels, conj=False, negate=False):
    ld = (k if kfast else rows) + pad
    slow = rows if kfast else k
    st = [ld, 1] if kfast else [1, ld]
    buf = rnd(rng, dt, shift + h * ld * slow)
    off = shift
    if negate:  # the rows in reverse order
        off += (rows - 1) * st[0]
        st = [-st[0], st[1]]
    ext, strides = [rows, k, h], st + [ld * slow]
    return Op(buf, ext[:3 if h > 1 else 2], strides[:3 if h > 1 else 2], labels[:3 if h > 1 else 2], off, conj)


@pytest.mark.parametrize("dt", DTYPES)
@pytest.mark.parametrize("form", FORMS, ids=lambda f: "x".join(str(x) for x in f[:4]))
def test_stream_tiles_over_layout_forms(tp, ex, torch_cuda, orc, dt, form):
    m, n, k, h, akf, bkf, dnf, pad, shift, beta, cmode = form
    torch = torch_cuda
    cplx = dt.startswith("complex")
    rng = np.random.default_rng(m + 3 * n + 7 * k)
    A = operand(rng, dt, m, k, h, akf, pad, shift, [0, 2, 9], conj=cplx, negate=pad == 3)
    B = operand(rng, dt, n, k, h, bkf, pad, 0, [1, 2, 9], conj=cplx and k % 2 == 1)
    est = [n, 1, m * n] if dnf else [1, m, m * n]
    ext = [m, n, h][:3 if h > 1 else 2]
    d0 = rnd(rng, dt, m * n * h) if cmode else np.zeros(m * n * h, dtype=dt)
    D = Op(d0, ext, est[:len(ext)], [0, 1, 9][:len(ext)], conj=cplx and k % 3 == 0)
    C = None
    if cmode == "own":
        C = Op(rnd(rng, dt, m * n * h), ext, ([1, m, m * n] if dnf else [n, 1, m * n])[:len(ext)], D.lab)
    elif cmode:
        C = D
    al = (complex(0.5, 0.25) if cplx else 1.5) if cmode else 1.0
    want = oracle_ref(orc, dt, A, B, C, D, al, beta, d0)
    tens = {x: torch.from_numpy(o.buf).cuda() for x, o in (("a", A), ("b", B)) + ((("c", C),) if cmode == "own" else ())}
    ptr = lambda x, o: tens[x].data_ptr() + o.offset * o.buf.itemsize
    p = make_product(tp, dt, A, B, C, D)
    got = {}
    for kernel in (0, DIRECT[dt]):
        p.set_kernel(kernel)
        td = torch.from_numpy(d0.copy()).cuda()
        c = None if cmode is None else td.data_ptr() if cmode == "in place" else ptr("c", C)
        assert p.execute(ex, al, ptr("a", A), ptr("b", B), beta, c, td.data_ptr()) == 0, tp.last_error()
        torch.cuda.synchronize()
        if kernel == 0:
            assert ".stream." in p.report()["family"], p.report()["family"]
        got[kernel] = td.cpu().numpy()
        assert orc.rel_frobenius(got[kernel], want) <= plain_tol(dt), (kernel, p.report()["family"])
    assert orc.rel_frobenius(got[0], got[DIRECT[dt]].astype(want.dtype)) <= plain_tol(dt)


def test_uncoalesced_operands_keep_the_other_families(tp, ex, torch_cuda, orc):
    """The rule's other side: a batch-innermost layout (every gather strided) is
    not given to the stream tiles."""
    h, m, n, k = 16, 130, 260, 20
    rng = np.random.default_rng(5)
    A = Op(rnd(rng, "float64", h * m * k), [h, k, m], [1, h, h * k], [9, 2, 0])
    B = Op(rnd(rng, "float64", h * n * k), [h, k, n], [1, h, h * k], [9, 2, 1])
    d0 = np.zeros(h * m * n)
    D = Op(d0, [h, m, n], [1, h, h * m], [9, 0, 1])
    p = make_product(tp, "float64", A, B, None, D)
    assert ".stream." not in p.report()["family"]


def test_grouped_list_of_stream_tiles(tp, torch_cuda):
    """A list of f64 contractions over either fast index, either output
    orientation, 16-byte groups or not, extents around a tile's edges, K from 1 to
    past a stage, with C in place: grouped (captured and replayed) against the same
    plans one by one on the direct tile and against float64 einsum."""
    torch = torch_cuda
    ex = tp.Executor()
    rng = np.random.default_rng(12)
    gen = torch.Generator(device="cuda").manual_seed(3)
    rand = lambda n: torch.randn(n, dtype=torch.float64, device="cuda", generator=gen)
    cases = [(m, n, k) for m in (1, 17, 64, 65, 200) for n in (3, 48, 64, 130) for k in (1, 4, 13, 16, 50)]
    items, singles, outs = [], [], []
    for i, (m, n, k) in enumerate(cases):
        akf, bkf, dnf = (bool(x) for x in rng.integers(0, 2, 3))
        beta = 0.5 if i % 3 == 0 else 0.0
        sa, sb, sd = [k, 1] if akf else [1, m], [1, k] if bkf else [n, 1], [n, 1] if dnf else [1, m]
        a, b, d0 = rand(m * k), rand(k * n), rand(m * n)
        spec = [tp.OperandSpec(tp.LayoutSpec(e, s)) for e, s in (([m, k], sa), ([k, n], sb), ([m, n], sd))]
        prob = tp.Problem.from_labels(tp.F64, *spec, [0, 2], [2, 1], [0, 1])
        want = a.as_strided([m, k], sa) @ b.as_strided([k, n], sb) + beta * d0.as_strided([m, n], sd)
        d1, d2 = d0.clone(), d0.clone()
        for d, plan, to in ((d1, tp.Plan(prob), items), (d2, tp.Plan(prob, tp.PlanConfig(kernel=3)), singles)):
            c = d.data_ptr() if beta else None
            to.append(tp.Item(plan, 1.0, a.data_ptr(), b.data_ptr(), d.data_ptr(), beta, c))
        outs.append((a, b, d0, d1, d2, want, sd, [m, n]))
    torch.cuda.synchronize()
    batch = tp.PreparedBatch(items)
    for rep in range(2):  # captured, then replayed
        for o in outs:
            o[3].copy_(o[2])
        torch.cuda.synchronize()
        batch.run(ex)
        ex.synchronize()
        for o, c in zip(outs, cases):
            got = o[3].as_strided(o[7], o[6])
            assert float((got - o[5]).norm() / o[5].norm()) <= 1e-13, (c, rep)
    ex.set_grouping(False)
    tp.PreparedBatch(singles).run(ex)
    ex.synchronize()
    for o, c in zip(outs, cases):
        assert float((o[3] - o[4]).norm() / o[4].norm()) <= 1e-13, c
    ex.close()

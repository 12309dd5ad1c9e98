"""f32 and c32 contractions on the tensor cores with the operands split on the way
into shared memory (csrc/k_tcstream.cu) or, where large, into BF16 planes first (csrc/k_split.cu), on a
B200.

Against the extended-precision label oracle at the plain bound (relative Frobenius
1e-6) over the forms the rule accepts: either index fast in each operand, 16-byte
groups or not, either output orientation, K at the ends of a 16-deep step, a
32-deep stage and a 128-deep chunk, one row or column past a tile, narrow outputs,
batches (outermost and innermost, through panels), negative strides, conjugation,
alpha / beta with C and in place. Then values that the BF16 planes cannot carry:
infinities, NaN, products near overflow and near underflow must come out as from
the FFMA tile."""
import numpy as np
import pytest

from test_gpu_parity import Op, make_product, oracle_ref, plain_tol, rnd

pytestmark = pytest.mark.gpu

DIRECT = {"float32": 1, "complex64": 5}


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


# (m, n, k, batch, A k-fast, B k-fast, D n-fast, leading pad, origin shift, beta, C: none / own / in place);
# f32 takes four times the larger of m and n.
FORMS = [
    (2900, 2900, 1, 1, False, True, False, 0, 0, 0.0, None),
    (1700, 1290, 4, 1, True, True, False, 0, 0, 0.0, None),
    (1281, 577, 15, 1, False, False, True, 1, 0, 0.0, None),
    (1281, 577, 16, 1, False, True, False, 0, 1, 0.5, "in place"),
    (1280, 640, 17, 1, True, False, False, 4, 0, -0.75, "own"),
    (1283, 600, 32, 1, True, True, True, 0, 0, 0.0, None),
    (1283, 600, 33, 1, False, False, False, 3, 0, 0.0, None),
    (641, 129, 128, 1, True, False, False, 0, 0, 0.0, None),
    (641, 129, 129, 1, True, True, False, 4, 0, 1.0, "own"),
    (30011, 31, 33, 1, False, True, False, 1, 0, 0.0, None),
    (120, 30000, 24, 1, True, True, False, 0, 0, 0.0, None),
    (130, 70, 100, 30, False, True, False, 2, 0, 0.0, None),
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


def form_ops(dt, form):
    m, n, k, h, akf, bkf, dnf, pad, shift, beta, cmode = form
    if dt == "float32":
        m, n = (4 * m, n) if m >= n else (m, 4 * n)
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
    return A, B, C, D, al


def execute(torch, p, ex, dt, A, B, C, D, al, beta):
    dev = [torch.from_numpy(o.buf).cuda() for o in (A, B)]
    ptr = [t.data_ptr() + o.offset * o.buf.itemsize for t, o in zip(dev, (A, B))]
    td = torch.from_numpy(D.buf.copy()).cuda()
    tc = None if C is None else td if C is D else torch.from_numpy(C.buf).cuda()
    return p.execute(ex, al, ptr[0], ptr[1], beta, tc.data_ptr() if C is not None else None, td.data_ptr()), td


@pytest.mark.parametrize("dt", sorted(DIRECT))
@pytest.mark.parametrize("form", FORMS, ids=lambda f: "x".join(str(x) for x in f[:4]))
def test_layout_forms(tp, ex, torch_cuda, orc, dt, form):
    beta = form[9]
    A, B, C, D, al = form_ops(dt, form)
    want = oracle_ref(orc, dt, A, B, C, D, al, beta, D.buf)
    p = make_product(tp, dt, A, B, C, D)
    assert ".tcgen05.stream." in p.report()["family"], p.report()["family"]
    status, td = execute(torch_cuda, p, ex, dt, A, B, C, D, al, beta)
    assert status == 0, tp.last_error()
    torch_cuda.cuda.synchronize()
    assert orc.rel_frobenius(td.cpu().numpy(), want) <= plain_tol(dt)


def dense(dt, rng, term, e, zero=False, conj=False):
    ext = [e[x] for x in term]
    st = np.cumprod([1] + ext[:-1]).tolist()
    n = int(np.prod(ext))
    return Op(np.zeros(n, dtype=dt) if zero else rnd(rng, dt, n), ext, st, [ord(x) for x in term], conj=conj)


@pytest.mark.parametrize("spec,sizes", [
    ("ikmb,mjac->abcijk", dict(a=12, b=11, c=20, i=13, j=11, k=12, m=9)),   # rows of A far apart in D's order
    ("hki,hkj->hij", dict(h=37, i=210, j=260, k=66)),                       # batch innermost
    ("cbka,kj->abjc", dict(a=50, b=21, c=22, j=60, k=40)),                  # the large operand through a panel
])
@pytest.mark.parametrize("beta", [0.0, 0.5])
@pytest.mark.parametrize("dt", sorted(DIRECT))
def test_panels(tp, ex, torch_cuda, orc, dt, beta, spec, sizes):
    """Operands whose gather is not coalesced go through dense panels, or take the
    families that need no panel where the workspace cap leaves no room."""
    rng = np.random.default_rng(8)
    cplx = dt.startswith("complex")
    ta, tb, td = spec.replace("->", ",").split(",")
    A, B, D = dense(dt, rng, ta, sizes, conj=cplx), dense(dt, rng, tb, sizes), dense(dt, rng, td, sizes, zero=beta == 0.0)
    C = D if beta else None
    want = oracle_ref(orc, dt, A, B, C, D, 1.0, beta, D.buf)
    p = make_product(tp, dt, A, B, C, D)
    small = tp.Executor()
    small.set_workspace_limit(4096)
    status, got = execute(torch_cuda, p, ex, dt, A, B, C, D, 1.0, beta)
    assert status == 0, tp.last_error()
    torch_cuda.cuda.synchronize()
    assert ".tcgen05.stream." in p.report()["family"], p.report()["family"]
    assert orc.rel_frobenius(got.cpu().numpy(), want) <= plain_tol(dt)
    status, got = execute(torch_cuda, p, small, dt, A, B, C, D, 1.0, beta)
    if spec.startswith("ik"):  # the general choice for it needs no workspace
        assert status == 0, tp.last_error()
    if status == 0:
        torch_cuda.cuda.synchronize()
        assert ".stream." not in p.report()["family"]
        assert orc.rel_frobenius(got.cpu().numpy(), want) <= plain_tol(dt)
    small.close()


@pytest.mark.parametrize("case", ["inf", "nan", "overflow", "tiny", "denormal", "graded", "zeros"])
@pytest.mark.parametrize("dt", sorted(DIRECT))
def test_values_outside_the_planes(tp, ex, torch_cuda, orc, dt, case):
    m, n, k = 4000, 390, 40
    rng = np.random.default_rng(3)
    A = operand(rng, dt, m, k, 1, False, 0, 0, [0, 2, 9])
    B = operand(rng, dt, n, k, 1, True, 0, 0, [1, 2, 9])
    a, b = A.buf, B.buf
    if case == "inf":
        a[5], a[777 * 3] = np.inf, -np.inf
    elif case == "nan":
        a[1234], b[77] = np.nan, np.nan
    elif case == "overflow":
        a[:4 * m:7] *= np.float32(3e38)
        b[::11] *= np.float32(3.0)
    elif case == "tiny":
        a *= np.float32(1e-17)
        b *= np.float32(1e-17)
    elif case == "denormal":
        a *= np.float32(1e-40)
    elif case == "graded":
        a *= (10.0 ** rng.uniform(-30, 0, a.size)).astype("float32")
        b *= (10.0 ** rng.uniform(-8, 8, b.size)).astype("float32")
    else:
        a[: a.size // 2] = 0
        b[::2] = 0
    D = Op(np.zeros(m * n, dtype=dt), [m, n], [1, m], [0, 1])
    p = make_product(tp, dt, A, B, None, D)
    got = {}
    for kernel in (0, DIRECT[dt]):
        p.set_kernel(kernel)
        status, td = execute(torch_cuda, p, ex, dt, A, B, None, D, 1.0, 0.0)
        assert status == 0, tp.last_error()
        torch_cuda.cuda.synchronize()
        if kernel == 0:
            assert ".tcgen05.stream." in p.report()["family"], p.report()["family"]
        got[kernel] = td.cpu().numpy().view("float32")
    x, y = got[0], got[DIRECT[dt]]
    assert np.array_equal(np.isnan(x), np.isnan(y))
    inf = np.isinf(y)
    assert np.array_equal(np.isinf(x), inf) and np.array_equal(x[inf], y[inf])
    ok = np.isfinite(y)
    if case in ("tiny", "denormal", "graded", "zeros"):
        # Each output within 40 roundings of the sum of its products' magnitudes
        # (and 40 steps of the smallest denormal).
        wide = np.complex128 if dt.startswith("complex") else np.float64
        am, bm = np.abs(a.astype(wide).reshape(k, m)), np.abs(b.astype(wide).reshape(n, k))
        mag = (bm @ am).reshape(-1)
        if dt.startswith("complex"):
            mag = np.repeat(mag, 2)
        lim = 40 * (2.0 ** -24 * mag + 2.0 ** -149)
        assert np.all(np.abs(x.astype("float64") - y.astype("float64")) <= 2 * lim)
    else:
        assert orc.rel_frobenius(x[ok], y[ok].astype("float64")) <= plain_tol(dt)


# (spec, extents, A conj, D permuted strides, beta): rows and columns past a tile, K past a
# chunk, an only wave whose depth is split, a last wave that is, batches, strided gathers.
SPLIT_FORMS = [
    ("km,kn->mn", dict(m=1100, n=1300, k=2500), True, False, 0.0),
    ("mk,nk->nm", dict(m=1025, n=1281, k=2411), False, False, 0.5),
    ("mk,kn->mn", dict(m=4100, n=2309, k=1530), True, False, 0.5),
    ("mkh,knh->mnh", dict(m=700, n=900, k=2090, h=9), False, False, 0.0),
    ("kmlo,nlpk->mnop", dict(k=47, m=40, l=50, o=36, n=33, p=40), True, False, 0.0),
]


def split_case(torch, tp, dt, form, seed=5):
    spec, e, conj, _, beta = form
    if dt == "float32":
        e = dict(e, m=2 * e["m"])  # enough work for the planes' pass
    ta, tb, td = spec.replace("->", ",").split(",")
    tdt = getattr(torch, dt)
    gen = torch.Generator(device="cuda").manual_seed(seed)

    def make(term):
        ext = [e[x] for x in term]
        st = np.cumprod([1] + ext[:-1]).tolist()
        return torch.randn(int(np.prod(ext)), dtype=tdt, device="cuda", generator=gen).as_strided(ext, st)

    A, B, D = make(ta), make(tb), make(td)
    conj = conj and dt.startswith("complex")
    lay = lambda t, c=False: tp.OperandSpec(tp.LayoutSpec(list(t.shape), list(t.stride())), c)
    code = {"float32": tp.F32, "complex64": tp.C32}[dt]
    lab = lambda t: [ord(x) for x in t]
    prob = tp.Problem.from_labels(code, lay(A, conj), lay(B), lay(D), lab(ta), lab(tb), lab(td))
    return A, B, D, conj, prob


@pytest.mark.parametrize("dt", sorted(DIRECT))
@pytest.mark.parametrize("form", SPLIT_FORMS, ids=lambda f: f[0])
def test_planes_packed_first(tp, torch_cuda, dt, form):
    torch = torch_cuda
    ex = tp.Executor(device=0, stream=torch.cuda.current_stream().cuda_stream, sync=False)
    A, B, D, conj, prob = split_case(torch, tp, dt, form)
    plan = tp.Plan(prob)
    assert ".tma.split." in plan.report()["family"], plan.report()["family"]
    wide = torch.complex128 if dt.startswith("complex") else torch.float64
    a = A.to(wide).conj() if conj else A.to(wide)
    want = torch.einsum(form[0], a, B.to(wide)) + form[4] * D.to(wide)
    if form[4]:
        plan.execute_into_accum(ex, 1.0, A, B, form[4], D, c=D)
    else:
        plan.execute_into(ex, 1.0, A, B, D)
    torch.cuda.synchronize()
    assert float((D.to(wide) - want).norm() / want.norm()) <= plain_tol(dt)
    ex.close()


@pytest.mark.parametrize("case", ["inf", "nan", "overflow", "tiny", "denormal"])
@pytest.mark.parametrize("form", [SPLIT_FORMS[0], SPLIT_FORMS[2]], ids=["split wave", "split tail"])
@pytest.mark.parametrize("dt", sorted(DIRECT))
def test_values_outside_the_packed_planes(tp, torch_cuda, dt, form, case):
    """As from the direct tile; a few rows and columns hold the values, so that the
    other tiles stay on the tensor cores."""
    torch = torch_cuda
    ex = tp.Executor(device=0, stream=torch.cuda.current_stream().cuda_stream, sync=False)
    A, B, D, conj, prob = split_case(torch, tp, dt, form[:4] + (0.0,))
    ta = form[0].split(",")[0]
    rows = A if ta[0] == "m" else A.transpose(0, 1)  # [m, k]
    cols = B.transpose(0, 1)                         # [n, k] of "kn"
    if case == "inf":
        rows[3, 5], rows[1000, 77] = float("inf"), float("-inf")
    elif case == "nan":
        rows[130, 1], cols[7, 9] = float("nan"), float("nan")
    elif case == "overflow":
        rows[64:70] *= 3e37
        cols[:9] *= 40.0
    elif case == "tiny":
        rows[200:300] *= 1e-17
        cols[100:200] *= 1e-17
    else:
        rows[:150] *= 1e-40
    res = []
    for kernel in (0, DIRECT[dt]):
        plan = tp.Plan(prob, tp.PlanConfig(kernel=kernel))
        D.zero_()
        plan.execute_into(ex, 1.0, A, B, D)
        torch.cuda.synchronize()
        res.append(torch.view_as_real(D).double() if dt.startswith("complex") else D.double())
    x, y = res
    assert torch.equal(torch.isnan(x), torch.isnan(y))
    inf = torch.isinf(y)
    assert torch.equal(torch.isinf(x), inf) and torch.equal(x[inf], y[inf])
    wide = torch.complex128 if dt.startswith("complex") else torch.float64
    mag = torch.einsum(form[0], A.abs().double(), B.abs().double())
    if dt.startswith("complex"):
        mag = mag.unsqueeze(-1).expand(x.shape)
    # Each output within 60 roundings of the sum of its products' magnitudes.
    ok = torch.isfinite(y) & torch.isfinite(mag)
    assert bool(((x - y).abs()[ok] <= 60 * (2.0 ** -24 * mag[ok] + 2.0 ** -149)).all())
    ex.close()

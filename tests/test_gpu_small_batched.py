"""Batches of small products on a B200 through the C ABI: whole products in
shared memory (csrc/k_small.cu), chosen by the model for M, N, K <= 32 and 256 or
more batch entries.

Against the extended-precision label oracle at the plain bounds, over the layout
forms the kernel takes (batch outermost and contiguous with an origin off the
16-byte boundary, k fast with odd and even K, batch innermost, padded, two batch
axes that do not fold), with conjugation, alpha, beta and C, sizes at the edges
of its blocks (1, 2, 4, 5, 31, 32), and a batch that ends inside a group."""
import numpy as np
import pytest

from test_gpu_parity import Op, make_product, oracle_ref, plain_tol, rnd

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


def dense(order, ext, pad=0):
    """Element strides of the labels `order` (fastest first), `pad` between the steps of the second."""
    st, acc = {}, 1
    for i, x in enumerate(order):
        st[x] = acc
        acc = acc * ext[x] + (pad if i == 0 else 0)
    return st, acc


# (m, n, k, batch axes, order of A, B, D labels fastest first, padding, origin shift, C)
FORMS = [
    (4, 4, 4, (300,), "mkh", "knh", "mnh", 0, 0, False),
    (5, 7, 13, (257,), "mkh", "knh", "mnh", 0, 1, False),
    (5, 7, 12, (401,), "kmh", "nkh", "nmh", 0, 0, False),
    (32, 4, 32, (259,), "kmh", "knh", "mnh", 0, 0, True),
    (31, 32, 32, (256,), "mkh", "nkh", "mnh", 1, 0, False),
    (32, 31, 17, (262,), "hmk", "hkn", "hmn", 0, 0, True),
    (1, 32, 5, (333,), "mhk", "khn", "mhn", 0, 3, False),
    (2, 30, 1, (511,), "mkh", "knh", "mnh", 0, 0, True),
    (16, 1, 31, (300,), "kmh", "knh", "nmh", 2, 0, False),
    (3, 6, 9, (20, 17), "mgkh", "hkng", "gmhn", 0, 0, True),
]


@pytest.mark.parametrize("dt", ["float32", "float64", "complex64", "complex128"])
@pytest.mark.parametrize("form", FORMS, ids=lambda f: "x".join(str(x) for x in f[:3]) + "-" + f[4])
def test_small_batches_over_layout_forms(tp, ex, torch_cuda, orc, dt, form):
    m, n, k, batch, oa, ob, od, pad, shift, with_c = form
    torch = torch_cuda
    cplx = dt.startswith("complex")
    ext = {"m": m, "n": n, "k": k, "h": batch[0], "g": batch[1] if len(batch) > 1 else 1}
    ids = {"m": 0, "n": 1, "k": 2, "h": 9, "g": 10}
    rng = np.random.default_rng(100 * m + 10 * n + k)

    def op(order, conj=False, init=True):
        st, total = dense(order, ext, pad)
        total += pad * int(np.prod([ext[x] for x in order[1:]]))
        buf = rnd(rng, dt, total + shift) if init else np.zeros(total + shift, dtype=dt)
        return Op(buf, [ext[x] for x in order], [st[x] for x in order], [ids[x] for x in order], shift, conj)

    A, B = op(oa, conj=cplx), op(ob, conj=cplx and k % 2 == 0)
    D = op(od, conj=cplx and with_c, init=with_c)
    C = op(od[::-1]) if with_c else None
    al, be = ((complex(0.5, 0.25), complex(-1.0, 0.5)) if cplx else (1.5, -0.75)) if with_c else (1.0, 0.0)
    want = oracle_ref(orc, dt, A, B, C, D, al, be, D.buf)
    p = make_product(tp, dt, A, B, C, D)
    assert "small-batched" in p.report()["family"], p.report()["family"]
    dev = {id(o): torch.from_numpy(o.buf.copy()).cuda() for o in (A, B, C, D) if o is not None}
    ptr = lambda o: None if o is None else dev[id(o)].data_ptr() + o.offset * o.buf.itemsize
    assert p.execute(ex, al, ptr(A), ptr(B), be, ptr(C), ptr(D)) == 0, tp.last_error()
    torch.cuda.synchronize()
    got = dev[id(D)].cpu().numpy()
    assert orc.rel_frobenius(got, want) <= plain_tol(dt), p.report()["family"]
    # Elements between the addressed ones keep their values.
    inside = np.zeros(D.buf.size, dtype=bool)
    idx = np.full([1] * len(D.ext), D.offset)
    for axis, (e, s) in enumerate(zip(D.ext, D.st)):
        idx = idx + (np.arange(e) * s).reshape([-1 if i == axis else 1 for i in range(len(D.ext))])
    inside[idx.ravel()] = True
    assert np.array_equal(got[~inside], D.buf[~inside])

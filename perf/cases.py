"""The measured workloads: what a program that uses this library has it do.

Every case goes through the public Python front end (`tprims_b200`): plans of
labelled contractions executed on torch CUDA tensors, the vector-Jacobian
product, and lists of N-ary networks. Shapes come from the repository's own
benchmark configurations (`bench.py`) and from the shape corpora under
`tests/golden/` (`corpus.json`: tensor-network and batched GEMM shapes;
`tccg.json`: the 49 TCCG contractions), or are generic members of the same
families; `draw` spreads sizes over the ranges those files span.

All tensors are column-major in the order their labels are written (the first
label has stride 1), as in both corpora; `a_lead` > 1 gives A a non-unit
leading stride. A contraction whose labels put the batch index first is
therefore batch-innermost.
"""
import math
import os
import sys

import torch

sys.path.insert(0, os.path.join(os.getcwd(), "tensoralgebra-rs_b200"))

import tprims_b200 as tp  # noqa: E402

TORCH = {"f32": torch.float32, "f64": torch.float64, "c32": torch.complex64, "c64": torch.complex128}
CODE = {"f32": tp.F32, "f64": tp.F64, "c32": tp.C32, "c64": tp.C64}
BYTES = {"f32": 4, "f64": 8, "c32": 8, "c64": 16}
SCHEME = {"plain": tp.PREC_PLAIN, "bf16x6": tp.PREC_BF16X6, "ozaki": tp.PREC_OZAKI_INT8}


def contraction(name, spec, sizes, dtype, scheme="plain", dist="uniform", conj=False, beta=0.0, a_lead=1, sync=False):
    """A binary contraction `spec` ("ak,kb->ab") with the extents `sizes`
    ("a=3,k=4,b=5"). `conj` conjugates A. `sync` uses a blocking executor (the
    C ABI's contract); otherwise the executor is asynchronous, as a GPU
    program that chains calls on one stream keeps it."""
    case = {"kind": "contract", "spec": spec, "sizes": sizes, "dtype": dtype, "scheme": scheme, "dist": dist,
            "conj": conj, "beta": beta, "a_lead": a_lead, "sync": sync}
    return dict(case, name=name) if name else case


def vjp(name, sizes, dtype):
    """Forward and cotangents of D[i,j] = sum_{k,l} A[i,k,k,l] B[l,j,k]."""
    case = {"kind": "vjp", "spec": "ikkl,ljk->ij", "sizes": sizes, "dtype": dtype}
    return dict(case, name=name) if name else case


def updates(name, count, dtype, list_seed):
    """A list of `count` environment updates
    E'[x,t,y] = sum E[a,s,b] M[a,p,x] W[s,p,t,q] conj(M2[b,q,y]), uneven bonds
    drawn from `list_seed` (the shapes belong to the case, the values do not)."""
    case = {"kind": "updates", "count": count, "dtype": dtype, "list_seed": list_seed}
    return dict(case, name=name) if name else case


def listed():
    return [
        # The smallest call: a 16 x 16 x 16 product of a tensor-network program
        # (corpus.json has it 32 times per run, among hundreds of its size),
        # through a blocking executor as a C ABI caller has it.
        contraction("small_f64", "ak,kb->ab", "a=16,b=16,k=16", "f64", sync=True),
        # The permuted product of bench.py's first configuration, accumulating
        # half of C: the ordinary mid-size call.
        contraction("permuted_f64", "aebf,fced->abcd", "a=24,b=24,c=24,d=24,e=24,f=24", "f64", beta=0.5),
        # bench.py's headline contraction in drop-in FP32, M = N = K = 4096
        # with a strided A: the largest.
        contraction("large_f32", "kmlo,nlpk->mnop", "k=64,m=64,l=64,o=64,n=64,p=64", "f32", dist="normal", a_lead=2),
        # The same contraction in split precision.
        contraction("large_bf16x6", "kmlo,nlpk->mnop", "k=64,m=64,l=64,o=64,n=64,p=64", "f32", scheme="bf16x6",
                    dist="normal", a_lead=2),
        # bench.py's batched conjugated complex product, batch innermost, on
        # the FP64 path and on the INT8 slices.
        contraction("batched_c64", "hki,hkj->hij", "h=64,i=384,j=384,k=384", "c64", conj=True),
        contraction("batched_ozaki_c64", "hki,hkj->hij", "h=64,i=384,j=384,k=384", "c64", scheme="ozaki", conj=True),
        # One sweep's worth of bench.py's uneven environment updates, as one
        # list of networks.
        updates("updates_f64", 256, "f64", 4000),
        # A short-K TCCG contraction (coupled-cluster triples) that writes a
        # permuted six-index output.
        contraction("triples_f32", "ikmb,mjac->abcijk", "a=24,b=16,c=16,i=24,j=16,k=16,m=24", "f32"),
        # A tall product of a tensor-network program with odd sizes
        # (corpus.json: M = 177147, N = 243, K = 50).
        contraction("tall_f64", "ak,kb->ab", "a=177147,b=243,k=50", "f64"),
        # An integral transformation (TCCG, 72-extent modes) on complex64 data.
        contraction("transform_c32", "kbac,jk->abjc", "a=72,b=52,j=72,c=52,k=72", "c32"),
        # Many small products in one call, batch outermost (corpus.json:
        # 8192 products of 32 x 4 x 32).
        contraction("batched_small_f64", "mkh,knh->mnh", "m=32,n=4,k=32,h=8192", "f64"),
        # A differentiable layer: forward and both cotangents with a repeated
        # index on A (bench.py's last configuration at a quarter of its k).
        vjp("vjp_f64", "i=512,j=512,k=32,l=256", "f64"),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _sizes(**ext):
    return ",".join(f"{k}={v}" for k, v in ext.items())


def draw(rng):
    kind = rng.choice(["small", "permuted", "gemm", "split", "batched", "ozaki", "updates", "triples", "tall",
                       "transform", "batched_small", "vjp"])
    any_dtype = rng.choice(["f32", "f64", "c32", "c64"])
    if kind == "small":
        a, b, k = (_log_int(rng, 2, 64) for _ in range(3))
        spec = rng.choice(["ak,kb->ab", "ka,kb->ab", "ak,bk->ba"])
        return contraction(None, spec, _sizes(a=a, b=b, k=k), any_dtype, sync=True)
    if kind == "permuted":
        e = {x: rng.randint(8, 28) for x in "abcdef"}
        spec = rng.choice(["aebf,fced->abcd", "eafb,cedf->cadb", "abef,efcd->dcba"])
        return contraction(None, spec, _sizes(**e), rng.choice(["f64", "f32", "c64"]), beta=rng.choice([0.0, 0.5]))
    if kind == "gemm":
        m, n, k = (_log_int(rng, 256, 4096) for _ in range(3))
        spec = rng.choice(["mk,kn->mn", "km,kn->mn", "mk,nk->nm"])
        if any_dtype != "f32":  # slower pipes: the same cost ceiling in time
            m, n, k = (min(x, 2048) for x in (m, n, k))
        return contraction(None, spec, _sizes(m=m, n=n, k=k), any_dtype, dist="normal")
    if kind == "split":
        e = {x: rng.randint(24, 64) for x in "kmlonp"}
        return contraction(None, "kmlo,nlpk->mnop", _sizes(**e), "f32", scheme="bf16x6", dist="normal",
                           a_lead=rng.choice([1, 2]))
    if kind in ("batched", "ozaki"):
        h = _log_int(rng, 8, 64)
        i, j, k = (rng.randint(64, 384) for _ in range(3))
        spec = rng.choice(["hki,hkj->hij", "kih,kjh->ijh"])
        if kind == "ozaki":
            return contraction(None, spec, _sizes(h=h, i=i, j=j, k=k), rng.choice(["f64", "c64"]), scheme="ozaki",
                               conj=False)
        return contraction(None, spec, _sizes(h=h, i=i, j=j, k=k), any_dtype, conj=any_dtype[0] == "c")
    if kind == "updates":
        dt = rng.choice(["f64", "c64"])
        return updates(None, _log_int(rng, 32, 256 if dt == "f64" else 128), dt, rng.randint(1, 10 ** 6))
    if kind == "triples":
        e = {x: rng.randint(12, 24) for x in "abcijkm"}
        spec = rng.choice(["ikmb,mjac->abcijk", "ijma,mkbc->abcijk", "ekab,ijec->abcijk"])
        if spec.startswith("e"):
            e["e"] = e.pop("m")
        if any_dtype[0] == "c" or any_dtype == "f64":
            e = {x: min(v, 20) for x, v in e.items()}
        return contraction(None, spec, _sizes(**e), any_dtype)
    if kind == "tall":
        a, b, k = _log_int(rng, 20000, 200000), _log_int(rng, 9, 256), _log_int(rng, 8, 256)
        spec = rng.choice(["ak,kb->ab", "ka,kb->ab", "bk,ka->ba"])
        return contraction(None, spec, _sizes(a=a, b=b, k=k), rng.choice(["f32", "f64"]))
    if kind == "transform":
        e = {x: rng.randint(24, 72) for x in "abjck"}
        spec = rng.choice(["kbac,jk->abjc", "cbka,kj->abjc", "pa,pqrs->aqrs"])
        if spec.startswith("p"):
            e = dict(zip("apqrs", e.values()))
        return contraction(None, spec, _sizes(**e), any_dtype)
    if kind == "batched_small":
        m, n, k = (_log_int(rng, 1, 32) for _ in range(3))
        h = min(_log_int(rng, 512, 262144), 2 ** 24 // max(m * k, k * n, m * n))
        spec = rng.choice(["mkh,knh->mnh", "hmk,hkn->hmn"])
        return contraction(None, spec, _sizes(m=m, n=n, k=k, h=h), any_dtype)
    i, j = (rng.randint(128, 512) for _ in range(2))
    k, l = rng.randint(8, 32), rng.randint(32, 256)
    return vjp(None, _sizes(i=i, j=j, k=k, l=l), rng.choice(["f32", "f64"]))


def _extents(case):
    return {k: int(v) for k, v in (kv.split("=") for kv in case["sizes"].split(","))}


def _terms(case):
    lhs, out = case["spec"].split("->")
    a, b = lhs.split(",")
    return a, b, out


def _strides(dims, lead=1):
    st, acc = [], lead
    for d in dims:
        st.append(acc)
        acc *= d
    return st


def _values(gen, n, dtype, dist):
    real = torch.float32 if dtype in ("f32", "c32") else torch.float64
    cplx = dtype[0] == "c"
    count = 2 * n if cplx else n
    if dist == "normal":
        x = torch.randn(count, dtype=real, device="cuda", generator=gen)
    else:
        x = torch.rand(count, dtype=real, device="cuda", generator=gen) * 2 - 1
    return torch.view_as_complex(x.view(n, 2)) if cplx else x


def _tensor(gen, labels, ext, dtype, dist="uniform", lead=1):
    dims = [ext[x] for x in labels]
    flat = _values(gen, math.prod(dims) * lead, dtype, dist)
    return flat.as_strided(dims, _strides(dims, lead))


def _empty(labels, ext, dtype):
    dims = [ext[x] for x in labels]
    return torch.zeros(math.prod(dims), dtype=TORCH[dtype], device="cuda").as_strided(dims, _strides(dims))


def _layout(t, conj=False):
    return tp.OperandSpec(tp.LayoutSpec(list(t.shape), list(t.stride())), conj)


def _plan(case, a, b, d, conj=False, scheme="plain"):
    la, lb, ld = ([ord(x) for x in term] for term in _terms(case))
    prob = tp.Problem.from_labels(CODE[case["dtype"]], _layout(a, conj), _layout(b), _layout(d), la, lb, ld)
    return tp.Plan(prob, tp.PlanConfig(precision=SCHEME[scheme]))


def _executor(sync):
    return tp.Executor(device=0, stream=torch.cuda.current_stream().cuda_stream, sync=sync)


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _inputs(case, seed):
    """The tensors of a case (values from `seed` alone)."""
    gen = _generator(seed)
    if case["kind"] == "updates":
        import random

        rng = random.Random(case["list_seed"])
        out = []
        for _ in range(case["count"]):
            e = {"a": _log_int(rng, 16, 256), "b": _log_int(rng, 16, 256), "s": rng.choice([4, 8, 16]),
                 "p": rng.choice([2, 4])}
            e.update(x=e["a"], y=e["b"], t=e["s"], q=e["p"])
            ops = []
            for term in ("asb", "apx", "sptq", "bqy"):
                t = _tensor(gen, term, e, case["dtype"], "normal")
                ops.append(t / torch.linalg.vector_norm(t))
            out.append((e, ops))
        return out
    ext = _extents(case)
    la, lb, ld = _terms(case)
    if case["kind"] == "vjp":
        return [_tensor(gen, x, ext, case["dtype"], "normal") for x in (la, lb, ld)]
    a = _tensor(gen, la, ext, case["dtype"], case["dist"], case["a_lead"])
    b = _tensor(gen, lb, ext, case["dtype"], case["dist"])
    c = _tensor(gen, ld, ext, case["dtype"], case["dist"]) if case["beta"] else None
    return [a, b, c]


UPDATE_TERMS = ("asb", "apx", "sptq", "bqy", "xty")


def prepare(case, seed):
    if case["kind"] == "updates":
        nets, ins, outs = [], [], []
        inputs_of = _inputs(case, seed)
        # The updated environments lie one after another in one buffer.
        result = torch.zeros(sum(math.prod(e[x] for x in "xty") for e, _ in inputs_of), dtype=TORCH[case["dtype"]],
                             device="cuda")
        offset = 0
        for ext, ops in inputs_of:
            dims = [ext[x] for x in "xty"]
            d = result[offset:offset + math.prod(dims)].as_strided(dims, _strides(dims))
            offset += math.prod(dims)
            labels = [[ord(x) for x in term] for term in UPDATE_TERMS]
            inputs = [(_layout(t, k == 3), labels[k]) for k, t in enumerate(ops)]
            nets.append(tp.Network(CODE[case["dtype"]], inputs, (_layout(d).layout, labels[4]),
                                   path=[(0, 1), (2, 0), (1, 0)]))
            ins.append(ops)
            outs.append(d)
        return {"case": case, "ex": _executor(False), "batch": tp.PreparedNetworks(nets, ins, outs), "nets": nets,
                "ins": ins, "result": result}
    ops = _inputs(case, seed)
    ext = _extents(case)
    la, lb, ld = _terms(case)
    d = _empty(ld, ext, case["dtype"])
    if case["kind"] == "vjp":
        a, b, dd = ops
        return {"case": case, "ex": _executor(False), "plan": _plan(case, a, b, d), "a": a, "b": b, "dd": dd, "d": d,
                "da": _empty(la, ext, case["dtype"]), "db": _empty(lb, ext, case["dtype"])}
    a, b, c = ops
    return {"case": case, "ex": _executor(case["sync"]), "plan": _plan(case, a, b, d, case["conj"], case["scheme"]),
            "a": a, "b": b, "c": c, "d": d}


def run(state):
    case, ex = state["case"], state["ex"]
    if case["kind"] == "updates":
        state["batch"].run(ex)
        return state["result"]
    plan = state["plan"]
    if case["kind"] == "vjp":
        plan.execute_into(ex, 1.0, state["a"], state["b"], state["d"])
        plan.vjp(ex, 1.0, state["a"], state["b"], state["dd"], state["da"], state["db"])
        return {"d": state["d"], "da": state["da"], "db": state["db"]}
    if case["beta"]:
        plan.execute_into_accum(ex, 1.0, state["a"], state["b"], case["beta"], state["d"], c=state["c"])
    else:
        plan.execute_into(ex, 1.0, state["a"], state["b"], state["d"])
    return state["d"]


def work(case):
    dtype = case["dtype"]
    elem, per_mac = BYTES[dtype], 8 if dtype[0] == "c" else 2
    if case["kind"] == "updates":
        import random

        rng = random.Random(case["list_seed"])
        nbytes = flops = 0
        for _ in range(case["count"]):
            a, b, s, p = _log_int(rng, 16, 256), _log_int(rng, 16, 256), rng.choice([4, 8, 16]), rng.choice([2, 4])
            nbytes += elem * (2 * a * s * b + a * p * a + s * p * s * p + b * p * b)
            flops += per_mac * (a * s * b * p * a + s * b * p * a * s * p + b * a * s * p * b)
        return {"bytes": nbytes, "flops": flops}
    ext = _extents(case)
    la, lb, ld = _terms(case)
    size = lambda labels: math.prod(ext[x] for x in labels)
    macs = size(set(la + lb))
    if case["kind"] == "vjp":
        diag, b, d = size(set(la)), size(lb), size(ld)
        # A's diagonal, B and dD read; D, dB and all of dA written.
        return {"bytes": elem * (diag + b + d + d + b + size(la)), "flops": 3 * per_mac * macs}
    touched = size(la) + size(lb) + size(ld) * (2 if case["beta"] else 1)
    return {"bytes": elem * touched, "flops": per_mac * macs}


def exact(case, seed):
    wide = torch.complex128 if case["dtype"][0] == "c" else torch.float64
    if case["kind"] == "updates":
        out = []
        for _, ops in _inputs(case, seed):
            e, m, w, m2 = (x.to(wide) for x in ops)
            t1 = torch.einsum("asb,apx->sbpx", e, m)
            t2 = torch.einsum("sbpx,sptq->bxtq", t1, w)
            out.append(torch.einsum("bxtq,bqy->ytx", t2, m2.conj()).reshape(-1))  # column-major "xty"
        return torch.cat(out)
    if case["kind"] == "vjp":
        a, b, dd = (x.to(wide) for x in _inputs(case, seed))
        diag = torch.diagonal(a, dim1=1, dim2=2)  # [i, l, k]
        da = torch.zeros_like(a)
        torch.diagonal(da, dim1=1, dim2=2).copy_(torch.einsum("ij,ljk->ilk", dd, b))
        return {"d": torch.einsum("ilk,ljk->ij", diag, b), "da": da, "db": torch.einsum("ij,ilk->ljk", dd, diag)}
    a, b, c = _inputs(case, seed)
    a = a.to(wide)
    out = torch.einsum(case["spec"], a.conj() if case["conj"] else a, b.to(wide))
    return out + case["beta"] * c.to(wide) if case["beta"] else out

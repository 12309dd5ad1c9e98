"""The layout facts that a plan keeps for its launch choice (report()["layout"]) follow
from the folded axes; here they are recomputed from the offset vectors, over the shape
corpora and over random strided problems, without a GPU."""
import numpy as np
import pytest

import bench

ITEM = {0: 4, 1: 8, 2: 8, 3: 16}


def facts(tp, plan, dtype):
    """What the plan should say, by passes over its offset vectors."""
    rep = plan.report()
    get = lambda name: np.array(tp.product_scatter(plan.product, name), dtype=np.int64)
    A = dict(r=get("a_m"), k=get("a_k"), h=get("h_a"))
    B = dict(r=get("b_n"), k=get("b_k"), h=get("h_b"))
    D = dict(r=get("d_m"), k=get("d_n"), h=get("h_d"))
    C = dict(r=get("c_m"), k=get("c_n"), h=get("h_c"))
    if rep["swapped"]:
        A, B = B, A
        D, C = dict(r=D["k"], k=D["r"], h=D["h"]), dict(r=C["k"], k=C["r"], h=C["h"])
    v = 16 // ITEM[dtype]

    def unit(x):
        d = np.abs(np.diff(x)) == 1
        return x.size < 2 or 4 * int(d.sum()) >= 3 * (x.size - 1)

    def groups(fast, slow, h):
        if v == 1:
            return True
        if np.any(slow % v) or np.any(h % v):
            return False
        i = np.arange(fast.size)
        inside = i[1:] % v != 0
        return not np.any((fast - i) % v) and bool(np.all(np.diff(fast)[inside] == 1))

    def vec(o, kfast):
        return groups(o["k"], o["r"], o["h"]) if kfast else groups(o["r"], o["k"], o["h"])

    step = lambda x: abs(int(x[1] - x[0])) if x.size > 1 else 1 << 64
    fits = lambda o: all(bool(np.all((x < 1 << 30) & (x >= -(1 << 30)))) for x in (o["r"], o["k"]))
    fast = lambda o: 2 if step(o["h"]) < min(step(o["r"]), step(o["k"])) else 1 if step(o["k"]) < step(o["r"]) else 0
    seq = lambda x: x.size > 0 and bool(np.all(x == np.arange(x.size) * (x[1] - x[0] if x.size > 1 else 0)))
    sizes = (A["r"].size, B["r"].size, A["k"].size)
    small = all(1 <= s <= 32 for s in sizes)
    return rep, {
        "a_vec": vec(A, rep["a_kfast"]), "b_vec": vec(B, rep["b_kfast"]),
        "a_gather": unit(A["k"] if rep["a_kfast"] else A["r"]), "b_gather": unit(B["k"] if rep["b_kfast"] else B["r"]),
        "off32": dtype in (0, 2) and fits(A) and fits(B),
        "h_inner": all(step(o["h"]) < min(step(o["r"]), step(o["k"])) for o in (A, B, D)),
        "small_regular": all(seq(x) for o in (A, B, D, C) for x in o.values()) if small else True,
        "a_fast": fast(A), "b_fast": fast(B)}


def check(tp, plan, dtype, what):
    rep, want = facts(tp, plan, dtype)
    assert rep["layout"] == want, (what, rep["layout"], want)


def test_dot_general_corpus(tp):
    for e in bench.corpus_entries():
        code, _ = bench.CORPUS_DT[e["dtype"]]
        if sum(np.prod(e[s]["dims"], dtype=float) for s in "abc") > 2e6:
            continue
        spec = lambda side: tp.OperandSpec(tp.LayoutSpec(list(e[side]["dims"]), list(e[side]["strides"])))
        dot = tp.DotGeneral(e["lc"], e["rc"], e["lb"], e["rb"])
        check(tp, tp.Plan(tp.Problem.from_dot_general(code, spec("a"), spec("b"), spec("c"), dot)), code, e["name"])


@pytest.mark.parametrize("seed", range(6))
def test_random_layouts(tp, seed):
    """Up to three labels per role in any order in each operand, padded, reversed and
    widened strides, extents of 1 and odd ones, every type."""
    rng = np.random.default_rng(seed)
    for case in range(60):
        dtype = int(rng.integers(4))
        roles = {}
        lab = 0
        for role in "mnkh":
            roles[role] = list(range(lab, lab + int(rng.integers(0, 4 if role != "h" else 3))))
            lab += len(roles[role])
        ext = {x: int(rng.choice([1, 2, 3, 4, 6, 8, 12, 16])) for x in range(lab)}

        def operand(parts):
            labels = [x for p in parts for x in roles[p]]
            order = list(rng.permutation(labels)) if rng.random() < 0.7 else labels
            st, acc = {}, int(rng.choice([1, 1, 1, 2, 3, 4, 1 << 20]))
            for x in order:
                st[x] = int(acc * rng.choice([1, 1, 1, -1]))
                acc = acc * ext[x] + int(rng.choice([0, 0, 0, 1, 2, 4])) * (acc > 1)
            return tp.OperandSpec(tp.LayoutSpec([ext[x] for x in labels], [st[x] for x in labels])), labels

        (a, la), (b, lb), (d, ld) = operand("mkh"), operand("knh"), operand("mnh")
        check(tp, tp.Plan(tp.Problem.from_labels(dtype, a, b, d, la, lb, ld)), dtype, (seed, case, ext, la, lb, ld))


def test_tccg_layouts(tp):
    for case in bench.tccg_cases():
        for size in ("small", "tccg64"):
            ext = case["extents"][size]
            lay = lambda s: tp.OperandSpec(tp.LayoutSpec(*bench.tccg_layout(s, ext)[:2]))
            lab = lambda s: [ord(x) for x in s]
            if size == "tccg64" and np.prod([ext[x] for x in case["c"]], dtype=float) > 1.5e7:
                continue
            for dtype in (0, 3):
                prob = tp.Problem.from_labels(dtype, lay(case["a"]), lay(case["b"]), lay(case["c"]), lab(case["a"]),
                                              lab(case["b"]), lab(case["c"]))
                check(tp, tp.Plan(prob), dtype, (case["name"], size))

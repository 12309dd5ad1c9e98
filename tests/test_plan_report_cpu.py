"""What a plan's report says about its launch choice, without a GPU."""


def plan(tp, dtype, m, n, k):
    lay = lambda d: tp.OperandSpec(tp.LayoutSpec.col_major(d))
    return tp.Plan(tp.Problem.from_labels(dtype, lay([m, k]), lay([k, n]), lay([m, n]), [0, 2], [2, 1], [0, 1]))


def test_report_names_the_model_beside_the_named_candidates(tp):
    """The autotuner times the model's choice, also where it is a tensor-core family that
    no caller can name, and the candidates are the families that a caller can."""
    for dtype in (tp.F32, tp.C32):
        for m, n, k in [(4096, 4096, 4096), (3000, 3000, 40), (64, 64, 64)]:
            r = plan(tp, dtype, m, n, k).report()
            assert r["autotune_model"].startswith(r["family"])
            assert not any(".tcgen05." in c for c in r["autotune_candidates"])
            assert (".tcgen05." in r["family"]) == (m > 64)
    r = plan(tp, tp.F64, 576, 576, 576).report()
    assert r["autotune_model"] == r["autotune_candidates"][0]


def strided(tp, dtype, m, n, k, lead):
    """A's rows `lead` apart: a gather that is not coalesced for lead > 1."""
    a = tp.OperandSpec(tp.LayoutSpec([m, k], [lead, lead * m]))
    lay = lambda d: tp.OperandSpec(tp.LayoutSpec.col_major(d))
    return tp.Plan(tp.Problem.from_labels(dtype, a, lay([k, n]), lay([m, n]), [0, 2], [2, 1], [0, 1]))


def test_report_names_the_family_inside_a_list(tp):
    """Coalesced f64 items take a stream tile, or the 32 x 32 direct tile where one of it
    holds the item; the others the direct and skinny tiles."""
    family = lambda *x: strided(tp, tp.F64, *x).report()["list_family"]
    for m, n, k in [(16, 16, 64), (32, 32, 512), (32, 8, 8)]:
        assert family(m, n, k, 1) == "sm100.f64.dmma884.32x32x16"
    for m, n, k in [(33, 32, 512), (64, 64, 64), (300, 16, 60), (16, 300, 60), (256, 256, 256)]:
        assert ".stream." in family(m, n, k, 1)
    skinny = {(130, 16, 32): "128x16xk32", (130, 17, 32): "128x32xk32", (128, 16, 33): "128x16xk64", (128, 32, 64): "128x32xk64",
              (999, 64, 64): "128x64xk64"}
    for (m, n, k), name in skinny.items():
        assert family(m, n, k, 2) == "sm100.f64.fma.skinny." + name
    assert family(256, 256, 256, 2) == "sm100.f64.dmma884.64x64x16"

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

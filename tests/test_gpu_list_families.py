"""Tile families of grouped f64 lists, on a B200: the skinny tiles (items whose gather is
not coalesced) against the oracle, and the choice against lists pinned to one family."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch_cuda():
    import torch

    assert torch.cuda.is_available(), "the -m gpu tests need a CUDA device"
    return torch


def test_list_on_every_skinny_tile(tp, torch_cuda, orc):
    """Short-K items whose rows of A lie two apart, around the extents where the skinny
    families change, with alpha, beta and C, at the plain bound."""
    torch = torch_cuda
    rng = np.random.default_rng(11)
    shapes = [(130, 8, 8), (257, 16, 32), (128, 17, 31), (300, 32, 32), (129, 16, 33), (512, 15, 64), (200, 32, 64),
              (131, 31, 40), (128, 33, 33), (999, 64, 64), (385, 50, 17)]
    items, keep, seen = [], [], set()
    for m, n, k in shapes:
        a, b, c = rng.uniform(-1, 1, 2 * m * k), rng.uniform(-1, 1, k * n), rng.uniform(-1, 1, m * n)
        lay = lambda d, s: tp.OperandSpec(tp.LayoutSpec(d, s))
        spec_d = lay([m, n], [1, m])
        plan = tp.Plan(tp.Problem.from_labels(tp.F64, lay([m, k], [2, 2 * m]), lay([k, n], [1, k]), spec_d, [0, 2], [2, 1],
                                              [0, 1], c=spec_d, lc=[0, 1]))
        family = plan.report()["list_family"]
        assert ".skinny." in family
        seen.add(family)
        dev = [torch.from_numpy(x).cuda() for x in (a, b, c)] + [torch.zeros(m * n, dtype=torch.float64, device="cuda")]
        keep.append((a, b, c, dev))
        items.append(tp.Item(plan, 0.75, dev[0].data_ptr(), dev[1].data_ptr(), dev[3].data_ptr(), beta=-1.5, c=dev[2].data_ptr()))
    assert len(seen) == 5
    ex = tp.Executor()
    ex.set_profiling(True)
    tp.PreparedBatch(items).run(ex)
    ex.synchronize()
    assert ex.kernel_times()["grouped"]["launches"] == 1
    ex.close()
    for (m, n, k), (a, b, c, dev) in zip(shapes, keep):
        want = np.zeros(m * n)
        orc.packed_contract(0.75, orc.View(a, [m, k], [2, 2 * m], [0, 2]), orc.View(b, [k, n], [1, k], [2, 1]), -1.5,
                            orc.View(c, [m, n], [1, m], [0, 1]), orc.View(want, [m, n], [1, m], [0, 1]))
        assert orc.rel_frobenius(dev[3].cpu().numpy(), want) <= 1e-13, (m, n, k)


def list_time(tp, torch, shapes, kernel):
    """Milliseconds of a list of column-major f64 products, and its results."""
    gen = torch.Generator(device="cuda").manual_seed(1)
    items, keep = [], []
    for m, n, k in shapes:
        a, b = (torch.rand(c, dtype=torch.float64, device="cuda", generator=gen) for c in (m * k, k * n))
        d = torch.zeros(m * n, dtype=torch.float64, device="cuda")
        lay = lambda x: tp.OperandSpec(tp.LayoutSpec.col_major(x))
        prob = tp.Problem.from_labels(tp.F64, lay([m, k]), lay([k, n]), lay([m, n]), [0, 2], [2, 1], [0, 1])
        items.append(tp.Item(tp.Plan(prob, tp.PlanConfig(kernel=kernel)), 1.0, a.data_ptr(), b.data_ptr(), d.data_ptr()))
        keep.append((a, b, d))
    batch, ex, best = tp.PreparedBatch(items), tp.Executor(), 1e9
    ex.set_profiling(True)
    for i in range(8):
        ex.kernel_times(reset=True)
        batch.run(ex)
        ex.synchronize()
        best = min(best, ex.kernel_times()["grouped"]["ms"])
    ex.close()
    return best, [d for _, _, d in keep]


# Pinned ids: the 64 x 64 (3) and 32 x 32 (4) direct tiles.
@pytest.mark.parametrize("name,kernel,shapes", [
    ("one 32 x 32 tile, deep", 4, [(32, 32, 512)] * 1500),
    ("one 32 x 32 tile, narrow", 4, [(16, 16, 256)] * 1500),
    ("mixed", 3, [(16 + 37 * i % 480, 16 + 61 * i % 450, 16 + 53 * i % 470) for i in range(300)]),
])
def test_model_is_no_slower_than_a_pinned_family(tp, torch_cuda, name, kernel, shapes):
    ms, got = list_time(tp, torch_cuda, shapes, 0)
    pinned, want = list_time(tp, torch_cuda, shapes, kernel)
    for x, y in zip(got, want):
        assert float((x - y).norm() / y.norm()) <= 1e-13
    assert ms <= 1.1 * pinned, (name, ms, pinned)

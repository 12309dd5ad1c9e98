"""Error of the plain f32 and c32 tensor-core kernels against 64 bits, beside the FFMA
tiles' on the same operands, on a B200.

Both sum K products with FP32 roundings: the FFMA tiles in chains of 16 (direct) or 64
(packed) between restarts, the tensor cores in steps of 16 that round once, the steps
in running sums of 8 to 32. On smooth data (of both signs or of one) the tensor cores
must not be further off; u^8 spreads the products of a step over many binades, which
the tensor core truncates: half as much again at most."""
import pytest

pytestmark = pytest.mark.gpu

CODE = {"f32": 0, "c32": 2}
# The family that the general choice takes at these sizes: direct below K = 64, else packed.
FFMA = {"f32": (1, 10), "c32": (5, 15)}


def draw(torch, n, dt, dist, gen):
    x = torch.rand(n * (2 if dt == "c32" else 1), device="cuda", generator=gen)
    if dist == "signed":
        x = x * 2 - 1
    elif dist == "heavy tail":
        x = x ** 8
    return torch.view_as_complex(x.view(-1, 2)) if dt == "c32" else x


@pytest.mark.parametrize("dist", ["signed", "one sign", "heavy tail"])
@pytest.mark.parametrize("m,n,k", [(2900, 2900, 3), (2900, 2900, 16), (2900, 2900, 32), (2900, 2900, 33), (2900, 2900, 64),
                                   (2048, 2048, 257), (2048, 2048, 512), (2048, 2048, 1024), (2048, 2048, 2048),
                                   (2048, 1024, 4100), (1024, 1024, 9000)])
@pytest.mark.parametrize("dt", sorted(CODE))
def test_error_beside_the_ffma_tiles(tp, dt, m, n, k, dist):
    import torch

    gen = torch.Generator(device="cuda").manual_seed(k)
    A = draw(torch, m * k, dt, dist, gen).as_strided([m, k], [1, m])
    B = draw(torch, k * n, dt, dist, gen).as_strided([k, n], [1, k])
    D = torch.zeros(m * n, dtype=A.dtype, device="cuda").as_strided([m, n], [1, m])
    wide = torch.complex128 if dt == "c32" else torch.float64
    want = A.to(wide) @ B.to(wide)
    ex = tp.Executor(device=0, stream=torch.cuda.current_stream().cuda_stream)
    lay = lambda t: tp.OperandSpec(tp.LayoutSpec(list(t.shape), list(t.stride())))
    prob = tp.Problem.from_labels(CODE[dt], lay(A), lay(B), lay(D), [0, 2], [2, 1], [0, 1])
    err = []
    for kernel in (0, FFMA[dt][k >= 64]):
        plan = tp.Plan(prob, tp.PlanConfig(kernel=kernel))
        plan.execute_into(ex, 1.0, A, B, D)
        err.append(float((D.to(wide) - want).norm() / want.norm()))
        if kernel == 0:
            assert ".tcgen05." in plan.report()["family"]
    ex.close()
    assert err[0] <= (1.5 if dist == "heavy tail" else 1.05) * err[1], err

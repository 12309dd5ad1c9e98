"""The estimate that chooses between the FFMA tiles, the in-flight and the packed tensor-core
family for plain f32 and c32 (choose_tc_kernel): shapes on both sides of each line, each with
the three times measured on a B200 (FFMA, in flight, packed; us). The family chosen is the
fastest of the three."""
import pytest

import tprims_b200 as tp

SHAPES = [
    ("f32", "ka,kb->ab", dict(a=198795, b=5, k=14), "stream", (92.6, 31.0, 213.1)),
    ("c32", "ka,kb->ab", dict(a=168696, b=12, k=3), "stream", (86.5, 44.9, 274.6)),
    ("f32", "bk,ka->ba", dict(a=72853, b=36, k=15), "stream", (31.0, 23.7, 53.6)),
    ("f32", "eafb,cedf->cadb", dict(a=29, b=19, c=22, d=24, e=27, f=24), "split", (37.1, 66.0, 35.1)),
    ("f32", "mk,kn->mn", dict(m=2940, n=190, k=979), "split", (67.8, 75.4, 47.1)),
    ("c32", "mk,kn->mn", dict(m=4280, n=68, k=3625), "split", (476.9, 387.3, 272.8)),
    ("c32", "abef,efcd->dcba", dict(a=31, b=18, c=19, d=20, e=16, f=25), "split", (59.7, 57.7, 39.2)),
    ("c32", "hki,hkj->hij", dict(h=9, i=150, j=207, k=498), "split", (83.0, 83.5, 54.3)),
    ("f32", "hki,hkj->hij", dict(h=37, i=49, j=103, k=95), "simt", (16.5, 27.9, 41.2)),
    ("f32", "aebf,fced->abcd", dict(a=27, b=19, c=26, d=28, e=9, f=9), "simt", (12.4, 20.6, 33.0)),
    ("f32", "abef,efcd->dcba", dict(a=28, b=14, c=29, d=21, e=6, f=24), "simt", (15.0, 23.8, 31.5)),
    ("f32", "mk,kn->mn", dict(m=40, n=2177, k=145), "simt", (15.5, 21.8, 30.9)),
]


def family(dtype, spec, ext):
    lhs, out = spec.split("->")
    a, b = lhs.split(",")
    layout = lambda s: tp.OperandSpec(tp.LayoutSpec.col_major([ext[x] for x in s]))
    labels = lambda s: [ord(x) for x in s]
    code = {"f32": 0, "c32": 2}[dtype]
    problem = tp.Problem.from_labels(code, layout(a), layout(b), layout(out), labels(a), labels(b), labels(out))
    return tp.Plan(problem).report()["family"]


@pytest.mark.parametrize("dtype,spec,ext,want,times", SHAPES)
def test_the_fastest_family_is_chosen(dtype, spec, ext, want, times):
    assert times[("simt", "stream", "split").index(want)] == min(times)
    name = family(dtype, spec, ext)
    assert (".%s." % want) in name or (want == "simt" and ".tcgen05." not in name), name

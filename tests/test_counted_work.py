"""The operations a plan reports (rsr_batch_describe), from which rates are
computed, are those it runs at every point: the register kernel runs a constant
subtree once an item, the other kernels run it at every point."""
import pytest

from rsr_b200 import _native as N
from rsr_b200 import evaluator as E
from rsr_b200 import isa as I
from rsr_b200 import workloads as W
from programs import _prog, cv, var
from rsr_b200.isa import FLOAT, VEC3

POINTS = 1000


def _pair():
    """(E + (c1 x c2)) . E + sqrt(3 * 4), and the same with each constant subtree folded to one constant."""
    c = lambda *v: cv(VEC3 if len(v) == 3 else FLOAT, v)  # noqa: E731
    e = var(VEC3, 0)
    tail = ["AddF"]
    return (_prog([e, c(1, 2, 3), c(3, 1, 2), "CrossV3", "AddV3", e, "DotV3", c(3), c(4), "MulF", "SqrtF"] + tail),
            _prog([e, c(1, 7, -5), "AddV3", e, "DotV3", c(12)] + tail))


def test_the_programs_operations_are_counted_whole():
    whole, folded = (E.analyze(p, 9)["flops_per_point"] for p in _pair())
    w = I.FLOP_WEIGHT
    assert whole - folded == w["CrossV3"] + w["MulF"] + w["SqrtF"]
    assert folded == w["AddV3"] + w["DotV3"] + w["AddF"] + I.MSE_EPILOGUE_FLOPS


def _described(e, pop, d, **kw):
    b = e.prepare(I.pack(pop), d, **kw)
    try:
        s = b.describe()
        assert s["flops"] == sum(g["flops"] for g in s["groups"])
        return s["flops"], {g["kernel"] for g in s["groups"]}
    finally:
        b.close()


@pytest.mark.gpu
def test_a_plan_counts_what_it_runs_at_every_point():
    whole, folded = _pair()
    per_point = [E.analyze(p, 9)["flops_per_point"] for p in (whole, folded)]
    with E.Engine() as e:
        d = e.upload(W.lorentz_dataset(POINTS, seed=2))
        assert _described(e, [whole], d) == (per_point[1] * POINTS, {"register"})
        assert _described(e, [whole, folded], d)[0] == 2 * per_point[1] * POINTS
        assert _described(e, [whole], d, kernel=N.KERNEL_PLAIN) == (per_point[0] * POINTS, {"slot"})
        g = [_described(e, [p], d, gradient=True)[0] // POINTS for p in (whole, folded)]
        assert g[0] - g[1] > per_point[0] - per_point[1]   # both sweeps run them

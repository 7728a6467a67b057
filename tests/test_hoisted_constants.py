"""Constant subtrees run once per work item (uops.h, hoisted constants): every
value of a program that holds some is bit for bit the oracle's, for subtrees
of every type, whole programs without a feature, full and partly filled items
and datasets from a few points to several items."""
import numpy as np
import pytest

from oracle import binding as O
from programs import _LEAF_OFF, _prog, cv, op_dataset, var
from rsr_b200 import isa as I
from rsr_b200.evaluator import Engine
from rsr_b200.isa import FLOAT, MAT2, MAT3, VEC2, VEC3

pytestmark = pytest.mark.gpu


def _programs():
    rng = np.random.default_rng(8)
    c = lambda t: cv(t, rng.normal(0, 1, I.KIND_WIDTH[t]))
    v = lambda t: var(t, _LEAF_OFF[t])
    red = {FLOAT: [], VEC2: ["NormV2"], VEC3: ["NormV3"], MAT2: ["DetM2"], MAT3: ["DetM3"]}
    out = []
    for name in I.BASIC_NAMES + I.LINALG_NAMES:
        args, ret = I.SIGNATURE[name]
        sub = [c(t) for t in args] + [name]              # one constant subtree of every operator
        add = {FLOAT: "MulF", VEC2: "AddV2", VEC3: "CrossV3", MAT2: "MulM2", MAT3: "MulM3"}[ret]
        out.append(_prog(sub + red[ret]))                # a program without a feature
        out.append(_prog(sub + [v(ret), add] + red[ret]))
        out.append(_prog([v(ret)] + sub + [add] + red[ret] + [c(FLOAT), c(FLOAT), "DivF", "AddF"]))  # two of them
    return out


@pytest.mark.parametrize("per_item", [0, 1, 3, 8])
@pytest.mark.parametrize("n", [7, 300, 4096 + 9])
def test_points_bit_identical(n, per_item):
    ds, pop = op_dataset(n), _programs()
    with Engine(programs_per_warp=per_item) as e:
        got = e.eval_points_batch(pop, ds)
    for i, p in enumerate(pop):
        want = O.eval_points(p, ds)
        nan = np.isnan(want)
        assert np.array_equal(np.isnan(got[i]), nan), i
        assert np.array_equal(got[i][~nan], want[~nan]), i


def test_a_fit_refolds_the_constants_it_moves():
    """2.5 x^2 - 1.2 with its 2.5 and 1.2 each the sum of two constants: L-BFGS moves all four."""
    from rsr_b200 import workloads as W
    ds = W.scalar_dataset(400)
    x = var(FLOAT, 0)
    cf = lambda u: cv(FLOAT, (u,))
    p = _prog([cf(0.3), cf(0.9), "AddF", x, "MulF", x, "MulF", cf(0.4), cf(0.2), "AddF", "SubF"])
    with Engine() as e:
        params, mse, _ = e.fit_lbfgs([p], ds, 20)
        assert mse[0] < 1e-8 and abs(params[0] + params[1] - 2.5) < 1e-3 and abs(params[2] + params[3] - 1.2) < 1e-3
        p.unflatten_params(params)
        assert e.compute_mse(p, ds) == mse[0]

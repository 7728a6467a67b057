"""Square roots and quotients of several points together (vm_ops.cuh): the
IEEE round-to-nearest results, bit for bit, on both sides of the range that
the shared test lets through -- numpy's float32 sqrt and divide are the
reference."""
import numpy as np
import pytest

from rsr_b200 import _native as N
from rsr_b200 import isa as I
from rsr_b200.dataset import Dataset
from rsr_b200.evaluator import Engine
from rsr_b200.isa import FLOAT, Program

pytestmark = pytest.mark.gpu
f32 = np.float32


def _around(v):
    v = f32(v)
    return [np.nextafter(v, f32(0)), v, np.nextafter(v, f32(np.inf))]


def _edges():
    e = [0.0, np.inf, np.nan, np.finfo(f32).max, np.finfo(f32).tiny, np.finfo(f32).smallest_subnormal, 1.0, 3.0]
    for k in (-149, -126, -101, -100, -61, -60, -59, -1, 0, 1, 59, 60, 61, 126, 127):
        e += _around(2.0 ** k)
    e = np.array(e, f32)
    return np.concatenate([e, -e])


def _columns():
    """x, y: whole tiles inside the range, tiles with one value outside, every pair of edges."""
    rng = np.random.default_rng(21)
    inside = (rng.uniform(1, 2, (2, 4096)) * 2.0 ** rng.integers(-58, 58, (2, 4096))).astype(f32)
    inside[1] *= rng.choice([-1, 1], 4096).astype(f32)
    mixed = inside[:, rng.permutation(4096)].copy()
    e = _edges()
    mixed[:, ::37] = rng.choice(e, (2, len(range(0, 4096, 37))))
    pairs = np.array(np.meshgrid(e, e)).reshape(2, -1)
    return np.concatenate([inside, mixed, pairs, inside[:, :77]], 1)


@pytest.mark.parametrize("points_per_lane", [2, 4, 8])
@pytest.mark.parametrize("kernel", [N.KERNEL_AUTO, N.KERNEL_PLAIN])
def test_bit_identical_to_ieee(points_per_lane, kernel):
    x, y = _columns()
    ds = Dataset.new(np.stack([x, y], 1), np.zeros(len(x), f32), [FLOAT, FLOAT])
    X, Y = I.load_var(FLOAT, 0), I.load_var(FLOAT, 1)
    pop = [Program([X, I.op("SqrtF")], []), Program([X, Y, I.op("DivF")], []), Program([Y, X, I.op("DivF")], [])]
    with Engine(points_per_thread=points_per_lane) as e:
        got = e.eval_points_batch(pop, ds, kernel=kernel)[:, :len(x)]
    with np.errstate(all="ignore"):
        want = np.stack([np.sqrt(x), x / y, y / x])
    nan = np.isnan(want)
    assert np.array_equal(np.isnan(got), nan)
    assert np.array_equal(got[~nan].view(np.uint32), want[~nan].view(np.uint32))

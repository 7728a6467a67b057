"""Products, sums and differences of two points in one instruction (vm_ops.cuh):
each rounded by itself, bit for bit as numpy's float32 gives it, never a product
contracted with the sum behind it."""
import numpy as np
import pytest

from rsr_b200 import _native as N
from rsr_b200 import isa as I
from rsr_b200.dataset import Dataset
from rsr_b200.evaluator import Engine
from rsr_b200.isa import FLOAT, VEC3, Program

pytestmark = pytest.mark.gpu
f32 = np.float32


def _columns(n):
    """x, y, z and three vectors: ordinary values, wide exponents, infinities, NaN, zeros and subnormals."""
    rng = np.random.default_rng(31)
    c = rng.standard_normal((n, 12)).astype(f32)
    wide = rng.random(c.shape) < 0.2
    c[wide] *= (2.0 ** rng.integers(-75, 64, wide.sum())).astype(f32)
    odd = rng.random(c.shape) < 0.02
    c[odd] = rng.choice(np.array([0, -0.0, np.inf, -np.inf, np.nan, 1e-45, -1e-40, 3e38], f32), odd.sum())
    return c


def _cross(a, b):
    return np.stack([a[1] * b[2] - a[2] * b[1], a[2] * b[0] - a[0] * b[2], a[0] * b[1] - a[1] * b[0]])


def _dot(a, b):
    return (a[0] * b[0] + a[1] * b[1]) + a[2] * b[2]


@pytest.mark.parametrize("points_per_lane", [2, 4, 8])
@pytest.mark.parametrize("kernel", [N.KERNEL_AUTO, N.KERNEL_PLAIN])
@pytest.mark.parametrize("n", [1, 255, 4099])
def test_bit_identical_to_float32(points_per_lane, kernel, n):
    c = _columns(n)
    ds = Dataset.new(c, np.zeros(n, f32), [FLOAT] * 3 + [VEC3] * 3)
    X, Y, Z = (I.load_var(FLOAT, i) for i in range(3))
    U, V, W = (I.load_var(VEC3, i) for i in (3, 6, 9))
    op = I.op
    pop = [Program(code, []) for code in (
        [X, Y, op("MulF"), Z, op("AddF")], [X, Y, op("MulF"), Z, op("SubF")], [Z, X, Y, op("MulF"), op("SubF")],
        [X, Y, op("MulF"), Y, Z, op("MulF"), op("AddF")],
        [U, V, op("CrossV3"), W, op("AddV3"), U, op("DotV3")],
        [W, X, U, op("ScaleV3"), op("SubV3"), V, op("DotV3")],
        [X, U, op("ScaleV3"), Y, V, op("ScaleV3"), op("AddV3"), op("NormV3")])]
    x, y, z = c.T[:3]
    u, v, w = c.T[3:6], c.T[6:9], c.T[9:12]
    with np.errstate(all="ignore"):
        s = x * u + y * v
        want = np.stack([x * y + z, x * y - z, z - x * y, x * y + y * z, _dot(_cross(u, v) + w, u),
                         _dot(w - x * u, v), np.sqrt(_dot(s, s))])
    with Engine(points_per_thread=points_per_lane) as e:
        got = e.eval_points_batch(pop, ds, kernel=kernel)[:, :n]
    nan = np.isnan(want)
    assert np.array_equal(np.isnan(got), nan)
    assert np.array_equal(got[~nan].view(np.uint32), want[~nan].view(np.uint32))

"""Square roots and quotients over the range that the shared test of vm_ops.cuh
lets through, bit for bit the IEEE results (numpy's float32 sqrt and divide):
every mantissa at exponents of both parities and at both ends, every mantissa of
a divisor with random dividends, and quotients next to the middle between two
floats, where a last step that is off rounds the wrong way.  And the reciprocals
of the matrix inverses, on both sides of their 1e-9 branch."""
import numpy as np
import pytest

from oracle import binding as O
from programs import _prog, cv, var
from rsr_b200 import isa as I
from rsr_b200.dataset import Dataset
from rsr_b200.evaluator import Engine
from rsr_b200.isa import FLOAT, MAT2, MAT3, Program

pytestmark = pytest.mark.gpu
f32, u32, u64 = np.float32, np.uint32, np.uint64
MANTISSAS = np.arange(1 << 23, dtype=u32)


def _floats(mantissa, exponent):
    return (mantissa | ((np.asarray(exponent) + 127).astype(u32) << u32(23))).view(f32)


@pytest.fixture(scope="module")
def engine():
    with Engine() as e:
        yield e


def _points(engine, prog, *columns):
    n = len(columns[0])
    d = engine.upload_rows(np.stack(columns, 1), np.zeros(n, f32))[0]
    try:
        return engine.eval_points_batch([prog], d)[0, :n]
    finally:
        d.release()


def _same(got, want):
    bad = np.flatnonzero(got.view(u32) != want.view(u32))
    assert bad.size == 0, (bad.size, bad[:3])


X, Y = I.load_var(FLOAT, 0), I.load_var(FLOAT, 1)
SQRT, DIV = Program([X, I.op("SqrtF")], []), Program([X, Y, I.op("DivF")], [])


@pytest.mark.parametrize("exponent", [-100, -99, -1, 0, 1, 62, 126, 127])
def test_roots_of_every_mantissa(engine, exponent):
    x = _floats(MANTISSAS, exponent)
    _same(_points(engine, SQRT, x), np.sqrt(x))


@pytest.mark.parametrize("seed", [0, 1, 2])
def test_quotients_by_every_mantissa(engine, seed):
    rng = np.random.default_rng(seed)
    n = len(MANTISSAS)
    b = _floats(MANTISSAS, rng.integers(-60, 60, n))
    a = _floats(rng.integers(0, 1 << 23, n).astype(u32), rng.integers(-60, 60, n)) * rng.choice([-1, 1], n).astype(f32)
    _same(_points(engine, DIV, a, b), a / b)


def _next_to_a_midpoint(n, seed):
    """24-bit A, B with A 2^25 = N B - r, N odd of 25 bits and r small: A / B is r / (B 2^25) from the
    middle between two floats."""
    rng = np.random.default_rng(seed)
    b = (rng.integers(1 << 22, 1 << 23, n).astype(u64) << u64(1)) | u64(1)
    r = rng.choice(np.array([-7, -5, -3, -1, 1, 3, 5, 7]), n)
    inv = b.copy()                                    # of b modulo 2^25
    for _ in range(5):
        inv = inv * (u64(2) - b * inv)
    m = u64((1 << 25) - 1)
    big_n = (inv * r.astype(np.int64).view(u64)) & m
    prod = big_n.astype(np.int64) * b.astype(np.int64) - r
    assert (prod % (1 << 25) == 0).all()
    a = prod >> 25
    keep = (big_n >= 1 << 24) & (a >= 1 << 23) & (a < 1 << 24)
    return a[keep].astype(f32), b[keep].astype(f32)


def test_quotients_next_to_a_midpoint(engine):
    a, b = _next_to_a_midpoint(1 << 23, 5)
    assert len(a) > 1 << 20
    q = a.astype(np.float64) / b.astype(np.float64)   # a quotient of 24-bit integers, to 53 bits
    scaled = q * 2.0 ** (24 - np.floor(np.log2(q)) - 1)
    assert (np.abs(scaled - np.floor(scaled) - 0.5) < 2.0 ** -19).all()
    _same(_points(engine, DIV, a, b), a / b)
    _same(_points(engine, DIV, a * f32(2.0 ** -70), b * f32(2.0 ** 20)), (a * f32(2.0 ** -70)) / (b * f32(2.0 ** 20)))


@pytest.mark.parametrize("kind,width", [(MAT2, 4), (MAT3, 9)])
def test_inverses_around_the_singular_branch(engine, kind, width):
    """Diagonal matrices with determinants of a few floats around 1e-9, and from 2^-40 to 2^70."""
    k = 2 if kind == MAT2 else 3
    rng = np.random.default_rng(3)
    edge = f32(1e-9)
    near = (edge.view(u32).astype(np.int64) + np.arange(-256, 256)).astype(u32).view(f32)
    wide = (rng.uniform(1, 2, 3584) * 2.0 ** rng.integers(-40, 70, 3584)).astype(f32)
    det = np.concatenate([near, -near, wide, -wide]).astype(f32)
    m = np.zeros((len(det), width), f32)
    m[:, ::k + 1] = 1.0
    m[:, 0] = det
    m[:, 1] = rng.uniform(-1, 1, len(det)).astype(f32)     # below the diagonal: no part of the determinant
    ds = Dataset.new(m, np.zeros(len(det), f32), [kind])
    name = "M2" if kind == MAT2 else "M3"
    v = cv(I.VEC2 if k == 2 else I.VEC3, (1.0, 0.5) if k == 2 else (1.0, 0.5, 0.25))
    for tail in ([f"Trace{name}"], [v, f"Mul{name}V{k}", f"NormV{k}"]):
        p = _prog([var(kind, 0), f"Inverse{name}"] + tail)
        got, want = engine.eval_points(p, ds), O.eval_points(p, ds)
        nan = np.isnan(want)
        assert np.array_equal(np.isnan(got), nan)
        _same(got[~nan], want[~nan])

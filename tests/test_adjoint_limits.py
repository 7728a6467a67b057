"""Shared memory of a register-adjoint block (kernels_adj.cu, adj_layout): which
gradients a block can take, and at how many points a lane, follows from it."""
import numpy as np
import pytest

from rsr_b200 import _native as N
from rsr_b200 import evaluator as E
from rsr_b200 import isa as I
from rsr_b200.dataset import Dataset
from rsr_b200.isa import FLOAT, Program, Scalar

pytestmark = pytest.mark.gpu
f32 = np.float32
LIMIT = 227 * 1024          # bytes of a block
WARPS = 16                  # of a block of the Float profile


def _sum(n_params, n_terms):
    """c_0 + .. + c_(n_params - 1) + x + .. + x, n_terms of the x."""
    code = [I.load_const(FLOAT, 0)]
    for k in range(1, n_params):
        code += [I.load_const(FLOAT, k), I.op("AddF")]
    code += [I.load_var(FLOAT, 0), I.op("AddF")] * n_terms
    return Program(code, [Scalar(FLOAT, (0.25,))] * n_params)


def _block_bytes(prog):
    """One part an item, no spilled value: code and a stop entry behind each sweep for the two header
    words, constants, the item, the cross-warp sums; and each warp's sums."""
    e = E.encoding(prog, 1, 5)
    assert e[0] == 0 and not e[2:7].any()
    words, n, up = len(e) - 7, prog.param_count(), lambda v: (v + 3) & ~3   # noqa: E731
    header = up(words + 1 + 2) + up(n) + 4 + 2 * WARPS * 33
    return 4 * (header + WARPS * (32 * min(n, 32) + 64))


@pytest.fixture(scope="module")
def engine():
    with E.Engine() as e:
        yield e


def _data():
    return Dataset.new(np.zeros((8, 1), f32), np.zeros(8, f32), [FLOAT])


@pytest.mark.parametrize("n_params", [1, 31, 32, 33, 40])
def test_block_size(engine, n_params):
    p = _sum(n_params, 7000)
    b = engine.prepare([p], _data(), gradient=True)
    try:
        b.run()
        mse, grad = b.results()
        g, = b.describe()["groups"]
    finally:
        b.close()
    assert g["kernel"] == "register_adjoint" and g["smem_bytes"] == _block_bytes(p) > 116_000
    s = f32(0.25) * n_params
    assert mse[0] == s * s and (grad[0, :min(n_params, 32)] == 2 * s).all() and not grad[0, n_params:].any()


@pytest.mark.parametrize("n_params", [3, 40])
def test_the_longest_program_a_block_takes(engine, n_params):
    """16 bytes a term; the one term more that does not fit is an error, not a launch."""
    n = (LIMIT - _block_bytes(_sum(n_params, 0))) // 16
    longest = _sum(n_params, n)
    assert LIMIT - 16 < _block_bytes(longest) <= LIMIT
    s = f32(0.25) * n_params
    mse, grad = engine.compute_mse_grad_batch([longest], _data())
    assert mse[0] == s * s and (grad[0, :min(n_params, 32)] == 2 * s).all()
    with pytest.raises(N.RsrError, match="shared memory"):
        engine.compute_mse_grad_batch([_sum(n_params, n + 1)], _data())

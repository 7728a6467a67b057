"""Shared memory of a register-kernel block (kernels_reg.cu, reg_layout): which
programs it can take, and at how many points a lane, follows from it."""
import numpy as np
import pytest

from rsr_b200 import evaluator as E
from rsr_b200 import isa as I
from rsr_b200 import workloads as W
from rsr_b200.dataset import Dataset
from rsr_b200.isa import FLOAT, VEC3, Program, Scalar

pytestmark = pytest.mark.gpu
f32 = np.float32
WARPS = 8


def _bytes(code_words, consts, stack_floats, per_item):
    """Code and constants of an item, 32 words for the item, the cross-warp sums; and each warp's
    spill stacks and running sums (a pair a lane and program)."""
    up = lambda v: (v + 3) & ~3   # noqa: E731
    return 4 * (up(code_words) + up(consts) + 32 + 2 * WARPS * 8 + WARPS * (stack_floats + 64 * per_item))


def _run(e, pop, d):
    b = e.prepare(I.pack(pop), d)
    try:
        b.run()
        return b.results(), b.describe()["groups"]
    finally:
        b.close()


@pytest.mark.parametrize("per_item", [1, 2, 8])
def test_block_size(per_item):
    x, y = I.load_var(FLOAT, 0), I.load_var(FLOAT, 1)
    c = [I.load_const(FLOAT, k) for k in range(5)]
    progs = [Program([x] + [w for k in c[:n] for w in (k, I.op("MulF"))], [Scalar(FLOAT, (2.0,))] * n)
             for n in range(6)]
    progs.append(Program([x, y, I.op("AddF"), x, y, I.op("MulF"), I.op("DivF")], []))   # one spilled value
    words = [len(E.encoding(p, 2, 1)) + 1 for p in progs]   # nothing to hoist; and the word behind a program
    with E.Engine(programs_per_warp=per_item) as e:
        d = e.upload(Dataset.new(np.ones((100, 2), f32), np.zeros(100, f32), [FLOAT, FLOAT]))
        for i, p in enumerate(progs):
            _, (g,) = _run(e, [p] * per_item, d)
            stack = 32 * g["points_per_thread"] * E.analyze(p, 2)["depth_fast"][0]
            assert g["kernel"] == "register" and g["programs_per_warp"] == per_item
            assert g["smem_bytes"] == _bytes(words[i] * per_item, p.param_count() * per_item, stack, per_item), i


def _with_prologue(n):
    """c_0 * c_1 + x + .. + x: as accumulator code n + 2 words, hoisted 3 more."""
    code = [I.load_const(FLOAT, 0), I.load_const(FLOAT, 1), I.op("MulF")] + [I.load_var(FLOAT, 0), I.op("AddF")] * n
    return Program(code, [Scalar(FLOAT, (1.5,)), Scalar(FLOAT, (2.0,))])


def test_a_prologue_does_not_push_a_program_off_the_kernel():
    """The longest program that fits without its constant subtree hoisted: it runs that way."""
    n = next(n for n in range(24_900, 25_000) if _bytes(n + 4, 2, 0, 1) > 100 * 1024)
    longest = _with_prologue(n)
    plain, hoisted = (len(E.encoding(longest, 1, 1)), len(E.encoding(longest, 1, 6)) - 3)
    assert (plain, hoisted) == (n + 2, n + 5)
    assert _bytes(plain + 1, 2, 0, 1) <= 100 * 1024 < _bytes(hoisted + 1, 3, 0, 1)
    with E.Engine() as e:
        d = e.upload(Dataset.new(np.zeros((8, 1), f32), np.zeros(8, f32), [FLOAT]))
        mse, (g,) = _run(e, [longest], d)
        assert g["kernel"] == "register" and mse[0] == 9.0
        assert e.compute_mse(longest, d) == 9.0
        short = _with_prologue(10)
        mse, groups = _run(e, [longest, short, longest, short], d)
        assert (mse == 9.0).all() and {g["kernel"] for g in groups} == {"register"}


def test_prologues_and_sums_share_their_room():
    """Eight programs an item, all with prologues, over items of many tiles: the sums of one item are
    taken where its prologues' addresses stood, and the next item's addresses are laid there again."""
    ds = W.lorentz_dataset(50_000, seed=8)
    gen = [Program([I.load_var(VEC3, 0), I.load_const(VEC3, 0), I.load_const(VEC3, 1), I.op("CrossV3"), I.op("AddV3"),
                    I.op("NormV3")], [Scalar(VEC3, (1.0, k, 2.0)), Scalar(VEC3, (0.5, 1.0, k))]) for k in range(64)]
    with E.Engine(programs_per_warp=8) as many, E.Engine(programs_per_warp=1) as one:
        a = many.compute_mse_batch(gen, ds)
        b = one.compute_mse_batch(gen, ds)
        pts = many.eval_points_batch(gen, ds).astype(np.float64)[:, :ds.num_samples]
    assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
    want = ((pts - one_target(ds)) ** 2).mean(1)
    np.testing.assert_allclose(a, want, rtol=1e-6)


def one_target(ds):
    return np.ascontiguousarray(ds.target_batches).reshape(-1)[:ds.num_samples].astype(np.float64)

"""Points per lane set the order of a program's sums, and are halved where a
register-kernel block would not fit its shared memory (runtime.cu end_plan).
A program whose stacks reach that edge has to get the same points per lane, and
the same bits, whatever the size of the plan it is in."""
import numpy as np
import pytest

from rsr_b200 import evaluator as E
from rsr_b200 import isa as I
from rsr_b200.dataset import Dataset
from rsr_b200.isa import FLOAT, VEC3, Program


def deep_program(n_scalars, n_vectors):
    """n_scalars floats and n_vectors Vec3 values spilled at once: nested scales
    of a balanced sum of 2^n_vectors two-leaf sums."""
    X, V, W = I.load_var(FLOAT, 0), I.load_var(VEC3, 1), I.load_var(VEC3, 4)
    code = [X, X, I.op("AddF")] * (n_scalars + 1)
    for i in range(2 ** n_vectors):
        code += [V, W, I.op("AddV3")]
        code += [I.op("AddV3")] * (((i + 1) & -(i + 1)).bit_length() - 1)
    return Program(code + [I.op("ScaleV3")] * (n_scalars + 1) + [I.op("NormV3")], [])


@pytest.mark.parametrize("n_scalars,n_vectors", [(15, 3), (4, 4)])
def test_the_program_spills_as_many_values_as_it_says(n_scalars, n_vectors):
    d = E.analyze(deep_program(n_scalars, n_vectors), 7)["depth_fast"]
    assert d[0] == n_scalars and d[2] == n_vectors and not d[1] and not d[3] and not d[4]


def _run(e, pop, d):
    b = e.prepare(I.pack(pop), d)
    try:
        b.run()
        g = [g for g in b.describe()["groups"] if g["kernel"] == "register"]
        return b.results(), {x["points_per_thread"] for x in g}, {x["programs_per_warp"] for x in g}
    finally:
        b.close()


# 24 stack slots of 8 KB at 8 points a lane: with four programs' sums an item
# past the 200 KB a block may take, with one program's within it.  16 slots fit either way.
@pytest.mark.gpu
@pytest.mark.parametrize("n_scalars,n_vectors,points_per_lane", [(15, 3, 4), (4, 4, 8)])
def test_sums_do_not_follow_the_plans_size(n_scalars, n_vectors, points_per_lane):
    rng = np.random.default_rng(5)
    n = 65_536
    ds = Dataset.new(rng.uniform(-1, 1, (n, 7)).astype(np.float32), rng.uniform(-1, 1, n).astype(np.float32),
                     [FLOAT, VEC3, VEC3])
    prog = deep_program(n_scalars, n_vectors)
    sms, chunks = 148, n // 4096
    with E.Engine() as e:
        d = e.upload(ds)
        seen = set()
        for k in (1, 18 * sms // chunks + 8, 72 * sms // chunks + 8):
            got, points, shared = _run(e, [prog] * k, d)
            if not seen:
                alone = got[0].view(np.uint32)
            assert (got.view(np.uint32) == alone).all()
            assert points == {points_per_lane}
            seen |= shared
        assert seen == {1, 2, 4}   # a plan of every step of the rule

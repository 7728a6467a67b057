"""Few programs on large data sets: an item holds one program until the plan has
chunks enough for the device several times over, or its data sets (F+V3) chunks
enough for every SM by themselves (runtime.cu programs_an_item)."""
import pytest

from rsr_b200 import isa as I
from rsr_b200 import workloads as W
from rsr_b200.evaluator import Engine

pytestmark = pytest.mark.gpu


def _items(e, pop, **kw):
    b = e.prepare(I.pack(pop), **kw)
    try:
        g = [g for g in b.describe()["groups"] if g["kernel"] == "register"]
        return sum(x["items"] for x in g), {x["programs_per_warp"] for x in g}
    finally:
        b.close()


@pytest.mark.parametrize("points", [262_136, 262_144, 600_000])
def test_one_program_an_item_while_the_plan_is_small(points):
    chunks = -(-points // 4096)
    pop = W.inverse_population(12, seed=7)
    with Engine() as e:
        d = e.upload(W.inverse_dataset(points, seed=9))
        for n in (1, 2, 4, 12):
            assert n * chunks < 18 * 148
            assert _items(e, pop[:n], dataset=d) == (n * chunks, {1})


def test_a_large_data_set_among_small_ones():
    pop = W.inverse_population(41, seed=7)
    small, large = W.inverse_dataset(5000, seed=1), W.inverse_dataset(262_144, seed=2)
    with Engine() as e:
        small, large = e.upload(small), e.upload(large)
        assert _items(e, pop, datasets=[small] * 40 + [large]) == (40 * 2 + 64, {1})


def test_data_sets_that_fill_the_device_by_themselves():
    """F+V3 on 1M points: 245 chunks are more than one and a half an SM."""
    pop = W.lorentz_population(44, seed=7)
    small, large = W.lorentz_dataset(5000, seed=1), W.lorentz_dataset(1_000_000, seed=2)
    with Engine() as e:
        small, large = e.upload(small), e.upload(large)
        assert _items(e, pop[:4], dataset=large)[1] == {4}
        assert _items(e, pop, datasets=[small] * 40 + [large] * 4)[1] == {1}   # not where most sets are small

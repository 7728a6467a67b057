"""How many programs share a work item follows from the plan's size
(runtime.cu programs_an_item); no result does."""
import numpy as np
import pytest

from rsr_b200 import isa as I
from rsr_b200 import workloads as W
from rsr_b200.evaluator import Engine

pytestmark = pytest.mark.gpu


def _run(e, pop, d):
    b = e.prepare(I.pack(pop), d)
    try:
        b.run()
        return b.results(), {g["programs_per_warp"] for g in b.describe()["groups"] if g["kernel"] == "register"}
    finally:
        b.close()


@pytest.mark.parametrize("family,points", [("scalar", 400), ("vector", 5000), ("matrix", 4097)])
def test_alone_as_in_plans_of_every_size(family, points):
    make_ds, make_pop = {"scalar": (W.scalar_dataset, W.scalar_population), "vector": (W.lorentz_dataset, W.lorentz_population),
                         "matrix": (W.transform_dataset, W.transform_population)}[family]
    pop = make_pop(12_000, seed=3)
    with Engine() as e:
        d = e.upload(make_ds(points, seed=4))
        whole, large = _run(e, pop, d)
        sms, chunks = 148, -(-points // 4096)
        sizes = set(large)
        for n in (1, 3, 18 * sms // chunks - 1, 18 * sms // chunks + 1, 72 * sms // chunks + 1):
            part, g = _run(e, pop[:n], d)
            assert np.array_equal(part.view(np.uint32), whole[:n].view(np.uint32))
            sizes |= g
        assert len(sizes) > 1   # the rule's branches were met

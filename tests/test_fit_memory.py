"""A context keeps a fit's device buffers for its next fit (lbfgs.cu), and gives
them back with its last data set."""
import numpy as np
import pytest

from rsr_b200 import isa as I
from rsr_b200 import workloads as W
from rsr_b200.evaluator import Engine

pytestmark = pytest.mark.gpu
MB = 1 << 20


def test_buffers_go_with_the_last_data_set():
    import torch
    free = lambda: torch.cuda.mem_get_info()[0]  # noqa: E731
    ds, pop = W.lorentz_dataset(100_000, seed=2), I.pack(W.lorentz_population(4096, seed=12))
    with Engine() as e:   # every kernel loaded
        first = e.fit_lbfgs(pop, ds, max_iterations=1)
    with Engine() as e:
        d = e.upload(ds)
        e.compute_mse_grad_batch(pop, d)
        e.compute_mse_batch(pop, d)
        d.release()
        before = free()
        d, other = e.upload(ds), e.upload(W.lorentz_dataset(1000, seed=3))
        with_data = free()
        e.fit_lbfgs(pop, d, max_iterations=1)
        kept = with_data - free()
        assert kept > 32 * MB   # the gradient sums of 4096 programs x 25 parts alone are 26 MB
        other.release()
        assert with_data - free() > 32 * MB   # still there for the next fit
        d.release()
        assert before - free() < 4 * MB
        # and a fit after that is the first one's, bit for bit
        again = e.fit_lbfgs(pop, e.upload(ds), max_iterations=1)
        assert all(np.array_equal(a.view(np.uint32), b.view(np.uint32)) for a, b in zip(first[:2], again[:2]))

"""GPU: a batch of many small systems runs one launch per kernel; each system's results are those of a
batch of its own, bit for bit, whatever its companions' sizes, trajectory counts and couplings.
"""
import numpy as np
import pytest

from molspin_b200 import systems as S
from molspin_b200.batching import BatchB200
from tests import helpers as h

pytestmark = pytest.mark.gpu

# (nuclei, trajectories): every kernel of the row and quartet forms, one trajectory to several hundred
SHAPES = [([], 1), ([2], 5), ([2, 2, 2], 33), ([2] * 4, 8), ([3, 2, 2], 3), ([2] * 5, 17), ([3, 3, 2, 2], 9), ([2] * 6, 2),
          ([3, 2, 2, 2, 2, 2], 4), ([2] * 7, 6), ([3, 3, 2, 2, 2, 2], 1), ([2] * 8, 3), ([3] + [2] * 7, 2), ([2] * 4, 300),
          ([3, 3], 40)]


def _systems(copies):
    out = []
    for k in range(copies):
        for nuc, M in SHAPES:
            half = len(nuc) // 2
            s = h.random_system(nuc[:half], nuc[half:], seed=50 * k + len(out), st_rate=0.02 * (k % 2)) if nuc else \
                S.radical_pair([], [], [], [], np.array([0.0, 2e-4, 5e-5]), sink_rate=2e-3)
            out.append((s, s.trace_samples(M, 1.0 + k), len(out)))
    return out


@pytest.mark.parametrize("copies,m", [(1, 3), (5, 12)])
def test_each_system_as_if_alone(copies, m):
    times = S.time_grid(4.0, 1.0)
    systems = _systems(copies)
    batch = BatchB200(0)
    for s, F, seed in systems:
        batch.add(s, F, seed=seed)
    batch.run(times, m)
    before = batch.launch_count()
    batch.run(times, m, accumulate=True, step_offset=4)
    assert batch.launch_count() - before <= 10  # three kernels of rows, seven of quartets
    got = [batch.yields(k)[0] for k in range(len(systems))]
    for (s, F, seed), per in zip(systems, got):
        one = BatchB200(0)
        one.add(s, F, seed=seed)
        one.run(times, m)
        one.run(times, m, accumulate=True, step_offset=4)
        np.testing.assert_array_equal(one.yields(0)[0], per)

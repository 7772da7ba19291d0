"""The path engine's columns where a chunk of pairs has more of them than the pinned staging holds: the kernels write
device memory, copied into host memory of the call."""

import numpy as np
import pytest

from optlab_b200 import engine
from optlab_b200.requests import paths_request

pytestmark = pytest.mark.gpu

STEPS, NAMES, REPEAT = 40, 5, 25  # 1000 observations of five names: 40 KB a pair in float, 1024 pairs a chunk at least


def _columns(repeat, precision, n_pairs):
    corr = np.full((NAMES, NAMES), 0.4) + 0.6 * np.eye(NAMES)
    obs = np.repeat(np.arange(1, STEPS + 1), repeat)
    held = paths_request(dt=np.full(STEPS, 1 / 52), t0=np.arange(STEPS) / 52, obs_step=obs, root=np.linalg.cholesky(corr),
                         kind=[1] * NAMES, cvar=np.zeros(NAMES), heston=np.tile([0.0, 1, 1, 0, 0], NAMES), same=1,
                         fwd=np.full((NAMES, len(obs)), 100.0), n_pairs=n_pairs, seed=5,
                         step_row=np.tile(np.arange(STEPS), (NAMES, 1)), lo=np.full(STEPS, -1.0),
                         inv_dx=np.full(STEPS, 10.0), table=np.linspace(0.03, 0.06, STEPS * 21).reshape(STEPS, 21), n_x=21)
    engine.paths(held, precision)
    return next(a for a in held.keep if isinstance(a, np.ndarray) and a.ndim == 3)


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("n_pairs", [1024, 2500])
def test_columns_without_the_staging_equal_those_through_it(precision, n_pairs):
    many, one = _columns(REPEAT, precision, n_pairs), _columns(1, precision, n_pairs)
    assert np.array_equal(many, np.repeat(one, REPEAT, axis=1))

"""Runs of several steps with the state on the chip, beside test_gpu_resident.py:
what the blocks tell each other, and what goes on around a run."""
import numpy as np
import pytest

from test_gpu_resident import _case, _compare

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("flux", ["upwind", "lax_wendroff"])
@pytest.mark.parametrize("runs", [(33,), (4,) * 8])
def test_non_finite_states_far_from_the_walls(runs, flux):
    """Non-finite values that travel through blocks without boundary nodes or
    ghost faces, whose import warps meet one barrier a step: about 100 of the 152
    blocks."""
    cfn = _case(60_000, flux)
    c = cfn[0]
    pdf = np.asarray(c.pdf, np.float32).copy()
    xy = np.asarray(c.centroids)
    span = xy.max(0) - xy.min(0)
    for at, q, v in (((0.3, 0.6), 1, np.nan), ((0.5, 0.5), 5, np.inf), ((0.7, 0.35), 3, -np.inf)):
        pdf[((xy - xy.min(0) - span * at) ** 2).sum(1).argmin(), q] = v
    c.pdf = pdf
    _compare(cfn, runs, "auto", "staged")

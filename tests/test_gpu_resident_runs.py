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


def test_two_handles_side_by_side():
    """A long run of one handle does not keep the steps of another from running, nor
    make its blocks give up, and both end as they do alone."""
    import torch

    from fvdbm_jax_gb300 import Environment
    cfn = [_case(3200, "upwind"), _case(60_000, "upwind")]
    alone = []
    for c in cfn:
        env = Environment(*c)
        env.init()
        env.step(64)
        alone.append(np.array(env.cells.pdf))
        env.close()
    a, b = (Environment(*c) for c in cfn)
    a.init()
    b.init()
    a.step(64)
    assert np.array_equal(a.cells.pdf, alone[0])
    a.step(500_000)  # more than a second
    b.step(64)
    b.sync()
    busy = not torch.cuda.ExternalStream(a.stream_ptr).query()
    assert np.array_equal(b.cells.pdf, alone[1])
    a.sync()
    assert busy
    a.close()
    b.close()


def test_beside_other_kernels():
    """Runs while another stream keeps the SMs busy."""
    import torch

    from fvdbm_jax_gb300 import Environment
    cfn = _case(60_000, "upwind")
    x = torch.randn((8192, 8192), device="cuda")
    other = torch.cuda.Stream()
    got = []
    for load in (0, 40):
        env = Environment(*cfn)
        env.init()
        torch.cuda.synchronize()
        with torch.cuda.stream(other):
            for _ in range(load):
                y = x @ x
        for _ in range(20):
            env.step(64)
        env.sync()
        got.append(np.array(env.cells.pdf))
        env.close()
    torch.cuda.synchronize()
    assert np.array_equal(*got)

"""How runs of several steps are carried out: which handles keep the state on the
chip, and that the launches they take otherwise (short runs, larger meshes, or
by fvdbm_run_config) still give the same bits."""
import ctypes as C

import numpy as np
import pytest

from test_gpu_resident import _case, _compare, _same

pytestmark = pytest.mark.gpu

LAUNCHES, TWO_COPIES, RING = 0, 1, 2


def _info(env):
    from fvdbm_jax_gb300 import _native as nat
    r = nat.RunInfo()
    nat.check(nat.lib().fvdbm_get_run_info(env.handle, C.byref(r)), env.handle)
    return r


def _launches_only(env):
    from fvdbm_jax_gb300 import _native as nat
    nat.check(nat.lib().fvdbm_run_config(env.handle, 0), env.handle)
    assert _info(env).path == LAUNCHES


@pytest.mark.parametrize("cells,flux,lattice,kernel,path,least", [
    (2, "upwind", "D2Q9", "auto", TWO_COPIES, 4), (2, "lax_wendroff", "D2Q13", "auto", TWO_COPIES, 4),
    (98, "upwind", "D2Q9", "fast", TWO_COPIES, 4), (3200, "upwind", "D2Q9", "persist", TWO_COPIES, 1),
    (96_000, "upwind", "D2Q9", "auto", TWO_COPIES, 4), (96_000, "lax_wendroff", "D2Q13", "auto", TWO_COPIES, 4),
    (120_000, "lax_wendroff", "D2Q9", "fast", TWO_COPIES, 4), (215_000, "upwind", "D2Q9", "auto", RING, 4),
    (240_000, "upwind", "D2Q9", "fast", RING, 6), (270_000, "upwind", "D2Q9", "auto", RING, 8),
    (300_000, "upwind", "D2Q9", "fast", RING, 8), (320_000, "upwind", "D2Q9", "persist", RING, 1),
    (400_000, "upwind", "D2Q9", "persist", RING, 2), (400_000, "upwind", "D2Q9", "auto", RING, 10),
    (400_000, "lax_wendroff", "D2Q9", "auto", TWO_COPIES, 8), (270_000, "upwind", "D2Q13", "auto", TWO_COPIES, 8),
    (420_000, "upwind", "D2Q9", "auto", RING, 16), (430_000, "upwind", "D2Q9", "persist", RING, 16),
    (490_000, "upwind", "D2Q9", "auto", RING, 18), (520_000, "upwind", "D2Q9", "fast", RING, 24), (600_000, "upwind", "D2Q9", "auto", RING, 48),
    (450_000, "lax_wendroff", "D2Q9", "auto", LAUNCHES, 0), (650_000, "upwind", "D2Q9", "auto", LAUNCHES, 0),
    (3200, "upwind", "D2Q9", "fused", LAUNCHES, 0), (3200, "upwind", "D2Q9", "fused_nodes", LAUNCHES, 0),
    (3200, "upwind", "D2Q9", "staged", LAUNCHES, 0), (3200, "upwind", "D2Q13", "staged", LAUNCHES, 0)])
def test_path_of_a_handle(cells, flux, lattice, kernel, path, least):
    from fvdbm_jax_gb300 import Environment
    env = Environment(*_case(cells, flux, lattice), kernel=kernel)
    env.init()
    r = _info(env)
    assert (r.path, r.min_steps) == (path, least)
    assert (r.blocks > 0) == (path != LAUNCHES)
    env.close()


def test_path_of_other_meshes():
    """Channel with outlet and cylinder, the finite-volume update, the cos stencil;
    no coordinates (device order: chunks' neighbours may be too far apart)."""
    from fvdbm_jax_gb300 import Batch, Environment
    for cfn, kw, path in ((_case(60_000, "upwind", mesh="channel"), {}, TWO_COPIES),
                          (_case(250_000, "upwind", mesh="channel"), {}, RING),
                          (_case(250_000, "upwind"), {"finite_volume": True}, RING),
                          (_case(5000, "upwind", cos=True), {}, TWO_COPIES)):
        env = Environment(*cfn, **kw)
        env.init()
        assert _info(env).path == path
        env.close()
    for sizes, path in (((2, 98, 3200, 20_000, 800), TWO_COPIES), ((2, 98, 3200, 200_000, 230_000), RING)):
        b = Batch([_case(n, "upwind", seed=k) for k, n in enumerate(sizes)])
        b.init()
        assert _info(b).path == path
        b.close()


@pytest.mark.parametrize("lattice,flux,kernel", [("D2Q9", "upwind", "persist"), ("D2Q9", "lax_wendroff", "persist"),
                                                 ("D2Q9", "upwind", "auto"), ("D2Q13", "upwind", "auto"),
                                                 ("D2Q9", "upwind", "fast")])
@pytest.mark.parametrize("cells,mesh,special", [(98, "cavity", 0.0), (3200, "cavity", 1e-3), (60_000, "channel", 0.0)])
def test_runs_by_launches(cells, mesh, special, lattice, flux, kernel):
    """Grid barriers between the steps of a persistent launch, and replayed graphs
    (runs of 32 and more), against single steps."""
    from fvdbm_jax_gb300 import Environment
    if kernel == "fast":
        special = 0.0  # (its bits are its own)
    cfn = _case(cells, flux, lattice, mesh, special=special)
    a, b = (Environment(*cfn, kernel=k) for k in (kernel, "fast" if kernel == "fast" else "staged"))
    a.init()
    b.init()
    _launches_only(a)
    for n in (5, 1, 70):
        a.step(n)
        for _ in range(n):
            b.step()
        _same(a, b, (kernel, n))
    a.close()
    b.close()


@pytest.mark.parametrize("cells,kernel,runs", [(400_000, "auto", (9, 10, 1, 17)), (520_000, "fast", (23, 24, 1, 31)),
                                               (600_000, "auto", (47, 48, 1, 53))])
def test_shortest_runs_of_the_ring(cells, kernel, runs):
    _compare(_case(cells, "upwind"), runs, kernel, "fast" if kernel == "fast" else "fused")


def test_persistent_runs_beyond_the_chip():
    _compare(_case(650_000, "upwind"), (2, 1, 5), "persist", "fused")


def test_long_horizon_by_launches():
    """2,000 steps of the 60k channel in persistent launches, on the chip and as
    replayed graphs."""
    from fvdbm_jax_gb300 import Environment
    cfn = _case(60_000, "upwind", mesh="channel")
    envs = [Environment(*cfn, kernel=k) for k in ("persist", "auto", "auto")]
    for e in envs:
        e.init()
    _launches_only(envs[0])
    _launches_only(envs[2])
    for e in envs:
        e.step(2000)
    _same(envs[0], envs[1], "persist")
    _same(envs[2], envs[1], "graphs")
    for e in envs:
        e.close()


@pytest.mark.parametrize("flux", ["upwind", "lax_wendroff"])
def test_batch_by_launches(flux):
    """Graphs of a batch, dropped and captured again as cases retire and return."""
    from fvdbm_jax_gb300 import Batch
    cs = [_case(n, flux, seed=k) for k, n in enumerate((2, 98, 3200, 20_000, 800))]
    for k, (c, _, _) in enumerate(cs):
        c.dynamics.tau = 0.55 + 0.05 * k
    a, b = Batch(cs), Batch(cs)
    a.init()
    b.init()
    _launches_only(a)
    for n, active in ((64, None), (37, (1, 0, 1, 1, 1)), (70, (1, 1, 0, 1, 0)), (33, (1, 1, 1, 1, 1))):
        if active is not None:
            a.set_active(active)
            b.set_active(active)
        a.step(n)
        for _ in range(n):
            b.step(1)
        sa, sb = a.state(), b.state()
        for k in sa:
            assert np.array_equal(sa[k], sb[k], equal_nan=True), (n, k)
    a.close()
    b.close()


@pytest.mark.parametrize("declined", [False, True])
def test_autotune_times_the_launches_it_tunes(declined, monkeypatch):
    from fvdbm_jax_gb300 import Batch
    b = Batch([_case(n, "upwind", seed=k) for k, n in enumerate((98, 3200))])
    b.init()
    if declined:
        _launches_only(b)
    seen, step = [], Batch.step
    monkeypatch.setattr(Batch, "step", lambda self, n=1: (seen.append(_info(self).path), step(self, n))[1])
    rec = b.autotune(steps=32, use_cache=False)
    assert set(seen) == {LAUNCHES} and len(seen) == 2 * len(rec["sec_per_step"])
    assert _info(b).path == (LAUNCHES if declined else TWO_COPIES)
    b.close()


def test_creation_without_memory_for_the_tables():
    """A handle whose launches fit in the device's memory and whose tables of the run on the
    chip do not: it is created, and its runs take the launches."""
    import torch

    from fvdbm_jax_gb300 import Environment
    cfn = _case(400_000, "lax_wendroff")
    need, got = [], []
    for kernel in ("fused_nodes", "auto"):  # without and with the tables
        env = Environment(*cfn, kernel=kernel)
        env.init()
        env.step(9)
        got.append(np.array(env.cells.pdf))
        need.append(env.info()["device_bytes"])
        env.close()
    tables = need[1] - need[0]
    assert tables > 30e6
    torch.cuda.empty_cache()
    ballast = torch.empty(int(torch.cuda.mem_get_info()[0] - need[0] - tables / 2), dtype=torch.uint8, device="cuda")
    env = Environment(*cfn)
    try:
        env.init()
        env.step(9)
        got.append(np.array(env.cells.pdf))
        path = _info(env).path
    finally:
        env.close()
        del ballast
        torch.cuda.empty_cache()
    assert path == LAUNCHES
    assert np.array_equal(got[0], got[1]) and np.array_equal(got[0], got[2])

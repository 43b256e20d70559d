"""Runs of several steps in one launch with the state on the chip against the
same number of single staged steps, bit for bit: one to many blocks, one and
several cells per thread, both lattices and flux schemes, the finite-volume
update and the cos stencil, runs that follow one another and single steps in
between, and states with non-finite values (whose steps take the literal form
block by block)."""
import numpy as np
import pytest

import goldens as G
from test_gpu_random_state import KEYS, SPECIAL

pytestmark = pytest.mark.gpu


def _case(cells, flux, lattice="D2Q9", mesh="cavity", special=0.0, cos=False, seed=3):
    from fvdbm_jax_gb300 import D2Q9, D2Q13, Mesher, meshgen
    if mesh == "cavity":
        raw = meshgen.cavity(n=int(round((cells / 2) ** 0.5)) + 1, seed=seed)
    else:
        raw = meshgen.channel_cylinder(n_target=cells, seed=seed)
    m = Mesher().import_meshpy(raw)
    m.calc_mesh_properties()
    dyn = (D2Q9 if lattice == "D2Q9" else D2Q13)(0.6, 0.25 * float(m.face_lengths.min()))
    c, f, n = m.to_env(dyn, flux)
    if cos:
        f.stencil_variant = "cos"
        f.alpha = np.random.default_rng(seed).uniform(0, 0.4, (f.n.shape[0], 1)).astype(np.float32)
    for mk in (1, 2, 4, 5):
        n = m.set_vel_node(n, mk, (0.0, 0.0))
    n = m.set_vel_node(n, 3, (0.1, 0.0))
    if mesh == "channel":
        n = m.set_rho_node(n, 2, 1.0)
    rng = np.random.default_rng(seed + 1)
    pdf = np.asarray(c.pdf, np.float32)
    pdf = (pdf * (1.0 + 0.1 * rng.standard_normal(pdf.shape))).astype(np.float32)
    if special:
        pick = rng.random(pdf.shape) < special
        pdf[pick] = SPECIAL[rng.integers(0, SPECIAL.size, int(pick.sum()))]
    c.pdf = pdf
    return c, f, n


def _same(a, b, what):
    ga, gb = G.env_state(a), G.env_state(b)
    for k in KEYS:
        assert np.array_equal(ga[k], gb[k], equal_nan=True), (what, k)


def _compare(cfn, runs, kernel, ref, fv=False):
    from fvdbm_jax_gb300 import Environment
    a, b = (Environment(*cfn, kernel=k, finite_volume=fv) for k in (kernel, ref))
    a.init()
    b.init()
    for n in runs:
        a.step(n)
        for _ in range(n):
            b.step()
        _same(a, b, (kernel, n))
    a.close()
    b.close()


@pytest.mark.parametrize("lattice", ["D2Q9", "D2Q13"])
@pytest.mark.parametrize("flux", ["upwind", "lax_wendroff"])
@pytest.mark.parametrize("cells,mesh", [(2, "cavity"), (18, "cavity"), (98, "cavity"), (3200, "cavity"),
                                        (60_000, "channel"), (96_000, "cavity")])
def test_runs_match_single_steps(cells, mesh, flux, lattice):
    _compare(_case(cells, flux, lattice, mesh), (4, 1, 7, 33), "auto", "staged")


@pytest.mark.parametrize("kernel", ["auto", "persist"])
@pytest.mark.parametrize("flux", ["upwind", "lax_wendroff"])
def test_cos_stencil_and_finite_volume(flux, kernel):
    _compare(_case(5000, flux, cos=True), (5, 8), kernel, "staged")
    _compare(_case(5000, flux), (5, 8), kernel, "staged", fv=True)


def test_many_cells_per_thread():
    """Beyond 2^18 cells (the single-launch family's node buffers) and near
    the capacity of the blocks' shared memory."""
    for cells in (270_000, 400_000):
        _compare(_case(cells, "upwind"), (4, 1, 6), "auto", "fused")


@pytest.mark.parametrize("cells,kernel,fv,special", [(215_000, "auto", False, 0.0), (250_000, "auto", True, 1e-6),
                                                     (300_000, "fast", False, 0.0), (420_000, "auto", True, 0.0),
                                                     (430_000, "fast", False, 0.0), (600_000, "auto", False, 0.0),
                                                     (430_000, "persist", False, 0.0)])
def test_in_place(cells, kernel, fv, special):
    """From the line where the ring is faster to its capacity: two and more
    chunks, runs that leave the ring at every offset."""
    ref = "fast" if kernel == "fast" else "fused"
    _compare(_case(cells, "upwind", special=special), (16, 1, 19), kernel, ref, fv=fv)


def test_two_copies_near_capacity():
    """What the ring does not take."""
    _compare(_case(400_000, "lax_wendroff"), (8, 9), "auto", "fused")
    _compare(_case(270_000, "upwind", lattice="D2Q13"), (8, 9), "auto", "fused")


def test_ring_without_coordinates():
    """The sweep's order needs them: the device order, or two copies."""
    import ctypes as C

    from fvdbm_jax_gb300 import _native as nat
    from fvdbm_jax_gb300.environment import pack
    cfn = _case(220_000, "upwind")
    pdf = np.ascontiguousarray(cfn[0].pdf, np.float32)
    out = []
    for runs in ((17,), (1,) * 17):
        mesh, params, keep, *_ = pack(*cfn, kernel="auto")
        mesh.cell_xy = None
        L, h = nat.lib(), C.c_void_p()
        nat.check(L.fvdbm_create(C.byref(mesh), C.byref(params), C.byref(h)), None)
        nat.check(L.fvdbm_set_state(h, nat.fptr(pdf), None, None, None), h)
        for n in runs:
            nat.check(L.fvdbm_step(h, n), h)
        got = np.empty_like(pdf)
        nat.check(L.fvdbm_get_cells(h, nat.fptr(got), None, None, None), h)
        L.fvdbm_destroy(h)
        out.append(got)
    assert np.array_equal(*out)


def test_in_place_batch():
    """Cases of one and of many blocks; one retires in between and comes back."""
    from fvdbm_jax_gb300 import Batch
    cs = [_case(n, "upwind", seed=k) for k, n in enumerate((2, 98, 3200, 200_000, 230_000))]
    for k, (c, _, _) in enumerate(cs):
        c.dynamics.tau = 0.55 + 0.05 * k
    a, b = Batch(cs), Batch(cs)
    a.init()
    b.init()
    for n, active in ((17, None), (16, (1, 0, 1, 0, 1)), (20, (1, 1, 1, 1, 1))):
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


@pytest.mark.parametrize("lattice", ["D2Q9", "D2Q13"])
@pytest.mark.parametrize("flux", ["upwind", "lax_wendroff"])
@pytest.mark.parametrize("share", [1e-4, 2e-3])
def test_non_finite_states(share, flux, lattice):
    _compare(_case(3200, flux, lattice, special=share), (6, 5), "auto", "staged")


@pytest.mark.parametrize("flux", ["upwind", "lax_wendroff"])
@pytest.mark.parametrize("cells", [98, 3200, 120_000])
def test_fast_family_runs_match_single_steps(cells, flux):
    _compare(_case(cells, flux), (4, 1, 20), "fast", "fast")


@pytest.mark.parametrize("flux", ["upwind", "lax_wendroff"])
def test_batch_runs_match_single_steps(flux):
    """Uneven cases with their own tau and dt, one of a few cells; one retires in
    between and comes back."""
    from fvdbm_jax_gb300 import Batch
    cs = [_case(n, flux, seed=k) for k, n in enumerate((2, 98, 3200, 20_000, 800))]
    for k, (c, _, _) in enumerate(cs):
        c.dynamics.tau = 0.55 + 0.05 * k
    a, b = Batch(cs), Batch(cs)
    a.init()
    b.init()
    for n, active in ((5, None), (6, (1, 0, 1, 1, 1)), (1, None), (12, (1, 1, 0, 1, 0)), (5, (1, 1, 1, 1, 1))):
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

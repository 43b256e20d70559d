"""Runs of several steps with the state on the chip, beside test_gpu_resident.py:
what the blocks tell each other, and what goes on around a run."""
import numpy as np
import pytest

from test_gpu_resident import _case, _compare, _same

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


def _beside(env):
    from test_gpu_run_paths import _info
    return bool(_info(env).readback_beside)


@pytest.mark.parametrize("cells", [3200, 270_000])
def test_which_single_steps_are_read_back_beside(cells):
    """rho and vel of the step's input, read while the step runs: after a step that
    follows other work, after the last of as many steps as the frame before had, and on
    large meshes after any; the values are those of a read-back that waits."""
    import torch

    from fvdbm_jax_gb300 import Environment
    from fvdbm_jax_gb300 import _native as nat
    L, large = nat.lib(), cells >= 1 << 18
    cfn = _case(cells, "upwind")
    env, ref = Environment(*cfn), Environment(*cfn, kernel="staged")
    env.init()
    ref.init()
    h = env.handle
    N = np.shape(cfn[0].pdf)[0]
    rho, vel = (torch.zeros(s).pin_memory().numpy() for s in ((N,), (N, 2)))
    rows = np.arange(4, dtype=np.int32)
    buf = torch.zeros((4, 9), device="cuda")

    def step(k, beside):
        for _ in range(k):
            env.step()
            ref.step()
        assert _beside(env) == beside

    def read():
        nat.check(L.fvdbm_get_cells(h, None, nat.fptr(rho), nat.fptr(vel), None), h)
        assert np.array_equal(rho, np.asarray(ref.cells.rho).reshape(-1))
        assert np.array_equal(vel, ref.cells.vel)

    for first, k in ((True, 1), (True, 1), (large, 3), (True, 3), (True, 3)):
        step(k, first)
        read()
    step(1, True)
    step(1, large)
    pack = lambda: nat.check(L.fvdbm_pack_cells(h, nat.iptr(rows), 4, buf.data_ptr()), h)
    unpack = lambda: nat.check(L.fvdbm_unpack_cells(h, nat.iptr(rows), 4, buf.data_ptr()), h)
    for other in (pack, lambda: (pack(), unpack()), env.residual, lambda: env.nodes.pdf):
        other()
        step(1, True)
        read()
    env.step(0)
    step(1, True)
    read()
    env.close()
    ref.close()


@pytest.mark.parametrize("cells,kernel", [(3200, "auto"), (3200, "fast"), (270_000, "auto")])
def test_replays_of_a_captured_graph_between_runs(cells, kernel):
    """Steps captured by the caller (which are launches, whatever their number) go on from
    the state that runs, single steps and setters leave, and the other way round."""
    import torch

    from fvdbm_jax_gb300 import Environment
    cfn = _case(cells, "upwind")
    a, b = (Environment(*cfn, kernel=kernel) for _ in range(2))
    a.init()
    b.init()
    a.step(2)
    a.sync()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=torch.cuda.ExternalStream(a.stream_ptr), capture_error_mode="thread_local"):
        a.step(20)
    done = 2

    def replay():
        with torch.cuda.stream(torch.cuda.ExternalStream(a.stream_ptr)):
            g.replay()

    for n, graph in ((0, True), (16, True), (2, True), (17, False), (1, True), (20, False), (6, True), (0, True)):
        a.step(n)
        done += n
        if graph:
            replay()
            done += 20
    a.sync()
    for _ in range(done):
        b.step()
    assert np.array_equal(a.cells.pdf, b.cells.pdf)
    pdf = np.array(cfn[0].pdf)
    a.cells.pdf = pdf
    b.cells.pdf = pdf
    replay()
    a.step(16)
    for _ in range(36):
        b.step()
    assert np.array_equal(a.cells.pdf, b.cells.pdf)
    a.close()
    b.close()


def _porous(cells, seed=5):
    from fvdbm_jax_gb300 import D2Q9, Mesher, meshgen
    m = Mesher().import_meshpy(meshgen.porous(n_obstacles=30, n_target=cells, porosity=0.8, seed=seed, gap_cells=1.0))
    m.calc_mesh_properties()
    c, f, n = m.to_env(D2Q9(0.6, 0.25 * float(m.face_lengths.min())), "upwind")
    for mk in (1, 3, 5):
        n = m.set_vel_node(n, mk, (0.0, 0.0))
    n = m.set_rho_node(m.set_rho_node(n, 4, 1.02), 2, 1.0)
    rng = np.random.default_rng(seed)
    pdf = np.asarray(c.pdf, np.float32)
    c.pdf = (pdf * (1.0 + 0.1 * rng.standard_normal(pdf.shape))).astype(np.float32)
    return c, f, n


def test_ring_with_density_nodes_and_obstacles():
    _compare(_case(250_000, "upwind", mesh="channel"), (16, 1, 19), "auto", "fused")
    _compare(_porous(230_000), (16, 1, 19), "auto", "fused")


def test_ring_batch_with_density_nodes_and_obstacles():
    from fvdbm_jax_gb300 import Batch
    cs = [_case(98, "upwind"), _porous(20_000), _case(150_000, "upwind", mesh="channel"), _porous(120_000, 6)]
    a, b = Batch(cs), Batch(cs)
    a.init()
    b.init()
    for n, active in ((17, None), (16, (1, 0, 1, 1)), (20, (1, 1, 0, 1))):
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


@pytest.mark.parametrize("cells,kernel", [(98, "auto"), (3200, "auto"), (3200, "fast"), (60_000, "auto"), (270_000, "auto")])
def test_single_steps_among_other_calls(cells, kernel):
    """A step's first launch may start beside the step before; in between come setters of
    cells and nodes, halo rows, read-backs and runs, in any order."""
    import torch

    from fvdbm_jax_gb300 import Environment
    from fvdbm_jax_gb300 import _native as nat
    L, rng = nat.lib(), np.random.default_rng(cells)
    cfn = _case(cells, "upwind")
    N = np.shape(cfn[0].pdf)[0]
    env = [Environment(*cfn, kernel=k) for k in (kernel, "fast" if kernel == "fast" else "staged")]
    for e in env:
        e.init()
    rows = rng.choice(N, min(N, 64), replace=False).astype(np.int32)
    buf = torch.zeros((rows.size, 9), device="cuda")
    pdf, vel = np.array(cfn[0].pdf), np.array(cfn[2].vel)

    def macros(e):
        nat.check(L.fvdbm_set_cells_eq(e.handle, nat.fptr(rho), nat.fptr(u)), e.handle)

    def halo(e):
        nat.check(L.fvdbm_pack_cells(e.handle, nat.iptr(rows), rows.size, buf.data_ptr()), e.handle)
        nat.check(L.fvdbm_unpack_cells(e.handle, nat.iptr(rows[::-1].copy()), rows.size, buf.data_ptr()), e.handle)
        e.sync()

    def cells_in(e):
        e.cells.pdf = pdf * scale

    def nodes_in(e):
        e.nodes.vel = vel * scale

    calls = [macros, halo, cells_in, nodes_in, lambda e: e.residual(), lambda e: e.nodes.pdf, lambda e: e.cells.rho,
             lambda e: e.sync(), lambda e: None]
    for k in range(40):
        call, steps, run = calls[rng.integers(len(calls))], int(rng.integers(1, 5)), int(rng.integers(4, 20))
        scale = np.float32(rng.uniform(0.98, 1.02))
        rho = (1.0 + 0.01 * rng.standard_normal(N)).astype(np.float32)
        u = (0.01 * rng.standard_normal((N, 2))).astype(np.float32)
        for i, e in enumerate(env):
            call(e)
            for _ in range(steps):
                e.step()
                if i:
                    e.sync()
        if k % 8 == 7:
            env[0].step(run)
            for _ in range(run):
                env[1].step()
                env[1].sync()
            _same(*env, (kernel, k))
    for e in env:
        e.close()


def test_single_batch_steps_among_other_calls():
    from fvdbm_jax_gb300 import Batch
    rng = np.random.default_rng(7)
    cs = [_case(n, "upwind", seed=k) for k, n in enumerate((2, 98, 3200, 20_000))]
    a, b = Batch(cs), Batch(cs)
    a.init()
    b.init()
    for k in range(24):
        active = rng.integers(0, 2, 4) if k % 3 else np.ones(4, int)
        for i, x in enumerate((a, b)):
            x.set_active(active)
            for _ in range(1 + k % 4):
                x.step(1)
                if i:
                    x.sync()
            if k % 5 == 4:
                x.residual()
        if k % 6 == 5:
            sa, sb = a.state(), b.state()
            for q in sa:
                assert np.array_equal(sa[q], sb[q], equal_nan=True), (k, q)
    a.close()
    b.close()

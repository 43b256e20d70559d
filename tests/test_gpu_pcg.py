"""The warm start's potential-flow estimate solved on the GPU
(``fvdbm_pcg``, Jacobi-preconditioned conjugate gradients, through
``warmstart.solve_potentials``): against the host's sparse direct solve of the
same systems, for several cases solved together as one block-diagonal
system, and bitwise reproducible."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _cases():
    from fvdbm_jax_gb300 import cases as CS
    out = []
    for i, (k, nt) in enumerate(((20, 6000), (60, 15000), (120, 30000))):
        rin, rout = 1.01 + 0.01 * i, 0.99 - 0.01 * i
        out.append((CS.porous_square(k, nt, 0.003, rho_in=rin, rho_out=rout, porosity=0.8, fv_dt=1.0,
                                     seed=700 + i, mesher=True), rin, rout))
    return out


def test_gpu_potential_matches_host_solve():
    from fvdbm_jax_gb300 import warmstart as WS
    cs = _cases()
    host = [WS.sample(case, rin, rout) for case, rin, rout in cs]
    runs = []
    for _ in range(2):
        dev = [WS.sample(case, rin, rout, defer_potential=True) for case, rin, rout in cs]
        assert all(s.pending is not None for s in dev)
        it, rel = WS.solve_potentials(dev, rtol=1e-6)
        assert all(s.pending is None for s in dev)
        assert 0 < it < 50_000 and rel <= 1e-6, (it, rel)
        runs.append(dev)
    for h, d, d2 in zip(host, runs[0], runs[1]):
        assert np.array_equal(d.x, d2.x)  # bitwise reproducible
        assert np.array_equal(h.x[:, :6], d.x[:, :6])  # the other features are untouched
        phi_h, phi_d = h.x[:, 6].astype(np.float64), d.x[:, 6].astype(np.float64)
        assert np.abs(phi_d - phi_h).max() <= 2e-4, np.abs(phi_d - phi_h).max()
        g_h, g_d = h.x[:, 7:9].astype(np.float64), d.x[:, 7:9].astype(np.float64)
        assert np.abs(g_d - g_h).max() <= 2e-3 * np.abs(g_h).max(), (np.abs(g_d - g_h).max(), np.abs(g_h).max())


def test_unsolved_samples_are_refused():
    from fvdbm_jax_gb300 import warmstart as WS
    case, rin, rout = _cases()[0]
    s = WS.sample(case, rin, rout, defer_potential=True)
    net = WS.MPNN(seed=0)
    with pytest.raises(ValueError, match="solve_potentials"):
        net.fit([s], epochs=1)


def test_predict_many_equals_predict():
    from fvdbm_jax_gb300 import warmstart as WS
    cs = _cases()
    smp = [WS.sample(case, rin, rout, defer_potential=True) for case, rin, rout in cs]
    WS.solve_potentials(smp)
    net = WS.MPNN(seed=3)
    one = [net.predict(s) for s in smp]
    for bc in (10**9, 20_000):  # one group; several groups on shared buffers
        many = net.predict_many(smp, batch_cells=bc)
        assert len(many) == len(one)
        for a, b in zip(one, many):
            assert np.array_equal(a, b)


def test_predict_cases_on_the_gpu_matches_the_host_path():
    """Features and stages built on the GPU (warmstart.predict_cases) give the
    network the same inputs as the host path (sample + solve_potentials +
    predict_many): the same predictions up to the potential solve's rounding,
    and the same bits on a repeat."""
    from fvdbm_jax_gb300 import warmstart as WS
    cs = _cases()
    smp = [WS.sample(case, rin, rout, defer_potential=True) for case, rin, rout in cs]
    WS.solve_potentials(smp, rtol=1e-6)
    net = WS.MPNN(seed=5)
    x = np.concatenate([s.x for s in smp])
    net.x_mu, net.x_sd = x.mean(0), np.maximum(x.std(0), 1e-12)
    host = net.predict_many(smp)
    rin, rout = [c[1] for c in cs], [c[2] for c in cs]
    for bc in (10 ** 9, 20_000):
        gpu, it, rel = WS.predict_cases(net, [c[0] for c in cs], rin, rout, batch_cells=bc)
        again, _, _ = WS.predict_cases(net, [c[0] for c in cs], rin, rout, batch_cells=bc)
        assert rel <= 1e-6 and it > 0
        for h, g, g2 in zip(host, gpu, again):
            assert np.array_equal(g, g2)
            assert g.shape == h.shape
            scale = np.abs(h).max(0)
            assert np.all(np.abs(g - h).max(0) <= 1e-3 * scale + 1e-6), (np.abs(g - h).max(0), scale)


@pytest.mark.parametrize("n", [1, 2, 255, 256, 257, 1025, 40_000, 155_648, 155_649, 311_296, 311_297])
def test_pcg_sizes(n):
    """One to many row groups per block and the launch-per-kernel form beyond
    them: rows of 1 to 9 entries in any column order, entries out of range
    (skipped), the residual it reports against float64, the same bits twice."""
    import ctypes as C

    import scipy.sparse as sp
    import torch

    from fvdbm_jax_gb300 import _native as nat
    rng = np.random.default_rng(n)
    m = 3 * n
    i, j = rng.integers(0, n, m), rng.integers(0, n, m)
    w = rng.uniform(0.1, 1.0, m)
    A = sp.coo_matrix((-np.concatenate([w, w]), (np.concatenate([i, j]), np.concatenate([j, i]))), shape=(n, n)).tocsr()
    A.setdiag(0.0)
    A.eliminate_zeros()
    A = (A + sp.diags(0.05 - np.asarray(A.sum(1)).reshape(-1))).tocsr().astype(np.float32)
    A.sum_duplicates()
    b = rng.standard_normal(n).astype(np.float32)
    ix, v, ip = A.indices.astype(np.int32), A.data.copy(), A.indptr.astype(np.int32)
    # an out-of-range entry at the end of the last row
    ix, v = np.append(ix, np.int32(n + 5)), np.append(v, np.float32(1e9))
    ip[-1] += 1
    dev = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (ip, ix, v, b)]
    L = nat.lib()
    wb = int(L.fvdbm_pcg_work_bytes(n))
    outs = []
    for _ in range(2):
        work = torch.full((wb,), 7, dtype=torch.uint8, device="cuda")
        x = torch.zeros(n, device="cuda")
        it, rel = C.c_int32(0), C.c_double(0.0)
        rc = L.fvdbm_pcg(n, *[t.data_ptr() for t in dev], x.data_ptr(), 2000, 1e-5, 7, work.data_ptr(), wb,
                         torch.cuda.current_stream().cuda_stream, C.byref(it), C.byref(rel))
        assert rc == 0
        outs.append((x.cpu().numpy(), it.value, rel.value))
    assert np.array_equal(outs[0][0], outs[1][0]) and outs[0][1:] == outs[1][1:]
    xs, its, rel = outs[0]
    assert its > 0 and its % 7 == 0 and rel <= 1e-5
    true = np.linalg.norm(b - A.astype(np.float64) @ xs) / np.linalg.norm(b)
    # the recurrence's residual drifts from the true one by rounding: a few
    # hundred float32 ulps of |A||x| at most on these well-conditioned systems
    assert true <= 1e-5 + 300 * 6e-8 * np.linalg.norm(abs(A).astype(np.float64) @ abs(xs)) / np.linalg.norm(b)


@pytest.mark.parametrize("n", [1, 31, 1023, 1024, 1025, 5000])
@pytest.mark.parametrize("bins", [1, 16, 300, (1 << 21) + 1])
def test_bin_rows(n, bins):
    """Each bin's cells in ascending order, against a stable sort by bin."""
    import torch

    from fvdbm_jax_gb300 import _native as nat
    rng = np.random.default_rng(n + bins)
    b = rng.integers(0, bins, n).astype(np.int32)
    start = np.concatenate([[0], np.cumsum(np.bincount(b, minlength=bins))]).astype(np.int32)
    w = rng.uniform(size=bins).astype(np.float32)
    dev = [torch.from_numpy(a).cuda() for a in (b, start, w)]
    pcol, ucol = (torch.full((n,), -1, dtype=torch.int32, device="cuda") for _ in range(2))
    pwt = torch.zeros(n, device="cuda")
    nat.check(nat.lib().fvdbm_ws_bin_rows(n, bins, *[t.data_ptr() for t in dev], 7, 3, pcol.data_ptr(), pwt.data_ptr(),
                                          ucol.data_ptr(), torch.cuda.current_stream().cuda_stream))
    order = np.argsort(b, kind="stable")
    assert np.array_equal(pcol.cpu().numpy(), order + 7)
    assert np.array_equal(pwt.cpu().numpy(), w[b[order]])
    assert np.array_equal(ucol.cpu().numpy(), b + 3)

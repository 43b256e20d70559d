"""The one-launch solve when its waits run out: the launch-per-kernel form takes
over from the caller's x and gives the same bits."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("polls", [0, 3])
@pytest.mark.parametrize("n", [1, 257, 40_000, 155_649, 311_296])
def test_solve_whose_waits_run_out(n, polls):
    import scipy.sparse as sp
    import torch

    from fvdbm_jax_gb300 import _native as nat
    rng = np.random.default_rng(n)
    i, j, w = rng.integers(0, n, 2 * n), rng.integers(0, n, 2 * n), rng.uniform(0.1, 1.0, 2 * n)
    A = sp.coo_matrix((-np.concatenate([w, w]), (np.concatenate([i, j]), np.concatenate([j, i]))), shape=(n, n)).tocsr()
    A = (A + sp.diags(0.05 - np.asarray(A.sum(1)).reshape(-1))).tocsr().astype(np.float32)
    dev = [torch.from_numpy(np.ascontiguousarray(a)).cuda()
           for a in (A.indptr.astype(np.int32), A.indices.astype(np.int32), A.data, rng.standard_normal(n).astype(np.float32))]
    x0 = torch.from_numpy(rng.standard_normal(n).astype(np.float32)).cuda()
    L = nat.lib()
    wb = int(L.fvdbm_pcg_work_bytes(n))
    out = []
    for limit in (1 << 20, polls):
        work = torch.full((wb,), 7, dtype=torch.uint8, device="cuda")
        x, it, rel = x0.clone(), C.c_int32(0), C.c_double(0.0)
        rc = L.fvdbm_pcg_bounded(n, *[t.data_ptr() for t in dev], x.data_ptr(), 60, 1e-6, 20, limit, work.data_ptr(), wb,
                                 torch.cuda.current_stream().cuda_stream, C.byref(it), C.byref(rel))
        assert rc == 0
        out.append((x.cpu().numpy(), it.value, rel.value))
    assert np.array_equal(out[0][0], out[1][0]) and out[0][1:] == out[1][1:]
    assert not np.array_equal(out[0][0], x0.cpu().numpy())

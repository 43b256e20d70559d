"""Chunked aggregation on either side of the lines between its routes: rows of every
length, against the same float32 fold in numpy."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("chunks,d,acc", [((127,), 64, 0), ((128,), 64, 1), ((129, 127), 128, 0), ((1, 255, 128), 64, 1),
                                          ((130, 126), 32, 0), ((200, 0, 340, 2), 64, 0), ((1,) * 50 + (300,), 64, 1),
                                          ((1,) * 200_000 + (62_144,), 64, 0), ((8,) * 256, 32, 1), ((400,), 7, 0)])
def test_rows_of_every_length(chunks, d, acc):
    import torch

    from fvdbm_jax_gb300 import _native as nat
    rng = np.random.default_rng(sum(chunks) + d)
    n, rows, nch = 500, len(chunks), sum(chunks)
    per = 3  # entries of a chunk
    col = rng.integers(0, n, nch * per).astype(np.int32)
    wt = rng.uniform(0, 1, nch * per).astype(np.float32)
    h = rng.standard_normal((n, d)).astype(np.float32)
    cs = (per * np.arange(nch + 1)).astype(np.int32)
    cp = np.concatenate([[0], np.cumsum(chunks)]).astype(np.int32)
    t = [torch.from_numpy(a).cuda() for a in (cs, cp, col, wt, h)]
    first = rng.standard_normal((rows, d)).astype(np.float32)
    out = torch.from_numpy(first.copy()).cuda()
    part = torch.zeros((nch, d), device="cuda")
    nat.check(nat.lib().fvdbm_mp_spmm_chunked(t[0].data_ptr(), t[1].data_ptr(), nch, t[2].data_ptr(), t[3].data_ptr(), rows,
                                              t[4].data_ptr(), d, out.data_ptr(), acc, part.data_ptr(),
                                              torch.cuda.current_stream().cuda_stream))
    p = part.cpu().numpy()
    ref = np.zeros((rows, d), np.float32)
    for k in range(max(chunks)):
        on = np.flatnonzero(np.diff(cp) > k)
        ref[on] = ref[on] + p[cp[on] + k]
    assert np.array_equal(out.cpu().numpy(), first + ref if acc else ref)

"""The warp search of the photon grid where its paths differ: lists up to and beyond 32 entries,
queries whose buckets hold many photons (nearest cells first, the rest only if they can matter),
photons at equal positions (equal distances, ordered by index) and buckets shared by several of a
query's cells (listed twice by the reference's grid, once by grids with narrower cells)."""
import numpy as np
import pytest

from oracle import oracle as O
from tests.test_hashgrid import photon_cloud, queries_near, run_gpu


@pytest.mark.gpu
@pytest.mark.parametrize("n,r,k,cf,table", [
    (30000, 0.9, 1, 2.0, 0),       # hundreds of photons in reach
    (30000, 0.9, 31, 1.0, 1 << 16),
    (30000, 0.9, 32, 1.0, 0),
    (30000, 0.9, 33, 2.0, 0),
    (30000, 0.7, 64, 1.0, 4099),
    (4000, 0.3, 10, 1.0, 13),      # range mode, every bucket shared
    (4000, 0.6, 40, 2.0, 5),       # reference mode, every bucket shared
    (33, 5.0, 64, 1.5, 0),         # fewer photons than list entries
])
def test_knn_paths_against_the_oracle(cuda, n, r, k, cf, table):
    pos = photon_cloud(n, 41)
    pos[n // 2:n // 2 + n // 8] = pos[: n // 8]          # photons at equal positions
    q = queries_near(pos, 3001, 42, 0.5 * r)
    g, ends, ids = O.hashgrid_build(pos, r, cf, table if table else None)
    want, wcnt, wd2 = O.hashgrid_query(g, ends, ids, pos, q, k)
    _, got, gcnt, gd2 = run_gpu(pos, q, r, k, cf, table)
    assert np.array_equal(wcnt, gcnt)
    assert np.array_equal(np.sort(wd2, 1), np.sort(gd2, 1))      # distances are the reference's bit for bit
    f = np.float32
    for i in range(len(q)):
        m = gcnt[i]
        have, d = got[i, :m], gd2[i, :m]
        p = pos[have]
        dx, dy, dz = (q[i, a] - p[:, a] for a in range(3))
        assert np.array_equal((f(1) * dx * dx + dy * dy) + dz * dz, d)      # each entry is its photon's distance
        order = np.lexsort((have, d))
        assert np.array_equal(order, np.arange(m)) or cf == 2.0 and np.array_equal(have[order], have)
        assert cf == 2.0 or len(set(have.tolist())) == m                    # once each, unless the reference's grid
        full = d[-1] if m == k else np.inf
        closer = d < full                                                   # below the k-th distance the set is fixed
        w = want[i, :m][wd2[i, :m] < full]
        assert np.array_equal(np.sort(have[closer]), np.sort(w))
        assert (got[i, m:] == -1).all() and (gd2[i, m:] == 0).all()

"""Photons without a position (NaN coordinates, of either sign): they lie in no radius and leave the
grid's box, and with it every answer about the others, as it is without them."""
import numpy as np
import pytest

from tests.test_hashgrid import photon_cloud, queries_near


@pytest.mark.gpu
@pytest.mark.parametrize("n,radius", [(4000, 0.4), (700001, 0.05)])      # one photon a thread, and several
@pytest.mark.parametrize("where", ["first", "middle", "last", "whole warps"])
@pytest.mark.parametrize("sign", [1.0, -1.0])
def test_nan_photons_are_nowhere(cuda, n, radius, where, sign):
    import torch
    from imbatracer_b200.hashgrid import HashGrid
    pos = photon_cloud(n, 31)
    q = queries_near(pos, 2000, 32, radius / 2)
    at = {"first": slice(0, 1), "middle": slice(1999, 2002), "last": slice(n - 1, n),
          "whole warps": slice(n - n // 4, n)}[where]
    nan = np.copysign(np.float32(np.nan), np.float32(sign))
    pos[5:7] = [[-40.0, -50.0, -60.0], [40.0, 50.0, 60.0]]     # the box's corners, before a thread's NaN
    bad = pos.copy()
    bad[at] = nan
    keep = np.ones(n, bool)        # the answers wanted: the grid of the other photons
    keep[at] = False
    d_q = torch.from_numpy(q).cuda()

    def answers(photons):
        g = HashGrid(0)
        g.build(torch.from_numpy(photons).cuda(), radius, 2.0, 2 * n + 9)
        ids, cnt, d2 = (t.cpu().numpy() for t in g.query(d_q, 32, with_d2=True))
        p = g.params()
        g.close()
        return ids, cnt, d2, np.concatenate([p["lo"], p["hi"]])

    ids, cnt, d2, box = answers(bad)
    index = np.nonzero(keep)[0]
    wids, wcnt, wd2, wbox = answers(np.ascontiguousarray(pos[keep]))
    assert (wcnt > 0).sum() > 1000
    assert np.array_equal(box, wbox)
    assert np.array_equal(cnt, wcnt) and np.array_equal(d2, wd2)
    assert np.array_equal(ids, np.where(wids >= 0, index[wids], -1))

"""The lat/lon search where its FP32 tests leave the decision to FP64: distances
and levels a little inside and outside the cut-offs, cut-offs at the antipode, a
vertical cut-off that excludes nothing, levels that have no FP32 logarithm.  Lists
equal to the oracle's entry for entry, so that the counting pass (FP32 where that
is certain) and the writing pass agree; a decision 1e-9 of the cut-off away from it
is far from FP64's rounding.  Weights exp(-y / 2) within 1e-13 and eight roundings of
y times the weight (y reaches 1,200 here)."""
import numpy as np
import pytest

from letkf_gb300 import synthetic as S
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _t(a, dt, dev):
    import torch

    return torch.as_tensor(np.ascontiguousarray(a), dtype=dt, device=dev)


@pytest.mark.parametrize("dist_zero,zerov_scale", [(1.8e6, 1.0), (1.8e6, 1.0e3), (2.0e7, 1.0), (2.1e7, 1.0),
                                                   (1.0e5, 1.0), (-1.8e6, 1.0)])
def test_speedy_search_bands(cuda, dist_zero, zerov_scale):
    import torch

    from letkf_gb300.core import search_speedy

    c = S.speedy_case(3, nstations=200)
    rng = np.random.default_rng(3)
    dist_zerov = c["dist_zerov"] * zerov_scale
    hp = np.arange(5, c["glon"].size, 61)
    lev = 4
    olon, olat, olev = c["olon"].copy(), c["olat"].copy(), c["olev"].copy()
    n = olon.size
    order = rng.permutation(n)
    deltas = [1e-3, -1e-3, 1e-5, -1e-5, 1e-7, -1e-7, 1e-9, -1e-9]
    at = 0
    for i, d in enumerate(deltas):  # at the cut-off's distance from a point, north of it
        for h in hp[i::8][:6]:
            lat = c["glat"][h] + abs(dist_zero) * (1.0 + d) / 6371.3e3 / 3.1415926535 * 180.0
            if lat < 89.0:
                olon[order[at]], olat[order[at]] = c["glon"][h], lat
                olev[order[at]] = np.exp(c["logpfm"][lev - 1, h])
            at += 1
    for i, d in enumerate(deltas):  # at the vertical cut-off beside a point
        for h in hp[i::8][:6]:
            o = order[at]
            olon[o], olat[o] = c["glon"][h], c["glat"][h]
            olev[o] = np.exp(min(600.0, c["logpfm"][lev - 1, h] + (-1.0) ** at * dist_zerov * (1.0 + d)))
            at += 1
    for v in (0.0, -5.0, 1.0e-310, 1.0e-35, 1.0e35, 1.0e300, np.nan, np.inf):
        for h in hp[:4]:
            o = order[at]
            olon[o], olat[o], olev[o] = c["glon"][h], c["glat"][h], v
            at += 1
    perm, grd = O.speedy_sort_obs(c["lon"], c["lat"], olon, olat)
    elm, odat, oerr = c["elm"][perm], c["odat"][perm], c["oerr"][perm]
    olon, olat, olev = olon[perm], olat[perm], olev[perm]
    dlat_zero = abs(dist_zero) / 3.1415926535 / 6371.3e3 * 180.0
    dlon_zero = dlat_zero / np.cos(3.1415926535 * c["glat"] / 180.0)
    so = O.SpeedyObs(c["lon"], c["lat"], grd, elm, olon, olat, olev, odat, oerr, dist_zero, dist_zerov, dlat_zero,
                     c["sigma_obs"], c["sigma_obsv"], c["var_local"])
    f = lambda a: _t(a, torch.float64, cuda)
    grid = {"lon": f(c["lon"]), "lat": f(c["lat"]), "nobsgrd": _t(grd, torch.int32, cuda)}
    obs = dict(elm=f(elm), lon=f(olon), lat=f(olat), lev=f(olev), dat=f(odat), err=f(oerr))
    logp = c["logpfm"][lev - 1, hp]
    pts = {"lon": f(c["glon"][hp]), "lat": f(c["glat"][hp]), "dlon_zero": f(dlon_zero[hp]),
           "ilev": _t(np.full(hp.size, lev, np.int32), torch.int32, cuda), "logpfm": f(logp)}
    offs, idx, rloc, rdiag = (x.cpu().numpy() for x in search_speedy(
        grid, obs, pts, (dist_zero, dist_zerov, dlat_zero, c["sigma_obs"], c["sigma_obsv"]), c["var_local"]))
    for p, h in enumerate(hp):
        ri, rl, rd = so.obs_local(c["glon"][h], c["glat"][h], dlon_zero[h], lev, logp[p])
        s = slice(offs[p], offs[p + 1])
        np.testing.assert_array_equal(idx[s], ri, err_msg=f"point {p}")
        with np.errstate(all="ignore"):
            bar = (1.0e-13 + 2.0 ** -49 * np.abs(np.log(rl))) * rl + 1.0e-300
        ok = (np.abs(rloc[s] - rl) <= bar) | (np.isnan(rl) & np.isnan(rloc[s])) | (rloc[s] == rl)
        assert ok.all(), f"point {p}"
        np.testing.assert_array_equal(rdiag[s], rd)

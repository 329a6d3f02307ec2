"""The FP64 updates, the obs-space analysis and EFSO at the sizes where their
tiles and chunks end: odd and even ensembles around the lane counts and the
64-wide tile, more variables than one chunk holds, the clipped variable in any
chunk, every number of EFSO terms, lists that leave a warp partly empty.

Reference: the formulas of scale/letkf/letkf_tools.f90:215-268 and
gfs/letkf/letkf_tools.f90:466-497,547-679 in numpy.  Tolerance 1e-12 of the
largest value: sums of at most 130 products of O(1) terms in another order."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

RTOL = 1e-12


def _t(a, dev, dt=None):
    import torch

    return torch.as_tensor(np.ascontiguousarray(a), dtype=dt or torch.float64, device=dev)


def _close(a, b):
    assert np.abs(a - b).max() <= RTOL * np.abs(b).max()


@pytest.mark.parametrize("ne,nv,mode,q_var", [(2, 1, 2, 0), (3, 5, 1, 4), (7, 17, 2, 16), (8, 16, 2, 0), (15, 33, 0, 20),
                                              (31, 4, 2, 3), (32, 3, 1, 1), (33, 11, 2, 2), (50, 18, 2, 17),
                                              (64, 6, 2, 0), (65, 2, 1, 1), (101, 11, 2, 5), (128, 1, 0, 0)])
def test_relaxed_update_edges(cuda, ne, nv, mode, q_var):
    from letkf_gb300.core import update_relax_f64

    rng = np.random.default_rng(100 * ne + nv)
    npts, alpha, q_max = 23, 0.7, 0.05
    w = rng.standard_normal((npts, ne, ne)) / ne + np.eye(ne)      # [p][m][k]
    pa = rng.standard_normal((npts, ne, ne)) * 0.1 / ne + np.eye(ne) / ne  # not symmetric: every element counts
    tm = rng.standard_normal((npts, ne)) * 0.1
    xb = rng.standard_normal((nv, npts, ne)) + 3.0
    beta = rng.uniform(0, 1, (nv, npts))
    beta[:, ::5] = 1.0
    beta[:, 1::7] = 0.0
    xa, infl = update_relax_f64(_t(xb, cuda), _t(w, cuda), _t(tm, cuda), _t(pa, cuda), mode=mode, alpha=alpha,
                                beta=_t(beta, cuda), q_var=q_var, q_sprd_max=q_max)
    mean = xb.mean(-1, keepdims=True)
    x = xb - mean
    fac = np.ones((nv, npts))
    inc = np.einsum("vpk,pmk->vpm", x, w)
    if mode == 1:
        inc = (1 - alpha) * inc + alpha * x
    if mode == 2:
        va = np.einsum("vpk,pmk,vpm->vp", x, pa, x)
        vg = (x * x).sum(-1)
        ok = (beta != 0) & (va > 0) & (vg > 0)
        fac[ok] = alpha * np.sqrt(vg[ok] / (va[ok] * (ne - 1))) - alpha + 1
        inc = inc * fac[..., None]
    inc = inc + np.einsum("vpk,pk->vp", x, tm)[..., None]
    want = mean + beta[..., None] * inc + (1 - beta)[..., None] * x
    q = want[q_var]
    qm = q.mean(-1, keepdims=True)
    sp = np.sqrt(((q - qm) ** 2).sum(-1, keepdims=True) / (ne - 1)) / qm
    want[q_var] = np.where(sp > q_max, qm + (q - qm) * q_max / sp, q)
    _close(xa.cpu().numpy(), want)
    if mode == 2:
        _close(infl.cpu().numpy(), fac)


@pytest.mark.parametrize("ne,nv,merged", [(2, 40, False), (31, 1, True), (33, 16, False), (64, 17, True), (127, 3, False),
                                          (7, 4, True), (32, 4, False), (40, 2, True), (55, 2, False), (56, 6, True),
                                          (64, 5, False), (128, 1, True), (101, 6, False)])
@pytest.mark.parametrize("npts", [1, 19, 20_000])
def test_update_f64_edges(cuda, ne, nv, merged, npts):
    from letkf_gb300.core import update_f64

    rng = np.random.default_rng(ne)
    npts = min(npts, 3_000_000 // (ne * ne))
    w = rng.standard_normal((npts, ne, ne)) / ne
    tm = rng.standard_normal((npts, ne)) * 0.1
    xb = rng.standard_normal((nv, npts, ne)) + 3.0
    xa = update_f64(_t(xb, cuda), _t(w, cuda), None if merged else _t(tm, cuda)).cpu().numpy()
    mean = xb.mean(-1, keepdims=True)
    x = xb - mean
    want = mean + np.einsum("vpk,pmk->vpm", x, w)
    if not merged:
        want = want + np.einsum("vpk,pk->vp", x, tm)[..., None]
    _close(xa, want)


@pytest.mark.parametrize("ne", [2, 31, 63, 64, 65, 96, 128, 129, 200])
def test_obs_analysis_edges(cuda, ne):
    import torch

    from letkf_gb300.core import obs_analysis

    rng = np.random.default_rng(ne)
    n, alpha, q_max = 41, 0.25, 0.1
    tr = rng.standard_normal((n, ne, ne)) / ne + np.eye(ne)
    h = rng.standard_normal((n, ne))
    y = rng.uniform(3.0, 6.0, n)
    mode = (np.arange(n) % 3).astype(np.int32)
    anal, mean = obs_analysis(_t(tr, cuda), _t(y, cuda), _t(h, cuda), alpha, _t(mode, cuda, torch.int32), q_max)
    a = y[:, None] + (1 - alpha) * np.einsum("pk,pmk->pm", h, tr) + alpha * h
    a[mode == 1] = (y[:, None] + h)[mode == 1]
    m = np.where(mode == 1, y, a.mean(1))
    sp = np.sqrt(((a - m[:, None]) ** 2).sum(1) / (ne - 1)) / m
    cut = (mode == 2) & (sp > q_max)
    a[cut] = (m[:, None] + (a - m[:, None]) * (q_max / sp)[:, None])[cut]
    _close(anal.cpu().numpy(), a)
    _close(mean.cpu().numpy(), m)


@pytest.mark.parametrize("ne,npts,nterm", [(2, 1, 1), (15, 7, 2), (16, 9, 3), (17, 2500, 4), (33, 40, 5), (64, 1300, 6),
                                           (96, 12, 7), (130, 20, 8)])
def test_efso_edges(cuda, ne, npts, nterm):
    import torch

    from letkf_gb300.core import efso

    rng = np.random.default_rng(ne + npts)
    nobs, nv = 300, nterm + 2
    cnt = rng.integers(0, 45, npts)
    cnt[0] = 33
    offs = np.concatenate([[0], np.cumsum(cnt)]).astype(np.int64)
    idx = rng.integers(0, nobs, int(offs[-1])).astype(np.int32)
    rd, rl = rng.uniform(0.5, 2.0, idx.size), rng.uniform(0.0, 1.0, idx.size)
    hdxa, dep = rng.standard_normal((nobs, ne)), rng.standard_normal(nobs)
    fcst, fcer = rng.standard_normal((nv, npts, ne)), rng.standard_normal((nv, npts))
    term = list(range(nterm)) + [0, -1]
    dj, sense = efso(ne, _t(offs, cuda, torch.int64), _t(idx, cuda, torch.int32), _t(rd, cuda), _t(rl, cuda),
                     _t(hdxa, cuda), _t(fcst, cuda), _t(fcer, cuda), term, _t(dep, cuda))
    want = np.zeros((nobs, nterm))
    point = np.repeat(np.arange(npts), cnt)
    for t in range(nterm):
        w1 = sum(fcst[v] * fcer[v][:, None] for v in range(nv) if term[v] == t)
        np.add.at(want[:, t], idx, (hdxa[idx] * w1[point]).sum(1) * rl / rd)
    _close(dj.cpu().numpy(), want)
    _close(sense.cpu().numpy(), want * dep[:, None])


@pytest.mark.parametrize("ne,nv", [(7, 2), (31, 9), (32, 3), (40, 1), (40, 8), (50, 11), (64, 6), (101, 18), (128, 2)])
@pytest.mark.parametrize("merged", [True, False])
def test_beta_of_one_is_the_plain_update_bit_for_bit(cuda, ne, nv, merged):
    import torch

    from letkf_gb300.core import update_f64, update_relax_f64

    rng = np.random.default_rng(ne + nv)
    npts = 37
    w = _t(rng.standard_normal((npts, ne, ne)) / ne, cuda)
    tm = None if merged else _t(rng.standard_normal((npts, ne)) * 0.1, cuda)
    xb = _t(rng.standard_normal((nv, npts, ne)) + 3.0, cuda)
    beta = np.ones((nv, npts))
    want = update_f64(xb, w, tm)
    assert torch.equal(update_relax_f64(xb, w, tm)[0], want)
    assert torch.equal(update_relax_f64(xb, w, tm, beta=_t(beta, cuda))[0], want)
    beta[rng.uniform(size=beta.shape) < 0.4] = 0.5  # interior points beside a boundary's ramp
    one = _t(beta == 1.0, cuda, torch.bool)
    assert torch.equal(update_relax_f64(xb, w, tm, beta=_t(beta, cuda))[0][one], want[one])


@pytest.mark.parametrize("ne,nv", [(127, 16), (127, 17), (128, 1), (128, 15), (128, 16), (128, 17), (128, 33)])
def test_rtps_of_the_largest_ensembles(cuda, ne, nv):
    """W and Pa of k = 128 leave room for fewer variables than a chunk holds."""
    test_relaxed_update_edges(cuda, ne, nv, 2, nv - 1)


@pytest.mark.parametrize("ne", [2, 7, 8, 15, 16, 21, 22, 24, 25, 33, 40, 46, 54, 55, 72, 79, 80, 83, 88, 96, 100, 104, 127])
@pytest.mark.parametrize("nv", [2, 3, 4, 5, 7, 16, 17])
def test_merged_weights_on_either_side_of_each_rule(cuda, ne, nv):
    """The forms of the plain update with merged weights, and the general
    kernel that the relaxed entry point takes, give the same bits."""
    import torch

    from letkf_gb300.core import update_f64, update_relax_f64

    rng = np.random.default_rng(10 * ne + nv)
    npts = 29
    w, xb = rng.standard_normal((npts, ne, ne)) / ne, rng.standard_normal((nv, npts, ne)) + 3.0
    dw, dx = _t(w, cuda), _t(xb, cuda)
    xa = update_f64(dx, dw)
    assert torch.equal(xa, update_relax_f64(dx, dw)[0])
    mean = xb.mean(-1, keepdims=True)
    _close(xa.cpu().numpy(), mean + np.einsum("vpk,pmk->vpm", xb - mean, w))


@pytest.mark.parametrize("ne,nv,npts,merged", [(8, 1, 160_001, True), (8, 1, 160_007, False), (5, 2, 170_003, True),
                                               (8, 3, 200_003, False), (7, 4, 90_002, False), (31, 1, 30_001, True),
                                               (32, 1, 30_001, False), (32, 4, 40_003, False),
                                               (58, 6, 19_501, False)])
def test_update_f64_batches_of_points(cuda, ne, nv, npts, merged):
    """A warp's batch of several points, up to 16 rows, the last batch short."""
    import torch

    from letkf_gb300.core import update_f64

    g = torch.Generator(device=cuda).manual_seed(ne + nv)
    r = lambda *s: torch.randn(*s, dtype=torch.float64, device=cuda, generator=g)
    w, tm, xb = r(npts, ne, ne) / ne, r(npts, ne) * 0.1, r(nv, npts, ne) + 3.0
    xa = update_f64(xb, w, None if merged else tm)
    for p in range(0, npts, 10_000):
        q = slice(p, p + 10_000)
        x = xb[:, q].cpu().numpy()
        mean = x.mean(-1, keepdims=True)
        x = x - mean
        want = mean + np.matmul(x.transpose(1, 0, 2), w[q].cpu().numpy().transpose(0, 2, 1)).transpose(1, 0, 2)
        if not merged:
            want = want + np.einsum("vpk,pk->vp", x, tm[q].cpu().numpy())[..., None]
        _close(xa[:, q].cpu().numpy(), want)


@pytest.mark.parametrize("ne", [3, 16, 40])
def test_efso_rounds_an_entry_twice(cuda, ne):
    """Small integers, so that the sums over the members are exact: an entry's
    rloc / rdiag and its product with the sum are the only roundings."""
    import torch

    from letkf_gb300.core import efso

    rng = np.random.default_rng(ne)
    npts, nobs = 40, 4000
    offs = np.linspace(0, nobs, npts + 1).astype(np.int64)
    idx = rng.permutation(nobs).astype(np.int32)
    rd, rl = rng.uniform(0.1, 9.0, nobs), rng.uniform(0.0, 1.0, nobs)
    i = lambda *s: rng.integers(-9, 10, s).astype(np.float64)
    hdxa, fcst, fcer, dep = i(nobs, ne), i(2, npts, ne), i(2, npts), i(nobs)
    dj, _ = efso(ne, _t(offs, cuda, torch.int64), _t(idx, cuda, torch.int32), _t(rd, cuda), _t(rl, cuda),
                 _t(hdxa, cuda), _t(fcst, cuda), _t(fcer, cuda), [0, 0], _t(dep, cuda))
    w1 = (fcst * fcer[..., None]).sum(0)
    point = np.repeat(np.arange(npts), np.diff(offs))
    want = np.empty(nobs)
    want[idx] = (hdxa[idx] * w1[point]).sum(1) * (rl / rd)
    assert np.array_equal(dj.cpu().numpy()[:, 0], want)


@pytest.mark.parametrize("ne", [2, 3, 7, 10, 21, 24, 25, 32, 33, 54, 55, 63, 64, 65, 71, 72, 79, 80, 88, 100])
@pytest.mark.parametrize("nv", [2, 3, 4, 5, 6, 7, 17, 40])
def test_mean_weights_on_either_side_of_each_rule(cuda, ne, nv):
    """The same with mean weights."""
    import torch

    from letkf_gb300.core import update_f64, update_relax_f64

    rng = np.random.default_rng(10 * ne + nv)
    npts = 29
    w, tm = rng.standard_normal((npts, ne, ne)) / ne, rng.standard_normal((npts, ne)) * 0.1
    xb = rng.standard_normal((nv, npts, ne)) + 3.0
    dw, dt, dx = _t(w, cuda), _t(tm, cuda), _t(xb, cuda)
    xa = update_f64(dx, dw, dt)
    assert torch.equal(xa, update_relax_f64(dx, dw, dt)[0])
    mean = xb.mean(-1, keepdims=True)
    x = xb - mean
    _close(xa.cpu().numpy(), mean + np.einsum("vpk,pmk->vpm", x, w) + np.einsum("vpk,pk->vp", x, tm)[..., None])


@pytest.mark.parametrize("ne", [3, 8, 16, 17, 30, 32, 33])
def test_obs_analysis_of_few_members(cuda, ne):
    test_obs_analysis_edges(cuda, ne)


@pytest.mark.parametrize("ne", [33, 34, 40, 47, 64, 65, 66, 96, 97, 101, 127, 128])
def test_obs_analysis_by_warps(cuda, ne):
    """A warp per location, up to four members a lane, rows aligned or not; the
    tile's sums in the same order, so few locations and many give the same bits."""
    import torch

    from letkf_gb300.core import obs_analysis

    test_obs_analysis_edges(cuda, ne)
    g = torch.Generator(device=cuda).manual_seed(ne)
    r = lambda *s: torch.randn(*s, dtype=torch.float64, device=cuda, generator=g)
    n = 1100
    tr, h, y = r(n, ne, ne) / ne, r(n, ne), r(n) + 4.0
    mode = (torch.arange(n, device=cuda) % 3).to(torch.int32)
    anal, mean = obs_analysis(tr, y, h, 0.25, mode, 0.1)
    for p in (0, 1, 1000):
        q = slice(p, p + 100)
        a, m = obs_analysis(tr[q].contiguous(), y[q].contiguous(), h[q].contiguous(), 0.25, mode[q].contiguous(), 0.1)
        assert torch.equal(a, anal[q]) and torch.equal(m, mean[q])


@pytest.mark.parametrize("ne,npts,nterm", [(3, 2500, 3), (8, 40, 1), (8, 1300, 8), (9, 40, 8), (900, 5, 8), (1024, 7, 8),
                                           (1024, 4, 7)])
def test_efso_of_few_and_of_many_members(cuda, ne, npts, nterm):
    """No tile up to eight members, half a tile where memory is short."""
    test_efso_edges(cuda, ne, npts, nterm)


@pytest.mark.parametrize("ne,nv", [(2, 1), (2, 41), (3, 6), (4, 11), (5, 1), (5, 17), (6, 3), (7, 16), (8, 10), (8, 11),
                                   (9, 10)])
@pytest.mark.parametrize("mode", [0, 1, 2])
def test_small_ensembles_by_threads(cuda, ne, nv, mode):
    """A thread per point and variable up to eight members, either side of its rules."""
    test_relaxed_update_edges(cuda, ne, nv, mode, nv - 1)
    for merged in (True, False):
        test_update_f64_edges(cuda, ne, nv, merged, 301)
        test_beta_of_one_is_the_plain_update_bit_for_bit(cuda, ne, nv, merged)


@pytest.mark.parametrize("ne,nv", [(9, 1), (20, 2), (24, 3), (32, 4), (54, 1), (63, 2), (64, 4), (82, 5), (101, 1),
                                   (101, 6), (127, 3), (128, 1), (128, 3), (128, 6)])
@pytest.mark.parametrize("merged", [True, False])
def test_few_points_and_many_have_the_same_bits(cuda, ne, nv, merged):
    """Batches of rows from a number of points on, a CTA per point below it."""
    import torch

    from letkf_gb300.core import update_f64

    g = torch.Generator(device=cuda).manual_seed(ne + nv)
    r = lambda *s: torch.randn(*s, dtype=torch.float64, device=cuda, generator=g)
    npts = 701
    w, xb = r(npts, ne, ne) / ne, r(nv, npts, ne) + 3.0
    tm = None if merged else r(npts, ne) * 0.1
    xa = update_f64(xb, w, tm)
    for p in (0, 1, 131, 700):
        q = slice(p, min(p + 130, npts))
        part = update_f64(xb[:, q].contiguous(), w[q].contiguous(), None if merged else tm[q].contiguous())
        assert torch.equal(part, xa[:, q])
    x, m = xb[:, :50].cpu().numpy(), xb[:, :50].mean(-1, keepdim=True).cpu().numpy()
    want = m + np.einsum("vpk,pmk->vpm", x - m, w[:50].cpu().numpy())
    if not merged:
        want = want + np.einsum("vpk,pk->vp", x - m, tm[:50].cpu().numpy())[..., None]
    _close(xa[:, :50].cpu().numpy(), want)


@pytest.mark.parametrize("ne,nv", [(60, 17), (72, 32), (90, 20), (100, 20), (100, 33), (127, 17)])
def test_more_variables_than_a_pass(cuda, ne, nv):
    for merged in (True, False):
        test_update_f64_edges(cuda, ne, nv, merged, 19)

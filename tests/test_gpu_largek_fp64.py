"""The FP64 pass of the large-ensemble core where its tiles, digit chunks, list
pieces and groups end: ensembles around multiples of 64, lists around the 512
rows up to which the digit sums are exact, more points than one group holds,
points that the core certifies beside points that it does not, values that are
not finite.

Tolerance: the pass's bar, 1e-5 of the oracle's largest entry for the FP32
transform and 1e-8 for the FP64 inflation."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _run(cuda, ne, Ls, err, seed, wloc=False):
    import torch

    from letkf_gb300.core import core_batch_largek

    rng = np.random.default_rng(seed)
    offs = np.concatenate([[0], np.cumsum(Ls)]).astype(np.int64)
    n = int(offs[-1])
    # smooth rows: a few directions with very different weights
    basis = rng.standard_normal((24, ne)) * (0.6 ** np.arange(24))[:, None]
    rows = (rng.standard_normal((n, 24)) @ basis).astype(np.float32)
    rows -= rows.mean(1, keepdims=True)
    rd = (rng.uniform(0.5, 2.0, n) * np.repeat(err, Ls)).astype(np.float32)
    rl = rng.uniform(0.05, 1.0, n).astype(np.float32)
    d = rng.standard_normal(n).astype(np.float32)
    infl = rng.uniform(0.95, 1.2, len(Ls))
    f = lambda a: a.astype(np.float64)
    ref = O.letkf_core_batch(ne, offs, f(rows), f(rd), f(rl), f(d), infl, want_transm=True, rdiag_wloc=wloc)
    t = lambda a, dt=torch.float32: torch.as_tensor(np.ascontiguousarray(a), dtype=dt, device=cuda)
    pinf = t(infl, torch.float64)
    out = core_batch_largek(ne, t(offs, torch.int64), t(rows), t(rd), t(rl), t(d), pinf, want_transm=True,
                            rdiag_wloc=wloc)
    torch.cuda.synchronize()
    # lambda_max / c of each point
    kappa = np.zeros(len(Ls))
    w = 1.0 / f(rd) if wloc else f(rl) / f(rd)
    for p in range(len(Ls)):
        y = f(rows[offs[p]:offs[p + 1]])
        kappa[p] = 1.0 + np.linalg.norm(y * np.sqrt(w[offs[p]:offs[p + 1], None]), 2) ** 2 * infl[p] / (ne - 1)
    ref["kappa"] = kappa
    return ref, {k: v.cpu().numpy() for k, v in out.items()}, pinf.cpu().numpy()


def _check(ref, out, pinf, points):
    """Up to lambda_max / c = 3e6 every point is answered.  Past it a point may
    stay reported instead: the certificate asks for 1e-8 where FP64 rounding
    times the condition number is as large, and from 3e7 on mtx_eigen's
    truncation could act."""
    from letkf_gb300.lib import LETKF_ERR_CAPACITY

    for p in points:
        assert out["status"][p] == 0 or (ref["kappa"][p] > 3.0e6 and out["status"][p] == LETKF_ERR_CAPACITY), p
    points = [p for p in points if out["status"][p] == 0]
    for p in points:
        for k in ("trans", "transm"):
            scale = np.abs(ref[k][p]).max()
            assert np.abs(out[k][p] - ref[k][p]).max() <= 1e-5 * scale, (k, p)
    np.testing.assert_allclose(pinf[points], ref["parm_infl"][points], rtol=1e-8)


@pytest.mark.parametrize("ne", [129, 191, 192, 193, 256, 300])
def test_ill_conditioned_points_at_the_edges(cuda, ne):
    Ls = [1, 31, 33, 511, 512, 513, 1024, 1025, 2000]
    ref, out, pinf = _run(cuda, ne, Ls, np.full(len(Ls), 1e-5), ne, wloc=ne % 2 == 0)
    _check(ref, out, pinf, list(range(len(Ls))))


def test_more_points_than_a_group(cuda):
    Ls = list(np.random.default_rng(3).integers(40, 300, 41))
    ref, out, pinf = _run(cuda, 130, Ls, np.full(len(Ls), 1e-5), 3)
    _check(ref, out, pinf, list(range(len(Ls))))


def test_certified_points_beside_others(cuda):
    """The pass touches only the points that the core leaves."""
    Ls = [200, 200, 150, 150, 300, 80]
    err = np.array([1.0, 1e-5, 1.0, 1e-5, 1e-5, 1.0])
    ref, out, pinf = _run(cuda, 160, Ls, err, 5)
    assert (out["status"][[0, 2, 5]] == 0).all()
    _check(ref, out, pinf, [1, 3, 4])
    for p in (0, 2, 5):
        assert np.abs(out["trans"][p] - ref["trans"][p]).max() <= 1e-4 * np.abs(ref["trans"][p]).max()


@pytest.mark.parametrize("err", [1e-2, 1e-4])
def test_long_lists_split_over_ctas(cuda, err):
    """Few points with long lists: the first core's Gram and the pass's are
    both split along K."""
    Ls = [6000, 4500]
    ref, out, pinf = _run(cuda, 132, Ls, np.array([err, 1.0]), 8)
    assert (out["status"][0] == 0) == (err == 1e-2)
    _check(ref, out, pinf, [0])
    assert out["status"][1] == 0
    assert np.abs(out["trans"][1] - ref["trans"][1]).max() <= 1e-4 * np.abs(ref["trans"][1]).max()


def test_values_that_are_not_finite_stay_reported(cuda):
    import torch

    from letkf_gb300.core import core_batch_largek

    rng = np.random.default_rng(9)
    ne, Ls = 136, [60, 60, 60]
    offs = np.concatenate([[0], np.cumsum(Ls)]).astype(np.int64)
    rows = rng.standard_normal((180, ne)).astype(np.float32)
    rows[70, 5] = np.nan
    rows[130, 7] = np.inf
    t = lambda a, dt=torch.float32: torch.as_tensor(np.ascontiguousarray(a), dtype=dt, device=cuda)
    one = np.ones(180, dtype=np.float32)
    out = core_batch_largek(ne, t(offs, torch.int64), t(rows), t(one), t(one), t(one),
                            t(np.ones(3), torch.float64), want_transm=True)
    torch.cuda.synchronize()
    st = out["status"].cpu().numpy()
    assert st[0] == 0 and st[1] != 0 and st[2] != 0
    assert np.isfinite(out["trans"][0].cpu().numpy()).all()


@pytest.mark.parametrize("ne", [513, 576, 640, 1000, 1024])
@pytest.mark.parametrize("alone", [True, False])
def test_ensembles_of_more_than_one_piece(cuda, ne, alone):
    """k x k products whose K is more than the 512 that one exact sum holds:
    every tile, its mirror and its transpose are the sum of all pieces."""
    Ls, err = ([700], [3e-4]) if alone else ([513, 200, 1100, 31], [1e-3, 1.0, 1e-3, 2e-5])
    ref, out, pinf = _run(cuda, ne, Ls, np.array(err), ne)
    hard = [0] if alone else [0, 2, 3]
    assert (ref["kappa"][hard] > 1.0e5).all() and (ref["kappa"][hard] < 3.0e6).all()
    assert (out["status"] == 0).all()
    _check(ref, out, pinf, hard)
    if not alone:
        assert np.abs(out["trans"][1] - ref["trans"][1]).max() <= 1e-4 * np.abs(ref["trans"][1]).max()


def test_lists_of_several_digit_chunks_in_a_full_group(cuda):
    """A group of 32 points holds 1,536 list entries' digits at a time at this
    ensemble; lists around one and two chunks, one point in a second group."""
    import torch

    from letkf_gb300.core import core_batch_largek_indexed

    ne, nobs = 513, 3300
    rng = np.random.default_rng(17)
    Ls = [1535, 1536, 1537, 600, 3071, 3072, 3073, 3200] + [int(x) for x in rng.integers(600, 1700, 25)]
    offs = np.concatenate([[0], np.cumsum(Ls)]).astype(np.int64)
    n = int(offs[-1])
    basis = rng.standard_normal((24, ne)) * (0.6 ** np.arange(24))[:, None]
    rows = (rng.standard_normal((nobs, 24)) @ basis).astype(np.float32)
    rows -= rows.mean(1, keepdims=True)
    idx = np.concatenate([np.sort(rng.choice(nobs, L, replace=False)) for L in Ls]).astype(np.int32)
    rd = (rng.uniform(0.5, 2.0, n) * 1e-3).astype(np.float32)
    rl = rng.uniform(0.05, 1.0, n).astype(np.float32)
    d = rng.standard_normal(nobs).astype(np.float32)
    infl = rng.uniform(0.95, 1.2, len(Ls))
    f = lambda a: a.astype(np.float64)
    ref = O.letkf_core_batch(ne, offs, f(rows)[idx], f(rd), f(rl), f(d)[idx], infl, want_transm=True)
    ref["kappa"] = np.zeros(len(Ls))
    t = lambda a, dt=torch.float32: torch.as_tensor(np.ascontiguousarray(a), dtype=dt, device=cuda)
    pinf = t(infl, torch.float64)
    out = core_batch_largek_indexed(ne, t(offs, torch.int64), t(idx, torch.int32), t(rows), t(d), t(rd), t(rl), pinf,
                                    want_transm=True)
    torch.cuda.synchronize()
    _check(ref, {k: v.cpu().numpy() for k, v in out.items()}, pinf.cpu().numpy(), list(range(len(Ls))))

"""The FP64 core without an eigendecomposition (k <= 64) at the sizes where it
can go wrong: every padded width's edges, lists around its staged chunk, points
that it hands to the eigensolver beside points that it keeps.

Tolerance: the FP64 plain form's 1e-10 of the largest entry.  The iteration
stops after a correction of a residual below 5e-10, which it reduces by five
orders, and FP64 rounding is amplified by lambda_max / c <= 1e5 at most."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

RTOL = 1e-10


def _run(cuda, ne, Ls, scale, infl, wloc, pao, seed):
    import torch

    from letkf_gb300.core import core_batch_f64

    rng = np.random.default_rng(seed)
    offs = np.concatenate([[0], np.cumsum(Ls)]).astype(np.int64)
    n = max(int(offs[-1]), 1)
    rows = rng.standard_normal((n, ne))
    rows -= rows.mean(1, keepdims=True)
    for p, s in enumerate(scale):
        rows[offs[p]:offs[p + 1]] *= s
    rd, rl, d = rng.uniform(0.3, 3.0, n), rng.uniform(0.01, 1.0, n), rng.standard_normal(n)
    ref = O.letkf_core_batch(ne, offs, rows, rd, rl, d, infl, want_transm=True, want_pao=True, rdiag_wloc=wloc)
    t = lambda a, dt=torch.float64: torch.as_tensor(np.ascontiguousarray(a), dtype=dt, device=cuda)
    pinf = t(infl)
    out = core_batch_f64(ne, t(offs, torch.int64), t(rows), t(rd), t(rl), t(d), pinf, want_transm=True,
                         want_pao=pao, rdiag_wloc=wloc)
    torch.cuda.synchronize()
    return ref, {k: None if v is None else v.cpu().numpy() for k, v in out.items()}, pinf.cpu().numpy()


def _check(ref, out, pinf, points):
    for p in points:
        for k in ("trans", "transm", "pao"):
            if out[k] is not None:
                tol = RTOL * max(np.abs(ref[k][p]).max(), 1e-300)
                assert np.abs(out[k][p] - ref[k][p]).max() <= tol, (k, p)
        assert abs(pinf[p] - ref["parm_infl"][p]) <= 1e-12 * abs(ref["parm_infl"][p])


@pytest.mark.parametrize("ne", [2, 3, 8, 15, 16, 17, 24, 31, 32, 33, 40, 47, 48, 49, 63, 64, 65])
def test_widths_and_chunk_edges(cuda, ne):
    Ls = [1, 7, 8, 9, 15, 16, 17, 0, 31, 32, 33, 200]
    ref, out, pinf = _run(cuda, ne, Ls, np.ones(len(Ls)), np.linspace(0.95, 1.3, len(Ls)), ne % 2 == 0, ne % 3 != 0,
                          ne)
    assert (out["status"] == 0).all()
    _check(ref, out, pinf, range(len(Ls)))


@pytest.mark.parametrize("ne", [12, 40, 64])
def test_more_points_than_ctas(cuda, ne):
    """Points taken from the counter: lists of very different lengths."""
    rng = np.random.default_rng(ne)
    Ls = list((rng.uniform(size=2500) ** 6 * 300).astype(int))
    ref, out, pinf = _run(cuda, ne, Ls, np.ones(len(Ls)), np.full(len(Ls), 1.05), True, False, 5)
    assert (out["status"] == 0).all()
    _check(ref, out, pinf, range(0, len(Ls), 7))


@pytest.mark.parametrize("ne", [16, 40, 64])
def test_points_left_to_the_eigensolver(cuda, ne):
    """Spectra past the iteration's range, and a negative inflation, beside
    ordinary points: c / lambda_max down to where mtx_eigen truncates."""
    Ls = [40, 200, 40, 200, 40, 33, 40]
    scale = [1.0, 1.0e2, 1.0e3, 1.0e5, 1.0e-6, 1.0, 1.0]
    infl = np.array([1.1, 1.0, 1.0, 1.0, 1.0, -1.0, 1.2])
    ref, out, pinf = _run(cuda, ne, Ls, scale, infl, False, True, 11)
    assert list(out["status"]) == list(ref["status"])
    _check(ref, out, pinf, [0, 1, 4, 6])
    # past the range the result is the eigensolver's own, entry for entry to its conditioning
    for p in (2, 3):
        assert np.isfinite(out["trans"][p]).all()
        assert np.abs(out["trans"][p] - ref["trans"][p]).max() <= 1e-6 * np.abs(ref["trans"][p]).max()

"""The batched mixed core at the sizes where its padded widths, thread tiles and
staged chunks end, beside points that it leaves to the eigensolver, and over
more points than its grid holds.

Tolerance: the mixed form's bar, 1e-4 of the background spread, on the analysis
of unit-spread members (FP32 sums of at most 300 terms over spectra of
lambda_max / c below 1e3 leave two orders of margin)."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _check(cuda, ne, Ls, infl, wloc, sep, points):
    import torch

    from letkf_gb300.core import core_batch_mixed

    rng = np.random.default_rng(7 * ne + len(Ls))
    offs = np.concatenate([[0], np.cumsum(Ls)]).astype(np.int64)
    n = max(int(offs[-1]), 1)
    rows = rng.standard_normal((n, ne)).astype(np.float32)
    rows -= rows.mean(1, keepdims=True)
    rd, rl = rng.uniform(0.5, 3.0, n).astype(np.float32), rng.uniform(0.01, 1.0, n).astype(np.float32)
    d = rng.standard_normal(n).astype(np.float32)
    f = lambda a: a.astype(np.float64)
    ref = O.letkf_core_batch(ne, offs, f(rows), f(rd), f(rl), f(d), infl, want_transm=sep, rdiag_wloc=wloc)
    t = lambda a, dt: torch.as_tensor(np.ascontiguousarray(a), dtype=dt, device=cuda)
    pinf = t(infl, torch.float64)
    out = core_batch_mixed(ne, t(offs, torch.int64), t(rows, torch.float32), t(rd, torch.float32),
                           t(rl, torch.float32), t(d, torch.float32), pinf, want_transm=sep, rdiag_wloc=wloc)
    torch.cuda.synchronize()
    assert list(out["status"].cpu().numpy()) == list(ref["status"])
    W = out["trans"].cpu().numpy().astype(np.float64)
    wb = out["transm"].cpu().numpy().astype(np.float64) if sep else None
    for p in points:
        if ref["status"][p]:
            continue
        x = rng.standard_normal((4, ne))
        x -= x.mean(1, keepdims=True)
        spread = np.sqrt((x ** 2).sum(1) / (ne - 1)).mean()
        assert np.sqrt(np.mean((x @ W[p].T - x @ ref["trans"][p].T) ** 2)) < 1e-4 * spread, p
        if sep:
            assert np.abs(x @ wb[p] - x @ ref["transm"][p]).max() < 1e-4 * spread, p
    np.testing.assert_allclose(pinf.cpu().numpy(), ref["parm_infl"], rtol=1e-4)


@pytest.mark.parametrize("ne", [2, 3, 15, 16, 17, 31, 32, 33, 47, 48, 49, 63, 64, 65, 95, 96, 97, 127, 128])
def test_widths_and_chunk_edges(cuda, ne):
    Ls = [1, 15, 16, 17, 0, 31, 32, 33, 48, 64, 65, 300]
    _check(cuda, ne, Ls, np.linspace(0.95, 1.3, len(Ls)), ne % 2 == 0, ne % 3 != 0, range(len(Ls)))


@pytest.mark.parametrize("ne", [12, 32, 40, 64])
def test_more_points_than_ctas(cuda, ne):
    rng = np.random.default_rng(ne)
    Ls = list((rng.uniform(size=4000) ** 6 * 200).astype(int))
    _check(cuda, ne, Ls, np.full(len(Ls), 1.05), True, True, range(0, len(Ls), 13))


@pytest.mark.parametrize("ne", [16, 50, 100])
def test_negative_inflation_beside_ordinary_points(cuda, ne):
    """c <= 0: the point goes to the eigensolver, which reports it or truncates
    as the reference does; its neighbours are not touched."""
    Ls = [20, 20, 20, 0, 20]
    _check(cuda, ne, Ls, np.array([1.1, -1.0, 1.0, 1.2, 0.9]), False, True, [0, 2, 3, 4])

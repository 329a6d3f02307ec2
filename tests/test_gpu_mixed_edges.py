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


@pytest.mark.parametrize("ne", [2, 4, 5, 6, 16, 17, 31, 32, 33, 47, 48, 49, 64, 65, 96, 97, 127, 128])
@pytest.mark.parametrize("sep", [True, False])
def test_points_the_iteration_is_not_tried_for(cuda, ne, sep):
    """tr(Gram) of 1e6 c and more: the eigensolver takes the point with the sums
    that the first launch leaves in its place (from five members on).  A row
    touches a pair of members, pairs by a permutation, so that the Gram matrix
    is 2 x 2 blocks of condition below 12 anywhere in the matrix, and an element
    in the wrong place changes the result by its own size.  Tolerance 1e-4 of
    the largest element: FP32 sums of at most 300 terms, the rounding of n terms
    about sqrt(n) 6e-8, times 12: 1.2e-5."""
    import torch

    from letkf_gb300.core import core_batch_mixed

    rng = np.random.default_rng(ne)
    Ls = [300, 40, 0, 200, 290]
    offs = np.concatenate([[0], np.cumsum(Ls)]).astype(np.int64)
    hard = [0, 3, 4]
    scale = np.repeat([2e-6, 1.0, 1.0, 2e-6, 2e-6], Ls)
    n = int(offs[-1])
    rows = np.zeros((n, ne), np.float32)
    for p, L in enumerate(Ls):
        order, half = rng.permutation(ne), (ne + 1) // 2
        for l in range(L):
            i, j = 2 * (l % half), 2 * (l % half) + 1
            big, small = rng.choice([-1.0, 1.0]) * rng.uniform(2.0, 2.5), rng.uniform(-1.0, 1.0)
            u, v = (big, small) if (l // half) % 2 else (small, big)
            rows[offs[p] + l, order[i]] = u if j < ne else big
            if j < ne:
                rows[offs[p] + l, order[j]] = v
    rd, rl = (rng.uniform(0.8, 1.2, n) * scale).astype(np.float32), rng.uniform(0.8, 1.0, n).astype(np.float32)
    d = rng.standard_normal(n).astype(np.float32)
    infl = np.linspace(0.95, 1.3, len(Ls))
    f = lambda a: a.astype(np.float64)
    for p in hard:
        q = slice(offs[p], offs[p + 1])
        assert (f(rl[q]) / f(rd[q]) * (f(rows[q]) ** 2).sum(1)).sum() > 2.0e6 * (ne - 1) / infl[p]
    ref = O.letkf_core_batch(ne, offs, f(rows), f(rd), f(rl), f(d), infl, want_transm=sep)
    t = lambda a, dt=torch.float32: torch.as_tensor(np.ascontiguousarray(a), dtype=dt, device=cuda)
    pinf = t(infl, torch.float64)
    out = core_batch_mixed(ne, t(offs, torch.int64), t(rows), t(rd), t(rl), t(d), pinf, want_transm=sep)
    torch.cuda.synchronize()
    assert list(out["status"].cpu().numpy()) == list(ref["status"]) == [0] * len(Ls)
    for p in range(len(Ls)):
        for k in ("trans", "transm") if sep else ("trans",):
            got, want = f(out[k].cpu().numpy())[p], ref[k][p]
            assert np.abs(got - want).max() <= 1e-4 * np.abs(want).max(), (p, k)
    np.testing.assert_allclose(pinf.cpu().numpy(), ref["parm_infl"], rtol=1e-4)

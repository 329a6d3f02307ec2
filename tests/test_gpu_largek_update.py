"""The FP32 update of large ensembles and the large-k core's Gram where their
tiles end: ensembles around multiples of 32 members, one and eight variables,
the analysis written over the background, lists around the 16 rows of a stage
and the 32 of a pair.

Tolerances: the update's FP32 sum of ne products may be off by (ne + 2) 2^-24 of
the sum of their magnitudes, and the stored member rounds once more; the core's
bar is 1e-4 of the transform's largest entry."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ne,nv,inplace", [(2, 1, False), (31, 8, False), (33, 3, True), (130, 8, True),
                                           (509, 2, False), (512, 8, True)])
def test_update_tiles(cuda, ne, nv, inplace):
    import torch

    from letkf_gb300.core import _dptr, _stream, lib, update_mixed

    rng = np.random.default_rng(ne + nv)
    npts = 5
    xb = (rng.standard_normal((nv, npts, ne)) + 10.0).astype(np.float32)
    tr = (rng.standard_normal((npts, ne, ne)) / np.sqrt(ne)).astype(np.float32)
    tm = (rng.standard_normal((npts, ne)) * 0.1).astype(np.float32)
    t = lambda a: torch.as_tensor(np.ascontiguousarray(a), device=cuda)
    gx, gt, gm = t(xb), t(tr), t(tm)
    if inplace:
        assert lib().letkf_update_mixed(ne, npts, nv, _dptr(gx), _dptr(gt), _dptr(gm), _dptr(gx), _stream(None)) == 0
        xa = gx
    else:
        xa = update_mixed(gx, gt, gm)
    torch.cuda.synchronize()
    x64 = xb.astype(np.float64)
    mean = x64.mean(-1, keepdims=True)
    xp = x64 - mean
    base = mean + np.einsum("vpk,pk->vp", xp, tm.astype(np.float64))[..., None]
    want = base + np.einsum("vpk,pmk->vpm", xp, tr.astype(np.float64))
    mag = np.einsum("vpk,pmk->vpm", np.abs(xp), np.abs(tr.astype(np.float64)))
    tol = (ne + 2) * 2.0 ** -24 * mag + 2.0 ** -24 * np.abs(want) * 1.01
    assert (np.abs(xa.cpu().numpy() - want) <= tol).all()


@pytest.mark.parametrize("ne", [129, 250])
def test_gram_stages(cuda, ne):
    import torch

    from letkf_gb300.core import core_batch_largek

    rng = np.random.default_rng(ne)
    Ls = [1, 15, 16, 17, 31, 32, 33, 0, 47, 48, 49, 64, 65]
    offs = np.concatenate([[0], np.cumsum(Ls)]).astype(np.int64)
    n = int(offs[-1])
    f32 = lambda a: a.astype(np.float32).astype(np.float64)
    rows = f32(rng.standard_normal((n, ne)))
    rd, rl, d = f32(rng.uniform(0.3, 3.0, n)), f32(rng.uniform(0.01, 1.0, n)), f32(rng.standard_normal(n))
    infl = rng.uniform(0.95, 1.3, len(Ls))
    ref = O.letkf_core_batch(ne, offs, rows, rd, rl, d, infl, want_transm=True)
    t = lambda a, dt=torch.float32: torch.as_tensor(np.ascontiguousarray(a), dtype=dt, device=cuda)
    out = core_batch_largek(ne, t(offs, torch.int64), t(rows), t(rd), t(rl), t(d), t(infl, torch.float64),
                            want_transm=True)
    torch.cuda.synchronize()
    assert (out["status"].cpu().numpy() == 0).all()
    for p in range(len(Ls)):
        scale = np.abs(ref["trans"][p]).max()
        assert np.abs(out["trans"][p].cpu().numpy() - ref["trans"][p]).max() <= 1e-4 * scale, Ls[p]
        if Ls[p]:
            assert np.abs(out["transm"][p].cpu().numpy() - ref["transm"][p]).max() <= 1e-4 * scale, Ls[p]

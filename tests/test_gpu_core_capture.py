"""The batched cores of ensembles up to LETKF_MAX_NE hold no device memory of
their own: a captured call is kernels only (a graph with allocation nodes
cannot be cloned or made a child), and its replay gives the call's bits."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

KERNEL_NODE = 0


def _ok(status):
    assert status == 0


@pytest.mark.parametrize("ne", [7, 20, 40, 64, 90])
@pytest.mark.parametrize("form", ["f64", "mixed"])
def test_captured_core_is_kernels_only(cuda, ne, form):
    import torch

    from letkf_gb300.core import core_batch_f64, core_batch_mixed
    from letkf_gb300.lib import lib

    lib()
    rt = C.CDLL("libcudart.so.13")
    rng = np.random.default_rng(ne)
    npts = 6000 if ne <= 40 else 1500 if ne == 64 or form == "mixed" else 40
    offs = np.concatenate([[0], np.cumsum(rng.integers(0, 6, npts))]).astype(np.int64)
    n = int(offs[-1])
    dt = torch.float64 if form == "f64" else torch.float32
    t = lambda a, d=dt: torch.as_tensor(np.ascontiguousarray(a), dtype=d, device=cuda)
    args = (t(offs, torch.int64), t(rng.standard_normal((n, ne))), t(rng.uniform(0.5, 2.0, n)),
            t(rng.uniform(0.1, 1.0, n)), t(rng.standard_normal(n)))
    infl = t(np.full(npts, 1.1), torch.float64)
    core = core_batch_f64 if form == "f64" else core_batch_mixed
    want = core(ne, *args, infl.clone(), want_transm=True)
    torch.cuda.synchronize()

    ptr = lambda x: C.c_void_p(x.data_ptr())
    inf2, trans, transm = infl.clone(), torch.empty_like(want["trans"]), torch.empty_like(want["transm"])
    status = torch.empty_like(want["status"])
    outs = [ptr(inf2), ptr(trans), ptr(transm)] + ([None] if form == "f64" else [])
    call = lib().letkf_core_batch_f64 if form == "f64" else lib().letkf_core_batch_mixed
    stream = torch.cuda.Stream()
    s = C.c_void_p(stream.cuda_stream)
    graph, clone, exe = C.c_void_p(), C.c_void_p(), C.c_void_p()
    torch.cuda.synchronize()
    _ok(rt.cudaStreamBeginCapture(s, 2))
    st = call(ne, npts, *[ptr(a) for a in args], *outs, 0, 0.0, ptr(status), s)
    _ok(rt.cudaStreamEndCapture(s, C.byref(graph)))
    _ok(st)
    count = C.c_size_t()
    _ok(rt.cudaGraphGetNodes(graph, None, C.byref(count)))
    nodes = (C.c_void_p * count.value)()
    _ok(rt.cudaGraphGetNodes(graph, nodes, C.byref(count)))
    kinds = []
    for node in nodes:
        kind = C.c_int()
        _ok(rt.cudaGraphNodeGetType(C.c_void_p(node), C.byref(kind)))
        kinds.append(kind.value)
    assert kinds and all(k == KERNEL_NODE for k in kinds)

    _ok(rt.cudaGraphClone(C.byref(clone), graph))
    _ok(rt.cudaGraphInstantiate(C.byref(exe), clone, C.c_ulonglong(0)))
    _ok(rt.cudaGraphLaunch(exe, s))
    torch.cuda.synchronize()
    assert torch.equal(trans, want["trans"]) and torch.equal(transm, want["transm"])
    assert torch.equal(inf2, want["parm_infl"]) and torch.equal(status, want["status"])
    _ok(rt.cudaGraphExecDestroy(exe))
    _ok(rt.cudaGraphDestroy(clone))
    _ok(rt.cudaGraphDestroy(graph))

"""FP64 products recorded into a CUDA graph: also an operator's first one, which may
allocate nothing and wait for nothing then."""
import ctypes as C

import numpy as np
import pytest
import torch

import aboria_gb300 as ab
from aboria_gb300._lib import lib

pytestmark = pytest.mark.gpu


def _operator(form, p, kern):
    """An operator as a C program makes it: FP64 by default, nothing prepared."""
    h = C.c_void_p()
    if form == "dense":
        st = lib().abx_create_dense_operator(p._h, p._h, C.byref(kern), C.byref(h))
    elif form == "sparse":
        st = lib().abx_create_sparse_operator(p._h, p._h, 0.2, C.byref(kern), C.byref(h))
    else:
        st = lib().abx_create_fmm_operator(p._h, C.byref(kern), 5 if form == "fmm5" else 3, C.byref(h))
    assert st == 0
    return ab.Operator(h, p, p)


@pytest.mark.parametrize("prepared", [False, True])
@pytest.mark.parametrize("kind,p0", [(ab.K_LAPLACE, 0.01), (ab.K_GAUSSIAN, 9.0), (ab.K_CONST, 2.0)])
@pytest.mark.parametrize("form", ["dense", "sparse", "fmm", "fmm5"])
def test_first_product(form, kind, p0, prepared):
    stream = torch.cuda.Stream()
    ctx = ab.Context(0, stream=stream.cuda_stream)
    rng = np.random.default_rng(0)
    p = ab.Particles(3, ctx).set(rng.uniform(0, 1, (3000, 3)))
    box = [0.0] * 3, [1.0] * 3, [False] * 3
    p.init_octree(*box, 20) if form.startswith("fmm") else p.init_neighbour_search(*box, 10)
    kern = ab.Kernel.make(kind, p0)
    b = torch.from_numpy(rng.uniform(0.5, 1.0, 3000)).cuda()
    want = _operator(form, p, kern) * b
    K = _operator(form, p, kern)
    if prepared:
        K.set_precision(ab.PREC_FP64)
    out = torch.zeros(3000, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        K.matvec(b, out=out, sync=False)
    assert not out.any()  # recorded, not run
    graph.replay()
    torch.cuda.synchronize()
    # the FP64 kernels and the integer ones
    assert torch.linalg.norm(out - want) <= 1e-12 * torch.linalg.norm(want)

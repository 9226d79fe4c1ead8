"""Whole solves in one thread-block cluster (k_pcg_cluster) against the same
solver as a sequence of launches (fm_project_noalloc never uses the cluster):
the smallest grids, slabs of unequal size, odd coarse extents, every number of
CTAs, the solution kept outside shared memory, both bottom orders and the
degenerate sweep counts.  Same arithmetic in the same order except for the inner
products (FP64 sums), so the kernel parity tolerances apply and the iteration
counts agree.  A masked grid too large for a cluster is checked by what a
projection must do."""
import ctypes as C
import importlib

import numpy as np
import pytest
import torch

TOL = {torch.float32: 2e-5, torch.float64: 1e-10}  # the kernel parity tolerances

# shape, levels, pre_post, bottom, bottom_mode
CASES = [
    ((4, 4), 2, 2, 10, 0), ((24, 40), 3, 1, 1, 0), ((20, 12), 3, 2, 0, 0), ((36, 52), 3, 3, 3, 1),
    ((64, 64), 4, 2, 20, 1), ((200, 72), 4, 2, 20, 1), ((336, 128), 4, 2, 20, 1), ((384, 384), 5, 2, 20, 1),
    ((4, 6, 10), 2, 2, 10, 0), ((20, 28, 36), 3, 2, 50, 0), ((32, 24, 40), 3, 3, 7, 1), ((48, 16, 48), 3, 1, 50, 0),
]


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("shape,levels,pre_post,bottom,mode", CASES)
def test_cluster_solve_equals_launch_sequence(fm, cuda, shape, levels, pre_post, bottom, mode, dtype):
    lib = fm._lib.lib()
    g = fm.GridSpec(shape)
    cg, code = g.c_grid(), fm._lib.dtype_code(dtype)
    P = fm._lib.MGParams(levels, pre_post, bottom, mode, 200, 0.0, 1e-8, 1e-12, 4, 0)
    handle = C.c_void_p()
    assert lib.fm_mgpcg_create(C.byref(cg), code, C.byref(P), C.byref(handle)) == 0
    stream = torch.cuda.current_stream().cuda_stream
    rng = np.random.default_rng(6)
    try:
        for _ in range(2):
            u = [torch.tensor(rng.uniform(-1, 1, size=g.face_shape(c)), dtype=dtype, device=cuda) for c in range(g.dim)]
            a, b = [x.clone() for x in u], [x.clone() for x in u]
            pa = [x.data_ptr() for x in a] + [None] * (3 - g.dim)
            pb = [x.data_ptr() for x in b] + [None] * (3 - g.dim)
            ia, ib, ra, rb = C.c_int(0), C.c_int(0), C.c_double(0), C.c_double(0)
            sa = lib.fm_project(handle, pa[0], pa[1], pa[2], None, stream, C.byref(ia), C.byref(ra))
            sb = lib.fm_project_noalloc(C.byref(cg), code, C.byref(P), pb[0], pb[1], pb[2], stream, C.byref(ib),
                                        C.byref(rb))
            torch.cuda.synchronize()
            assert sa == sb
            assert ia.value == ib.value
            for x, y in zip(a, b):
                assert float((x - y).abs().max() / y.abs().max()) < TOL[dtype]
    finally:
        lib.fm_mgpcg_destroy(handle)


@pytest.mark.gpu
def test_masked_solve_of_a_grid_too_large_for_a_cluster(fm, cuda):
    M = importlib.import_module("differentiable-flowmap_b200.mgpcg")
    Cf = importlib.import_module("differentiable-flowmap_b200.configs")
    n = 512
    mask = torch.tensor(Cf.leaf_mask(n), device=cuda)
    S = M.SolidMGPCG((n, n), mask, torch.float64, levels=6, abs_tol=0.0, rel_tol=1e-16, check_every=0)
    gen = torch.Generator(device=cuda).manual_seed(3)
    u = [torch.randn(s, generator=gen, device=cuda, dtype=torch.float64) for s in ((n + 1, n), (n, n + 1))]
    fluid = (mask <= 0).double()

    def divergence(v):
        return (v[0][1:] - v[0][:-1] + v[1][:, 1:] - v[1][:, :-1]) * fluid

    before = float(divergence(u).norm())
    S.project(u)
    assert S.stats()["not_converged"] == 0
    # |r|^2 < 1e-16 z0.r0 and z0.r0 <= |r0|^2 / (smallest eigenvalue ~ (pi / n)^2): |r| < 2e-6 |r0|
    assert float(divergence(u).norm()) < 2e-6 * before
    assert float((u[0][1:] * (1 - fluid)).abs().max()) == 0 and float((u[1][:, :-1] * (1 - fluid)).abs().max()) == 0

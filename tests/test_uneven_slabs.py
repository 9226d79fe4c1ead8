"""Whole solves of 2D FP32 grids whose largest slab holds over 10 500 cells, a fifth more
than the mean, run as a sequence of launches; even slabs, smaller ones and grids whose
launches have no coarse-level kernel stay in one cluster."""
import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,levels,cluster", [
    ((320, 448), 5, False), ((288, 448), 5, False), ((400, 320), 5, True),
    ((480, 320), 5, True), ((304, 384), 5, True), ((400, 352), 4, True), ((384, 384), 5, True)])
def test_path(fm, cuda, shape, levels, cluster):
    lib, h, it = fm._lib.lib(), C.c_void_p(), C.c_int(0)
    P = fm._lib.MGParams(levels, 2, 10, 1, 200, 0.0, 1e-8, 1e-12, 4, 0)
    cg, s = fm.GridSpec(shape).c_grid(), torch.cuda.current_stream().cuda_stream
    u = [torch.linspace(-1, 1, a * b, device=cuda).sin().reshape(a, b) for a, b in
         ((shape[0] + 1, shape[1]), (shape[0], shape[1] + 1))]
    assert lib.fm_mgpcg_create(C.byref(cg), 0, C.byref(P), C.byref(h)) == 0
    a, b = ([x.clone() for x in u] for _ in range(2))
    before = fm._lib.launch_count()
    assert lib.fm_project(h, a[0].data_ptr(), a[1].data_ptr(), None, None, s, C.byref(it), None) == 0
    n = fm._lib.launch_count() - before
    torch.cuda.synchronize()
    lib.fm_mgpcg_destroy(h)
    assert (n == 3) == cluster
    assert lib.fm_project_noalloc(C.byref(cg), 0, C.byref(P), b[0].data_ptr(), b[1].data_ptr(), None, s, None, None) == 0
    for x, y in zip(a, b):  # the kernel parity tolerance
        assert float((x - y).abs().max() / y.abs().max()) < 2e-5

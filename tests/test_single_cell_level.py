"""A coarsest level of one cell has no neighbours: its smoothing divides by zero, as the
reference's does, and a solve over such levels ends as non-finite in every type and on
every path (whole solves and coarse levels in one cluster, and launch by launch)."""
import ctypes as C

import numpy as np
import pytest
import torch

from oracle import MGParams, Oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", ["f32", "f64"])
@pytest.mark.parametrize("shape,levels", [((4, 4), 3), ((16, 16), 5), ((8, 8, 8), 4)],
                         ids=lambda v: "x".join(map(str, v)) if isinstance(v, tuple) else str(v))
def test_one_cell_level(fm, cuda, shape, levels, name):
    o = Oracle(shape, name)
    dtype = torch.float32 if name == "f32" else torch.float64
    r = np.random.default_rng(3).uniform(0.5, 1.5, size=shape).astype(o.dtype)
    want = np.zeros(shape, o.dtype)
    with np.errstate(all="ignore"):
        o.mg_vcycle(MGParams(levels, 2, 10, 1, 1, 0.0, 0.0, 0.0), r.copy(), want)
    assert not np.isfinite(want).all()
    sol = fm.MGPCG(shape, dtype, levels=levels, pre_post=2, bottom=10, bottom_mode=1)
    assert np.array_equal(sol.apply_preconditioner(torch.tensor(r, device=cuda)).cpu().numpy(), want, equal_nan=True)

    lib, g = fm._lib.lib(), fm.GridSpec(shape)
    P = fm._lib.MGParams(levels, 2, 10, 1, 50, 0.0, 1e-8, 1e-12, 0, 0)
    cg, h, it, rtr = g.c_grid(), C.c_void_p(), C.c_int(0), C.c_double(0)
    assert lib.fm_mgpcg_create(C.byref(cg), fm._lib.dtype_code(dtype), C.byref(P), C.byref(h)) == 0
    gen = torch.Generator(device=cuda).manual_seed(1)
    u = [torch.rand(g.face_shape(c), generator=gen, device=cuda, dtype=dtype) for c in range(g.dim)]
    st = lib.fm_project(h, *[x.data_ptr() for x in u], *[None] * (3 - g.dim), None,
                        torch.cuda.current_stream().cuda_stream, C.byref(it), C.byref(rtr))
    lib.fm_mgpcg_destroy(h)
    assert st == 4  # FM_ERR_NONFINITE

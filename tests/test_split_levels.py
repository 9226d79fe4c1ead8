"""3D levels stored by colour, and the 3D kernels that walk along axis 0, where they
change their split: one group of 16 cells a row, rows not a multiple of a block, few
and many planes, odd coarse extents, a second level that keeps (or does not keep) the
rule on the row length, one smoothing step.  A V-cycle equals the sequential oracle's
bit for bit; a projection equals the one without allocations (which keeps the natural
order) within the kernel parity tolerances, with the same number of iterations."""
import ctypes as C

import numpy as np
import pytest
import torch

from oracle import MGParams, Oracle

pytestmark = pytest.mark.gpu
TOL = {"f32": 2e-5, "f64": 1e-10}  # the kernel parity tolerances

# shape, levels, pre_post, bottom; every grid is too large for one cluster
CASES = [
    ((72, 64, 96), 3, 1, 3), ((36, 200, 64), 3, 2, 4), ((8, 512, 128), 3, 2, 4), ((512, 8, 128), 2, 3, 4),
    ((256, 256, 16), 2, 2, 2), ((68, 84, 80), 3, 2, 4), ((100, 72, 72), 3, 2, 4), ((60, 52, 272), 2, 1, 2),
]


@pytest.mark.parametrize("name", ["f32", "f64"])
@pytest.mark.parametrize("shape,levels,pre_post,bottom", CASES)
def test_vcycle_and_projection(fm, cuda, shape, levels, pre_post, bottom, name):
    o = Oracle(shape, name)
    dtype = torch.float32 if name == "f32" else torch.float64
    rng = np.random.default_rng(sum(shape))
    r = rng.standard_normal(shape).astype(o.dtype)
    want = np.zeros(shape, o.dtype)
    o.mg_vcycle(MGParams(levels, pre_post, bottom, 0, 1, 0.0, 0.0, 0.0), r.copy(), want)
    sol = fm.MGPCG(shape, dtype, levels=levels, pre_post=pre_post, bottom=bottom, bottom_mode=0, abs_tol=0.0,
                   rel_tol=1e-6, max_iters=200, check_every=4)
    for _ in range(2):  # the solver's buffers are dirty the second time
        assert np.array_equal(sol.apply_preconditioner(torch.tensor(r, device=cuda)).cpu().numpy(), want)

    lib, g = fm._lib.lib(), fm.GridSpec(shape)
    P = fm._lib.MGParams(levels, pre_post, bottom, 0, 200, 0.0, 1e-6, 1e-12, 4, 0)
    u = [torch.tensor(rng.uniform(-1, 1, size=g.face_shape(c)), dtype=dtype, device=cuda) for c in range(3)]
    a, b = [x.clone() for x in u], [x.clone() for x in u]
    sol.project(a)
    ib, rb, cg = C.c_int(0), C.c_double(0), g.c_grid()
    assert lib.fm_project_noalloc(C.byref(cg), fm._lib.dtype_code(dtype), C.byref(P), *[x.data_ptr() for x in b],
                                  torch.cuda.current_stream().cuda_stream, C.byref(ib), C.byref(rb)) == 0
    torch.cuda.synchronize()
    assert sol.last_iters == ib.value
    for x, y in zip(a, b):
        assert float((x - y).abs().max() / y.abs().max()) < TOL[name]

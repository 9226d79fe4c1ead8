"""2D V-cycles on both sides of the line between the two coarse-level kernels (rows of the
coarsest level a multiple of 32 cells; 512 pairs of cells or more, in FP64 at most 1024)
equal the sequential V-cycle bit for bit."""
import numpy as np
import pytest
import torch

from oracle import MGParams, Oracle

pytestmark = pytest.mark.gpu


# coarsest level: 32x32 (512 pairs), 16x64 (512), 64x32 (1024), 64x64 (2048), 30x32 (480), 32x36, 36x32
@pytest.mark.parametrize("shape,levels", [((128, 128), 3), ((64, 256), 3), ((256, 128), 3), ((256, 256), 3), ((120, 128), 3),
                                          ((128, 144), 3), ((144, 128), 3), ((256, 256), 4)],
                         ids=lambda v: "x".join(map(str, v)) if isinstance(v, tuple) else str(v))
@pytest.mark.parametrize("pname", ["f64", "f32"])
@pytest.mark.parametrize("mode", [0, 1])
def test_vcycle_bitwise(fm, cuda, shape, levels, pname, mode):
    o = Oracle(shape, pname)
    r = np.random.default_rng(sum(shape)).standard_normal(shape).astype(o.dtype)
    ref = np.zeros(shape, o.dtype)
    o.mg_vcycle(MGParams(levels, 2, 6, mode, 1, 0.0, 0.0, 0.0), r.copy(), ref)
    S = fm.MGPCG(shape, torch.float64 if pname == "f64" else torch.float32, levels=levels, pre_post=2, bottom=6,
                 bottom_mode=mode)
    z = S.apply_preconditioner(torch.tensor(r, device=cuda)).cpu().numpy()
    assert np.array_equal(z, ref), np.abs(z - ref).max()

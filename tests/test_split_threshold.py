"""FP32 3D solvers store their levels by colour from a size on (850 000 cells); on either
side of that size, and in FP64, which keeps the natural order, a V-cycle equals the
sequential oracle's bit for bit, also on a second call with dirty buffers."""
import numpy as np
import pytest
import torch

from oracle import MGParams, Oracle

pytestmark = pytest.mark.gpu

# shape, levels, pre_post: just below, just above, one group of 16 cells a row, few rows, many planes, a
# coarse level whose rows break the rule of 16 n cells
CASES = [((92, 96, 96), 3, 2), ((96, 96, 96), 4, 1), ((96, 96, 96), 3, 3), ((244, 220, 16), 2, 2), ((420, 8, 256), 3, 1),
         ((8, 428, 256), 3, 2), ((24, 100, 368), 2, 2), ((100, 96, 96), 3, 2), ((116, 92, 80), 3, 2)]


@pytest.mark.parametrize("name", ["f32", "f64"])
@pytest.mark.parametrize("shape,levels,pre_post", CASES, ids=lambda v: "x".join(map(str, v)) if isinstance(v, tuple) else str(v))
def test_vcycle_equals_the_oracle(fm, cuda, shape, levels, pre_post, name):
    o = Oracle(shape, name)
    r = np.random.default_rng(sum(shape)).standard_normal(shape).astype(o.dtype)
    want = np.zeros(shape, o.dtype)
    o.mg_vcycle(MGParams(levels, pre_post, 3, 0, 1, 0.0, 0.0, 0.0), r.copy(), want)
    sol = fm.MGPCG(shape, torch.float32 if name == "f32" else torch.float64, levels=levels, pre_post=pre_post, bottom=3,
                   bottom_mode=0)
    for _ in range(2):
        assert np.array_equal(sol.apply_preconditioner(torch.tensor(r, device=cuda)).cpu().numpy(), want)

"""New obstacle masks: setting one costs a launch per level, whether or not the solve runs
in one cluster (which reads packed masks), and a solver with a new mask equals one
created with it bit for bit -- square and odd coarse rows, two levels, 2D and 3D, in a
cluster and as a sequence of launches (512x256 in FP64)."""
import importlib

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64], ids=["f32", "f64"])
@pytest.mark.parametrize("shape,levels", [((8, 10), 2), ((40, 24), 3), ((36, 52), 3), ((128, 64), 4), ((512, 256), 5),
                                          ((8, 12, 10), 2), ((16, 24, 20), 3), ((32, 32, 32), 4)],
                         ids=lambda v: "x".join(map(str, v)) if isinstance(v, tuple) else str(v))
def test_set_mask(fm, cuda, shape, levels, dtype):
    M = importlib.import_module("differentiable-flowmap_b200.mgpcg")
    kw = dict(levels=levels, max_iters=30, abs_tol=0.0, rel_tol=1e-9, check_every=0)
    gen = torch.Generator(device=cuda).manual_seed(11)
    masks = [(torch.rand(shape, generator=gen, device=cuda) < q).float() for q in (0.0, 0.3, 0.9, 0.02)]
    u = [torch.rand(fm.GridSpec(shape).face_shape(c), generator=gen, device=cuda, dtype=dtype) for c in range(len(shape))]
    old = M.SolidMGPCG(shape, masks[0], dtype, **kw)
    for m in masks[1:] + masks[:1]:
        before = fm._lib.launch_count()
        old.set_mask(m)
        assert fm._lib.launch_count() - before == levels
        a, b = [x.clone() for x in u], [x.clone() for x in u]
        old.project(a)
        M.SolidMGPCG(shape, m, dtype, **kw).project(b)
        for x, y in zip(a, b):
            assert torch.equal(x.nan_to_num(7.0), y.nan_to_num(7.0))  # NaN: a fluid cell without fluid neighbours

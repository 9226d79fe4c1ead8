"""The transposed samples add the overlapping taps of neighbouring lanes up before
they reach memory.  Checked where such chains begin, break and end: along rows of
near-identity maps, at masked (zero) adjoints, at jumps of the map, at row ends and
in the last, partly filled warp, against the FP64 oracle's forward kernel by
<A f, lam> = <f, A^T lam>.
"""
import numpy as np
import pytest
import torch

from oracle import Oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kept", [1.0, 0.7, 0.1, 0.0])
@pytest.mark.parametrize("shape", [(4, 4, 4), (5, 4, 67), (6, 33, 31), (4, 4), (7, 129), (33, 30)],
                         ids=lambda s: "x".join(map(str, s)))
def test_chained_scatter_is_the_transpose(fm, cuda, shape, kept):
    rng = np.random.default_rng(31)
    o, g, d, dx = Oracle(shape, "f64"), fm.GridSpec(shape), len(shape), 1.0 / shape[1]
    p = np.stack(np.meshgrid(*[(np.arange(n) + 0.5) * dx for n in shape], indexing="ij"))
    p += 0.3 * dx * np.sin(7 * p[::-1])            # neighbours mostly one entry apart
    p[:, shape[0] // 2:] += rng.uniform(-2, 2) * dx  # and a jump
    flat = p.reshape(d, -1)
    flat[:, ::13] = rng.uniform(-0.2, 1.2, size=flat[:, ::13].shape)
    s0 = rng.uniform(-1, 1, size=shape)
    lam = rng.uniform(-1, 1, size=shape) * (rng.uniform(size=shape) < kept)
    out = np.zeros(shape)
    o.advect_scalar(s0, out, p, dx)
    T = lambda a: torch.tensor(a, dtype=torch.float64, device=cuda)  # noqa: E731
    gs = torch.zeros(shape, dtype=torch.float64, device=cuda)
    fm.kernels.pullback_scalar_adj(g, dx, T(s0), T(p), T(lam), 1.0, 0.0, gs, None)
    got = gs.cpu().numpy()
    # sums of at most 27 n products of |.| <= 1, each a few roundings: 64 eps of the absolute sum
    bound = 64 * np.finfo(np.float64).eps * np.abs(lam).sum()
    assert abs((out * lam).sum() - (s0 * got).sum()) <= bound
    # the weights of a sample add up to one
    assert abs(lam.sum() - got.sum()) <= bound

"""FP64 gradient stencils where dx is no power of two, on grids that take tiles 4 and 8
high (few and many of them), with the pairs between the passes in memory of their own and
over the footprints: the oracle's values."""
import numpy as np
import pytest
import torch

from oracle import Oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", [3, 4])
@pytest.mark.parametrize("shape", [(8, 9, 31), (7, 16, 33), (35, 78, 31), (25, 49, 122)], ids=lambda s: "x".join(map(str, s)))
def test_values(fm, cuda, shape, order):
    rng, o, g, dx = np.random.default_rng(61), Oracle(shape, "f64"), fm.GridSpec(shape), 1.0 / 23
    u, w = ([rng.uniform(-1, 1, size=g.face_shape(c)) for c in range(3)] for _ in range(2))
    ref = [np.zeros(g.face_shape(c)) for c in range(3)]
    o.calculate_nabla_u_w([x.copy() for x in u], [x.copy() for x in w], ref, dx, order)
    T = lambda a: torch.tensor(a, device=cuda)  # noqa: E731
    out = [torch.full(g.face_shape(c), float("nan"), dtype=torch.float64, device=cuda) for c in range(3)]
    fm.kernels.nabla_u_w(g, dx, [T(x) for x in u], [T(x) for x in w], out, order)
    for a, b in zip(out, ref):  # the FP64 kernel parity tolerance
        assert np.abs(a.cpu().numpy() - b).max() <= 1e-11 * np.abs(b).max()

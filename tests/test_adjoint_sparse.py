"""Adjoints that are zero at most nodes: a lane without an adjoint samples nothing and adds
nothing, so the gradients of the parts of an adjoint add up to those of the whole."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kept", [0.01, 0.5])
@pytest.mark.parametrize("rk", [2, 4])
@pytest.mark.parametrize("shape", [(9, 7, 35), (13, 70)], ids=lambda s: "x".join(map(str, s)))
def test_parts_add_up(fm, cuda, shape, rk, kept):
    k, g, d, dx = fm.kernels, fm.GridSpec(shape), len(shape), 1.0 / shape[1]
    gen = torch.Generator(device=cuda)
    gen.manual_seed(41)
    R = lambda s: torch.rand(s, generator=gen, device=cuda, dtype=torch.float64) * 2 - 1  # noqa: E731
    faces = [g.face_shape(c) for c in range(d)]
    u, f, lam = ([R(s) for s in faces] for _ in range(3))
    T, psi = ([R((d,) + s) for s in faces] for _ in range(2))
    s1, ls = R(shape), R(shape)
    keep = [torch.rand(s, generator=gen, device=cuda) < kept for s in faces + [shape]]

    def grads(lm, l):
        Z = lambda s: torch.zeros(s, device=cuda, dtype=torch.float64)  # noqa: E731
        a, b, c, e, h = ([Z(s) for s in faces] for _ in range(5))
        gT, gp = ([Z((d,) + s) for s in faces] for _ in range(2))
        gs = Z(shape)
        k.advect_u_grid_adj(g, rk, dx, 0.7 * dx, u, f, lm, a, b)
        k.advect_scalar_grid_adj(g, rk, dx, 0.7 * dx, u, s1, l, c, gs)
        k.pullback_u_adj(g, dx, u, T, psi, lm, 1.0, 0.5, e, gT, gp, h)
        return a + b + c + e + h + gT + gp + [gs]

    whole = grads(lam, ls)
    part = grads([x * m for x, m in zip(lam, keep)], ls * keep[-1])
    rest = grads([x * ~m for x, m in zip(lam, keep)], ls * ~keep[-1])
    # an entry is a sum of up to some thousand products; each order of them is within 1e-12 of the largest
    for w, x, y in zip(whole, part, rest):
        assert float((w - x - y).abs().max()) <= 1e-12 * max(float(w.abs().max()), 1.0)

"""Where the Gaussian sums change their split: supports longer than one table along
the middle, the outer or the column axis (the last takes the per-face path),
ragged ends of the steps of 8 faces, and the order in which blocks take the
Gaussians, which must not show in the results.
"""
import importlib

import numpy as np
import pytest
import torch

import force_oracle as FO

pytestmark = pytest.mark.gpu
K = importlib.import_module("differentiable-flowmap_b200.kernels")


def _dev(a, dtype=torch.float64):
    return torch.tensor(np.ascontiguousarray(a), device="cuda", dtype=dtype)


@pytest.mark.parametrize("res", [(530, 9), (9, 530), (270, 7, 9), (7, 270, 9), (9, 7, 270), (5, 4, 4), (17, 15)],
                         ids=lambda s: "x".join(map(str, s)))
def test_long_supports_match_oracle(cuda, res):
    d, dx, rng = len(res), 1.0 / res[0], np.random.default_rng(41)
    c = rng.uniform(-0.1, 1.1, size=(6, d)) * np.array(res) * dx
    # support radii: the whole box and more, beyond one table, half the box, a few cells, less than a cell
    R = np.array([2.0 * max(res), 0.9 * max(res), 0.5 * max(res), 6.0, 2.3, 0.4]) * dx
    r, s = 5.0 / R ** 2, rng.uniform(-1, 1, size=(6, d))
    g = K.GridSpec(res)
    adj = [rng.normal(size=g.face_shape(k)) for k in range(d)]
    want = FO.gaussian_force_grad(res, dx, c, r, s, adj)
    got = K.gaussian_force_grad(g, dx, _dev(c), _dev(r), _dev(s), [_dev(a) for a in adj])
    for gv, wv in zip(got, want):
        # FP64 sums of at most 3 * 17010 terms, each a few roundings, relative to the largest sum
        np.testing.assert_allclose(gv.cpu().numpy(), wv, rtol=0, atol=1e-10 * np.abs(wv).max())
    f = [torch.empty(g.face_shape(k), device="cuda", dtype=torch.float64) for k in range(d)]
    K.gaussian_force(g, dx, _dev(c), _dev(r), _dev(s), f)
    for a, b in zip(f, FO.gaussian_force(res, dx, c, r, s)):
        np.testing.assert_allclose(a.cpu().numpy(), b, rtol=0, atol=1e-12)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64], ids=["f32", "f64"])
def test_order_of_the_gaussians_does_not_show(cuda, dtype):
    """8193 Gaussians are taken as they come, 8192 or fewer widest first."""
    res, dx, rng = (40, 24), 1.0 / 40, np.random.default_rng(43)
    n = 8193
    c = _dev(rng.uniform(0, 1, size=(n, 2)) * np.array([1.0, 0.6]), dtype)
    r = _dev(1.0 / (rng.choice([0.3, 1, 2, 5, 9], size=n) * dx) ** 2, dtype)
    r[5], r[77], r[300], r[4000] = -1.0, float("nan"), 0.0, float("inf")
    s = _dev(rng.uniform(-1, 1, size=(n, 2)), dtype)
    g = K.GridSpec(res)
    adj = [_dev(rng.normal(size=g.face_shape(k)), dtype) for k in range(2)]
    whole = K.gaussian_force_grad(g, dx, c, r, s, adj)
    for a, b in ((0, 8192), (1, 8193), (0, 1), (70, 327), (300, 301), (4000, 4001)):
        part = K.gaussian_force_grad(g, dx, c[a:b].contiguous(), r[a:b].contiguous(), s[a:b].contiguous(), adj)
        for x, y in zip(whole, part):
            assert torch.equal(x[a:b].nan_to_num(7.0), y.nan_to_num(7.0))
            assert torch.isfinite(y).all()

"""FP32 parameter sums of the Gaussians against 64 bits on the same inputs: no further off
than weights of two factors (a joint exponential of two axes times a table entry of
the third) whose sums over faces are kept in FP64.  Three factors, one table entry per
axis, share their roundings among all faces of a plane and are 1.2 to 1.4 times further off."""
import importlib

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
K = importlib.import_module("differentiable-flowmap_b200.kernels")
N, COUNT = 64, 512


def _relative_errors(c, r, weights_of):
    """Relative error of sum e^2 over the faces of each Gaussian and component, for the
    FP32 weights that weights_of(offsets squared, r, mask) gives; None: the exact sums alone."""
    dx, exact, got = np.float32(1.0 / N), [], []
    for I in range(len(r)):
        for cc in range(3):
            d = []
            for a in range(3):
                i = np.arange(int(c[I, a] * N) - 12, int(c[I, a] * N) + 13).astype(np.float32)
                d.append((i if a == cc else i + np.float32(0.5)) * dx - c[I, a])
            s2 = (d[0] ** 2)[:, None, None] + (d[1] ** 2)[:, None] + d[2] ** 2
            h = np.sqrt(s2)
            m = (h * h) * r[I] < np.float32(5)
            d64 = [x.astype(np.float64) ** 2 for x in d]
            e64 = np.exp(-(d64[0][:, None, None] + d64[1][:, None] + d64[2]) * float(r[I]))
            exact.append((e64[m] ** 2).sum())
            if weights_of is not None:
                got.append((weights_of(d, r[I])[m].astype(np.float64) ** 2).sum())
    return np.array(exact).reshape(-1, 3), np.array(got).reshape(-1, 3) if got else None


def _two_factors(d, r):
    joint = np.exp(-(((d[0] ** 2)[:, None] + d[2] ** 2) * r))
    return joint[:, None, :] * np.exp(-((d[1] ** 2) * r))[:, None]


@pytest.mark.parametrize("radius", [1.5, 3.0, 6.0], ids=lambda v: f"{v:g}cells")
def test_penalty_sums_as_close_to_64_bits_as_two_factors(cuda, radius):
    rng = np.random.default_rng(47)
    c = rng.uniform(0.3, 0.7, size=(COUNT, 3)).astype(np.float32)
    r = (5.0 / (radius / N * rng.uniform(0.97, 1.03, size=COUNT)) ** 2).astype(np.float32)
    exact, model = _relative_errors(c, r, _two_factors)
    rms = lambda x: np.sqrt(np.mean((x / exact - 1) ** 2))  # noqa: E731
    g = K.GridSpec((N, N, N))
    adj = [torch.ones(g.face_shape(k), device=cuda) for k in range(3)]
    dev = lambda a: torch.tensor(a, device=cuda)  # noqa: E731
    out = K.gaussian_force_grad(g, 1.0 / N, dev(c), dev(r), dev(np.ones((COUNT, 3), np.float32)), adj)
    pen = out[3].cpu().numpy()  # 2 s sum e^2 with s = 1
    assert pen.shape == exact.shape
    # two estimates of one rms from 1536 sums each differ by 2.6 % (one deviation): four of them, and
    # as much again for another exponential function
    assert rms(pen / 2) < 1.15 * rms(model)

"""Control forces and their parameter sums on FP32 grids with axes so long that the
position of a face is rounded by hundredths of a cell: a face that the exact test
reaches must not be lost by the index range worked out for its Gaussian."""
import importlib

import numpy as np
import pytest
import torch

from force_oracle import face_positions

pytestmark = pytest.mark.gpu
K = importlib.import_module("differentiable-flowmap_b200.kernels")


@pytest.mark.parametrize("res", [(6, 1500000), (1500000, 6), (5, 4, 400000), (400000, 4, 5)],
                         ids=lambda s: "x".join(map(str, s)))
def test_no_face_is_lost(cuda, res):
    d, dx, count = len(res), np.float32(1e-3), 600
    rng = np.random.default_rng(53)
    long = int(np.argmax(res))
    c = (rng.uniform(0, 1, size=(count, d)) * np.array(res) * dx).astype(np.float32)
    c[:, long] = rng.uniform(0.9, 0.99999, size=count) * res[long] * dx
    # nearly whole multiples of half a cell around the centre: faces near the cutoff on both sides
    radius = rng.integers(2, 9, size=count) * 0.5 * (1 + rng.uniform(-0.03, 0.03, size=count)) * dx
    r = (5.0 / radius ** 2).astype(np.float32)
    s = np.ones((count, d), np.float32)
    want = np.zeros((count, d))
    for k in range(d):
        P = face_positions(res, k, dx, np.float32)
        for I in range(count):
            near = []
            for a in range(d):
                x = P[a].reshape(-1)
                m = int(c[I, a] / dx)
                near.append(x[max(m - 12, 0):m + 13] - c[I, a] if a == long else x - c[I, a])
            s2 = np.zeros((), np.float32)
            for a in range(d):
                s2 = s2 + (near[a] ** 2).reshape([-1 if b == a else 1 for b in range(d)])
            h = np.sqrt(s2)
            q = (h * h) * r[I]
            want[I, k] = np.exp(-q[q < 5].astype(np.float64)).sum()
    g = K.GridSpec(res)
    dev = lambda a: torch.tensor(a, device=cuda)  # noqa: E731
    adj = [torch.ones(g.face_shape(k), device=cuda) for k in range(d)]
    _, got, _, _ = K.gaussian_force_grad(g, float(dx), dev(c), dev(r), dev(s), adj)
    # a lost face takes exp(-5) = 6.7e-3 away; the FP32 weights are good to a few times 1e-7 of sums below 300
    assert np.abs(got.cpu().numpy() - want).max() < 1e-3

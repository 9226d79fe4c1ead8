"""Which path a projection takes, and that both agree: a solve in one cluster is three
launches (front, solve, back); grids that do not fit it, or whose coarse levels have
fewer planes than it has CTAs, run as a sequence of launches.  Slabs of unequal size
on 2, 4, 8 and 16 CTAs, in 2D and 3D, with and without masks, and, above the limit, the
host-polled, device-side and captured forms."""
import ctypes as C

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
TOL = {torch.float32: 2e-5, torch.float64: 1e-10}  # the kernel parity tolerances
DTYPES = pytest.mark.parametrize("dtype", [torch.float32, torch.float64], ids=["f32", "f64"])


def _params(fm, levels, check_every, max_iters=200):
    return fm._lib.MGParams(levels, 2, 10, 1, max_iters, 0.0, 1e-8, 1e-12, check_every, 0)


def _project(fn, h, u, stream, outcome=True):
    it, rtr = C.c_int(0), C.c_double(0)
    st = fn(h, *[x.data_ptr() for x in u], *[None] * (3 - len(u)), None, stream, C.byref(it) if outcome else None,
            C.byref(rtr) if outcome else None)
    return st, it.value


class _Solver:
    """A plain (mask None) or masked handle."""

    def __init__(self, fm, shape, dtype, P, mask=None):
        self.lib, self.masked = fm._lib.lib(), mask is not None
        self.h, g = C.c_void_p(), fm.GridSpec(shape)
        cg, code = g.c_grid(), fm._lib.dtype_code(dtype)
        if self.masked:
            st = self.lib.fm_solid_create(C.byref(cg), code, C.byref(P), mask.data_ptr(), C.byref(self.h))
        else:
            st = self.lib.fm_mgpcg_create(C.byref(cg), code, C.byref(P), C.byref(self.h))
        assert st == 0

    @property
    def project(self):
        return self.lib.fm_solid_project if self.masked else self.lib.fm_project

    def __enter__(self):
        return self

    def __exit__(self, *_):
        torch.cuda.synchronize()
        (self.lib.fm_solid_destroy if self.masked else self.lib.fm_mgpcg_destroy)(self.h)


def _velocity(fm, shape, dtype, cuda):
    rng = np.random.default_rng(sum(shape))
    return [torch.tensor(rng.uniform(-1, 1, size=fm.GridSpec(shape).face_shape(c)), dtype=dtype, device=cuda)
            for c in range(len(shape))]


def _mask(shape, cuda):
    m = torch.zeros(shape, device=cuda)
    m[tuple(slice(n // 3, n // 2 + 1) for n in shape)] = 1
    m[(0,) * len(shape)] = 1
    return m


# CTAs and the planes that are split over them: 2D 56x40 28 over 2, 100x44 50 over 4, 92x116 46 over 8, 200x72 100 over 8,
# 104x264 26 over 16; 3D 16x18x14 8 over 2, 20^3 10 over 4, 22^3 11 over 8, 24^3 12 over 8
IN_CLUSTER = [((56, 40), 2), ((100, 44), 2), ((92, 116), 3), ((200, 72), 4), ((104, 264), 4), ((16, 18, 14), 2),
              ((20, 20, 20), 3), ((22, 22, 22), 2), ((24, 24, 24), 3)]


@DTYPES
@pytest.mark.parametrize("shape,levels", IN_CLUSTER, ids=lambda v: "x".join(map(str, v)) if isinstance(v, tuple) else str(v))
def test_in_cluster(fm, cuda, shape, levels, dtype):
    stream = torch.cuda.current_stream().cuda_stream
    P, u = _params(fm, levels, 4), _velocity(fm, shape, dtype, cuda)
    a, b = [x.clone() for x in u], [x.clone() for x in u]
    with _Solver(fm, shape, dtype, P) as S:
        before = fm._lib.launch_count()
        sa, ia = _project(S.project, S.h, a, stream)
        assert fm._lib.launch_count() - before == 3
    cg, it = fm.GridSpec(shape).c_grid(), C.c_int(0)
    sb = fm._lib.lib().fm_project_noalloc(C.byref(cg), fm._lib.dtype_code(dtype), C.byref(P), *[x.data_ptr() for x in b],
                                          *[None] * (3 - len(b)), stream, C.byref(it), None)
    assert sa == sb == 0 and ia == it.value
    for x, y in zip(a, b):
        assert float((x - y).abs().max() / y.abs().max()) < TOL[dtype]


@DTYPES
@pytest.mark.parametrize("shape,levels", IN_CLUSTER, ids=lambda v: "x".join(map(str, v)) if isinstance(v, tuple) else str(v))
def test_masked_in_cluster(fm, cuda, shape, levels, dtype):
    """The divergence of the fluid cells goes, closed faces are zero, and an all-fluid mask
    gives the plain solver's velocity."""
    stream = torch.cuda.current_stream().cuda_stream
    mask, u = _mask(shape, cuda), _velocity(fm, shape, dtype, cuda)
    P = _params(fm, levels, 0)
    a, b, c = ([x.clone() for x in u] for _ in range(3))
    with _Solver(fm, shape, dtype, P, mask) as S:
        before = fm._lib.launch_count()
        assert _project(S.project, S.h, a, stream)[0] == 0
        assert fm._lib.launch_count() - before == 3
    fluid = (mask <= 0).to(dtype)
    div = lambda v: sum(x.diff(dim=k) for k, x in enumerate(v)) * fluid  # noqa: E731
    closed = [x.clone() for x in u]
    for k, x in enumerate(closed):
        n = shape[k]
        x.narrow(k, 0, 1).zero_(), x.narrow(k, n, 1).zero_()
        x.narrow(k, 0, n).mul_(fluid), x.narrow(k, 1, n).mul_(fluid)
    # |r|^2 < 1e-8 z0.r0 and z0.r0 <= |r0|^2 / (smallest eigenvalue, about (pi / n)^2); FP32 rounding on top
    bound = 1e-4 * max(shape) / np.pi + (1e-4 if dtype == torch.float32 else 0.0)
    r = div(a)
    assert float((r - r.sum() / fluid.sum() * fluid).norm()) < bound * float(div(closed).norm())
    for k, x in enumerate(a):
        assert float((x.narrow(k, 1, shape[k]) * (1 - fluid)).abs().max()) == 0
    with _Solver(fm, shape, dtype, P, torch.zeros(shape, device=cuda)) as S, _Solver(fm, shape, dtype, P) as R:
        assert _project(S.project, S.h, b, stream)[0] == 0 and _project(R.project, R.h, c, stream)[0] == 0
    for x, y in zip(b, c):
        assert float((x - y).abs().max() / y.abs().max()) < TOL[dtype]


# too large, too few planes (28^3, 12x28x40), and FP64 grids that do not fit
SEQUENCE = [((512, 128), 4, torch.float64), ((416, 416), 4, torch.float32), ((28, 28, 28), 3, torch.float32),
            ((12, 28, 40), 3, torch.float64), ((40, 40, 40), 4, torch.float32), ((256, 256), 4, torch.float64)]


@pytest.mark.parametrize("masked", [False, True], ids=["plain", "masked"])
@pytest.mark.parametrize("shape,levels,dtype", SEQUENCE, ids=lambda v: "x".join(map(str, v)) if isinstance(v, tuple) else str(v))
def test_above_the_limit(fm, cuda, shape, levels, dtype, masked):
    """Host-polled, device-side and captured: the same velocity."""
    mask = _mask(shape, cuda) if masked else None
    u, out = _velocity(fm, shape, dtype, cuda), []
    for every in (3, 0):
        with _Solver(fm, shape, dtype, _params(fm, levels, every), mask) as S:
            for captured in ([False, True] if every == 0 else [False]):
                a, side = [x.clone() for x in u], torch.cuda.Stream()
                side.wait_stream(torch.cuda.current_stream())
                if captured:
                    graph = torch.cuda.CUDAGraph()
                    with torch.cuda.graph(graph, stream=side):
                        assert _project(S.project, S.h, a, side.cuda_stream, outcome=False)[0] == 0
                    for x, y in zip(a, u):
                        x.copy_(y)
                    graph.replay()
                else:
                    before = fm._lib.launch_count()
                    assert _project(S.project, S.h, a, side.cuda_stream, outcome=every != 0)[0] == 0
                    assert every == 0 or fm._lib.launch_count() - before > 20
                torch.cuda.synchronize()
                out.append(a)
                if captured:
                    del graph
    for a in out[1:]:
        for x, y in zip(a, out[0]):
            assert torch.equal(x, y)

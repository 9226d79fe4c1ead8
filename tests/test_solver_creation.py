"""A solver handle is ready when its creation returns: the first solve may run on a stream
that is not ordered behind the default stream, where creation puts its set-up."""
import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("masked", [False, True], ids=["plain", "masked"])
@pytest.mark.parametrize("shape", [(32, 48), (256, 320), (16, 16, 16)], ids=lambda s: "x".join(map(str, s)))
def test_first_solve_on_another_stream(fm, cuda, shape, masked):
    lib, g = fm._lib.lib(), fm.GridSpec(shape)
    cg = g.c_grid()
    P = fm._lib.MGParams(3, 2, 10, 0, 30, 0.0, 1e-8, 1e-12, 0, 0)
    side = torch.cuda.Stream()
    gen = torch.Generator(device=cuda).manual_seed(5)
    u = [torch.rand(g.face_shape(c), generator=gen, device=cuda, dtype=torch.float64) for c in range(g.dim)]
    out = []
    for busy in (False, True):
        h, a = C.c_void_p(), [x.clone() for x in u]
        torch.cuda.synchronize()
        if busy:
            torch.cuda._sleep(200_000_000)  # the default stream: about 0.1 s
        if masked:
            assert lib.fm_solid_create(C.byref(cg), 1, C.byref(P), None, C.byref(h)) == 0
        else:
            assert lib.fm_mgpcg_create(C.byref(cg), 1, C.byref(P), C.byref(h)) == 0
        assert torch.cuda.current_stream().query()  # nothing of the creation is left to run
        p = [x.data_ptr() for x in a] + [None] * (3 - g.dim)
        project = lib.fm_solid_project if masked else lib.fm_project
        assert project(h, *p, None, side.cuda_stream, None, None) == 0
        torch.cuda.synchronize()
        (lib.fm_solid_destroy if masked else lib.fm_mgpcg_destroy)(h)
        out.append(a)
    for x, y in zip(*out):
        assert torch.equal(x, y)

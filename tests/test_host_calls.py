"""The grid description that calls share: equal, hashable and picklable whether or
not a call has used it, with the face shapes and C struct of its cell counts."""
import copy
import pickle

import pytest


@pytest.mark.parametrize("shape", [(4, 5), (7, 4, 6)])
def test_grid_spec_after_use(fm, shape):
    g = fm.GridSpec(shape)
    g._ref, g._faces
    assert g._faces == tuple(g.face_shape(c) for c in range(g.dim))
    assert list(g._cgrid.n) == list(shape) + [1] * (3 - len(shape)) and g._cgrid.dim == len(shape)
    for h in (pickle.loads(pickle.dumps(g)), copy.deepcopy(g), fm.GridSpec(shape)):
        assert h == g and hash(h) == hash(g) and list(h._cgrid.n) == list(g._cgrid.n)

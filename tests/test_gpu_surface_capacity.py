"""A mesh that does not fit: the error names the counts that the mesh has, so that a tool made
with them holds it."""
import re

import numpy as np
import pytest
import torch

from nonnewton_b200 import _abi
from nonnewton_b200.engine import NNError
from nonnewton_b200.surface import SRTool

from .surf_cases import ball

pytestmark = pytest.mark.gpu


def _run(method, pos, vertices, indices):
    sr = SRTool([[0, 0, 0], [1, 1, 1]], voxel_size=0.01, particle_radius=0.02, max_num_vertices=vertices,
                max_num_indices=indices, max_num_particles=len(pos))
    getattr(sr, method)(0.0, 0.06, len(pos), torch.from_numpy(pos).cuda())
    return sr.mesh_vertex.cpu().numpy(), sr.mesh_index.cpu().numpy()


@pytest.mark.parametrize("method", ["dual_contouring", "marching_cubes"])
@pytest.mark.parametrize("short", ["vertices", "indices", "both"])
def test_error_names_the_counts_of_the_mesh(cuda_lib, method, short):
    pos = ball(seed=7, radius=0.12)
    v, f = _run(method, pos, 200000, 2000000)
    nv, ni = len(v), len(f)
    assert ni > 1000
    with pytest.raises(NNError) as e:
        _run(method, pos, nv - 1 if short != "indices" else nv, ni - 1 if short != "vertices" else ni)
    assert e.value.code == _abi.NN_ERR_CAPACITY
    assert re.search(r"\((\d+) vertices, (\d+) indices\)", str(e.value)).groups() == (str(nv), str(ni))
    with pytest.raises(NNError) as e:
        _run(method, pos, 100, 600)
    assert re.search(r"\((\d+) vertices, (\d+) indices\)", str(e.value)).groups() == (str(nv), str(ni))
    w, g = _run(method, pos, nv, ni)
    assert np.array_equal(w, v) and np.array_equal(g, f)

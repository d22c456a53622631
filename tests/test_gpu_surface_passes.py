"""The surface passes' own edges, against results that need no tolerance:
  - grids whose x extent leaves ragged rows of blocks, and meshes of a few particles
    (several warps share a particle's columns) equal the same set inside a larger grid,
    shifted by whole blocks: the field is fixed-point sums of values that do not depend on
    the grid's size;
  - a set given in another order has the same mesh (the sums are order-free; particle 0,
    which the pre-pass skips, stays first)."""
import numpy as np
import pytest
import torch

from nonnewton_b200.surface import SRTool

from .surf_cases import ball, block

pytestmark = pytest.mark.gpu


def _mesh(pos, box, method="dual_contouring", voxel=0.01, smooth=0.03):
    sr = SRTool([[0.0] * 3, box], voxel_size=voxel, particle_radius=0.02, record_normals=True,
                max_num_vertices=2000000, max_num_indices=6000000, max_num_particles=max(len(pos), 1))
    getattr(sr, method)(0.0, smooth, len(pos), torch.from_numpy(pos).cuda())
    return [t.cpu().numpy() for t in (sr.mesh_vertex, sr.mesh_index, sr.mesh_normal)]


@pytest.mark.parametrize("method", ["dual_contouring", "marching_cubes"])
@pytest.mark.parametrize("n,box", [((2, 1, 1), (0.5, 0.6, 0.55)), ((7, 5, 9), (0.61, 0.64, 0.7)),
                                   ((15, 17, 20), (0.83, 0.7, 0.95)), ((31, 30, 28), (1.02, 1.0, 1.0))])
def test_mesh_does_not_depend_on_the_grid_or_the_order(cuda_lib, n, box, method):
    pos = block(seed=3, n=n, corner=(0.2, 0.2, 0.2))
    v, f, nrm = _mesh(pos, list(box), method)
    assert (len(f) > 0) == (len(pos) > 100)  # two particles have no inside (and no smoothing width)
    big = _mesh(pos, [b + 0.37 for b in box], method)
    assert np.array_equal(v, big[0]) and np.array_equal(f, big[1]) and np.array_equal(nrm, big[2])
    order = np.concatenate([[0], 1 + np.random.default_rng(0).permutation(len(pos) - 1)])
    other = _mesh(pos[order], list(box), method)
    # the moments of the pre-pass are summed in another order: rounding only
    assert other[0].shape == v.shape and np.abs(other[0] - v).max(initial=0.0) <= 1e-5

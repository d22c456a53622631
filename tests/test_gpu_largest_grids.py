"""Grids of almost 2^31 cells, the largest that are accepted: loops over cells and the scan of
their counts end at the last cell, so a small set of particles has there what it has in a
grid that just holds it."""
import numpy as np
import pytest
import torch

from nonnewton_b200 import _abi
from nonnewton_b200 import scene as S
from nonnewton_b200.batch import Batch, scene_grid_cells
from nonnewton_b200.surface import SRTool

from .surf_cases import ball

pytestmark = pytest.mark.gpu


def _mesh(dims, pos, voxel=0.01, smooth=0.03):
    reach = 11  # vertices that the tool adds to the box at this smoothing radius
    sr = SRTool([[0.0] * 3, [(d - reach - 0.5) * voxel for d in dims]], voxel_size=voxel, particle_radius=0.02,
                record_normals=True, max_num_vertices=100000, max_num_indices=600000, max_num_particles=len(pos))
    assert sr.grid_dims(smooth) == list(dims)
    sr.dual_contouring(0.0, smooth, len(pos), torch.from_numpy(pos).cuda())
    out = [t.cpu().numpy() for t in (sr.mesh_vertex, sr.mesh_index, sr.mesh_normal)]
    sr.close()
    return out


@pytest.mark.parametrize("dims", [(1263, 1291, 1317), (1263, 1293, 1315)])  # 32 bytes a vertex
def test_surface_of_the_largest_grid(cuda_lib, dims):
    torch.cuda.empty_cache()
    if torch.cuda.mem_get_info()[0] < 90e9:
        pytest.skip("needs 69 GB of device memory")
    pos = ball(seed=5, radius=0.1)
    want = _mesh((111, 110, 109), pos)
    got = _mesh(dims, pos)
    assert len(want[1]) > 0
    for a, b in zip(got, want):
        assert np.array_equal(a, b)


def test_surface_of_the_most_particles(cuda_lib):
    """238,712,400 particles, whose 9 words of the anisotropic kernel each pass 2^31: the last
    particles' kernels are those of the last planes alone."""
    torch.cuda.empty_cache()
    if torch.cuda.mem_get_info()[0] < 90e9:
        pytest.skip("needs 50 GB of device memory")
    side, planes, vs = 620, 621, 0.01
    assert 9 * side * side * planes >= 2 ** 31

    def kernels(first):  # of the particles from plane `first` on
        i = torch.arange(first * side * side, planes * side * side, dtype=torch.int32, device="cuda")
        pos = torch.empty((len(i), 3), device="cuda")
        for k, c in enumerate((i % side, i // side % side, i // (side * side))):
            # on the lattice but for a tenth of a voxel, a hash of the index
            pos[:, k] = (c.float() + 0.4 + 0.1 * ((i % 1009) * (k + 7) % 101).float() / 101) * vs
        del i, c
        sr = SRTool([[0.0] * 3, [side * vs, side * vs, planes * vs]], voxel_size=vs, particle_radius=0.005,
                    max_num_vertices=1000, max_num_indices=6000, max_num_particles=len(pos))
        sr.dual_contouring(1e9, 0.0095, len(pos), pos)  # 26 neighbours; no surface at that level
        out = sr.stage(0, len(pos))["G"][-side * side:].clone()
        sr.close()
        return out

    got, want = kernels(0), kernels(planes - 8)
    torch.cuda.empty_cache()
    assert float(want.std()) > 0
    assert torch.allclose(got, want, rtol=1e-5, atol=1e-5 * float(want.abs().max()))


def _dam(extra=(0, 0, 0)):
    """A dam break whose domain goes on past its box by `extra` cells of the search grid."""
    sc = S.dam_break(seed=4, n_side=(9, 7, 8), box=0.4)
    edge = np.array([0.5, 1, 1]) * sc.param.support_radius * (1 + 1e-3)  # x cells are half as long
    sc.param.domain_end = np.asarray(sc.param.domain_end) + np.asarray(extra) * edge
    return sc


def _lists(scenes):
    b = Batch(sum(sc.particles.n for sc in scenes), len(scenes))
    b.set(scenes)
    b.engine.run_pass(_abi.NN_PASS_SEARCH)
    assert all(b.stats(k)["status"] == 0 for k in range(len(scenes)))
    out = b.engine.neighbors(b.n, 64)
    b.engine.close()
    return out


def test_lists_in_the_largest_search_grid(cuda_lib):
    """32,767 cells of 256 x 256 rows, a channel of 656 m: lists as in the box alone."""
    nx = scene_grid_cells(_dam(), x_split=2) // 1024  # 32 x 32 rows in the box's own grid
    far = _dam((32767 - nx, 200, 200))
    assert scene_grid_cells(far, x_split=2) == 32767 * 65536
    for a, b in zip(_lists([far]), _lists([_dam()])):
        assert torch.equal(a, b)
    # with a second scene the cells are 2^31 - 6,144: a scan tile (16,384) more would not fit an int
    assert scene_grid_cells(_dam((25, 0, 0)), x_split=2) == 58 * 1024
    for a, b in zip(_lists([far, _dam((25, 0, 0))]), _lists([_dam(), _dam()])):
        assert torch.equal(a, b)

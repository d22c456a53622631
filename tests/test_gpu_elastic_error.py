"""The elastic passes against the double build of the same kernels, on the same positions: the
kernel and its gradient take a correctly rounded square root and divisions. In a block
deformed by a tenth of its size and more, the strain does not cancel and what is left is the
rounding of these terms: a pair's gradient is about 8 roundings of 6e-8 and 26 pairs are
added, so a few 1e-7 (root mean square, of the field's). At a strain of 1 % the displacement
is what remains of positions a hundred times its size; it must not round at theirs (6e-6 a
component, 1 / sqrt(26) of it after the sum, more than twice that from R's own rounding)."""
import numpy as np
import pytest
import torch

from nonnewton_b200 import scene as S
from nonnewton_b200 import sph
from nonnewton_b200.config import SimConfig

pytestmark = pytest.mark.gpu


def _pass(sc, x, precision):
    m = sph.initialize(SimConfig(config=sc.config), particles=sc.particles, precision=precision)
    solver = sph.build_solver()
    solver.initialize()
    m.pd.x.copy_(x)
    m.ns.run_search()
    m.pd.acceleration.zero_()
    solver.elasticity_substep()
    el = m.pd.phase_id >= 3000
    return [getattr(m.pd, f)[el].double() for f in ("acceleration", "stress")]


@pytest.mark.parametrize("n_el,amplitude,bounds", [(12, 0.1, (5.4e-7, 3.4e-7)), (20, 0.3, (5.4e-7, 2.2e-7)),
                                                    (10, 0.01, (2.1e-6, 3.9e-6))])
def test_error_of_the_elastic_passes(cuda_lib, n_el, amplitude, bounds):
    sc = S.fluid_elastic(seed=0, n_el=n_el)
    x = torch.from_numpy(sc.particles.x).cuda()
    el = torch.from_numpy(sc.particles.phase_id).cuda() >= 3000
    c = x[el].double()
    side = float((c.amax(0) - c.amin(0)).amax())
    x[el] = (c + amplitude * side * torch.sin(2 * np.pi * (c[:, [1, 2, 0]] - c.amin(0)) / side)).float()
    for a, b, bound in zip(_pass(sc, x, "f32"), _pass(sc, x, "f64"), bounds):
        err = float((a - b).pow(2).mean().sqrt() / b.pow(2).mean().sqrt())
        assert err <= bound, err

"""Where the conjugate gradients reach their rounding level before the tolerance, the loop gives up soon and a further
correction follows: 1e4 in permeability between cells, a load on every row, a tolerance of 1e-12."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import vemgpu  # noqa: E402
from vemgpu import meshgen  # noqa: E402


@pytest.mark.parametrize("check_every", [0, 10])
@pytest.mark.parametrize("mode", ["fp64", "mixed"])
def test_loop_ends_at_its_rounding_level(mode, check_every):
    m = meshgen.voronoi_mesh(33, "disk", seed=4)
    rng = np.random.default_rng(33)
    theta = np.log(1e4) * (rng.random(33) < 0.3)
    g = vemgpu.DarcyGpu(m, k=0, geometry="arcs", problem="sinsin", bc="flux", theta=theta)
    for _ in range(8):
        b = torch.from_numpy(rng.standard_normal(g.N)).cuda()
        _, info = g.solve(b, mode=mode, tol=1e-12, check_every=check_every)
        # a loop takes some 25 iterations to its rounding level and 100 to give up; four corrections are enough
        assert info["residual"] <= 1e-12 and info["iterations"] <= 500
    g.close()

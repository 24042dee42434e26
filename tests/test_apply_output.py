"""vg_apply writes every row of its output, whatever the output held: flux rows are zeroed and summed into, each pressure row
and the multiplier's is stored by its owner."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import vemgpu  # noqa: E402
from vemgpu import meshgen  # noqa: E402
from test_edge_system import wheel  # noqa: E402


@pytest.mark.parametrize("bc", ["pressure", "flux"])
@pytest.mark.parametrize("mesh,k", [("wheel", 0), ("wheel", 1), ("wheel", 2), ("voronoi", 0), ("voronoi", 1),
                                    ("voronoi", 2), ("voronoi", 4)])  # a 16-gon of degree 4 exceeds the set-up kernel
def test_output_held_nan(k, mesh, bc):
    m = wheel() if mesh == "wheel" else meshgen.voronoi_mesh(97, "disk", seed=6)
    g = vemgpu.DarcyGpu(m, k=k, geometry="arcs" if "arc_nodes" in m else "identity", problem="sinsin", bc=bc)
    rng = np.random.default_rng(k)
    for dtype in (torch.float64, torch.float32):
        x = torch.from_numpy(rng.standard_normal(g.N)).cuda().to(dtype)
        for constrained in (True, False):
            for internal in (True, False):
                y = g.apply(x, constrained=constrained, out=torch.full_like(x, float("nan")), internal_order=internal)
                z = g.apply(x, constrained=constrained, out=torch.zeros_like(x), internal_order=internal)
                assert torch.isfinite(y).all() and torch.equal(y, z)
    g.close()

"""Small meshes of the problem without sources (csrc/vg_minres.cu). There ||div u_h|| is 0 and what vg_errors reports for
it is what the solve leaves in the pressure rows at its tolerance: a figure of the solver, kept what it has been."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import vemgpu  # noqa: E402
from vemgpu import fields, meshgen  # noqa: E402

# div_phys of one solve to 1e-10 on the seeded Voronoi annulus with the lognormal field (sigma 2, correlation length 0.1)
# of the given seed, as the library's MINRES has left it. Coarsest level below and above the finest, one and two loops.
RECORDED = {
    (500, "mixed", 3): 2.35796521e-10,
    (500, "fp64", 4): 1.80533479e-10,
    (1000, "mixed", 5): 1.06280976e-09,
    (2400, "mixed", 4): 1.36126941e-08,
    (2600, "fp64", 4): 1.52478647e-09,
    (8000, "mixed", 3): 5.58860573e-09,
    (8000, "fp64", 4): 3.13069769e-09,
}


def handle(cells, seed=None, **kw):
    m = meshgen.voronoi_mesh(cells, "annulus", seed=2026)
    theta = None
    if seed is not None:
        theta = fields.gaussian_field(fields.cell_centroids(m), sigma=2.0, corr=0.1, seed=seed, grid=512)
    return vemgpu.DarcyGpu(m, k=0, geometry="arcs", problem="annulus", bc="pressure", theta=theta, **kw), theta


@pytest.mark.parametrize("cells,mode,seed", sorted(RECORDED))
def test_divergence_figure_on_record(cells, mode, seed):
    """Rounding in the loop's FP64 scalars moves the figure by up to 1e-6 of itself, a bit of the coarsest inverse by
    1e-4 and more, another solver by a factor: 1e-5."""
    g, _ = handle(cells, seed)
    x, _ = g.solve(mode=mode)
    assert g.errors(x)["div_phys"] == pytest.approx(RECORDED[cells, mode, seed], rel=1e-5)
    g.close()


@pytest.mark.parametrize("cells", [1 << 15, (1 << 15) + 1])
def test_line_between_the_solvers(cells):
    """MINRES takes 80 to 100 iterations with the lognormal field, the conjugate gradients above the line 20 to 30; both
    end at the tolerance, and so they do after an update and from a guess."""
    g, theta = handle(cells, 5)
    for mode in ("fp64", "mixed"):
        x, info = g.solve(mode=mode)
        assert (info["iterations"] >= 60) == (cells <= 1 << 15)
        b = g.rhs()
        assert float((b - g.apply(x)).norm() / b.norm()) <= 2e-10
    g.set_log_permeability(-theta)
    y, info = g.solve(x=x.clone(), guess=True)
    b = g.rhs()
    assert info["residual"] <= 1e-10 and float((b - g.apply(y)).norm() / b.norm()) <= 2e-10
    g.close()


@pytest.mark.parametrize("cells", [5, 40, 2600])
def test_host_driven_batches(cells):
    """Batches of plain launches (check_every) do what the captured loop does, to the bit where both stop at the same
    iteration: with one iteration a batch."""
    g, _ = handle(cells, 7)
    for mode in ("fp64", "mixed"):
        x, a = g.solve(mode=mode)
        y, b = g.solve(mode=mode, check_every=1)
        assert a["iterations"] == b["iterations"] and torch.equal(x, y)
    g.close()

"""Maxwell-Stefan steps from states that are one pure species or another, cell by cell, with diffusivities far apart: the
friction of neighbouring cells differs by four to eight orders, and so does what the flux rows see of a jump between the
two sides of an edge (csrc/vg_ms.cu, ms_share)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from vemgpu import meshgen  # noqa: E402
from vemgpu.maxwell_stefan import MaxwellStefan  # noqa: E402


def pure(ms, seed=1):
    x1 = (np.random.default_rng(seed).random(ms.nc) < 0.5).astype(float)
    return ms.state(x1, 1.0 - x1)


@pytest.mark.parametrize("mode", ["fp64", "mixed"])
@pytest.mark.parametrize("dt", [1e-6, 1e-3, 1.0])
@pytest.mark.parametrize("D", [(1.0, 0.5, 0.2), (1.0, 1e-3, 1e2), (1e-4, 1e-4, 1.0)])
@pytest.mark.parametrize("cells", [33, 1500])
def test_linear_step(cells, D, dt, mode):
    ms = MaxwellStefan(meshgen.voronoi_mesh(cells, "disk", seed=4), D=D, dt=dt)
    s = pure(ms)
    out, info = ms.step(s, mode=mode, tol=1e-10)
    assert info["residual"] <= 1e-10
    b = torch.zeros_like(s)
    b[2 * ms.nf:] = s[2 * ms.nf:] * ms.areas.repeat(2) / dt
    # the step's own figure, to the rounding of the other summation order
    assert float((ms.apply(s, out) - b).norm() / b.norm()) <= 2e-10
    ms.close()


@pytest.mark.parametrize("mode", ["fp64", "mixed"])
@pytest.mark.parametrize("cells,D,dt", [(33, (1.0, 1e-3, 1e2), 1e-3), (33, (1.0, 1e-3, 1e2), 1.0),
                                        (1500, (1.0, 1e-3, 1e2), 1e-3), (1500, (1e-4, 1e-4, 1.0), 1.0)])
def test_picard_where_forced_solves_contract_slowly(cells, D, dt, mode):
    """Solved linear systems take two to six iterations here; with forced ones the iteration contracts by a half. In
    place and out of place are the same step, also where it starts again."""
    ms = MaxwellStefan(meshgen.voronoi_mesh(cells, "disk", seed=6), D=D, dt=dt, picard=20)
    s = pure(ms)
    out, info = ms.step(s, mode=mode, tol=1e-11)
    assert info["picard"] <= 20 and info["residual"] <= 1e-11
    assert info["picard_change"] <= 1e-10 and info["nonlinear_residual"] <= 1e-10
    t = s.clone()
    ms.step(t, out=t, mode=mode, tol=1e-11)
    assert torch.equal(out, t)
    ms.close()

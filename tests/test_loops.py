"""The three forms of the conjugate gradient loop: one cooperative launch (small meshes), a captured graph (above the line),
and host-driven batches of plain launches (check_every), which run the graph's kernels on any mesh."""
import numpy as np
import pytest
import scipy.sparse.linalg as spla

import oracle as O
from test_edge_system import CASES, MESHES, constrained_matrix, tolerance

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import vemgpu  # noqa: E402
from vemgpu import meshgen  # noqa: E402
from vemgpu.core import default_nq  # noqa: E402


@pytest.mark.parametrize("bc", ["pressure", "flux"])
@pytest.mark.parametrize("name,k", CASES)
def test_host_driven_batches_match_sparse_lu(name, k, bc):
    """The streamed and strided applies, records larger than a stage (the 16-gon at degree 1), and the loop's kernels on
    odd and tiny sizes, against a sparse LU; the bound of test_edge_system.test_solve_matches_sparse_lu."""
    m = MESHES[name]()
    nc = len(m["cell_ptr"]) - 1
    rng = np.random.default_rng(10 * k + nc + 1)
    theta = rng.normal(0, 1.0, nc)
    arcs = "arc_nodes" in m
    o = O.Oracle(m, k=k, nq=default_nq(k), ng=9, geom=O.GEOM_ARCS if arcs else O.GEOM_IDENTITY, problem=O.PROB_SINSIN,
                 bc=O.BC_PRESSURE if bc == "pressure" else O.BC_FLUX, theta=theta)
    g = vemgpu.DarcyGpu(m, k=k, geometry="arcs" if arcs else "identity", problem="sinsin", bc=bc, theta=theta)
    K = constrained_matrix(o)
    b = rng.standard_normal(g.N)
    lu = spla.splu(K)
    ref = lu.solve(b)
    ref += lu.solve(b - K @ ref)
    smin = np.linalg.svd(K.toarray(), compute_uv=False)[-1]
    tol = tolerance(k)
    for mode in ("fp64", "mixed"):
        for check_every in (1, 7):
            x, info = g.solve(torch.from_numpy(b).cuda(), mode=mode, tol=tol, check_every=check_every)
            assert info["residual"] <= tol
            assert np.linalg.norm(x.cpu().numpy() - ref) <= 2 * tol * np.linalg.norm(b) / smin, (mode, check_every, info)
    g.close()


# just above 64,000 / (k + 1) cells; at degree 4 above 148 pieces of 32 cells
@pytest.mark.parametrize("bc", ["pressure", "flux"])
@pytest.mark.parametrize("k,cells", [(0, 64001), (1, 32001), (2, 21334), (3, 16001), (4, 5500)])
def test_graph_above_the_line(k, cells, bc):
    """The graph runs two iterations a body, the second one empty where the first converged: to the bit what batches of
    one iteration do."""
    g = vemgpu.DarcyGpu(meshgen.voronoi_mesh(cells, "disk", seed=7), k=k, geometry="arcs", problem="sinsin", bc=bc)
    b = g.rhs()
    for mode in ("fp64", "mixed"):
        if k == 4 and mode == "mixed":
            continue  # FP32 blocks of this mesh still fit the single launch
        x, info = g.solve(b, mode=mode, tol=1e-10)
        y, batches = g.solve(b, mode=mode, tol=1e-10, check_every=1)
        assert info["residual"] <= 1e-10 and info["iterations"] == batches["iterations"]
        assert torch.equal(x, y)
        assert float((b - g.apply(x)).norm() / b.norm()) <= 2e-10
    g.close()


@pytest.mark.parametrize("k,cells", [(3, 3600), (4, 3600), (3, 5500), (4, 5500)])
def test_high_degrees_on_both_sides_of_the_line(k, cells):
    """FP64 and mixed, each by one launch or the graph as the blocks of its precision fit: both end at the tolerance and
    agree to the error it allows in the pressures (condition of the mean rows, 1e4 at these sizes)."""
    g = vemgpu.DarcyGpu(meshgen.voronoi_mesh(cells, "disk", seed=7), k=k, geometry="arcs", problem="sinsin", bc="pressure")
    b = g.rhs()
    xs = []
    for mode in ("fp64", "mixed"):
        x, info = g.solve(b, mode=mode, tol=1e-11)
        assert info["residual"] <= 1e-11
        xs.append(x)
    assert float((xs[0] - xs[1]).norm()) <= 2e-7 * float(xs[0].norm())
    g.close()

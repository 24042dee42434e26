// MINRES on the saddle-point form of small meshes without sources.
//
// Replaces the PETSc FGMRES of vem/CurvedVEM_Darcy_gpu/src/krylov.cu:49-175, as vg_hybrid.cu does on every other
// system. Preconditioned MINRES (Paige-Saunders) on the symmetric form
//     [A, -W^T; -W, 0] [u; p] = [g; -f]
// with the inverse diagonal of A on the flux rows and a multigrid V-cycle for S = W diag(A)^{-1} W^T, the cells' graph
// with conductances 1 / A_ii across an edge, on the pressure rows. Per iteration:
//   apply       y = K z_j and delta_j = z_j^T K z_j (fused, vg_apply.cu)
//   update      v_{j+1} = y/g_j - (delta_j/g_j^2) v_j - (g_j/g_{j-1}) v_{j-1}, y = 0; the flux rows (with their z and
//               z.v) on a second stream beside the pressure rows and the V-cycle
//   finish      gamma_{j+1} = sqrt(z_{j+1}.v_{j+1}), Givens rotation, residual estimate (device scalars)
//   step        w_{j+1} = (z_j/g_j - a3 w_{j-1} - a2 w_j)/a1, x += c_{j+1} eta_j w_{j+1}
// FP64, or FP32 under FP64 refinement; the true FP64 residual decides in both modes.
//
// Why it stays beside the conjugate gradients of vg_hybrid.cu, which need a fifth of its time (8,000 cells, mixed: 0.55
// against 2.9 ms a solve): on a problem without sources the divergence that vg_errors reports has nothing but the solve
// in it, ||div u_h|| being the residual of the pressure rows at the tolerance. The figures on record of such meshes are
// MINRES's (8,000 cells, mixed: 5.6e-9), and another solver's residual at the same tolerance is another number (1.0e-9),
// although the solutions agree to 1e-12. The figures are kept; the price is time.
#include <algorithm>
#include <cmath>

#include "vg_krylov.cuh"
#include "vg_solver.hpp"

namespace vg {

namespace {

// Largest mesh that keeps MINRES: figures are on record up to 30,000 cells. A mesh that is created, built and solved once
// takes, in ms, MINRES against conjugate gradients: 500 cells 10.6 against 6.7, 2,400 87 against 14 (its graph is the
// coarsest level, which is inverted pivot by pivot), 8,000 33 against 23, 30,000 76 against 70. Larger meshes are solved
// many times rather than once, and there the solve decides (250,000 cells: 6.6 against 2.5 ms, 1,000,000: 14.3 against 4.9).
constexpr int MINRES_CELLS = 1 << 15;
constexpr int MT = 256;

// d += A_ii on every flux row (two addends at most onto zero)
__global__ void k_flux_diagonal(const double* A, const int* map, const Piece* pieces, int npieces, double* d) {
    const long long t = blockIdx.x * (long long)MT + threadIdx.x;
    const int pc = int(t / PIECE), lane = int(t % PIECE);
    if (pc >= npieces) return;
    const Piece& P = pieces[pc];
    if (lane >= P.count) return;
    for (int i = 0; i < P.n; ++i) {
        const int g = map[P.map_off + (long long)i * PIECE + lane];
        atomicAdd(d + (g < 0 ? ~g : g), A[P.a_off + (long long)(i * P.n - i * (i - 1) / 2) * PIECE + lane]);
    }
}

__global__ void k_flux_inverse(double* d, float* d32, long long n) {
    for (long long i = blockIdx.x * (long long)MT + threadIdx.x; i < n; i += (long long)gridDim.x * MT) {
        const double v = 1.0 / fmax(fabs(d[i]), 1e-300);
        d[i] = v;
        d32[i] = float(v);
    }
}

// the conductances in the edges' own order (vg_hybrid.cu)
__global__ void k_flux_conductance(const double* dinv, const int* map, const int* emap, const Piece* pieces, int npieces,
                                   double* cond) {
    const long long t = blockIdx.x * (long long)MT + threadIdx.x;
    const int pc = int(t / PIECE), lane = int(t % PIECE);
    if (pc >= npieces) return;
    const Piece& P = pieces[pc];
    if (lane >= P.count) return;
    for (int i = 0; i < P.ne; ++i) {
        const int g = map[P.map_off + (long long)i * PIECE + lane];
        cond[emap[P.e_off + (long long)i * PIECE + lane]] = dinv[g < 0 ? ~g : g];  // both cells write the same value
    }
}

template <typename T>
auto& of(DevBuf<double>& d64, DevBuf<float>& d32) {
    if constexpr (sizeof(T) == 8)
        return d64;
    else
        return d32;
}

}  // namespace

bool Solver::minres_mesh() const {
    return k == 0 && bc == VG_BC_PRESSURE && problem == VG_PROBLEM_ANNULUS && m.nc <= MINRES_CELLS;
}

// preconditioner for the current permeability: on the first call after vg_build the whole hierarchy, the values alone
// (same addresses, so that captured loops stay valid) after an update. False when the cells' graph does not coarsen.
bool Solver::prepare_minres() {
    ArenaScope scope(arena_);
    auto& M = minres_;
    const int npieces = int(pieces_.size()), blocks = int(((long long)npieces * PIECE + MT - 1) / MT);
    M.dinv64.resize(nf);
    M.dinv32.resize(nf);
    M.dinv64.zero();
    k_flux_diagonal<<<blocks, MT>>>(d_A64_.data(), d_map_int_.data(), d_pieces_.data(), npieces, M.dinv64.data());
    k_flux_inverse<<<148, MT>>>(M.dinv64.data(), M.dinv32.data(), nf);
    VG_CUDA(cudaGetLastError());
    if (M.ready) {
        if (!edges_planned_) {
            plan_edges();
            edges_planned_ = true;
        }
        M.cond.resize(m.ne);
        M.values.resize(size_t(M.amg.level0_nnz()));
        k_flux_conductance<<<blocks, MT>>>(M.dinv64.data(), d_map_int_.data(), d_emap_.data(), d_pieces_.data(), npieces,
                                           M.cond.data());
        VG_CUDA(cudaGetLastError());
        laplacian_values(M.amg, M.cond.data(), M.values.data());
        M.amg.refresh(M.values.data());
        return true;
    }
    destroy_minres_graphs();  // they hold the previous hierarchy's addresses
    const std::vector<double> inner = M.dinv64.download();
    std::vector<double> cond(m.ne);
    for (int e = 0; e < m.ne; ++e) cond[e] = inner[e2i_host_[e]];
    const HostCsr S = cell_graph(cond);
    const std::vector<int> order = rank_order();
    try {
        M.amg.setup(S, d_errp_, &order, false, true);
    } catch (const Error& e) {
        if (e.code == VG_ENOMEM || e.code == VG_ECUDA) throw;
        return false;
    }
    for (auto& b : M.w64) b.resize(N);
    for (auto& b : M.w32) b.resize(N);
    M.r32.resize(N);
    M.scal.resize(sizeof(MinresScalars) / sizeof(double));
    M.flags.resize(NFLAGS);
    return M.ready = true;
}

template <typename T>
MinresVecs<T> Solver::minres_vecs() {
    T* p[8];
    for (int i = 0; i < 8; ++i) p[i] = of<T>(minres_.w64[i], minres_.w32[i]).data();
    return MinresVecs<T>{p[0], p[1], p[2], p[3], p[4], p[5], p[6], p[7],
                         of<T>(minres_.dinv64, minres_.dinv32).data(), nf, N};
}

template <typename T>
void Solver::minres_iteration(MinresVecs<T>& v, cudaStream_t s) {
    MinresScalars* sc = reinterpret_cast<MinresScalars*>(minres_.scal.data());
    int* flags = minres_.flags.data();
    double* part = d_partials_.data();
    unsigned* ctr = d_counter_.data();
    launch_apply(apply_args<T>(v.z_cur, v.y, true, T(-1), &sc->delta, flags), s);
    // the flux rows of the update (bandwidth-bound) run on a second stream beside the pressure rows and the V-cycle
    // (latency-bound); both join before the scalar update
    VG_CUDA(cudaEventRecord(ev_fork_, s));
    VG_CUDA(cudaStreamWaitEvent(side_, ev_fork_, 0));
    minres_update<T>(v, true, sc, flags, part, ctr, side_);
    VG_CUDA(cudaEventRecord(ev_join_, side_));
    minres_update<T>(v, false, sc, flags, part, ctr, s);
    minres_.amg.vcycle(v.v_old + nf, v.z_new + nf, s);
    VG_CUDA(cudaStreamWaitEvent(s, ev_join_, 0));
    minres_finish<T>(v.z_new, v.v_old, nf, N, false, 0.0, sc, flags, part, ctr, s);
    minres_step<T>(v, sc, flags, s);
    std::swap(v.v_cur, v.v_old);
    std::swap(v.z_cur, v.z_new);
    std::swap(v.w_cur, v.w_old);
}

// the loop as a CUDA graph: a conditional while node whose body is two iterations (the vector roles repeat with period
// two) followed by the condition kernel, the body count capped on the device
template <typename T>
void Solver::minres_build_graph(int p) {
    auto& M = minres_;
    VG_CUDA(cudaGraphCreate(&M.graph[p], 0));
    cudaGraphConditionalHandle h;
    VG_CUDA(cudaGraphConditionalHandleCreate(&h, M.graph[p], 1, cudaGraphCondAssignDefault));
    cudaGraphNodeParams cp{};
    cp.type = cudaGraphNodeTypeConditional;
    cp.conditional.handle = h;
    cp.conditional.type = cudaGraphCondTypeWhile;
    cp.conditional.size = 1;
    cudaGraphNode_t node;
    VG_CUDA(cudaGraphAddNode(&node, M.graph[p], nullptr, 0, &cp));
    cudaGraph_t body = cp.conditional.phGraph_out[0];
    VG_CUDA(cudaStreamBeginCaptureToGraph(stream_, body, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal));
    MinresVecs<T> v = minres_vecs<T>();
    const long long saved = M.amg.launches;
    try {
        minres_iteration<T>(v, stream_);
        minres_iteration<T>(v, stream_);
        loop_check(h, M.flags.data(), d_loop_.data(), stream_);
    } catch (...) {
        cudaGraph_t dummy;
        cudaStreamEndCapture(stream_, &dummy);
        throw;
    }
    M.amg.launches = saved;
    VG_CUDA(cudaStreamEndCapture(stream_, &body));
    VG_CUDA(cudaGraphInstantiate(&M.gexec[p], M.graph[p], 0));
}

void Solver::destroy_minres_graphs() {
    for (int p = 0; p < 2; ++p) {
        if (minres_.gexec[p]) cudaGraphExecDestroy(minres_.gexec[p]);
        if (minres_.graph[p]) cudaGraphDestroy(minres_.graph[p]);
        minres_.gexec[p] = nullptr;
        minres_.graph[p] = nullptr;
    }
}

// the symmetric system for the right-hand side r from zero, into the loop's vector x (minres_vecs); the iterations
template <typename T>
int Solver::minres_loop(const T* r, double tol, int maxit, int check_every, cudaStream_t s) {
    auto& M = minres_;
    MinresScalars* sc = reinterpret_cast<MinresScalars*>(M.scal.data());
    int* flags = M.flags.data();
    const int p = sizeof(T) == 4 ? 1 : 0;
    const bool graph = check_every <= 0;
    if (graph && !M.gexec[p]) minres_build_graph<T>(p);
    MinresVecs<T> v = minres_vecs<T>();
    VG_CUDA(cudaMemsetAsync(v.x, 0, sizeof(T) * N, s));
    minres_init<T>(r, v, sc, d_partials_.data(), d_counter_.data(), s);
    M.amg.vcycle(v.v_cur + nf, v.z_cur + nf, s);
    minres_finish<T>(v.z_cur, v.v_cur, nf, N, true, tol, sc, flags, d_partials_.data(), d_counter_.data(), s);
    int h_flags[NFLAGS] = {0, 0, 0, 0};
    if (graph) {
        const int loop[2] = {0, (maxit + 1) / 2};
        VG_CUDA(cudaMemcpyAsync(d_loop_.data(), loop, sizeof(loop), cudaMemcpyHostToDevice, s));
        VG_CUDA(cudaGraphLaunch(M.gexec[p], s));
        VG_CUDA(cudaMemcpyAsync(h_flags, flags, sizeof(h_flags), cudaMemcpyDeviceToHost, s));
        VG_CUDA(cudaStreamSynchronize(s));
    } else {
        // host-driven batches of check_every iterations (every kernel is a plain launch)
        for (int done = 0; done < maxit;) {
            const int batch = std::min(check_every, maxit - done);
            for (int it = 0; it < batch; ++it) minres_iteration<T>(v, s);
            done += batch;
            VG_CUDA(cudaMemcpyAsync(h_flags, flags, sizeof(h_flags), cudaMemcpyDeviceToHost, s));
            VG_CUDA(cudaStreamSynchronize(s));
            if (h_flags[0]) break;
        }
    }
    const int iters = h_flags[2];
    // start and the first cycle; per iteration apply, the two updates, cycle (residual, restriction, prolongation per
    // level, dense product), finish, step; the condition kernel per body
    const long long vc = 3LL * (M.amg.levels() - 1) + 1;
    n_launch += 2 + vc + (5 + vc) * iters + (iters + 2) / 2;
    n_apply += iters;
    n_iter += iters;
    return iters;
}

// corrections of x (internal order) until the true residual is at most the tolerance: FP64 to a tenth of it (the
// reference's KSP factor, krylov.cu:142) with at most two restarts (krylov.cu:136-170), or FP32 ones, each asked for
// inner_tol, or less when less reaches the tolerance. residual() leaves the residual in r and returns its relative norm.
void Solver::minres_solve(double* x, const double* r, double nb, const vg_solve_opts& o,
                          const std::function<double()>& residual, double& rel, int& total, int& outer, cudaStream_t s) {
    const bool fp64 = o.mode == VG_SOLVE_FP64;
    const int steps = fp64 ? 3 : o.max_outer;
    for (outer = 0; outer < steps && rel > o.tol && total < o.maxit; ++outer) {
        const double rn = rel * nb;
        if (fp64) {
            total += minres_loop<double>(r, std::min(0.5, 0.1 * o.tol * nb / rn), o.maxit - total, o.check_every, s);
            axpy64(x, minres_vecs<double>().x, 1.0, s);
            n_launch += 1;
        } else {
            to_float(r, minres_.r32.data(), 1.0 / rn, N, s);
            const double itol = std::min(0.5, std::max(o.inner_tol, 0.1 * o.tol / rel));
            total += minres_loop<float>(minres_.r32.data(), itol, o.maxit - total, o.check_every, s);
            axpy_from_float(x, minres_vecs<float>().x, rn, N, s);
            n_launch += 2;
        }
        rel = residual();
    }
}

}  // namespace vg

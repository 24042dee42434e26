// The hybridised system: conjugate gradients on edge pressures.
//
// With the fluxes of each cell taken apart (v_i = outward moments of the cell's own edges, then the
// interior moments) and one pressure unknown lambda per edge moment that ties the two sides together,
// a cell's rows of the saddle-point system read
//     A_E v - W_E^T p + c lambda = beta,   W_E v = f,      sum over the sides of c v = 0,
// with c = +1 on even moments and +-1 by the side's direction on odd ones. A cell alone gives
//     v = T (beta - c lambda) + Y f,   p = Z f - Y^T (beta - c lambda),
//     Z = (W A^{-1} W^T)^{-1},  Y = A^{-1} W^T Z,  T = A^{-1} - Y W A^{-1},
// and what is left is  S lambda = h,  S = sum c T c  over the edge moments: symmetric, positive definite
// (the pressure condition fixes lambda on the boundary) or semi-definite with the constants as its
// kernel (normal flux given, the multiplier then fixes the mean). K_E = e^theta I scales T by e^theta
// and Z by e^-theta and leaves Y.
//
// Why: MINRES on the saddle-point form with a block-diagonal preconditioner pays for its indefinite
// spectrum; on S the same multigrid serves conjugate gradients in a third of the iterations, on
// vectors of 3 instead of 4 unknowns per cell (k = 0). With T's diagonal in the place of T, S has the
// exact inverse  D^{-1} + Pi L^{-1} Pi^T: Pi takes a cell's pressure to its edges with the weights
// T_ii / D and L is the graph Laplacian of the cells with conductances 1 / (1 / T_ii + 1 / T_jj) across
// an edge. That is the preconditioner, with a V-cycle for L^{-1} (mean moments only: the higher moments
// have the diagonal), so one scalar hierarchy on the cells serves every degree and both conditions.
// The spectrum of T against its diagonal bounds the iterations whatever the mesh and the contrast.
//
// Right-hand side, back substitution and residuals are FP64 in both modes; MIXED runs the conjugate
// gradients in FP32. Loads on a shared edge are split between its cells, and the two sides' fluxes
// averaged, with the weights 1 - T_ii / D: the side of the higher resistance counts more, so that the
// remaining jump disturbs the flux rows least.
#include <algorithm>
#include <cmath>

#include "vg_apply.cuh"
#include "vg_krylov.cuh"
#include "vg_small.cuh"
#include "vg_solver.hpp"

namespace vg {

namespace {

// Largest mesh of degree 0 whose loop runs as one launch (vg_small.cu), and at degree k a (k + 1)th of it. What ends the
// gain is that a CTA's constants no longer fit its shared memory and that its pieces follow one another. At degree 4 the
// condensed blocks alone decide, which grow with (k + 1)^2 and come in whole pieces: a CTA holds SMALL_BLOCKS bytes of
// them at most (one piece in FP64, two in FP32). One launch against one kernel per phase, ms per solve to 1e-10 (disk;
// FP64, then mixed; the graph's vary by a tenth and more with the handle's place in memory at degrees 2 to 4):
//   k = 0   30,000 0.67 : 0.91, 0.67 : 0.96    60,000 0.95 : 1.03, 0.95 : 1.14    64,000 1.15 : 1.02, 1.15 : 1.07
//   k = 1   16,000 1.33 : 1.90, 1.07 : 1.51    32,000 2.04 : 2.16, 1.89 : 2.28    45,000 2.70 : 2.33, 2.37 : 2.49
//   k = 2   12,000 6.8 : 9.1, 6.2 : 8.1        21,000 12.1 : 14.4, 8.5 : 9.1      30,000 12.5 : 10.7, 9.5 : 9.2
//   k = 3    4,000 15.7 : 28.2, 15.9 : 22.2     8,000 36 : 31, 20 : 26            16,000 46 : 60, 26 : 30
//   k = 4    4,000 55 : 105, 43 : 64            8,000 134 : 110, 59 : 73          12,800 157 : 142, 126 : 84
constexpr long long SMALL_BLOCKS = 120 << 10;
constexpr int SMALL_CELLS = 64000;
constexpr int HT = 256;
inline int hblocks(long long n) { return int((n + HT - 1) / HT); }

__device__ __forceinline__ bool hyb_slot(const Piece* pieces, int npieces, Piece& P, int& lane) {
    const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    const int pc = int(t / PIECE);
    lane = int(t % PIECE);
    if (pc >= npieces) return false;
    P = pieces[pc];
    return lane < P.count;
}

__device__ __forceinline__ int tri(int i, int j, int n) { return i * n - i * (i - 1) / 2 + (j - i); }  // i <= j

// sign c of a side's moment i (i / ne the moment's degree)
__device__ __forceinline__ double side_sign(const signed char* esgn, const Piece& P, int i, int lane) {
    return esgn && (i / P.ne) % 2 ? double(esgn[P.e_off + (long long)(i % P.ne) * PIECE + lane]) : 1.0;
}

// in-place sweep of a symmetric positive definite matrix, one warp: a <- -a^{-1}; col: n scratch values
__device__ bool warp_sweep(double* a, double* col, int n, int lane) {
    bool ok = true;
    for (int k = 0; k < n; ++k) {
        for (int i = lane; i < n; i += 32) col[i] = a[i * n + k];
        __syncwarp();
        const double d = col[k], inv = 1.0 / d;
        if (!(d > 0) || !isfinite(inv)) ok = false;
        for (int z = lane; z < n * n; z += 32) {
            const int i = z / n, j = z % n;
            if (i == k && j == k)
                a[z] = -inv;
            else if (i == k)
                a[z] = col[j] * inv;
            else if (j == k)
                a[z] = col[i] * inv;
            else
                a[z] -= col[i] * col[j] * inv;
        }
        __syncwarp();
    }
    return ok;
}

// T (packed like A_E), Y (n x q, stored r n + i) and Z (packed) of every cell for K = I: one warp a cell,
// matrices in shared memory (n^2 + 2 n q + q^2 + n doubles). Set-up only.
__global__ void k_condense(const double* A, const double* W, const Piece* pieces, int npieces, int k, int words,
                           double* T, double* Y, double* Z, unsigned long long* status, const int* slot_cell) {
    extern __shared__ double hsm[];
    const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31, wpb = blockDim.x >> 5;
    const long long c = blockIdx.x * (long long)wpb + wid;
    if (c >= (long long)npieces * PIECE) return;
    const Piece P = pieces[c / PIECE];
    const int l = int(c % PIECE);
    if (l >= P.count) return;
    const int n = P.n, q = (k + 1) * (k + 2) / 2, nz = q * (q + 1) / 2;
    double* a = hsm + (size_t)wid * words;
    double *y = a + n * n, *w = y + n * q, *m = w + n * q, *col = m + q * q;
    for (int z = lane; z < n * n; z += 32) {
        const int i = z / n, j = z % n;
        a[z] = A[P.a_off + (long long)tri(min(i, j), max(i, j), n) * PIECE + l];
    }
    for (int z = lane; z < q * n; z += 32) w[z] = k == 0 ? 1.0 : W[P.w_off + (long long)z * PIECE + l];
    __syncwarp();
    bool ok = warp_sweep(a, col, n, lane);
    for (int z = lane; z < q * n; z += 32) {  // y = A^{-1} W^T, stored r n + i
        const int r = z / n, i = z % n;
        double s = 0;
        for (int j = 0; j < n; ++j) s -= a[i * n + j] * w[r * n + j];
        y[z] = s;
    }
    __syncwarp();
    for (int z = lane; z < q * q; z += 32) {
        const int r = z / q, t = z % q;
        double s = 0;
        for (int j = 0; j < n; ++j) s += w[r * n + j] * y[t * n + j];
        m[z] = s;
    }
    __syncwarp();
    ok = warp_sweep(m, col, q, lane) && ok;
    if (!ok && lane == 0) set_status(status, ST_SINGULAR, slot_cell[P.slot + l]);
    for (int z = lane; z < q * n; z += 32) {  // Y = y Z, into w
        const int r = z / n, i = z % n;
        double s = 0;
        for (int t = 0; t < q; ++t) s -= y[t * n + i] * m[t * q + r];
        w[z] = s;
    }
    __syncwarp();
    for (int z = lane; z < n * n; z += 32) {
        const int i = z / n, j = z % n;
        if (j < i) continue;
        double s = -a[z];
        for (int t = 0; t < q; ++t) s -= w[t * n + i] * y[t * n + j];
        T[P.a_off + (long long)tri(i, j, n) * PIECE + l] = s;
    }
    for (int z = lane; z < q * n; z += 32) Y[P.hw_off + (long long)z * PIECE + l] = w[z];
    for (int z = lane; z < q * q; z += 32) {
        const int i = z / q, j = z % q;
        if (j >= i) Z[P.slot * nz + (long long)tri(i, j, q) * PIECE + l] = -m[z];
    }
}

// D += e^theta T_ii per edge moment; R += 1 / (e^theta T_ii) per edge (means). Two addends at most onto zero.
__global__ void k_edge_diag(const double* T, const double* theta, const int* slot_cell, const int* emap,
                            const Piece* pieces, int npieces, int k, long long edges, double* D, double* R) {
    Piece P;
    int lane;
    if (!hyb_slot(pieces, npieces, P, lane)) return;
    const double et = exp(theta[slot_cell[P.slot + lane]]);
    for (int i = 0; i < (k + 1) * P.ne; ++i) {
        const long long g = (i / P.ne) * edges + emap[P.e_off + (long long)(i % P.ne) * PIECE + lane];
        const double t = et * T[P.a_off + (long long)tri(i, i, P.n) * PIECE + lane];
        atomicAdd(D + g, t);
        if (i < P.ne) atomicAdd(R + g, 1.0 / t);
    }
}

// inverse diagonal (0 on a boundary edge whose pressure is given), and as the preconditioner uses it; conductances of the cells' graph: 1 / R,
// on a boundary edge T_ii to the given pressure or none with the flux given
__global__ void k_edge_scale(const double* D, const double* R, const int2* ecell, long long edges, long long n,
                             int flux_bc, double* dinv, double* relaxed, float* relaxed32, double* cond) {
    for (long long i = blockIdx.x * (long long)HT + threadIdx.x; i < n; i += (long long)gridDim.x * HT) {
        const long long e = i % edges;
        const int2 c = ecell[e];
        const bool boundary = c.x == c.y;
        const double d = D[i];
        const double v = !(boundary && !flux_bc) && d > 0 && isfinite(d) ? 1.0 / d : 0.0;
        dinv[i] = v;
        relaxed[i] = EDGE_RELAX * v;
        relaxed32[i] = float(EDGE_RELAX * v);
        if (i < edges) cond[i] = boundary && flux_bc ? 0.0 : 1.0 / R[i];
    }
}

// condensed blocks into the record streams (and the strided arrays, where a kernel reads them), interpolation
// weights per (cell, edge) and per edge
struct ValueArgs {
    const double *T, *theta, *dinv;
    const int *slot_cell, *emap;
    const signed char* esgn;
    const Piece* pieces;
    int npieces, k;
    long long edges;
    const int2* ecell;
    unsigned char *rec64, *rec32;
    const long long *roff64, *roff32;
    double *S64, *cw64, *ew64;
    float *S32, *cw32, *ew32;
};
__global__ void k_edge_values(ValueArgs a) {
    const long long t = blockIdx.x * (long long)HT + threadIdx.x;
    const int pc = int(t / PIECE), lane = int(t % PIECE);
    if (pc >= a.npieces) return;
    const Piece P = a.pieces[pc];
    const int ne = P.ne, ed = (a.k + 1) * ne;
    const bool live = lane < P.count;
    double *r64 = nullptr;
    float* r32 = nullptr;
    if (a.rec64) {
        unsigned char *b64 = a.rec64 + a.roff64[pc], *b32 = a.rec32 + a.roff32[pc];
        if (lane == 0) {
            *reinterpret_cast<int4*>(b64) = make_int4(ne, 0, P.count, int(a.roff64[pc + 1] - a.roff64[pc]));
            *reinterpret_cast<int4*>(b32) = make_int4(ne, 0, P.count, int(a.roff32[pc + 1] - a.roff32[pc]));
        }
        r64 = reinterpret_cast<double*>(b64 + 16) + lane;
        r32 = reinterpret_cast<float*>(b32 + 16) + lane;
        int* m64 = reinterpret_cast<int*>(b64 + 16 + 8ll * PIECE * (ed * (ed - 1) / 2)) + lane;
        int* m32 = reinterpret_cast<int*>(b32 + 16 + 4ll * PIECE * (ed * (ed - 1) / 2)) + lane;
        for (int e = 0; e < ne; ++e) {
            const int g = live ? a.emap[P.e_off + (long long)e * PIECE + lane] : 0;
            m64[e * PIECE] = g;
            m32[e * PIECE] = g;
        }
    }
    const double et = live ? exp(a.theta[a.slot_cell[P.slot + lane]]) : 0.0;
    if (live)
        for (int e = 0; e < ne; ++e) {
            const long long o = P.e_off + (long long)e * PIECE + lane;
            const int g = a.emap[o];
            const double w = et * a.T[P.a_off + (long long)tri(e, e, P.n) * PIECE + lane] * a.dinv[g];
            a.cw64[o] = w;
            a.cw32[o] = float(w);
            if (a.ecell[g].x == P.rank0 + lane) {
                a.ew64[g] = w;
                a.ew32[g] = float(w);
            }
        }
    long long z = 0;
    for (int i = 1; i < ed; ++i)
        for (int j = i; j < ed; ++j, ++z) {
            const double v = live ? et * a.T[P.a_off + (long long)tri(i, j, P.n) * PIECE + lane] *
                                        (side_sign(a.esgn, P, i, lane) * side_sign(a.esgn, P, j, lane))
                                  : 0.0;
            if (r64) {
                r64[z * PIECE] = v;
                r32[z * PIECE] = float(v);
            }
            if (a.S64) {
                a.S64[P.s_off + z * PIECE + lane] = v;
                a.S32[P.s_off + z * PIECE + lane] = float(v);
            }
        }
}

// values of the cells' graph Laplacian on its stored pattern (rows and columns are ranks)
__global__ void k_laplacian(const int* ptr, const int* col, int n, const int* rank_slot, const Piece* pieces,
                            const int* emap, const int2* ecell, const double* cond, double* val) {
    const int t = blockIdx.x * HT + threadIdx.x;
    if (t >= n) return;
    const int lo = ptr[t], hi = ptr[t + 1];
    for (int j = lo; j < hi; ++j) val[j] = 0.0;
    const int slot = rank_slot[t];
    const Piece P = pieces[slot / PIECE];
    double diag = 0;
    for (int e = 0; e < P.ne; ++e) {
        const int g = emap[P.e_off + (long long)e * PIECE + slot % PIECE];
        const int2 c = ecell[g];
        const int other = c.x == t ? c.y : c.x;
        diag += cond[g];
        if (other != t)
            for (int j = lo; j < hi; ++j)
                if (col[j] == other) val[j] -= cond[g];
    }
    for (int j = lo; j < hi; ++j)
        if (col[j] == t) val[j] = diag;
}

// per-cell data of the right-hand side and the back substitution
struct CellArgs {
    const double *T, *Y, *Z, *theta, *dinv, *L;  // L: multiplier vector per (rank, r), null without a multiplier
    const int *slot_cell, *emap, *map, *mask;  // mask: given flux rows (null: none); map, mask: internal order
    const signed char* esgn;
    const Piece* pieces;
    int npieces, k;
    long long edges, nf, N;
    const double* mult;  // device: the multiplier (k_mult)
};

// One cell of the condensed right-hand side (BACK false: out[l] += c (T beta + Y f), out zero on entry) or of the
// back substitution (BACK true: out = the correction (u, p), fluxes zero on entry; lam the edge pressures in units of
// stop.scale()). r: residual of the symmetric form (pressure rows negated). K and NE compile-time, or NE = 0: any degree
// and edge count, local arrays in thread-local memory. Memory-bound on T (21 doubles of about 38 a hexagonal cell
// reads at k = 0): with the loops unrolled the local vectors stay in registers and every load of a cell is in flight
// before the first gather returns (1M cells, k = 0: right-hand side 161 -> 100 us, back substitution 257 -> 166 us).
constexpr int GEN_N = (MAX_K + 1) * MAX_NE + 24;
template <int K, int NE, bool BACK, typename T>
__device__ __forceinline__ void cell_system(const CellArgs& a, const Piece& P, int lane, const double* __restrict__ r,
                                            const T* __restrict__ lam, const CgStop& stop, double* __restrict__ out) {
    constexpr bool FIX = NE > 0;
    constexpr int Qc = (K + 1) * (K + 2) / 2, EDc = (K + 1) * NE, Nc = EDc + Qc - 1 + K * (K + 1) / 2;
    constexpr int MN = FIX ? Nc : GEN_N, MQ = FIX ? Qc : 15;
    const int ne = FIX ? NE : P.ne, q = FIX ? Qc : (a.k + 1) * (a.k + 2) / 2, ed = FIX ? EDc : (a.k + 1) * P.ne;
    const int n = FIX ? Nc : P.n;
    const double et = exp(a.theta[a.slot_cell[P.slot + lane]]), lscale = BACK ? stop.scale() : 0.0;
    const double* Tc = a.T + P.a_off + lane;
    int g[MN], l[MN];
    double b[MN], v[MN], w[BACK ? MN : 1], f[MQ], p[BACK ? MQ : 1];
#pragma unroll
    for (int i = 0; i < n; ++i) g[i] = a.map[P.map_off + (long long)i * PIECE + lane];
#pragma unroll
    for (int i = 0; i < ed; ++i) l[i] = (i / ne) * int(a.edges) + a.emap[P.e_off + (long long)(i % ne) * PIECE + lane];
#pragma unroll
    for (int i = 0; i < n; ++i) {
        const int gi = g[i] < 0 ? ~g[i] : g[i];
        double x = g[i] < 0 ? -r[gi] : r[gi];
        if (i < ed) {
            // a side's share of the edge's load, and its weight in the edge's flux
            const double share = 1.0 - et * Tc[(long long)tri(i, i, n) * PIECE] * a.dinv[l[i]];
            if (BACK) w[BACK ? i : 0] = share;
            x = a.mask && a.mask[gi] ? 0.0 : share * x;
            if (BACK) x -= side_sign(a.esgn, P, i, lane) * (lscale * double(lam[l[i]]));
        }
        b[i] = x;
        v[i] = 0;
    }
    const long long row = a.nf + (long long)(P.rank0 + lane) * q;
#pragma unroll
    for (int t = 0; t < q; ++t) {
        f[t] = -r[row + t];
        if (a.mult) f[t] -= a.L[row - a.nf + t] * *a.mult;
    }
    int z = 0;
#pragma unroll
    for (int i = 0; i < n; ++i)
#pragma unroll
        for (int j = i; j < n; ++j) {
            const double t = Tc[(long long)(z++) * PIECE];
            v[i] += t * b[j];
            if (j != i) v[j] += t * b[i];
        }
    if (BACK) {
        const int nz = q * (q + 1) / 2;
#pragma unroll
        for (int t = 0; t < q; ++t) p[BACK ? t : 0] = 0;
        int e = 0;
#pragma unroll
        for (int t = 0; t < q; ++t)
#pragma unroll
            for (int u = t; u < q; ++u) {
                const double zz = a.Z[P.slot * nz + (long long)(e++) * PIECE + lane] / et;
                p[BACK ? t : 0] += zz * f[u];
                if (u != t) p[BACK ? u : 0] += zz * f[t];
            }
    }
#pragma unroll
    for (int i = 0; i < n; ++i) {
        if (!BACK && i >= ed) continue;
        double s = et * v[i];
#pragma unroll
        for (int t = 0; t < q; ++t) {
            const double y = a.Y[P.hw_off + (long long)(t * n + i) * PIECE + lane];
            s += y * f[t];
            if (BACK) p[BACK ? t : 0] -= y * b[i];
        }
        if (!BACK) {
            atomicAdd(out + l[i], side_sign(a.esgn, P, i, lane) * s);  // at most two addends onto zero
            continue;
        }
        const int gi = g[i] < 0 ? ~g[i] : g[i];
        if (i >= ed) {
            out[gi] = s;
        } else if (a.mask && a.mask[gi]) {
            out[gi] = r[gi];  // identity row
        } else {
            const double x = w[BACK ? i : 0] * s;
            atomicAdd(out + gi, g[i] < 0 ? -x : x);  // two addends onto zero
        }
    }
    if (BACK)
#pragma unroll
        for (int t = 0; t < q; ++t) out[row + t] = p[BACK ? t : 0];
}

template <int K, bool BACK, typename T>
__global__ void __launch_bounds__(HT) k_cell_system(CellArgs a, const double* r, const T* lam, CgStop stop, double* out) {
    Piece P;
    int lane;
    if (!hyb_slot(a.pieces, a.npieces, P, lane)) return;
    if constexpr (K >= 0) {
        switch (P.ne) {
        case 3: cell_system<K, 3, BACK, T>(a, P, lane, r, lam, stop, out); return;
        case 4: cell_system<K, 4, BACK, T>(a, P, lane, r, lam, stop, out); return;
        case 5: cell_system<K, 5, BACK, T>(a, P, lane, r, lam, stop, out); return;
        case 6: cell_system<K, 6, BACK, T>(a, P, lane, r, lam, stop, out); return;
        case 7: cell_system<K, 7, BACK, T>(a, P, lane, r, lam, stop, out); return;
        case 8: cell_system<K, 8, BACK, T>(a, P, lane, r, lam, stop, out); return;
        default: break;
        }
    }
    cell_system<0, 0, BACK, T>(a, P, lane, r, lam, stop, out);
}

template <bool BACK, typename T>
void launch_cell_system(const CellArgs& a, const double* r, const T* lam, const CgStop& stop, double* out,
                        cudaStream_t s) {
    const int blocks = hblocks((long long)a.npieces * PIECE);
    if (a.k == 0)
        k_cell_system<0, BACK, T><<<blocks, HT, 0, s>>>(a, r, lam, stop, out);
    else if (a.k == 1)
        k_cell_system<1, BACK, T><<<blocks, HT, 0, s>>>(a, r, lam, stop, out);
    else
        k_cell_system<-1, BACK, T><<<blocks, HT, 0, s>>>(a, r, lam, stop, out);
    VG_CUDA(cudaGetLastError());
}

}  // namespace

// ---- set-up ---------------------------------------------------------------------------------------

// numbering of the edges (first touch in piece order) and the tables that follow from the mesh alone
void Solver::plan_edges() {
    const size_t per_edge = size_t(e_total_);
    std::vector<int> emap(per_edge, 0), rank_slot(m.nc, 0);
    std::vector<signed char> esgn(k >= 1 ? per_edge : 0, 1);
    std::vector<int2> ecell(m.ne, make_int2(-1, -1));
    edge_order_.assign(m.ne, -1);
    int next = 0;
    for (const auto& P : pieces_) {
        for (int e = 0; e < P.ne; ++e)
            for (int j = 0; j < P.count; ++j) {
                const int c = slot_cell_[P.slot + j], at = m.cptr[c] + e, ge = m.gedges[at];
                if (edge_order_[ge] < 0) edge_order_[ge] = next++;
                const int g = edge_order_[ge];
                const long long o = P.e_off + (long long)e * PIECE + j;
                emap[o] = g;
                if (k >= 1 && m.cnodes[at] != m.eend[2 * ge]) esgn[o] = -1;
                (ecell[g].x < 0 ? ecell[g].x : ecell[g].y) = P.rank0 + j;
            }
        for (int j = 0; j < P.count; ++j) rank_slot[P.rank0 + j] = int(P.slot + j);
    }
    if (next != m.ne) throw Error(VG_EMESH, "edge numbering does not cover every edge");
    for (auto& c : ecell)
        if (c.y < 0) c.y = c.x;  // boundary
    d_emap_.upload(emap);
    d_esgn_.upload(esgn);
    d_ecell_.upload(ecell);
    d_rank_slot_.upload(rank_slot);
}

// streams, values and loop vectors of the Darcy solve
void Solver::plan_hybrid() {
    const size_t per_edge = size_t(e_total_);
    if (k <= 1) {
        eplan64_ = plan_stream(pieces_, k, 8, sm_count_, RECORD_EDGE);
        eplan32_ = plan_stream(pieces_, k, 4, sm_count_, RECORD_EDGE);
        d_erec64_.resize(size_t(eplan64_.bytes));
        d_erec32_.resize(size_t(eplan32_.bytes));
        d_eroff64_.upload(eplan64_.rec_off);
        d_eroff32_.upload(eplan32_.rec_off);
        d_ebat64_.upload(eplan64_.batches);
        d_ebat32_.upload(eplan32_.batches);
        d_ecta64_.upload(eplan64_.cta_batch);
        d_ecta32_.upload(eplan32_.cta_batch);
    }
    // strided blocks: small meshes (one launch, vg_small.cu), degrees without a stream, and pieces too large for a
    // stage of either precision
    const long long per_cta = (long long)(pieces_.size() + sm_count_ - 1) / sm_count_;
    auto small = [&](size_t elem) {
        return m.nc <= SMALL_CELLS / (k + 1) &&
               (k < 4 || s_total_ / (long long)pieces_.size() * per_cta * (long long)elem <= SMALL_BLOCKS);
    };
    small_ctas_[0] = small(sizeof(double)) ? small_cg_ctas<double>(k, int(pieces_.size()), (long long)(k + 1) * m.ne, m.nc) : 0;
    small_ctas_[1] = k >= 1 && small(sizeof(float)) ? small_cg_ctas<float>(k, int(pieces_.size()), (long long)(k + 1) * m.ne, m.nc) : 0;
    bool strided = k > 1 || small_ctas_[0] > 0 || small_ctas_[1] > 0;
    for (const auto* pl : {&eplan64_, &eplan32_})
        for (const auto& b : pl->batches) strided = strided || b.bytes == 0;
    d_eS64_.resize(strided ? size_t(s_total_) : 0);
    d_eS32_.resize(strided ? size_t(s_total_) : 0);
    const size_t n = size_t(k + 1) * m.ne;
    d_edinv64_.resize(n);
    d_eh_.resize(n + 1);  // + the barrier word of the single-launch loop, which correct() clears with it
    d_erelax64_.resize(n);
    d_erelax32_.resize(n);
    d_econd_.resize(m.ne);
    d_ecw64_.resize(per_edge);
    d_ecw32_.resize(per_edge);
    d_eew64_.resize(m.ne);
    d_eew32_.resize(m.ne);
    for (auto& b : cg64_) b.resize(n);
    for (auto& b : cg32_) b.resize(n);
    for (auto& b : cgc64_) b.resize(m.nc);
    for (auto& b : cgc32_) b.resize(m.nc);
    d_mult_.resize(2);
    d_small_part_.resize(SMALL_SLOTS * SMALL_MAX_CTAS);
}

// mesh tables and the condensation of the cells for K = I (once after vg_build)
void Solver::prepare_condensation() {
    PhaseTimer pt;
    const int npieces = int(pieces_.size());
    if (!edges_planned_) {
        plan_edges();
        edges_planned_ = true;
        pt.mark("edge system: plan");
    }
    if (hybrid_condensed_) return;
    d_T_.resize(size_t(a_total_));
    d_Y_.resize(size_t(hw_total_));
    d_Z_.resize(pieces_.size() * PIECE * size_t(q * (q + 1) / 2));
    const int words = maxn * maxn + 2 * maxn * q + q * q + std::max(maxn, q);
    const int warps = std::max(1, std::min(8, int((96 << 10) / (words * sizeof(double)))));
    const size_t smem = size_t(warps) * words * sizeof(double);
    VG_CUDA(cudaFuncSetAttribute(k_condense, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)));
    d_status_.zero();
    const long long cells = (long long)npieces * PIECE;
    k_condense<<<int((cells + warps - 1) / warps), 32 * warps, smem>>>(
        d_A0_.data(), d_W64_.data(), d_pieces_.data(), npieces, k, words, d_T_.data(), d_Y_.data(), d_Z_.data(),
        d_status_.data(), d_slot_cell_.data());
    VG_CUDA(cudaGetLastError());
    check_status("condensation");
    hybrid_condensed_ = true;
    pt.mark("edge system: condensation");
}

// the condensed system and its multigrid, for the current permeability: everything on the first call
// after vg_build, the values alone (same addresses, so captured loops stay valid) after an update
void Solver::prepare_hybrid() {
    ArenaScope scope(arena_);
    PhaseTimer pt;
    const int npieces = int(pieces_.size());
    const long long n = (long long)(k + 1) * m.ne;
    prepare_condensation();
    if (!hybrid_planned_) {
        plan_hybrid();
        hybrid_planned_ = true;
    }
    pt.mark("edge system: cells");
    {
        // scratch: no solve is under way, and a vector of one holds (k + 1) ne values and more
        double *const D = sv64_[0].data(), *const R = sv64_[1].data();
        VG_CUDA(cudaMemsetAsync(D, 0, sizeof(double) * n, nullptr));
        VG_CUDA(cudaMemsetAsync(R, 0, sizeof(double) * m.ne, nullptr));
        k_edge_diag<<<hblocks((long long)npieces * PIECE), HT>>>(d_T_.data(), d_theta_.data(), d_slot_cell_.data(),
                                                                 d_emap_.data(), d_pieces_.data(), npieces, k, m.ne,
                                                                 D, R);
        k_edge_scale<<<148 * 8, HT>>>(D, R, d_ecell_.data(), m.ne, n, bc == VG_BC_FLUX,
                                      d_edinv64_.data(), d_erelax64_.data(), d_erelax32_.data(), d_econd_.data());
        VG_CUDA(cudaGetLastError());
        ValueArgs a{};
        a.T = d_T_.data();
        a.theta = d_theta_.data();
        a.dinv = d_edinv64_.data();
        a.slot_cell = d_slot_cell_.data();
        a.emap = d_emap_.data();
        a.esgn = k >= 1 ? d_esgn_.data() : nullptr;
        a.pieces = d_pieces_.data();
        a.npieces = npieces;
        a.k = k;
        a.edges = m.ne;
        a.ecell = d_ecell_.data();
        if (k <= 1) {
            a.rec64 = d_erec64_.data();
            a.rec32 = d_erec32_.data();
            a.roff64 = d_eroff64_.data();
            a.roff32 = d_eroff32_.data();
        }
        a.S64 = d_eS64_.data();
        a.S32 = d_eS32_.data();
        a.cw64 = d_ecw64_.data();
        a.cw32 = d_ecw32_.data();
        a.ew64 = d_eew64_.data();
        a.ew32 = d_eew32_.data();
        k_edge_values<<<hblocks((long long)npieces * PIECE), HT>>>(a);
        VG_CUDA(cudaGetLastError());
        VG_CUDA(cudaDeviceSynchronize());
    }
    pt.mark("edge system: values");
    if (use_amg) {
        d_lap_.resize(size_t(amg_.level0_nnz()));
        laplacian_values(amg_, d_econd_.data(), d_lap_.data());
        amg_.refresh(d_lap_.data());
        pt.mark("multigrid refresh");
    } else {
        destroy_graphs();  // a captured loop holds the hierarchy's addresses
        build_amg();
        pt.mark("multigrid");
    }
    amg_safe_ = false;
    hybrid_ready_ = true;
}

// every weight of the current hierarchy below the bound that keeps the cycle definite, until the next update
void Solver::make_amg_safe() {
    ArenaScope scope(arena_);
    VG_CUDA(cudaStreamSynchronize(stream_));
    d_lap_.resize(size_t(amg_.level0_nnz()));
    laplacian_values(amg_, d_econd_.data(), d_lap_.data());
    amg_.refresh(d_lap_.data(), true);
    amg_safe_ = true;
}

std::vector<int> Solver::rank_order() const {
    std::vector<int> order(m.nc);
    for (const auto& P : pieces_)
        for (int j = 0; j < P.count; ++j) order[slot_cell_[P.slot + j]] = P.rank0 + j;
    return order;
}

// multigrid of the cells' graph Laplacian (see the head of the file); without it (a hierarchy that does
// not coarsen) the diagonal alone preconditions
void Solver::build_amg() {
    const std::vector<double> own = d_econd_.download();
    std::vector<double> cond(m.ne);
    for (int e = 0; e < m.ne; ++e) cond[e] = own[edge_order_[e]];
    const HostCsr S = cell_graph(cond);
    const std::vector<int> order = rank_order();
    use_amg = false;
    amg_levels = 0;
    try {
        amg_.setup(S, d_errp_, &order, bc == VG_BC_FLUX);
    } catch (const Error& e) {
        if (e.code == VG_ENOMEM || e.code == VG_ECUDA) throw;
        return;
    }
    amg_levels = amg_.levels();
    use_amg = true;
}

HostCsr Solver::cell_graph(const std::vector<double>& cond) const {
    std::vector<int> ec(2 * size_t(m.ne), -1);
    for (int c = 0; c < m.nc; ++c)
        for (int j = m.cptr[c]; j < m.cptr[c + 1]; ++j) {
            const int e = m.gedges[j];
            (ec[2 * e] < 0 ? ec[2 * e] : ec[2 * e + 1]) = c;
        }
    HostCsr S;
    S.n = S.m = m.nc;
    S.ptr.assign(m.nc + 1, 0);
    std::vector<std::pair<int, double>> row;
    for (int c = 0; c < m.nc; ++c) {
        row.clear();
        double diag = 0;
        for (int j = m.cptr[c]; j < m.cptr[c + 1]; ++j) {
            const int e = m.gedges[j];
            const double d = cond[e];
            diag += d;
            const int o = ec[2 * e] == c ? ec[2 * e + 1] : ec[2 * e];
            if (o >= 0) row.push_back({o, -d});
        }
        row.push_back({c, diag});
        std::sort(row.begin(), row.end());
        for (size_t i = 0; i < row.size(); ++i) {
            if (i > 0 && row[i].first == row[i - 1].first) {
                S.val.back() += row[i].second;
                continue;
            }
            S.col.push_back(row[i].first);
            S.val.push_back(row[i].second);
        }
        S.ptr[c + 1] = int(S.col.size());
    }
    return S;
}

void Solver::laplacian_values(const Amg& amg, const double* cond, double* val) {
    k_laplacian<<<hblocks(m.nc), HT>>>(amg.level0_ptr(), amg.level0_col(), m.nc, d_rank_slot_.data(), d_pieces_.data(),
                                       d_emap_.data(), d_ecell_.data(), cond, val);
    VG_CUDA(cudaGetLastError());
}

// ---- solve ----------------------------------------------------------------------------------------

template <typename T>
CgVecs<T> Solver::cg_vecs() {
    CgVecs<T> v{};
    auto take = [&](auto& d64, auto& d32) {
        if constexpr (sizeof(T) == 8)
            return d64.data();
        else
            return d32.data();
    };
    v.p = take(cg64_[0], cg32_[0]);
    v.q = take(cg64_[1], cg32_[1]);
    v.x = take(cg64_[2], cg32_[2]);
    v.r_old = take(cg64_[3], cg32_[3]);
    v.r_new = take(cg64_[4], cg32_[4]);
    v.rc = take(cgc64_[0], cgc32_[0]);
    v.zc = use_amg ? take(cgc64_[1], cgc32_[1]) : nullptr;
    v.dinv = take(d_erelax64_, d_erelax32_);
    v.emap = d_emap_.data();
    v.cw = take(d_ecw64_, d_ecw32_);
    v.ecell = d_ecell_.data();
    v.ew = take(d_eew64_, d_eew32_);
    v.pieces = d_pieces_.data();
    v.npieces = int(pieces_.size());
    v.edges = m.ne;
    v.n = (long long)(k + 1) * m.ne;
    return v;
}

template <typename T>
EdgeArgs<T> Solver::edge_args(const CgVecs<T>& v) {
    EdgeArgs<T> a{};
    constexpr bool d = sizeof(T) == 8;
    a.x = v.p;
    a.y = v.q;
    if constexpr (d)
        a.S = d_eS64_.data();
    else
        a.S = d_eS32_.data();
    a.emap = d_emap_.data();
    a.pieces = d_pieces_.data();
    a.npieces = int(pieces_.size());
    a.k = k;
    a.edges = m.ne;
    a.flags = solve_flags();
    a.partials = d_partials_.data();
    a.counter = d_counter_.data();
    a.red = &scalars()->pq;
    if (k <= 1) {
        const StreamPlan& pl = d ? eplan64_ : eplan32_;
        a.rec = d ? d_erec64_.data() : d_erec32_.data();
        a.batches = d ? d_ebat64_.data() : d_ebat32_.data();
        a.cta_batch = d ? d_ecta64_.data() : d_ecta32_.data();
        a.ncta = pl.ncta;
        a.stages = pl.stages;
        a.stage_bytes = pl.stage_bytes;
        a.err = d_errp_;
    }
    return a;
}

// V-cycle on the restricted residual, r.z and the next direction
template <typename T>
void Solver::cg_tail(CgVecs<T>& v, int first, cudaStream_t s) {
    Scalars* sc = scalars();
    cg_finish<T>(v, first, m.nc, sc, solve_flags(), d_partials_.data(), d_counter_.data(), s);
    cg_direction<T>(v, sc, solve_flags(), s);
}

template <typename T>
void Solver::iteration(CgVecs<T>& v, cudaStream_t s) {
    Scalars* sc = scalars();
    int* flags = solve_flags();
    launch_edge_apply(edge_args<T>(v), s);
    std::swap(v.r_old, v.r_new);
    // the edge update (bandwidth-bound) runs on a second stream beside the restriction to the cells and
    // the V-cycle (latency-bound); both join before the scalar update
    VG_CUDA(cudaEventRecord(ev_fork_, s));
    VG_CUDA(cudaStreamWaitEvent(side_, ev_fork_, 0));
    cg_edges<T>(v, sc, flags, d_partials_.data(), d_counter_.data(), side_);
    VG_CUDA(cudaEventRecord(ev_join_, side_));
    if (use_amg) {
        cg_cells<T>(v, 0, sc, flags, s);
        amg_.vcycle(v.rc, v.zc, s);
    }
    VG_CUDA(cudaStreamWaitEvent(s, ev_join_, 0));
    cg_tail<T>(v, 0, s);
}

// the loop as a CUDA graph: a conditional while node whose body is two iterations (the residual's two
// buffers) followed by the condition kernel; the body count is capped on the device, so the loop ends
// even if the convergence flag is never raised
template <typename T>
void Solver::build_graph(int p) {
    VG_CUDA(cudaGraphCreate(&graph_[p], 0));
    cudaGraphConditionalHandle h;
    VG_CUDA(cudaGraphConditionalHandleCreate(&h, graph_[p], 1, cudaGraphCondAssignDefault));
    cudaGraphNodeParams cp{};
    cp.type = cudaGraphNodeTypeConditional;
    cp.conditional.handle = h;
    cp.conditional.type = cudaGraphCondTypeWhile;
    cp.conditional.size = 1;
    cudaGraphNode_t node;
    VG_CUDA(cudaGraphAddNode(&node, graph_[p], nullptr, 0, &cp));
    cudaGraph_t body = cp.conditional.phGraph_out[0];
    VG_CUDA(cudaStreamBeginCaptureToGraph(stream_, body, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal));
    CgVecs<T> v = cg_vecs<T>();
    const long long saved = amg_.launches;
    try {
        iteration<T>(v, stream_);
        iteration<T>(v, stream_);
        loop_check(h, solve_flags(), d_loop_.data(), stream_);
    } catch (...) {
        cudaGraph_t dummy;
        cudaStreamEndCapture(stream_, &dummy);
        throw;
    }
    amg_.launches = saved;
    VG_CUDA(cudaStreamEndCapture(stream_, &body));
    VG_CUDA(cudaGraphInstantiate(&gexec_[p], graph_[p], 0));
}

template <typename T>
bool Solver::takes_one_launch() {
    AmgView<T> v;
    return small_ctas_[sizeof(T) == 4 ? 1 : 0] > 0 && (!use_amg || amg_.view_levels<T>(v));
}

// conjugate gradients for the correction d of the residual r (symmetric form, internal order): condensed
// right-hand side, loop, back substitution (d's flux rows zero on entry). The caller reads the outcome with
// finish_correction once more work is queued behind it.
template <typename T>
void Solver::correct(const double* r, double* d, const CgStop& stop, int maxit, int check_every, cudaStream_t s) {
    Scalars* sc = scalars();
    int* flags = solve_flags();
    const int p = sizeof(T) == 4 ? 1 : 0;
    const bool graph = check_every <= 0;
    SmallCg<T> one{};
    one.amg.levels = -1;
    const bool small = graph && takes_one_launch<T>();
    if (small && use_amg) amg_.view_levels<T>(one.amg);
    if (graph && !small && !gexec_[p]) build_graph<T>(p);
    CellArgs a{};
    a.T = d_T_.data();
    a.Y = d_Y_.data();
    a.Z = d_Z_.data();
    a.theta = d_theta_.data();
    a.dinv = d_edinv64_.data();
    a.slot_cell = d_slot_cell_.data();
    a.emap = d_emap_.data();
    a.map = d_map_int_.data();
    a.esgn = k >= 1 ? d_esgn_.data() : nullptr;
    a.pieces = d_pieces_.data();
    a.npieces = int(pieces_.size());
    a.k = k;
    a.edges = m.ne;
    a.nf = nf;
    a.N = N;
    if (bc == VG_BC_FLUX) {
        a.mask = d_mask_int_.data();
        a.L = d_Lint_.data();
        a.mult = d_mult_.data();
        flux_multiplier(r, nullptr, d_Lint_.data(), m.nc, q, nf, N, d_mult_.data(), d_partials_.data(), d_counter_.data(), s);
        ++n_launch;
    }
    d_eh_.zero(s);
    launch_cell_system<false, T>(a, r, nullptr, stop, d_eh_.data(), s);
    CgVecs<T> v = cg_vecs<T>();
    if (small) {
        one.v = v;
        one.e = edge_args<T>(v);
        one.h = d_eh_.data();
        one.stop = stop;
        one.sc = sc;
        one.flags = flags;
        one.maxit = maxit;
        one.partials = d_small_part_.data();
        one.barrier = reinterpret_cast<unsigned*>(d_eh_.data() + v.n);
        one.err = d_errp_;
        launch_small_cg<T>(one, small_ctas_[p], s);
    } else {
        cg_init<T>(d_eh_.data(), v, sc, flags, stop, d_partials_.data(), d_counter_.data(), s);
        if (use_amg) {
            cg_cells<T>(v, 1, sc, flags, s);
            amg_.vcycle(v.rc, v.zc, s);
        }
        cg_tail<T>(v, 1, s);
    }
    if (graph && !small) {
        const int loop[2] = {0, (maxit + 1) / 2};
        VG_CUDA(cudaMemcpyAsync(d_loop_.data(), loop, sizeof(loop), cudaMemcpyHostToDevice, s));
        VG_CUDA(cudaGraphLaunch(gexec_[p], s));
    } else if (!small) {
        // host-driven batches of check_every iterations (every kernel is a plain launch)
        int h_flags[NFLAGS] = {0, 0, 0, 0};
        for (int done = 0; done < maxit;) {
            const int batch = std::min(check_every, maxit - done);
            for (int it = 0; it < batch; ++it) iteration<T>(v, s);
            done += batch;
            VG_CUDA(cudaMemcpyAsync(h_flags, flags, sizeof(h_flags), cudaMemcpyDeviceToHost, s));
            VG_CUDA(cudaStreamSynchronize(s));
            if (h_flags[0]) break;
        }
    }
    launch_cell_system<true, T>(a, r, v.x, stop, d, s);
    if (bc == VG_BC_FLUX) {
        flux_multiplier(r, d, d_Lint_.data(), m.nc, q, nf, N, d_mult_.data(), d_partials_.data(), d_counter_.data(), s);
        n_launch += 2;
    }
    last_small_ = small;
}

// the outcome of the last correction, from the copy of the solve's device scalars: iterations, gain
double Solver::finish_correction(const SolveOut& out, int& iters) {
    iters = out.flags[2];
    // per iteration: edge apply, edge update, finish, direction; with multigrid the restriction to the
    // cells and the composite V-cycle (residual, restriction, prolongation per level, dense product)
    const long long vc = use_amg ? 1 + 3LL * (amg_levels - 1) + 1 : 0;
    n_launch += last_small_ ? 3 : 2 + (3 + vc) + (4 + vc) * iters + (iters + 2) / 2;
    n_iter += iters;
    n_apply += iters;
    const double gain2 = out.sc.rz / out.sc.rz0;
    return gain2 > 0 && gain2 < 1 ? std::max(1e-16, std::sqrt(gain2)) : 1.0;
}

void Solver::solve(const double* b, double* x, const vg_solve_opts& o, vg_solve_info& info, cudaStream_t s) {
    if (!built) throw Error(VG_ESTATE, "vg_build must run before vg_solve");
    if (!b || !x) throw Error(VG_EINVAL, "null vector");
    if (!(o.tol > 0) || o.maxit < 1 || o.check_every < 0 || (o.mode == VG_SOLVE_MIXED && !(o.inner_tol > 0 && o.inner_tol < 1)))
        throw Error(VG_EINVAL, "invalid solve options");
    info = vg_solve_info{};
    if (!hybrid_ready_ && !minres_.ready) prepare_hybrid();
    (void)s;
    s = stream_;
    // order after the caller's work on the legacy default stream
    VG_CUDA(cudaEventRecord(ev_in_, nullptr));
    VG_CUDA(cudaStreamWaitEvent(s, ev_in_, 0));
    VG_CUDA(cudaEventRecord(ev0_, s));
    const bool cons = bc == VG_BC_FLUX;
    // symmetric form: pressure / multiplier rows negated
    DevBuf<double>&bs = sv64_[0], &r = sv64_[1], &y = sv64_[2], &d = sv64_[3];
    // the solve runs in the internal order: b and the initial x are permuted in, x out
    double* const x_ext = x;
    x = d_xi_.data();
    const bool guess = o.nonzero_guess != 0;
    start_residual(b, d_i2e_.data(), nf, N, bs.data(), r.data(), guess ? nullptr : x, solve_red(), d_partials_.data(),
                   d_counter_.data(), s);
    n_launch += 1;
    ++n_solve;
    SolveOut out{};
    // the solve's device scalars on the host: |r|^2 and |b|^2, and the outcome of the last loop
    auto read = [&] {
        VG_CUDA(cudaMemcpyAsync(&out, d_out_.data(), sizeof(out), cudaMemcpyDeviceToHost, s));
        VG_CUDA(cudaStreamSynchronize(s));
        const double nb = std::sqrt(out.red[1]);
        return std::sqrt(out.red[0]) / (nb > 0 ? nb : 1.0);
    };
    auto true_residual = [&] {
        y.zero(s);
        apply_int<double>(x, y.data(), cons, -1.0, s, nullptr);
        residual64(bs.data(), y.data(), r.data(), N, solve_red(), d_partials_.data(), d_counter_.data(), s);
        n_launch += 1;
    };
    // from x = 0 the residual is b, relative 1, and nothing has to be read before the first loop
    double rel = 1.0;
    if (guess) {
        permute<double>(x_ext, x, true, s);
        true_residual();
        rel = read();
    }
    int total = 0, outer = 0;
    if (minres_.ready) {
        if (!guess) rel = read();  // |b|
        const double nb = std::sqrt(out.red[1]);
        minres_solve(x, r.data(), nb > 0 ? nb : 1.0, o,
                     [&] {
                         true_residual();
                         return read();
                     },
                     rel, total, outer, s);
    }
    // A correction aims at a tenth of the tolerance (the reference's KSP factor, krylov.cu:142), in the
    // preconditioned norm and in the flux jumps, which are what the residual's rows will see of the error; the true FP64
    // residual then decides (krylov.cu:136-170) and a further correction follows while they gain. A loop's gain in its
    // norm and the residual's need not agree (high degrees): their ratio in one correction of a residual adjusts
    // what is asked of the next. An FP32 loop gains at most inner_tol.
    // Mixed at degree 0 on a mesh whose loop is one launch: an iteration is round trips, which FP32 does not shorten, and
    // one FP64 loop spares a second launch, its set-up and the residual between (mixed with FP32 loops -> with this one,
    // us: 100 cells 328 -> 263, 1,000 386 -> 305, 8,000 549 -> 452, 45,000 923 -> 806). From degree 1 on the FP64
    // blocks cost what they spare (10,000 cells 981 against 1,052, degree 2 40,000 cells 14,851 against 16,482).
    bool fp64 = o.mode == VG_SOLVE_FP64 || (k == 0 && o.check_every <= 0 && takes_one_launch<double>());
    const int steps = minres_.ready ? 0 : o.mode == VG_SOLVE_FP64 ? 12 : o.max_outer;
    double ratio = 1.0;
    int idle = 0;
    bool careful = false;  // loops end after six digits
    for (; outer < steps && rel > o.tol && total < o.maxit; ++outer) {
        const double want = 0.1 * o.tol / (rel * ratio), before = rel;
        CgStop stop;
        stop.raw = 0.1 * o.tol;
        stop.b2 = solve_red() + 1;
        // the first correction from x = 0 is x itself
        const bool direct = outer == 0 && !guess;
        double* const to = direct ? x : d.data();
        if (!direct) d.zero(s);
        if (fp64) {
            stop.unit = 0.0;
            stop.tol = std::min(0.5, want);
            stop.floor = careful ? 1e-6 : 1e-15;
            correct<double>(r.data(), to, stop, o.maxit - total, o.check_every, s);
        } else {
            stop.unit = rel;
            stop.tol = std::min(0.5, std::max(o.inner_tol, want));
            stop.floor = o.inner_tol;
            correct<float>(r.data(), to, stop, o.maxit - total, o.check_every, s);
        }
        if (!direct) {
            axpy64(x, d.data(), 1.0, s);
            n_launch += 1;
        }
        true_residual();
        rel = read();
        int it = 0;
        const double gain = finish_correction(out, it);
        total += it;
        // A correction that did harm is taken back. Where r.z was not positive, the cycle, whose coarse levels have
        // estimated weights, is not definite on these values, and the hierarchy is made safe; else the loop went on below
        // its rounding level, and FP64 loops of six digits each follow.
        const bool harm = !(rel <= 2.0 * before), indefinite = use_amg && !amg_safe_ && !(out.sc.rz > 0 && out.sc.rz0 > 0);
        if (rel > o.tol && (harm || indefinite)) {
            if (!(rel < before)) {
                if (direct)
                    VG_CUDA(cudaMemsetAsync(x, 0, sizeof(double) * N, s));
                else
                    axpy64(x, d.data(), -1.0, s);
                true_residual();
                rel = read();
                n_launch += 1;
            }
            if (indefinite) {
                make_amg_safe();
            } else if (careful) {
                ++outer;
                break;
            } else {
                fp64 = careful = true;
            }
            continue;
        }
        if (!direct) ratio = std::min(1e8, std::max(1.0, rel / (before * gain)));
        idle = rel <= 0.5 * before ? 0 : idle + 1;
        if (fp64 && idle >= 3) {  // rounding level
            ++outer;
            break;
        }
    }
    permute<double>(x, x_ext, false, s);
    VG_CUDA(cudaEventRecord(ev1_, s));
    VG_CUDA(cudaEventSynchronize(ev1_));
    check_pipeline();
    float ms = 0;
    VG_CUDA(cudaEventElapsedTime(&ms, ev0_, ev1_));
    info.iterations = total;
    info.outer = outer;
    info.residual = rel;
    info.seconds = ms * 1e-3;
    if (!(rel <= o.tol))
        throw Error(VG_ENOCONV, "Krylov solve did not converge: iterations=" + std::to_string(total) +
                                    " true_relative_residual=" + std::to_string(rel));
}

}  // namespace vg

// Conjugate gradients on the edge pressures of a small mesh as one cooperative launch.
//
// The loop of vg_krylov.cu runs 5 dependent kernels an iteration plus 2 per multigrid level. On a small mesh (the
// line is in vg_hybrid.cu: 64,000 cells at degree 0) each of them has work for a microsecond or two and costs 5 to 6
// of launch, drain and grid reduction (1,000 cells FP64: 33 us an iteration). Here the grid stays resident, one CTA per SM, and the phases
// of an iteration are separated by grid barriers:
//   apply      q += S p, p.q                                  (one lane per cell, red.global.add into zeroed q)
//   update     x += alpha p, r' = r - alpha q, sums; rc = Pi^T (r - alpha q)
//   down       per level: b' = Pt^T b and the smoothed residual
//   dense      x' = A^{-1} b'
//   up         per level: z = residual term + Pt x'; rc.zc
//   direction  beta, p = D^{-1} r' + Pi zc + beta p, q = 0
// Sums are block partials that every CTA adds in the same fixed order after the barrier, so that no CTA waits for
// a broadcast and results are bitwise reproducible. Vectors written inside the loop are read with plain loads behind
// the barrier's fences (never the read-only path). A barrier wait is bounded (1 s); one that gives up sets an error
// word and the kernel returns.
#include <algorithm>

#include "vg_small.cuh"
#include "vg_edge.cuh"
#include "vg_pipe.cuh"

namespace vg {

namespace {

constexpr int ST = 256;                   // threads per CTA
constexpr int SMALL_SMEM = 216 << 10;     // dynamic shared memory per CTA (one CTA per SM)
constexpr int SW = ST / 32;
// gathers of a row in flight at once. A phase of a small mesh is a chain of L2 round trips (0.6 us each): a loop unrolled
// by the compiler takes its last entries, which are most rows' only ones, one round trip each.
constexpr int BATCH = 8;
constexpr int PRE = 2;  // edges of a thread whose loads go out before a sum over the grid is known

struct Grid {
    unsigned* counter;
    unsigned round = 0;
    int* err;
    bool ok = true;

    // all CTAs of the grid; false when the wait gave up
    __device__ bool sync() {
        __syncthreads();
        ++round;
        __shared__ int good;
        if (threadIdx.x == 0) {
            // release and acquire at GPU scope; the CTA's barriers extend both to its other threads
            asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(counter) : "memory");
            const unsigned want = round * gridDim.x;
            good = 1;
            const unsigned long long t0 = globaltimer();
            for (unsigned it = 1;; ++it) {
                unsigned seen;
                asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(counter) : "memory");
                if (int(seen - want) >= 0) break;
                if (((it & 255u) == 0 && globaltimer() - t0 > WAIT_NS) || it >= (1u << 26)) {
                    good = 0;
                    *reinterpret_cast<volatile int*>(err) = 1;
                    break;
                }
            }
        }
        __syncthreads();
        ok = good != 0;
        return ok;
    }
};

// block sums of NS values into partials[slot ..][blockIdx]; a grid barrier follows before the next ones
template <int NS>
__device__ void put_partials(double (&v)[NS], double* partials, int slot) {
    __shared__ double sh[NS][SW];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 16; o; o >>= 1)
#pragma unroll
        for (int i = 0; i < NS; ++i) v[i] += __shfl_down_sync(0xffffffffu, v[i], o);
    if (lane == 0)
#pragma unroll
        for (int i = 0; i < NS; ++i) sh[i][warp] = v[i];
    __syncthreads();
    if (warp < NS) {
        double s = lane < SW ? sh[warp][lane] : 0.0;
#pragma unroll
        for (int o = SW / 2; o; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
        if (lane == 0) partials[(slot + warp) * SMALL_MAX_CTAS + blockIdx.x] = s;
    }
}

// the grid's sum of NS consecutive slots, the same in every thread (called behind a grid barrier, and another one
// before the next call). The loads are issued by open_sums; what does not need the sums goes between the two.
struct Partials {
    double v[SMALL_MAX_CTAS / 32];
};
template <int NS>
__device__ Partials open_sums(const double* partials, int slot) {
    const int s = slot + (threadIdx.x >> 5), l = threadIdx.x & 31;
    Partials p;
#pragma unroll
    for (int j = 0; j < SMALL_MAX_CTAS / 32; ++j) {
        const int b = l + 32 * j;
        p.v[j] = s < slot + NS && b < (int)gridDim.x ? __ldcg(partials + s * SMALL_MAX_CTAS + b) : 0.0;
    }
    return p;
}
template <int NS>
__device__ void get_sums(const Partials& p, double (&out)[NS]) {
    __shared__ double tot[NS];
    if (threadIdx.x < 32 * NS) {
        double v = 0;
#pragma unroll
        for (int j = 0; j < SMALL_MAX_CTAS / 32; ++j) v += p.v[j];
        for (int o = 16; o; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
        if ((threadIdx.x & 31) == 0) tot[threadIdx.x >> 5] = v;
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < NS; ++i) out[i] = tot[i];
}

// Shared memory of a CTA handed out front to back; null when the rest does not hold the request. Every thread makes
// the same requests, so every thread holds the same pointers.
struct Arena {
    unsigned char* base;
    int used, size;
    template <typename U>
    __device__ U* take(int n) {
        const int bytes = (n * int(sizeof(U)) + 15) & ~15;
        if (bytes > size - used) return nullptr;
        U* p = reinterpret_cast<U*>(base + used);
        used += bytes;
        return p;
    }
};

// rows blockIdx.x, + gridDim.x, ... of a matrix, copied into shared memory where they fit (local), else read in place
template <typename T>
struct Rows {
    const int *ptr, *col;
    const T* val;
    int n, rows;
    bool local;
};

template <typename T, class Len, class At>
__device__ Rows<T> stage_rows(Arena& ar, int n, const int* gptr, const int* gcol, const T* gval, Len len, At at) {
    const int G = gridDim.x, b = blockIdx.x, rows = n > b ? (n - b + G - 1) / G : 0;
    Rows<T> R{gptr, gcol, gval, n, rows, false};
    const Arena before = ar;
    int* ptr = ar.take<int>(rows + 1);
    if (!ptr) return R;
    for (int k = threadIdx.x; k < rows; k += ST) ptr[k + 1] = len(b + k * G);
    __syncthreads();
    if (threadIdx.x == 0) {
        ptr[0] = 0;
        for (int k = 0; k < rows; ++k) ptr[k + 1] += ptr[k];
    }
    __syncthreads();
    const int nnz = ptr[rows];
    T* val = ar.take<T>(nnz);
    int* col = val ? ar.take<int>(nnz) : nullptr;
    if (!col) {
        __syncthreads();  // ptr read by everyone before its space is handed out again
        ar = before;
        return R;
    }
    for (int k = threadIdx.x >> 3; k < rows; k += ST / 8)
        for (int j = threadIdx.x & 7; j < ptr[k + 1] - ptr[k]; j += 8) at(b + k * G, j, col[ptr[k] + j], val[ptr[k] + j]);
    R.ptr = ptr;
    R.col = col;
    R.val = val;
    R.local = true;
    return R;
}

template <typename T>
__device__ Rows<T> stage_csr(Arena& ar, int n, const int* ptr, const int* col, const T* val) {
    return stage_rows<T>(
        ar, n, ptr, col, val, [&](int r) { return ptr[r + 1] - ptr[r]; },
        [&](int r, int j, int& c, T& v) {
            c = col[ptr[r] + j];
            v = val[ptr[r] + j];
        });
}

// LANES lanes a row (strided sums, fixed shuffle tree): f(row, sum) on the row's first lane. Short rows (prolongations,
// the finest operator) take one lane: eight would leave a row's few gathers on as many lanes and need several passes
// where one does (30k cells FP64: 43 -> 38 us an iteration).
template <int LANES, typename T, class F>
__device__ __forceinline__ void row_sums(const Rows<T>& R, const T* x, F f) {
    const int sub = threadIdx.x % LANES;
    for (int k = threadIdx.x / LANES; LANES == 1 ? k < R.rows : __any_sync(0xffffffffu, k < R.rows); k += ST / LANES) {
        const int row = blockIdx.x + k * gridDim.x;
        T s = T(0);
        if (k < R.rows) {
            const int at = R.local ? k : row, hi = R.ptr[at + 1];
            for (int j = R.ptr[at] + sub; j < hi; j += BATCH * LANES) {
                T xv[BATCH];
#pragma unroll
                for (int u = 0; u < BATCH; ++u) xv[u] = j + u * LANES < hi ? x[R.col[j + u * LANES]] : T(0);
#pragma unroll
                for (int u = 0; u < BATCH; ++u)
                    if (j + u * LANES < hi) s += R.val[j + u * LANES] * xv[u];
            }
        }
#pragma unroll
        for (int o = LANES / 2; o; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o, LANES);
        if (k < R.rows && sub == 0) f(row, s);
    }
}
template <typename T, class F>
__device__ __forceinline__ void row_sums(const Rows<T>& R, bool wide, const T* x, F f) {
    if (wide)
        row_sums<8>(R, x, f);
    else
        row_sums<1>(R, x, f);
}

template <typename T, int K>
__global__ void __launch_bounds__(ST, 1) k_small_cg(SmallCg<T> a) {
    extern __shared__ __align__(16) unsigned char small_smem[];
    CgVecs<T> v = a.v;
    Grid grid{a.barrier, 0u, a.err};
    const int tid = threadIdx.x, G = gridDim.x, warp = tid >> 5, lane = tid & 31;
    const bool coarse = a.amg.levels >= 0;
    const int L = coarse ? a.amg.levels : 0;
    double rz = 0, rz0 = 0, best = 0, rr = 0, raw = 0, pq = 0;
    int its = 0, best_it = 0;
    bool stop = false;
    const double scale = 1.0 / a.stop.scale(), raw2 = a.stop.raw_abs() * a.stop.raw_abs();

    // ---- what this CTA reads in every iteration, in shared memory as far as it fits
    Arena ar{small_smem, 0, a.smem};
    // its edges: a contiguous range; x is only read and written here and stays local until the end
    const int e0 = int(v.n * blockIdx.x / G), en = int(v.n * (blockIdx.x + 1) / G) - e0;
    T* const xl = ar.take<T>(en);       // the host gives at least this much (and the next three)
    T* const dinv = ar.take<T>(en);
    T* const ew = ar.take<T>(en);
    int2* const ecell = ar.take<int2>(en);
    for (int i = tid; i < en; i += ST) {
        dinv[i] = v.dinv[e0 + i];
        const bool mean = e0 + i < v.edges;
        ew[i] = mean ? v.ew[e0 + i] : T(0);
        ecell[i] = mean ? v.ecell[e0 + i] : make_int2(0, 0);
    }
    // its pieces blockIdx.x, + G, ...: {edges, cells, first rank, byte offset or -1} and S | edge indices | weights
    const int np = v.npieces > (int)blockIdx.x ? (v.npieces - blockIdx.x + G - 1) / G : 0;
    int4* const piece = ar.take<int4>(np);
    for (int k = tid; k < np; k += ST) {
        const Piece& P = v.pieces[blockIdx.x + k * G];
        piece[k] = make_int4(P.ne, P.count, P.rank0, -1);
    }
    __syncthreads();
    for (int k = 0; k < np; ++k) {
        const int ne = piece[k].x, ed = (a.e.k + 1) * ne, nS = ed * (ed - 1) / 2 * PIECE, nE = ne * PIECE;
        const Arena before = ar;
        T* S = ar.take<T>(nS);
        T* w = S ? ar.take<T>(nE) : nullptr;
        int* m = w ? ar.take<int>(nE) : nullptr;
        if (!m) {
            ar = before;
            continue;
        }
        const Piece& P = v.pieces[blockIdx.x + k * G];
        for (int z = tid; z < nS; z += ST) S[z] = a.e.S[P.s_off + z];
        for (int z = tid; z < nE; z += ST) {
            w[z] = v.cw[P.e_off + z];
            m[z] = v.emap[P.e_off + z];
        }
        if (tid == 0) piece[k].w = int(reinterpret_cast<unsigned char*>(S) - small_smem);
    }
    Rows<T> Rt[AMG_VIEW_LEVELS], As[AMG_VIEW_LEVELS], Pt[AMG_VIEW_LEVELS];
#pragma unroll
    for (int l = 0; l < AMG_VIEW_LEVELS; ++l) {
        if (l >= L) break;
        const AmgLevelView<T>& A = a.amg.level[l];
        Rt[l] = stage_csr<T>(ar, A.nc, A.rptr, A.rcol, A.rval);
        Pt[l] = stage_csr<T>(ar, A.n, A.pptr, A.pcol, A.pval);
        if (A.sell.val)
            As[l] = stage_rows<T>(
                ar, A.n, nullptr, nullptr, nullptr, [&](int r) { return A.sell.width[r >> 5]; },
                [&](int r, int j, int& c, T& w) {
                    const long long o = A.sell.soff[r >> 5] + (r & 31) + 32 * j;
                    c = A.sell.col[o];
                    w = A.sell.val[o];
                });
        else
            As[l] = stage_csr<T>(ar, A.n, A.aptr, A.acol, A.aval);
    }
    T* const bd = coarse ? ar.take<T>(a.amg.ncoarse) : nullptr;  // the dense level's right-hand side
    const int nd = coarse ? a.amg.ncoarse : 0, drows = nd > (int)blockIdx.x ? (nd - blockIdx.x + G - 1) / G : 0;
    T* const dense = nd <= 16384 && (long long)drows * nd < (1 << 26) ? ar.take<T>(drows * nd) : nullptr;
    if (dense)
        for (int z = tid; z < drows * nd; z += ST)
            dense[z] = a.amg.inverse[(long long)(blockIdx.x + (z / nd) * G) * nd + z % nd];
    __syncthreads();

    // the edge indices, weights and block of a piece
    auto fields = [&](int k, int4 f, const T*& S, const T*& w, const int*& m) {
        if (f.w >= 0) {
            const int ed = (a.e.k + 1) * f.x;
            const unsigned char* at = small_smem + f.w;
            S = reinterpret_cast<const T*>(at) + lane;
            w = S + ed * (ed - 1) / 2 * PIECE;
            m = reinterpret_cast<const int*>(w - lane + f.x * PIECE) + lane;
        } else {
            const Piece& P = v.pieces[blockIdx.x + k * G];
            S = a.e.S + P.s_off + lane;
            w = v.cw + P.e_off + lane;
            m = v.emap + P.e_off + lane;
        }
    };
    // Pi^T r and Pi^T q on piece k, one lane per cell: rc = Pi^T (r - alpha q) is their combination, so that the
    // gathers need not wait for alpha
    auto restrict_piece = [&](int k, const T* r, bool start, T& sr, T& sq) {
        sr = sq = T(0);
        if (k >= np) return;
        const int4 f = piece[k];
        if (lane >= f.y) return;
        const T *S, *w;
        const int* m;
        fields(k, f, S, w, m);
        for (int e0 = 0; e0 < f.x; e0 += BATCH) {
            T rv[BATCH], qv[BATCH];
#pragma unroll
            for (int u = 0; u < BATCH; ++u) {
                const bool in = e0 + u < f.x;
                const int g = in ? m[(e0 + u) * PIECE] : 0;
                rv[u] = in ? r[g] : T(0);
                qv[u] = in && !start ? v.q[g] : T(0);
            }
#pragma unroll
            for (int u = 0; u < BATCH; ++u)
                if (e0 + u < f.x) {
                    sr += w[(e0 + u) * PIECE] * rv[u];
                    sq += w[(e0 + u) * PIECE] * qv[u];
                }
        }
    };
    auto put_cell = [&](int k, T value) {
        if (k < np && lane < piece[k].y) v.rc[piece[k].z + lane] = value;
    };
    // zc = V rc behind a barrier; leaves the partial sums of rc.zc in slot 3 (no barrier after them)
    auto vcycle = [&]() -> bool {
        const T* b = v.rc;
#pragma unroll
        for (int l = 0; l < AMG_VIEW_LEVELS; ++l) {
            if (l >= L) break;
            const AmgLevelView<T>& A = a.amg.level[l];
            row_sums(Rt[l], A.r_wide, b, [&](int row, T s) { A.b[row] = s; });
            auto smooth = [&](int row, T s) {
                const T bi = b[row];
                A.r[row] = __ldg(A.S + row) * (bi + (bi - s));
            };
            if (As[l].local || !A.sell.val)
                row_sums(As[l], A.a_wide, b, smooth);
            else
                for (int k = tid; k < As[l].rows; k += ST) {
                    const int row = blockIdx.x + k * G, w = __ldg(A.sell.width + (row >> 5));
                    const long long o = __ldg(A.sell.soff + (row >> 5)) + (row & 31);
                    T s = T(0);
                    for (int j = 0; j < w; ++j) s += __ldg(A.sell.val + o + 32 * j) * b[__ldg(A.sell.col + o + 32 * j)];
                    smooth(row, s);
                }
            if (!grid.sync()) return false;
            b = A.b;
        }
        double dot[1] = {};
        T* const xd = L ? a.amg.level[L - 1].x : v.zc;
        if (bd) {
            for (int j = tid; j < nd; j += BATCH * ST) {
                T t[BATCH];
#pragma unroll
                for (int u = 0; u < BATCH; ++u) t[u] = j + u * ST < nd ? b[j + u * ST] : T(0);
#pragma unroll
                for (int u = 0; u < BATCH; ++u)
                    if (j + u * ST < nd) bd[j + u * ST] = t[u];
            }
            __syncthreads();
            b = bd;
        }
        for (int k = warp; k < drows; k += SW) {  // dense coarsest level, one warp per row
            const int row = blockIdx.x + k * G;
            const T* A = dense ? dense + k * nd : a.amg.inverse + (long long)row * nd;
            T s = T(0);
#pragma unroll 8
            for (int j = lane; j < nd; j += 32) s += A[j] * b[j];  // shared memory both, as far as they fit
            for (int o = 16; o; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
            if (lane == 0) {
                xd[row] = s;
                if (!L) dot[0] += double(s) * double(b[row]);
            }
        }
#pragma unroll
        for (int l = AMG_VIEW_LEVELS - 1; l >= 0; --l) {
            if (l >= L) continue;
            if (!grid.sync()) return false;
            const AmgLevelView<T>& A = a.amg.level[l];
            T* const z = l ? a.amg.level[l ? l - 1 : 0].x : v.zc;
            row_sums(Pt[l], A.p_wide, A.x, [&](int row, T s) {
                const T y = A.r[row] + s;
                z[row] = y;
                if (l == 0) dot[0] += double(y) * double(v.rc[row]);
            });
        }
        put_partials(dot, a.partials, 3);
        return true;
    };
    // stop test and direction, behind a barrier; every thread of the grid takes the same decision
    auto finish = [&](bool start) {
        const Partials part = open_sums<3>(a.partials, 1);
        // D^{-1} r + Pi zc and the old direction, for as many edges as registers hold
        auto precond = [&](int i) {
            const T di = dinv[i];
            T z = di * v.r_new[e0 + i];
            if (coarse && e0 + i < v.edges && di != T(0)) {
                const T zy = v.zc[ecell[i].y];
                z += zy + ew[i] * (v.zc[ecell[i].x] - zy);
            }
            return z;
        };
        T zv[PRE], pv[PRE];
#pragma unroll
        for (int u = 0; u < PRE; ++u) {
            const int i = tid + u * ST;
            zv[u] = i < en ? precond(i) : T(0);
            pv[u] = i < en && !start ? v.p[e0 + i] : T(0);
        }
        double t[3];
        get_sums<3>(part, t);
        rr = t[0];
        raw = t[1];
        const double now = rr + (coarse ? t[2] : 0.0);
        const bool fine = now > 0 && isfinite(now);
        double beta = 0;
        if (start) {
            rz0 = best = now;
            stop = !fine;
        } else {
            beta = rz > 0 ? now / rz : 0.0;
            ++its;
            if (now < best) {
                best = now;
                best_it = its;
            }
            stop = !fine || !(pq > CG_BREAK * rz) || cg_spent(now, best, its - best_it, rz0) ||
                   (now <= a.stop.tol * a.stop.tol * rz0 && raw <= raw2) ||
                   now <= a.stop.floor * a.stop.floor * rz0 || its >= a.maxit;
        }
        rz = now;
        if (stop) return;
        const T bt = T(beta);
#pragma unroll
        for (int u = 0; u < PRE; ++u) {
            const int i = tid + u * ST;
            if (i >= en) break;
            v.p[e0 + i] = zv[u] + bt * pv[u];
            v.q[e0 + i] = T(0);
        }
        for (int i = tid + PRE * ST; i < en; i += ST) {
            const T z = precond(i);
            v.p[e0 + i] = start ? z : z + bt * v.p[e0 + i];
            v.q[e0 + i] = T(0);
        }
    };
    auto sums = [&](T r, T di, double (&s)[2]) {
        const double z = double(di * r);
        s[0] += z * double(r);
        if (di != T(0)) s[1] += double(r) * double(r) + z * z;
    };

    {
        double s[2] = {};
        for (int i = tid; i < en; i += ST) {
            const T r = T(scale * a.h[e0 + i]);
            sums(r, dinv[i], s);
            v.r_new[e0 + i] = r;
            xl[i] = T(0);
        }
        put_partials(s, a.partials, 1);
        if (!grid.sync()) return;
        if (coarse) {
            for (int k = warp; k < np; k += SW) {
                T sr, sq;
                restrict_piece(k, v.r_new, true, sr, sq);
                put_cell(k, sr);
            }
            if (!grid.sync()) return;
            if (!vcycle()) return;
            if (!grid.sync()) return;
        }
        finish(true);
    }
    while (!stop) {
        if (!grid.sync()) return;
        double quad[1] = {};
        for (int k = warp; k < np; k += SW) {
            const int4 f = piece[k];
            if (lane >= f.y) continue;
            const T *S, *w;
            const int* m;
            fields(k, f, S, w, m);
            edge_piece<T, K>(a.e, f.x, S, m, quad[0]);
        }
        put_partials(quad, a.partials, 0);
        if (!grid.sync()) return;
        const Partials part = open_sums<1>(a.partials, 0);
        T* const old = v.r_new;
        v.r_new = v.r_old;
        v.r_old = old;
        T pv[PRE], qv[PRE], rv[PRE];
#pragma unroll
        for (int u = 0; u < PRE; ++u) {
            const int i = tid + u * ST;
            pv[u] = i < en ? v.p[e0 + i] : T(0);
            qv[u] = i < en ? v.q[e0 + i] : T(0);
            rv[u] = i < en ? old[e0 + i] : T(0);
        }
        T sr = T(0), sq = T(0);
        if (coarse) restrict_piece(warp, old, false, sr, sq);
        double t[1];
        get_sums<1>(part, t);
        pq = t[0];
        const T alpha = T(pq > CG_BREAK * rz && isfinite(pq) ? rz / pq : 0.0);
        if (coarse) {
            put_cell(warp, sr - alpha * sq);
            for (int k = warp + SW; k < np; k += SW) {
                restrict_piece(k, old, false, sr, sq);
                put_cell(k, sr - alpha * sq);
            }
        }
        double s[2] = {};
        auto step = [&](int i, T p, T q, T r0) {
            xl[i] += alpha * p;
            const T r = r0 - alpha * q;
            sums(r, dinv[i], s);
            v.r_new[e0 + i] = r;
        };
#pragma unroll
        for (int u = 0; u < PRE; ++u)
            if (tid + u * ST < en) step(tid + u * ST, pv[u], qv[u], rv[u]);
        for (int i = tid + PRE * ST; i < en; i += ST) step(i, v.p[e0 + i], v.q[e0 + i], old[e0 + i]);
        put_partials(s, a.partials, 1);
        if (!grid.sync()) return;
        if (coarse) {
            if (!vcycle()) return;
            if (!grid.sync()) return;
        }
        finish(false);
    }
    for (int i = tid; i < en; i += ST) v.x[e0 + i] = xl[i];
    if (blockIdx.x == 0 && tid == 0) {
        a.sc->rz = rz;
        a.sc->rz0 = rz0;
        a.sc->rr = rr;
        a.sc->raw = raw;
        a.flags[0] = 1;
        a.flags[2] = its;
    }
}

template <typename T>
const void* small_kernel(int k) {
    if constexpr (sizeof(T) == 8)  // FP32 is asked for from degree 1 on (Solver::solve)
        if (k == 0) return reinterpret_cast<const void*>(k_small_cg<T, 0>);
    return k == 1 ? reinterpret_cast<const void*>(k_small_cg<T, 1>) : reinterpret_cast<const void*>(k_small_cg<T, 2>);
}

}  // namespace

// CTAs of the cooperative grid (0: this device or mesh does not take it)
template <typename T>
int small_cg_ctas(int k, int npieces, long long n, int cells) {
    int dev = 0, coop = 0, sms = 0, per = 0;
    VG_CUDA(cudaGetDevice(&dev));
    VG_CUDA(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev));
    VG_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    if (!coop) return 0;
    VG_CUDA(cudaFuncSetAttribute(small_kernel<T>(k), cudaFuncAttributeMaxDynamicSharedMemorySize, SMALL_SMEM));
    VG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, small_kernel<T>(k), ST, SMALL_SMEM));
    if (per < 1) return 0;
    const int ctas = std::min(std::min(sms, SMALL_MAX_CTAS), std::max({16, npieces, std::min(cells, COARSE_MAX) / 8}));
    // every CTA holds at least its edges' vectors and its list of pieces
    const long long need = (n / ctas + 1) * (3 * (long long)sizeof(T) + 8) + (npieces / ctas + 1) * 16 + 64;
    return need <= SMALL_SMEM ? ctas : 0;
}

template <typename T>
void launch_small_cg(const SmallCg<T>& a, int ctas, cudaStream_t s) {
    SmallCg<T> args = a;
    args.smem = SMALL_SMEM;
    void* p[] = {&args};
    VG_CUDA(cudaLaunchCooperativeKernel(small_kernel<T>(a.e.k), dim3(ctas), dim3(ST), p, SMALL_SMEM, s));
}

template int small_cg_ctas<double>(int, int, long long, int);
template int small_cg_ctas<float>(int, int, long long, int);
template void launch_small_cg<double>(const SmallCg<double>&, int, cudaStream_t);
template void launch_small_cg<float>(const SmallCg<float>&, int, cudaStream_t);

}  // namespace vg

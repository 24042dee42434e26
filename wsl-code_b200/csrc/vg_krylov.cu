// Preconditioned conjugate gradients on the edge pressures (vg_hybrid.cu: fluxes and cell pressures are
// eliminated cell by cell), replacing the PETSc FGMRES of vem/CurvedVEM_Darcy_gpu/src/krylov.cu:49-175.
// The preconditioner is
//     z = D^{-1} r + Pi V Pi^T r      (D: the diagonal over EDGE_RELAX),
// the diagonal plus one multigrid V-cycle V on the cell pressures, which Pi interpolates to the edges.
// Per iteration:
//   apply       q = S p and p.q (fused, vg_apply.cu)
//   edges       x += alpha p, r' = r - alpha q, r'.D^{-1} r' and the jump's norm   } two streams, the
//   cells       rc = Pi^T (r - alpha q), then the V-cycle  zc = V rc               } edges beside the cycle
//   finish      r'.z = r'.D^{-1} r' + rc.zc, beta, stop test (device scalars)
//   direction   p = D^{-1} r' + Pi zc + beta p, q = 0
// rc is formed from r and q, not from r', so the cycle does not wait for the edge update; r' goes to
// a second buffer. All scalars stay on the device; convergence sets a stop flag that turns the
// remaining kernels of a body into no-ops. Every reduction is a fixed-shape two-level sum (block
// partials, last block sums them in order): results are bitwise reproducible.
#include <algorithm>

#include "vg_krylov.cuh"
#include "vg_pipe.cuh"

namespace vg {

namespace {

// [lo, hi) split into a scalar head up to a multiple of 4, 4-wide body, scalar tail; grid-stride
template <class F4, class F1>
__device__ __forceinline__ void for_range(long long lo, long long hi, F4 body4, F1 body1) {
    const long long tid = blockIdx.x * (long long)blockDim.x + threadIdx.x, nth = (long long)gridDim.x * blockDim.x;
    long long a = (lo + 3) & ~3LL;
    if (a > hi) a = hi;
    const long long b = a + ((hi - a) & ~3LL);
    for (long long i = lo + tid; i < a; i += nth) body1(i);
    for (long long i = a + 4 * tid; i < b; i += 4 * nth) body4(i);
    for (long long i = b + tid; i < hi; i += nth) body1(i);
}

// block + grid reduction of NV values; the last block to finish calls fin(total)
template <int NV, class F>
__device__ void grid_reduce(double (&v)[NV], double* partials, unsigned* counter, F fin) {
    __shared__ double sh[VEC_THREADS / 32][NV];
    __shared__ double tot[VEC_THREADS][NV];
    __shared__ bool last;
    const int t = threadIdx.x, w = t >> 5, l = t & 31;
#pragma unroll
    for (int i = 0; i < NV; ++i)
        for (int off = 16; off; off >>= 1) v[i] += __shfl_down_sync(0xffffffffu, v[i], off);
    if (l == 0)
#pragma unroll
        for (int i = 0; i < NV; ++i) sh[w][i] = v[i];
    __syncthreads();
    if (t == 0) {
        for (int i = 0; i < NV; ++i) {
            double s = 0;
            for (int k = 0; k < VEC_THREADS / 32; ++k) s += sh[k][i];
            partials[NV * blockIdx.x + i] = s;
        }
        __threadfence();
        last = atomicAdd(counter, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    double acc[NV];
#pragma unroll
    for (int i = 0; i < NV; ++i) acc[i] = 0;
    for (int b = t; b < (int)gridDim.x; b += VEC_THREADS)
#pragma unroll
        for (int i = 0; i < NV; ++i) acc[i] += __ldcg(partials + NV * b + i);
#pragma unroll
    for (int i = 0; i < NV; ++i) tot[t][i] = acc[i];
    __syncthreads();
    for (int s = VEC_THREADS / 2; s; s >>= 1) {
        if (t < s)
#pragma unroll
            for (int i = 0; i < NV; ++i) tot[t][i] += tot[t + s][i];
        __syncthreads();
    }
    if (t == 0) {
        double r[NV];
        for (int i = 0; i < NV; ++i) r[i] = tot[0][i];
        fin(r);
        *counter = 0u;
    }
}

__device__ __forceinline__ double cg_alpha(const Scalars* sc) {
    return sc->pq > CG_BREAK * sc->rz && isfinite(sc->pq) ? sc->rz / sc->pq : 0.0;
}

// an entry's share of r.D^{-1} r and of |r|^2 + |D^{-1} r|^2 (the jump's effect on the pressure and on the flux rows);
// edges whose pressure is given (dinv 0) have no residual
template <typename T>
__device__ __forceinline__ void cg_sums(T r, T dinv, double (&acc)[2]) {
    const double z = double(dinv * r);
    acc[0] += z * double(r);
    if (dinv != T(0)) acc[1] += double(r) * double(r) + z * z;
}

template <typename T>
__global__ void __launch_bounds__(VEC_THREADS) k_cg_init(const double* h, CgVecs<T> v, Scalars* sc,
                                                         int* flags, CgStop stop, double* partials, unsigned* counter) {
    const double scale = 1.0 / stop.scale();
    double acc[2] = {0, 0};
    for_range(
        0, v.n,
        [&](long long i) {
            double h4[4];
            T r4[4], di[4], z0[4] = {T(0), T(0), T(0), T(0)};
            ld4(h + i, h4);
            ld4(v.dinv + i, di);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                r4[j] = T(scale * h4[j]);
                cg_sums(r4[j], di[j], acc);
            }
            st4(v.r_new + i, r4);
            st4(v.x + i, z0);
            st4(v.p + i, z0);
            st4(v.q + i, z0);
        },
        [&](long long i) {
            const T r = T(scale * h[i]);
            cg_sums(r, v.dinv[i], acc);
            v.r_new[i] = r;
            v.x[i] = v.p[i] = v.q[i] = T(0);
        });
    grid_reduce<2>(acc, partials, counter, [&](double* tot) {
        sc->rr = tot[0];
        sc->raw = tot[1];
        sc->tol2 = stop.tol * stop.tol;
        sc->raw2 = stop.raw_abs() * stop.raw_abs();
        sc->floor2 = stop.floor * stop.floor;
        sc->pq = 0.0;
        sc->beta = 0.0;
        flags[0] = 0;
        flags[2] = 0;
    });
}

template <typename T>
__global__ void __launch_bounds__(VEC_THREADS) k_cg_edges(CgVecs<T> v, Scalars* sc, int* flags, double* partials,
                                                          unsigned* counter) {
    if (flags[0]) return;
    const T a = T(cg_alpha(sc));
    double acc[2] = {0, 0};
    for_range(
        0, v.n,
        [&](long long i) {
            T p4[4], q4[4], x4[4], r4[4], di[4];
            ld4(v.p + i, p4);
            ld4(v.q + i, q4);
            ld4(v.x + i, x4);
            ld4(v.r_old + i, r4);
            ld4(v.dinv + i, di);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                x4[j] += a * p4[j];
                r4[j] -= a * q4[j];
                cg_sums(r4[j], di[j], acc);
            }
            st4(v.x + i, x4);
            st4(v.r_new + i, r4);
        },
        [&](long long i) {
            v.x[i] += a * v.p[i];
            const T r = v.r_old[i] - a * v.q[i];
            cg_sums(r, v.dinv[i], acc);
            v.r_new[i] = r;
        });
    grid_reduce<2>(acc, partials, counter, [&](double* tot) {
        sc->rr = tot[0];
        sc->raw = tot[1];
    });
}

// one warp per piece, one lane per cell. The edge indices and weights of up to CELL_PRE edges are
// loaded before the gathers, so that a lane has all its gathers in flight at once.
constexpr int CELL_PRE = 8;
template <typename T>
__global__ void __launch_bounds__(VEC_THREADS) k_cg_cells(CgVecs<T> v, int first, const Scalars* sc, const int* flags) {
    // the V-cycle's first kernel (programmatic dependent launch) may start and copy its matrix rows
    pdl_trigger();
    const int w = int((blockIdx.x * (long long)VEC_THREADS + threadIdx.x) >> 5), lane = threadIdx.x & 31;
    if (flags[0] || w >= v.npieces) return;
    const Piece& P = v.pieces[w];
    if (lane >= P.count) return;
    const T a = first ? T(0) : T(cg_alpha(sc));
    const T* r = first ? v.r_new : v.r_old;
    const int* m = v.emap + P.e_off + lane;
    const T* cw = v.cw + P.e_off + lane;
    const int ne = P.ne;
    int g[CELL_PRE];
    T c[CELL_PRE], rv[CELL_PRE], qv[CELL_PRE];
#pragma unroll
    for (int e = 0; e < CELL_PRE; ++e) {
        g[e] = e < ne ? m[e * PIECE] : 0;
        c[e] = e < ne ? cw[e * PIECE] : T(0);
    }
#pragma unroll
    for (int e = 0; e < CELL_PRE; ++e) {
        rv[e] = e < ne ? r[g[e]] : T(0);
        qv[e] = e < ne ? v.q[g[e]] : T(0);
    }
    T s = T(0);
#pragma unroll
    for (int e = 0; e < CELL_PRE; ++e) s += c[e] * (rv[e] - a * qv[e]);
    for (int e = CELL_PRE; e < ne; ++e) s += cw[e * PIECE] * (r[m[e * PIECE]] - a * v.q[m[e * PIECE]]);
    v.rc[P.rank0 + lane] = s;
}

template <typename T>
__global__ void __launch_bounds__(VEC_THREADS) k_cg_finish(CgVecs<T> v, int first, long long cells, Scalars* sc,
                                                           int* flags, double* partials, unsigned* counter) {
    if (flags[0]) return;
    double acc[1] = {0};
    if (v.zc)
        for_range(
            0, cells,
            [&](long long i) {
                T z4[4], r4[4];
                ld4(v.zc + i, z4);
                ld4(v.rc + i, r4);
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[0] += double(z4[j]) * double(r4[j]);
            },
            [&](long long i) { acc[0] += double(v.zc[i]) * double(v.rc[i]); });
    grid_reduce<1>(acc, partials, counter, [&](double* tot) {
        const double rz = tot[0] + sc->rr;
        const bool ok = rz > 0 && isfinite(rz);
        if (first) {
            sc->rz0 = rz;
            sc->best = rz;
            sc->best_it = 0;
            sc->beta = 0.0;
            if (!ok) flags[0] = 1;
        } else {
            sc->beta = sc->rz > 0 ? rz / sc->rz : 0.0;
            flags[2] += 1;
            if (rz < sc->best) {
                sc->best = rz;
                sc->best_it = flags[2];
            }
            if (!ok || !(sc->pq > CG_BREAK * sc->rz) || cg_spent(rz, sc->best, flags[2] - sc->best_it, sc->rz0) || (rz <= sc->tol2 * sc->rz0 && sc->raw <= sc->raw2) || rz <= sc->floor2 * sc->rz0)
                flags[0] = 1;
        }
        sc->rz = rz;
    });
}

template <typename T>
__global__ void __launch_bounds__(VEC_THREADS) k_cg_direction(CgVecs<T> v, const Scalars* sc, const int* flags) {
    if (flags[0]) return;
    const T b = T(sc->beta);
    const long long tid = blockIdx.x * (long long)VEC_THREADS + threadIdx.x, nth = (long long)gridDim.x * VEC_THREADS;
    long long done = 0;
    if (v.zc) {  // the edges' mean moments, four per thread
        const long long body = v.edges & ~3LL;
        // written as a difference: a constant zc gives the same constant on the edges
        auto mean = [&](int cx, int cy, T w, T dinv) {
            const T zy = v.zc[cy], zx = v.zc[cx];
            return dinv != T(0) ? zy + w * (zx - zy) : T(0);
        };
        for (long long i = 4 * tid; i < body; i += 4 * nth) {
            T r4[4], p4[4], w4[4], di[4], z0[4] = {T(0), T(0), T(0), T(0)};
            const int4 ca = reinterpret_cast<const int4*>(v.ecell + i)[0], cb = reinterpret_cast<const int4*>(v.ecell + i)[1];
            ld4(v.ew + i, w4);
            ld4(v.dinv + i, di);
            ld4(v.r_new + i, r4);
            ld4(v.p + i, p4);
            const T m4[4] = {mean(ca.x, ca.y, w4[0], di[0]), mean(ca.z, ca.w, w4[1], di[1]),
                             mean(cb.x, cb.y, w4[2], di[2]), mean(cb.z, cb.w, w4[3], di[3])};
#pragma unroll
            for (int j = 0; j < 4; ++j) p4[j] = di[j] * r4[j] + m4[j] + b * p4[j];
            st4(v.p + i, p4);
            st4(v.q + i, z0);
        }
        for (long long i = body + tid; i < v.edges; i += nth) {
            const int2 c = v.ecell[i];
            v.p[i] = v.dinv[i] * v.r_new[i] + mean(c.x, c.y, v.ew[i], v.dinv[i]) + b * v.p[i];
            v.q[i] = T(0);
        }
        done = v.edges;
    }
    for_range(
        done, v.n,
        [&](long long i) {
            T r4[4], p4[4], di[4], z0[4] = {T(0), T(0), T(0), T(0)};
            ld4(v.r_new + i, r4);
            ld4(v.dinv + i, di);
            ld4(v.p + i, p4);
#pragma unroll
            for (int j = 0; j < 4; ++j) p4[j] = di[j] * r4[j] + b * p4[j];
            st4(v.p + i, p4);
            st4(v.q + i, z0);
        },
        [&](long long i) {
            v.p[i] = v.dinv[i] * v.r_new[i] + b * v.p[i];
            v.q[i] = T(0);
        });
}

// ---- MINRES (Paige-Saunders, unnormalised Lanczos vectors, symmetric positive definite preconditioner) ----
__device__ void minres_start(MinresScalars* sc, int* flags, double g2, double tol) {
    const double g = sqrt(fmax(g2, 0.0));
    sc->gam = g;
    sc->gam_prev = 1.0;
    sc->c_prev = 1.0;
    sc->c = 1.0;
    sc->s_prev = 0.0;
    sc->s = 0.0;
    sc->eta = g;
    sc->eta0 = g;
    sc->tol = tol;
    flags[0] = (g > 0 && isfinite(g)) ? 0 : 1;
    flags[1] = 0;
    flags[2] = 0;
}

// Givens rotation and residual estimate once gamma_{j+1}^2 is known
__device__ void minres_scalars(MinresScalars* sc, int* flags, double gn2) {
    const double g = sc->gam, dl = sc->delta / (g * g);
    const double gn = sqrt(fmax(gn2, 0.0));
    const double c = sc->c, cp = sc->c_prev, s = sc->s, sp = sc->s_prev, eta = sc->eta;
    const double a0 = c * dl - cp * s * g;
    const double a1 = sqrt(a0 * a0 + gn * gn);
    const double a2 = s * dl + cp * c * g;
    const double a3 = sp * g;
    const bool ok = a1 > 0 && isfinite(a1);
    const double cn = ok ? a0 / a1 : 1.0, sn = ok ? gn / a1 : 0.0;
    sc->a1 = ok ? a1 : 1.0;
    sc->a2 = a2;
    sc->a3 = a3;
    sc->zscale = 1.0 / g;
    sc->xcoef = ok ? cn * eta : 0.0;
    sc->eta = -sn * eta;
    sc->c_prev = c;
    sc->c = cn;
    sc->s_prev = s;
    sc->s = sn;
    sc->gam_prev = g;
    sc->gam = gn;
    flags[1] = ok ? 1 : 0;
    flags[2] += 1;
    if (!ok || !(gn > 0) || fabs(sc->eta) <= sc->tol * sc->eta0) flags[0] = 1;
}

template <typename T>
__global__ void __launch_bounds__(VEC_THREADS) k_minres_init(const T* r, MinresVecs<T> v, MinresScalars* sc,
                                                             double* partials, unsigned* counter) {
    double acc[1] = {0};
    auto one = [&](long long i) {
        const T ri = r[i];
        v.v_cur[i] = ri;
        v.v_old[i] = v.w_cur[i] = v.w_old[i] = v.y[i] = T(0);
        if (i < v.nf) {
            const T zi = v.dinv[i] * ri;
            v.z_cur[i] = zi;
            acc[0] += double(zi) * double(ri);
        }
    };
    for_range(
        0, v.n,
        [&](long long i) {
            if (i < v.nf && i + 3 >= v.nf) {  // the four entries at the end of the flux rows
                for (int j = 0; j < 4; ++j) one(i + j);
                return;
            }
            T r4[4], z0[4] = {T(0), T(0), T(0), T(0)};
            ld4(r + i, r4);
            st4(v.v_cur + i, r4);
            st4(v.v_old + i, z0);
            st4(v.w_cur + i, z0);
            st4(v.w_old + i, z0);
            st4(v.y + i, z0);
            if (i >= v.nf) return;
            T d4[4], zi[4];
            ld4(v.dinv + i, d4);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                zi[j] = d4[j] * r4[j];
                acc[0] += double(zi[j]) * double(r4[j]);
            }
            st4(v.z_cur + i, zi);
        },
        one);
    grid_reduce<1>(acc, partials, counter, [&](double* tot) { sc->dot = tot[0]; });
}

template <bool FLUX, typename T>
__global__ void __launch_bounds__(VEC_THREADS) k_minres_update(MinresVecs<T> v, MinresScalars* sc, int* flags,
                                                               double* partials, unsigned* counter) {
    // the first V-cycle kernel after this one (launched with programmatic dependent launch) may
    // start now and copy its matrix rows while the update runs; it waits for the update's results
    pdl_trigger();
    if (flags[0]) {
        if (FLUX && blockIdx.x == 0 && threadIdx.x == 0) flags[1] = 0;
        return;
    }
    const double g = sc->gam, gp = sc->gam_prev, dl = sc->delta / (g * g);
    const T f1 = T(1.0 / g), f2 = T(dl / g), f3 = T(g / gp);
    double acc[1] = {0};
    for_range(
        FLUX ? 0 : v.nf, FLUX ? v.nf : v.n,
        [&](long long i) {
            T y4[4], vc[4], vo[4], vn[4], z0[4] = {T(0), T(0), T(0), T(0)};
            ld4(v.y + i, y4);
            ld4(v.v_cur + i, vc);
            ld4(v.v_old + i, vo);
#pragma unroll
            for (int j = 0; j < 4; ++j) vn[j] = y4[j] * f1 - f2 * vc[j] - f3 * vo[j];
            st4(v.v_old + i, vn);
            st4(v.y + i, z0);
            if (!FLUX) return;
            T d4[4], zn[4];
            ld4(v.dinv + i, d4);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                zn[j] = d4[j] * vn[j];
                acc[0] += double(zn[j]) * double(vn[j]);
            }
            st4(v.z_new + i, zn);
        },
        [&](long long i) {
            const T vn = v.y[i] * f1 - f2 * v.v_cur[i] - f3 * v.v_old[i];
            v.v_old[i] = vn;
            v.y[i] = T(0);
            if (!FLUX) return;
            const T zn = v.dinv[i] * vn;
            v.z_new[i] = zn;
            acc[0] += double(zn) * double(vn);
        });
    if (FLUX) grid_reduce<1>(acc, partials, counter, [&](double* tot) { sc->dot = tot[0]; });
}

template <typename T>
__global__ void __launch_bounds__(VEC_THREADS) k_minres_finish(const T* z, const T* vv, long long nf, long long n,
                                                               int first, double tol, MinresScalars* sc, int* flags,
                                                               double* partials, unsigned* counter) {
    if (!first && flags[0]) return;
    double acc[1] = {0};
    for_range(
        nf, n,
        [&](long long i) {
            T z4[4], v4[4];
            ld4(z + i, z4);
            ld4(vv + i, v4);
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[0] += double(z4[j]) * double(v4[j]);
        },
        [&](long long i) { acc[0] += double(z[i]) * double(vv[i]); });
    grid_reduce<1>(acc, partials, counter, [&](double* tot) {
        const double g2 = tot[0] + sc->dot;
        if (first)
            minres_start(sc, flags, g2, tol);
        else
            minres_scalars(sc, flags, g2);
    });
}

template <typename T>
__global__ void __launch_bounds__(VEC_THREADS) k_minres_step(MinresVecs<T> v, MinresScalars* sc, int* flags) {
    if (!flags[1]) return;
    const T zs = T(sc->zscale), a2 = T(sc->a2), a3 = T(sc->a3), ia1 = T(1.0 / sc->a1), xc = T(sc->xcoef);
    for_range(
        0, v.n,
        [&](long long i) {
            T z4[4], wo[4], wc[4], x4[4], wn[4];
            ld4(v.z_cur + i, z4);
            ld4(v.w_old + i, wo);
            ld4(v.w_cur + i, wc);
            ld4(v.x + i, x4);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                wn[j] = (z4[j] * zs - a3 * wo[j] - a2 * wc[j]) * ia1;
                x4[j] += xc * wn[j];
            }
            st4(v.w_old + i, wn);
            st4(v.x + i, x4);
        },
        [&](long long i) {
            const T wn = (v.z_cur[i] * zs - a3 * v.w_old[i] - a2 * v.w_cur[i]) * ia1;
            v.w_old[i] = wn;
            v.x[i] += xc * wn;
        });
}

__global__ void k_to_float(const double* in, float* out, double scale, long long n) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        out[i] = float(scale * in[i]);
}

__global__ void k_axpy_from_float(double* x, const float* d, double scale, long long n) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        x[i] += scale * double(d[i]);
}

// end of one body of the graph's while loop: continue while not converged and below the cap
__global__ void k_loop_check(cudaGraphConditionalHandle h, const int* flags, int* loop) {
    int c = ++loop[0];
    cudaGraphSetConditional(h, (flags[0] == 0 && c < loop[1]) ? 1u : 0u);
}

__global__ void __launch_bounds__(VEC_THREADS) k_residual64(const double* b, const double* y, double* r, long long n,
                                                            double* red, double* partials, unsigned* counter) {
    double acc[2] = {0, 0};
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        double bi = b[i], ri = bi - y[i];
        r[i] = ri;
        acc[0] += ri * ri;
        acc[1] += bi * bi;
    }
    grid_reduce<2>(acc, partials, counter, [&](double* tot) {
        red[0] = tot[0];
        red[1] = tot[1];
    });
}

__global__ void __launch_bounds__(VEC_THREADS) k_start_residual(const double* b, const int* i2e, long long nf,
                                                                long long n, double* bs, double* r, double* x,
                                                                double* red, double* partials, unsigned* counter) {
    double acc[1] = {0};
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const double v = b[i2e[i]], w = i < nf ? v : -v;
        bs[i] = w;
        r[i] = w;
        if (x) x[i] = 0.0;
        acc[0] += w * w;
    }
    grid_reduce<1>(acc, partials, counter, [&](double* tot) { red[0] = red[1] = tot[0]; });
}

// sums over the cells for flux_multiplier (grid-wide, fixed order)
__global__ void __launch_bounds__(VEC_THREADS) k_flux_sums(const double* r, const double* p, const double* L,
                                                           long long cells, int q, long long nf, long long n,
                                                           double* out, double* partials, unsigned* counter) {
    double acc[2] = {0, 0};
    for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < cells; c += (long long)gridDim.x * blockDim.x) {
        if (p)
            for (int t = 0; t < q; ++t) acc[0] += L[c * q + t] * p[nf + c * q + t];
        else
            acc[0] -= r[nf + c * q];
        acc[1] += L[c * q];
    }
    grid_reduce<2>(acc, partials, counter, [&](double* tot) {
        if (p)
            out[1] = (-r[n - 1] - tot[0]) / tot[1];
        else
            out[0] = tot[0] / tot[1];
    });
}

__global__ void k_flux_shift(const double* out, long long cells, int q, long long nf, long long n, double* p) {
    for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < cells; c += (long long)gridDim.x * blockDim.x)
        p[nf + c * q] += out[1];
    if (blockIdx.x == 0 && threadIdx.x == 0) p[n - 1] = out[0];
}

__global__ void k_flip(const double* in, double* out, long long nf, long long n) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        out[i] = i < nf ? in[i] : -in[i];
}

}  // namespace

// grid of a vector kernel over n entries, 4 a thread, a function of n alone (fixed-shape reductions); small meshes
// do not pay for 592 block partials
static int vec_blocks(long long n) {
    return int(std::max<long long>(1, std::min<long long>(VEC_BLOCKS, (n + 4 * VEC_THREADS - 1) / (4 * VEC_THREADS))));
}

// the 4-wide kernels need every vector on a 16-byte boundary (cudaMalloc gives 256)
template <typename T>
void check_aligned(const CgVecs<T>& v) {
    const void* ps[] = {v.p, v.q, v.x, v.r_old, v.r_new, v.rc, v.zc, v.dinv, v.ecell, v.ew};
    for (const void* p : ps)
        if (reinterpret_cast<uintptr_t>(p) % 16) throw Error(VG_EINVAL, "Krylov vectors must be 16-byte aligned");
}

template <typename T>
void cg_init(const double* h, CgVecs<T> v, Scalars* sc, int* flags, CgStop stop, double* partials, unsigned* counter,
             cudaStream_t st) {
    check_aligned(v);
    k_cg_init<T><<<vec_blocks(v.n), VEC_THREADS, 0, st>>>(h, v, sc, flags, stop, partials, counter);
    VG_CUDA(cudaGetLastError());
}

template <typename T>
void cg_edges(CgVecs<T> v, Scalars* sc, int* flags, double* partials, unsigned* counter, cudaStream_t s) {
    k_cg_edges<T><<<vec_blocks(v.n), VEC_THREADS, 0, s>>>(v, sc, flags, partials, counter);
    VG_CUDA(cudaGetLastError());
}

template <typename T>
void cg_cells(CgVecs<T> v, int first, Scalars* sc, int* flags, cudaStream_t s) {
    const int blocks = int(((long long)v.npieces * 32 + VEC_THREADS - 1) / VEC_THREADS);
    k_cg_cells<T><<<blocks, VEC_THREADS, 0, s>>>(v, first, sc, flags);
    VG_CUDA(cudaGetLastError());
}

template <typename T>
void cg_finish(CgVecs<T> v, int first, long long cells, Scalars* sc, int* flags, double* partials, unsigned* counter,
               cudaStream_t s) {
    k_cg_finish<T><<<vec_blocks(cells), VEC_THREADS, 0, s>>>(v, first, cells, sc, flags, partials, counter);
    VG_CUDA(cudaGetLastError());
}

template <typename T>
void cg_direction(CgVecs<T> v, Scalars* sc, int* flags, cudaStream_t s) {
    const int blocks = int(std::max<long long>(1, std::min<long long>(VEC_BLOCKS * 2, (v.n / 4 + VEC_THREADS) / VEC_THREADS)));
    k_cg_direction<T><<<blocks, VEC_THREADS, 0, s>>>(v, sc, flags);
    VG_CUDA(cudaGetLastError());
}

#define VG_CG_INSTANCES(T)                                                                                          \
    template void cg_init<T>(const double*, CgVecs<T>, Scalars*, int*, CgStop, double*, unsigned*,                  \
                             cudaStream_t);                                                                         \
    template void cg_edges<T>(CgVecs<T>, Scalars*, int*, double*, unsigned*, cudaStream_t);                         \
    template void cg_cells<T>(CgVecs<T>, int, Scalars*, int*, cudaStream_t);                                        \
    template void cg_finish<T>(CgVecs<T>, int, long long, Scalars*, int*, double*, unsigned*, cudaStream_t);        \
    template void cg_direction<T>(CgVecs<T>, Scalars*, int*, cudaStream_t);
VG_CG_INSTANCES(double)
VG_CG_INSTANCES(float)
#undef VG_CG_INSTANCES

template <typename T>
void check_aligned(const MinresVecs<T>& v, const T* extra = nullptr) {
    const void* ps[] = {v.v_cur, v.v_old, v.z_cur, v.z_new, v.w_cur, v.w_old, v.y, v.x, v.dinv, extra};
    for (const void* p : ps)
        if (reinterpret_cast<uintptr_t>(p) % 16) throw Error(VG_EINVAL, "Krylov vectors must be 16-byte aligned");
}

template <typename T>
void minres_init(const T* r, MinresVecs<T> v, MinresScalars* sc, double* partials, unsigned* counter, cudaStream_t s) {
    check_aligned(v, r);
    k_minres_init<T><<<VEC_BLOCKS, VEC_THREADS, 0, s>>>(r, v, sc, partials, counter);
    VG_CUDA(cudaGetLastError());
}

template <typename T>
void minres_update(MinresVecs<T> v, bool flux, MinresScalars* sc, int* flags, double* partials, unsigned* counter,
                   cudaStream_t s) {
    if (flux)
        k_minres_update<true, T><<<VEC_BLOCKS, VEC_THREADS, 0, s>>>(v, sc, flags, partials, counter);
    else
        k_minres_update<false, T><<<vec_blocks(v.n - v.nf), VEC_THREADS, 0, s>>>(v, sc, flags, partials, counter);
    VG_CUDA(cudaGetLastError());
}

template <typename T>
void minres_finish(const T* z, const T* v, long long nf, long long n, bool first, double tol, MinresScalars* sc,
                   int* flags, double* partials, unsigned* counter, cudaStream_t s) {
    k_minres_finish<T><<<VEC_BLOCKS, VEC_THREADS, 0, s>>>(z, v, nf, n, first, tol, sc, flags, partials, counter);
    VG_CUDA(cudaGetLastError());
}

template <typename T>
void minres_step(MinresVecs<T> v, MinresScalars* sc, int* flags, cudaStream_t s) {
    k_minres_step<T><<<VEC_BLOCKS, VEC_THREADS, 0, s>>>(v, sc, flags);
    VG_CUDA(cudaGetLastError());
}

#define VG_MINRES_INSTANCES(T)                                                                                      \
    template void minres_init<T>(const T*, MinresVecs<T>, MinresScalars*, double*, unsigned*, cudaStream_t);        \
    template void minres_update<T>(MinresVecs<T>, bool, MinresScalars*, int*, double*, unsigned*, cudaStream_t);    \
    template void minres_finish<T>(const T*, const T*, long long, long long, bool, double, MinresScalars*, int*,    \
                                   double*, unsigned*, cudaStream_t);                                               \
    template void minres_step<T>(MinresVecs<T>, MinresScalars*, int*, cudaStream_t);
VG_MINRES_INSTANCES(double)
VG_MINRES_INSTANCES(float)
#undef VG_MINRES_INSTANCES

void to_float(const double* in, float* out, double scale, long long n, cudaStream_t s) {
    k_to_float<<<vec_blocks(n), VEC_THREADS, 0, s>>>(in, out, scale, n);
    VG_CUDA(cudaGetLastError());
}

void axpy_from_float(double* x, const float* d, double scale, long long n, cudaStream_t s) {
    k_axpy_from_float<<<vec_blocks(n), VEC_THREADS, 0, s>>>(x, d, scale, n);
    VG_CUDA(cudaGetLastError());
}

void loop_check(cudaGraphConditionalHandle h, const int* flags, int* loop, cudaStream_t s) {
    k_loop_check<<<1, 1, 0, s>>>(h, flags, loop);
    VG_CUDA(cudaGetLastError());
}

void residual64(const double* b, const double* y, double* r, long long n, double* red, double* partials,
                unsigned* counter, cudaStream_t s) {
    k_residual64<<<vec_blocks(n), VEC_THREADS, 0, s>>>(b, y, r, n, red, partials, counter);
    VG_CUDA(cudaGetLastError());
}

void flux_multiplier(const double* r, double* p, const double* L, long long cells, int q, long long nf, long long n,
                     double* out, double* partials, unsigned* counter, cudaStream_t s) {
    k_flux_sums<<<vec_blocks(cells), VEC_THREADS, 0, s>>>(r, p, L, cells, q, nf, n, out, partials, counter);
    if (p) k_flux_shift<<<vec_blocks(cells), VEC_THREADS, 0, s>>>(out, cells, q, nf, n, p);
    VG_CUDA(cudaGetLastError());
}

void start_residual(const double* b, const int* i2e, long long nf, long long n, double* bs, double* r, double* x,
                    double* red, double* partials, unsigned* counter, cudaStream_t s) {
    k_start_residual<<<vec_blocks(n), VEC_THREADS, 0, s>>>(b, i2e, nf, n, bs, r, x, red, partials, counter);
    VG_CUDA(cudaGetLastError());
}

void flip_pressure(const double* in, double* out, long long nf, long long n, cudaStream_t s) {
    k_flip<<<vec_blocks(n), VEC_THREADS, 0, s>>>(in, out, nf, n);
    VG_CUDA(cudaGetLastError());
}

}  // namespace vg

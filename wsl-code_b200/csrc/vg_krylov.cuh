// Krylov kernels: preconditioned conjugate gradients on the edge pressures (the hybridised system,
// vg_hybrid.cu), FP64 residuals for iterative refinement, small vector kernels.
#pragma once
#include "vg_common.cuh"

namespace vg {

// CG scalars, device resident (double precision for both FP64 and FP32 inner solves)
struct Scalars {
    double rz, rz0;    // r.z of the current residual and of the first one
    double pq;         // p.S p (written by the edge apply)
    double beta;       // r.z / previous r.z
    double rr, raw;    // r.D^{-1} r and |r|^2 + |D^{-1} r|^2: what the flux jumps leave in the pressure and flux rows
    double tol2;       // stop at rz <= tol2 rz0 and raw <= raw2, or at rz <= floor2 rz0
    double raw2, floor2;
    double best;       // smallest r.z so far, reached at iteration best_it
    int best_it;
};
// flags[0] = stop (converged or breakdown), flags[2] = iterations
constexpr int NFLAGS = 4;

// What ends a loop that has not met its test: r.z far above the smallest one so far, or no new smallest one for long. A
// loop that has gained ten digits is at its rounding level and is given neither. With the flux given the constants are in
// the kernel of S; what rounding has put of them into r then grows from step to step and takes the digits of x with it, so
// that such a loop has to end at once (33 cells, 1e4 in permeability between them, tolerance 1e-12: residual 3e16 after
// 1,136 iterations; now 5e-14 after 33). Solves of degree 4 take 400 to 600 iterations either way.
__host__ __device__ inline bool cg_spent(double rz, double best, int since, double rz0) {
    const bool deep = best <= 1e-20 * rz0;
    return rz > (deep ? 1e2 : 1e8) * best || since >= (deep ? 100 : 1000);
}
// A step of more than 1 / CG_BREAK along p is none: p is a constant then and p.q rounding.
constexpr double CG_BREAK = 1e-10;

constexpr int VEC_BLOCKS = 148 * 4;  // grid of the vector kernels (fixed: deterministic reductions)
constexpr int VEC_THREADS = 256;

// weight of the diagonal beside the cells' V-cycle in the preconditioner z = EDGE_RELAX D^{-1} r + Pi V Pi^T r (k = 0:
// 23 iterations with 1, 21 with 0.75 to 0.85 at 60k cells; k >= 1 does not care between 0.75 and 1)
constexpr double EDGE_RELAX = 0.85;

// vectors and fixed data of the solve on the edge pressures
template <typename T>
struct CgVecs {
    T *p, *q, *x, *r_old, *r_new;  // (k + 1) * edges
    T *rc, *zc;                    // cells: restricted residual, V-cycle's result (null: diagonal only)
    const T* dinv;                 // EDGE_RELAX / diagonal, 0 on edges whose pressure is given
    const int* emap;               // edge per (cell, local edge), piece layout
    const T* cw;                   // weight of the cell in the edge's interpolated pressure, piece layout
    const int2* ecell;             // the (one or two) cells of an edge, as ranks
    const T* ew;                   // weight of the first of them (the second has 1 - it)
    const Piece* pieces;
    int npieces;
    long long edges, n;            // edges, (k + 1) * edges
};

// what ends a loop, and the unit its vectors are in. |b| (of the solve's right-hand side) is on the device, so that
// a solve from a zero guess starts its loop without a host round trip.
struct CgStop {
    double tol, floor;   // relative preconditioned norm and its floor
    double raw;          // jump norm over |b|
    double unit;         // residual over |b| that the loop's vectors are scaled by, 0: not scaled
    const double* b2;    // |b|^2
    __device__ double norm_b() const { return *b2 > 0 ? sqrt(*b2) : 1.0; }
    __device__ double scale() const { return unit > 0 ? unit * norm_b() : 1.0; }
    __device__ double raw_abs() const { return raw * norm_b() / scale(); }
};

// x = p = q = 0, r_new = h / unit, edge sums of the first residual
template <typename T>
void cg_init(const double* h, CgVecs<T> v, Scalars* sc, int* flags, CgStop stop, double* partials, unsigned* counter,
             cudaStream_t st);
// x += alpha p, r_new = r_old - alpha q, edge sums (alpha = rz / pq)
template <typename T>
void cg_edges(CgVecs<T> v, Scalars* sc, int* flags, double* partials, unsigned* counter, cudaStream_t s);
// rc = restriction of r_old - alpha q to the cells (first: of r_new)
template <typename T>
void cg_cells(CgVecs<T> v, int first, Scalars* sc, int* flags, cudaStream_t s);
// rz = rr + rc.zc, beta, stop test
template <typename T>
void cg_finish(CgVecs<T> v, int first, long long cells, Scalars* sc, int* flags, double* partials, unsigned* counter,
               cudaStream_t s);
// p = z + beta p with z = D^{-1} r_new + (interpolated zc), q = 0
template <typename T>
void cg_direction(CgVecs<T> v, Scalars* sc, int* flags, cudaStream_t s);

// graph while-loop condition: loop[0] = bodies run (incremented here), loop[1] = cap on bodies
void loop_check(cudaGraphConditionalHandle h, const int* flags, int* loop, cudaStream_t s);
// r = b - y (FP64), red[0] = ||r||^2, red[1] = ||b||^2 (deterministic)
void residual64(const double* b, const double* y, double* r, long long n, double* red, double* partials,
                unsigned* counter, cudaStream_t s);
// out = sign-flip of the pressure / multiplier block: out[i] = (i < nf ? 1 : -1) * in[i]
void flip_pressure(const double* in, double* out, long long nf, long long n, cudaStream_t s);
// ---- MINRES on the saddle-point form (vg_minres.cu) ----
// scalars, device resident (double precision for both FP64 and FP32 inner solves)
struct MinresScalars {
    double gam_prev, gam, delta;   // gamma_{j-1}, gamma_j, raw z_j^T K z_j (from the apply)
    double c_prev, c, s_prev, s;   // Givens c_{j-1}, c_j, s_{j-1}, s_j
    double eta, eta0, tol;         // residual estimate |eta| (preconditioner norm), stop at tol * eta0
    double a1, a2, a3, xcoef, zscale;
    double dot;                    // z.v of the flux rows, until the pressure rows' share is known
};
// flags[0] = stop (converged or breakdown), flags[1] = current iteration valid, flags[2] = iterations

// vectors of n entries, internal order: nf flux rows (dinv: their inverse diagonal), then pressure rows, whose part of
// z is written by the V-cycle between the calls below
template <typename T>
struct MinresVecs {
    T *v_cur, *v_old, *z_cur, *z_new, *w_cur, *w_old, *y, *x;
    const T* dinv;
    long long nf, n;
};
// v_cur = r, z = dinv r on the flux rows, everything else zero
template <typename T>
void minres_init(const T* r, MinresVecs<T> v, MinresScalars* sc, double* partials, unsigned* counter, cudaStream_t s);
// v_new = y/g - (d/g) v_cur - (g/g_prev) v_old (into v_old), y = 0; flux: the flux rows, with z_new = dinv v_new and its
// share of gamma^2; else the pressure rows
template <typename T>
void minres_update(MinresVecs<T> v, bool flux, MinresScalars* sc, int* flags, double* partials, unsigned* counter,
                   cudaStream_t s);
// the pressure rows' share of gamma^2 = z.v after the V-cycle, then the scalar recurrences (first: their start)
template <typename T>
void minres_finish(const T* z, const T* v, long long nf, long long n, bool first, double tol, MinresScalars* sc,
                   int* flags, double* partials, unsigned* counter, cudaStream_t s);
// w_new = (z_cur/g - a3 w_old - a2 w_cur)/a1 (into w_old), x += xcoef w_new
template <typename T>
void minres_step(MinresVecs<T> v, MinresScalars* sc, int* flags, cudaStream_t s);
// out32 = float(scale in64); x64 += scale double(d32)
void to_float(const double* in, float* out, double scale, long long n, cudaStream_t s);
void axpy_from_float(double* x, const float* d, double scale, long long n, cudaStream_t s);

// start of a solve: bs = r = b in the internal order (i2e) with the pressure and multiplier rows negated, x = 0 (null:
// left alone), red[0] = red[1] = |b|^2 (deterministic)
void start_residual(const double* b, const int* i2e, long long nf, long long n, double* bs, double* r, double* x,
                    double* red, double* partials, unsigned* counter, cudaStream_t s);
// flux condition, internal order, L the multiplier vector (q per cell). p null: out[0] = the multiplier that makes the
// mean rows of the residual r compatible. With p, the correction so far: its mean pressures are shifted so that the
// multiplier row holds, and the multiplier is stored
void flux_multiplier(const double* r, double* p, const double* L, long long cells, int q, long long nf, long long n,
                     double* out, double* partials, unsigned* counter, cudaStream_t s);
// x += a d (FP64)
void axpy64_kernel_launch(double* x, const double* d, double a, long long n, cudaStream_t s);

}  // namespace vg

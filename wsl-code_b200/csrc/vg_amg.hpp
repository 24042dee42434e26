// Smoothed-aggregation algebraic multigrid for a weighted graph Laplacian S on the cells: the coarse
// part of the edge-pressure preconditioner (vg_hybrid.cu); per species that of a Maxwell-Stefan step
// (vg_ms.cu: conductances 1 / (sum over an edge's sides of 1 / (T_ii (B^{-1})_ss)), plus |E|/dt); and the
// pressure rows of MINRES (vg_minres.cu: conductances 1 / A_ii).
//
// The reference preconditions with a PETSc ILU(0) on the CPU or, matrix-free, with the diagonal
// |rate M| + sum W^2/d (vem/CurvedVEM_Darcy_gpu/src/krylov.cu:99-117, src/equation_gpu.cu:282-315),
// which its own notes call weak for large meshes. Here one symmetric V-cycle on S (Jacobi pre- and
// post-smoothing with the same weight, exact coarsest solve), built on the host once per operator and
// applied on the device.
//
// The cycle runs in a composite form with the same operator. With S_l = smooth_l D_l^{-1}, one
// pre-smoothing step from zero, the residual, the restriction, the coarse correction and one
// post-smoothing step give, level by level,
//     r = b - A S b,   b_c = Pt^T b,   z = S (b + r) + Pt x_c,   Pt = (I - S A) P,
// because P^T (I - A S) = ((I - S A) P)^T for a symmetric A. Per level this is two dependent
// products on the cycle's critical path (the restriction by Pt^T and the prolongation by Pt)
// instead of four, and the residual, which only the prolongation of the same level reads, runs on
// a second stream beside the coarser levels.
#pragma once
#include <vector>

#include "vg_common.cuh"

namespace vg {

struct HostCsr {
    int n = 0, m = 0;  // rows, columns
    std::vector<int> ptr, col;
    std::vector<double> val;
};

// sliced ELL with slice height 32: entry k of row r lives at soff[r / 32] + k * 32 + r % 32,
// padding entries have col = 0 and val = 0
template <typename T>
struct DevSell {
    int n = 0, nslices = 0;
    const long long* soff = nullptr;
    const int* width = nullptr;
    const int* col = nullptr;
    const T* val = nullptr;
};

// CSR for the rectangular transfer operators and the coarse Galerkin operators, processed in row
// blocks: block b covers rows [rb[b].x, rb[b + 1].x) and entries [rb[b].y, rb[b + 1].y)
template <typename T>
struct DevCsr {
    int n = 0, nblk = 0;
    int slots = 1;  // CTAs of the kernel resident at once on the device (grid cap)
    int lpr = 1;    // threads per row in the row-block kernel's sums (1, or 8 for long rows)
    const int2* rb = nullptr;
    int* err = nullptr;  // set to 1 when a staged copy never lands (never in a correct run)
    const int* ptr = nullptr;
    const int* col = nullptr;
    const T* val = nullptr;
    int nwb = 0;                // warp blocks: block w covers rows [wb[w].x, wb[w + 1].x), entries [wb[w].y, wb[w + 1].y)
    const int2* wb = nullptr;
};

// one level of the cycle as plain pointers (the single-launch solve walks the hierarchy inside its kernel)
template <typename T>
struct AmgLevelView {
    int n, nc;                     // rows here and on the next level
    DevSell<T> sell;               // A S in slices, or (sell.val null) as CSR:
    const int *aptr, *acol;
    const T* aval;
    const int *rptr, *rcol, *pptr, *pcol;  // Rt, Pt
    const T *rval, *pval, *S;
    bool a_wide, r_wide, p_wide;   // rows of ten entries and more on average
    T *r, *b, *x;                  // this level's smoothed residual; the next level's right-hand side and solution
};
constexpr int AMG_VIEW_LEVELS = 4;
template <typename T>
struct AmgView {
    int levels = 0, ncoarse = 0;   // levels above the dense one
    AmgLevelView<T> level[AMG_VIEW_LEVELS];
    const T* inverse = nullptr;
};

// coarsest level: at most this many rows, inverted densely (2500^2 doubles = 50 MB)
constexpr int COARSE_MAX = 2500;
// largest coarsest level accepted when coarsening stops early (level cap)
constexpr int DENSE_MAX = 4096;

class Amg {
public:
    Amg() = default;
    Amg(const Amg&) = delete;
    Amg& operator=(const Amg&) = delete;
    ~Amg();
    // build the hierarchy of S (host CSR, symmetric positive definite or semi-definite); fine_order, when
    // given, renumbers the finest level's rows for the vectors the cycle acts on (row i -> fine_order[i])
    // after S has been coarsened in its own order; err: the device address of
    // the owner's error word; constant_kernel: S has the constants as its kernel (so
    // has every coarse matrix, whose aggregates' prolongator keeps them), and the coarsest one is inverted
    // with the mean of its diagonal as the constants' eigenvalue; saddle: the hierarchy of MINRES (vg_minres.cu),
    // whose figures are to the bit those of the prolongator's weight in the smoother and of a coarsest inverse
    // formed pivot by pivot
    void setup(const HostCsr& S, int* err, const std::vector<int>* fine_order = nullptr, bool constant_kernel = false,
               bool saddle = false);
    bool ready() const { return !levels_.empty(); }
    int levels() const { return int(levels_.size()); }
    long long nnz() const;
    // z = V-cycle(b) on the device (b, z of length n0); FP64 or FP32 copy of the hierarchy
    void vcycle(const double* b, double* z, cudaStream_t s);
    void vcycle(const float* b, float* z, cudaStream_t s);
    long long launches = 0;
    // false when the hierarchy has more levels than a view holds
    template <typename T>
    bool view_levels(AmgView<T>& out);
    // Recompute every value of the hierarchy on the device for a new finest-level operator with the
    // same sparsity: the aggregates and sparsity patterns of setup() are kept, the weights follow the new values'
    // rho(D^{-1} A) (a bound on it on the finest level, an estimate on the others; the captured cycle's device addresses
    // do not change).
    // a0: the finest level's values in the order of its stored pattern (level0_ptr / level0_col).
    // safe: every level's weights held below the bound.
    void refresh(const double* a0, bool safe = false);
    const int* level0_ptr() const { return levels_.empty() ? nullptr : levels_[0].dpa_ptr.data(); }
    const int* level0_col() const { return levels_.empty() ? nullptr : levels_[0].dpa_col.data(); }
    long long level0_nnz() const { return levels_.empty() ? 0 : (long long)levels_[0].pa_col.size(); }

private:
    struct Sell {
        int n = 0, nslices = 0;
        std::vector<long long> soff;
        std::vector<int> width, col;
        std::vector<double> val;
        // CSR copy used instead of the slices when rows are long
        bool csr = false;
        std::vector<int> cptr, ccol;
        int lpr = 1;          // threads per row of the row-block sums
        std::vector<int> rb;  // row blocks: (first row, first entry) pairs, one past the last block included
        std::vector<int> wb;  // warp blocks (at most 32 rows and WS_CAP entries), same layout
        std::vector<double> cval;
    };
    struct CsrBufs {  // one CSR matrix on the device: row blocks, pattern, FP64 and FP32 values
        DevBuf<int> ptr, col, rb, wb;
        DevBuf<double> v64;
        DevBuf<float> v32;
    };
    struct Level {
        int n = 0, nc = 0;
        double omega = 0;   // prolongator smoothing, 4 / (3 rho(D^{-1} A))
        double rho = 0;     // the estimate of rho(D^{-1} A) that both come from
        double smooth = 0;  // the cycle's Jacobi smoothing, SMOOTH_WEIGHT / rho
        // A: the level's operator with its columns scaled by S = smooth D^{-1} (A S, for the residual
        // r = b - A S b); Pt = (I - S A) P: n x nc, Rt = Pt^T: nc x n (absent on the coarsest level)
        Sell A, Pt, Rt;
        std::vector<double> dinv;
        // structure kept for refresh(): stored CSR pattern of A, aggregate of every stored row, position in P of every R entry and in Pt of every Rt entry,
        // SELL slot of every CSR entry of A (SELL storage), patterns of P and R = P^T (FP64 values:
        // the Galerkin product of the next level is R A P)
        std::vector<int> pa_ptr, pa_col, agg, r2p, rt2pt;
        std::vector<long long> sellpos;
        DevBuf<int> dpa_ptr, dpa_col, dagg, dr2p, drt2pt;
        DevBuf<int> dpa_row, dpt_row;  // row of every stored entry of A and of Pt (first refresh)
        DevBuf<double> dap;            // A P on Pt's pattern (refresh)
        DevBuf<long long> dsellpos;
        DevBuf<double> dvals;  // unscaled stored values of A (levels below the finest; refresh)
        CsrBufs cP, cR;        // P and R (FP64 values only; refresh)
        // device storage of the cycle's matrices
        DevBuf<long long> dA_soff;
        DevBuf<int> dA_w, dA_col;
        DevBuf<double> dA_v64;
        DevBuf<float> dA_v32;
        CsrBufs cA, cPt, cRt;
        DevBuf<double> power;  // start of the power iteration (refresh)
        DevBuf<double> dinv64, s64, x64, b64, r64;  // s: S = smooth D^{-1}
        DevBuf<float> s32, x32, b32, r32;
    };
    template <typename T>
    void cycle(int l, const T* b, T* z, cudaStream_t s);
    // CSR -> dinvc64_ / dinvc32_, by panels or pivot by pivot
    void dense_inverse(const int* ptr, const int* col, const double* val, int n, bool pivotwise = false);
    template <typename T>
    DevSell<T> view(const Level& L) const;
    template <typename T>
    DevCsr<T> cview(const Sell& S, const CsrBufs& B) const;

    std::vector<Level> levels_;
    int ncoarse_ = 0;
    bool constant_kernel_ = false, saddle_ = false;
    DevBuf<double> rho_;  // refresh: rho(D^{-1} A) of every level, estimate and bound
    int* err_ = nullptr;  // the owner's error word: set when a cycle kernel gave up on a copy (never in a correct run)
    int csr_slots_[2] = {1, 1};  // resident CTAs of the CSR kernels on this hierarchy's device (FP32, FP64)
    DevBuf<double> dinvc64_;  // dense inverse of the coarsest matrix
    DevBuf<float> dinvc32_;
    // its workspace, kept for the next refresh: a second copy of the matrix, two panels' inverses, the outcome
    DevBuf<double> gj_work_, gj_d_;
    DevBuf<unsigned long long> gj_bad_;
    // second stream of the cycle (the residuals) and, per level, the events that fork it after the
    // level's right-hand side is written and join it before the level's prolongation
    cudaStream_t side_ = nullptr;
    std::vector<cudaEvent_t> ev_fork_, ev_join_;
    void release_streams();
};

}  // namespace vg

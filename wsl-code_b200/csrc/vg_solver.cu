// vemgpu Solver: host orchestration of the device setup, apply, Krylov solve, adjoint and errors.
#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstring>
#include <unordered_map>

#include "vg_apply.cuh"
#include "vg_krylov.cuh"
#include "vg_setup.cuh"
#include "vg_solver.hpp"

namespace vg {

void lift_rhs(const int* mask, const double* g, const double* y, double* b, long long N, cudaStream_t s);
void rescale_ops(const double* theta, const int* slot_cell, const Piece* pieces, int npieces, const double* A0,
                 double* A64, float* A32, cudaStream_t s);
void assemble_values(const double* A, const double* W, const int* map, const int* slot_cell, const int* mask,
                     const double* L, const Piece* pieces, int npieces, int k, long long nf, long long N,
                     int constrained, int mult, const long long* rp, const int* ci, double* val, int* bad,
                     cudaStream_t s);
template <typename T>
void gather_launch(const T* in, const int* idx, long long off, T* out, long long n, cudaStream_t s);
void contract_adjoint(const double* A, const int* map, const int* slot_cell, const int* mask, const Piece* pieces,
                      int npieces, int k, const double* x, const double* mu, int constrained, double* g,
                      cudaStream_t s);
long long first_nonfinite(const double* v, long long n, unsigned long long* scratch);

namespace {

// Gauss-Legendre rules on [-1, 1] (vem/CurvedVEM_Darcy_gpu/core/gauss_quadrature.cpp:74-167)
std::vector<double> gauss_legendre(int n) {
    struct H {
        double x, w;
    };
    std::vector<H> half;
    bool centre = false;
    double wc = 0;
    switch (n) {
    case 1: return {0.0, 2.0};
    case 2: half = {{0.5773502691896257645091488, 1.0}}; break;
    case 3: half = {{0.7745966692414833770358531, 0.5555555555555556}}; centre = true; wc = 0.8888888888888889; break;
    case 4: half = {{0.8611363115940526, 0.3478548451374539}, {0.3399810435848563, 0.6521451548625461}}; break;
    case 5:
        half = {{0.9061798459386640, 0.2369268850561891}, {0.5384693101056831, 0.4786286704993665}};
        centre = true;
        wc = 0.5688888888888889;
        break;
    case 6:
        half = {{0.9324695142031520, 0.1713244923791703}, {0.6612093864662645, 0.3607615730481386},
                {0.2386191860831969, 0.4679139345726910}};
        break;
    case 7:
        half = {{0.9491079123427585, 0.1294849661688697}, {0.7415311855993944, 0.2797053914892767},
                {0.4058451513773972, 0.3818300505051190}};
        centre = true;
        wc = 0.4179591836734694;
        break;
    case 8:
        half = {{0.9602898564975362, 0.1012285362903763}, {0.7966664774136267, 0.2223810344533745},
                {0.5255324099163290, 0.3137066458778873}, {0.1834346424956498, 0.3626837833783620}};
        break;
    case 9:
        half = {{0.9681602395076261, 0.0812743883615744}, {0.8360311073266358, 0.1806481606948574},
                {0.6133714327005904, 0.2606106964029355}, {0.3242534234038089, 0.3123470770400028}};
        centre = true;
        wc = 0.3302393550012598;
        break;
    case 10:
        half = {{0.9739065285171717, 0.0666713443086881}, {0.8650633666889845, 0.1494513491505806},
                {0.6794095682990244, 0.2190863625159820}, {0.4333953941292472, 0.2692667193099964},
                {0.1488743389816312, 0.2955242247147529}};
        break;
    default: throw Error(VG_EINVAL, "Gauss-Legendre order must be 1..10");
    }
    std::vector<double> out;
    for (auto& h : half) {
        out.push_back(-h.x);
        out.push_back(h.w);
    }
    if (centre) {
        out.push_back(0.0);
        out.push_back(wc);
    }
    for (auto it = half.rbegin(); it != half.rend(); ++it) {
        out.push_back(it->x);
        out.push_back(it->w);
    }
    return out;
}

// triangle rules as (xi, eta, w) on the reference triangle (gauss_quadrature.cpp:258-305) and the
// 36-point Duffy rule of vem/CurvedVEM_Darcy_gpu/src/mesh_pack.cpp:110-124 written the same way
std::vector<double> triangle_rule(int n) {
    std::vector<double> r;
    auto add = [&](double a, double b, double w) {
        r.push_back(a);
        r.push_back(b);
        r.push_back(w);
    };
    switch (n) {
    case 1: add(1.0 / 3.0, 1.0 / 3.0, 0.5); break;
    case 3:
        add(0.5, 0.0, 1.0 / 6.0);
        add(0.5, 0.5, 1.0 / 6.0);
        add(0.0, 0.5, 1.0 / 6.0);
        break;
    case 4: {
        double s = 1.0 / std::sqrt(3.0);
        add((1 + s) / 2, (1 - s) * (1 + s) / 4, (1 - s) / 8.0);
        add((1 + s) / 2, (1 - s) * (1 - s) / 4, (1 - s) / 8.0);
        add((1 - s) / 2, (1 + s) * (1 + s) / 4, (1 + s) / 8.0);
        add((1 - s) / 2, (1 + s) * (1 - s) / 4, (1 + s) / 8.0);
        break;
    }
    case 7: {
        add(1.0 / 3.0, 1.0 / 3.0, 0.1125);
        double a = 0.797426985353087, b = 0.101286507323456, w1 = 0.0629695902724135;
        add(a, b, w1);
        add(b, a, w1);
        add(b, b, w1);
        double c = 0.059715871789770, d = 0.470142064105115, w2 = 0.0661970763907399;
        add(c, d, w2);
        add(d, c, w2);
        add(d, d, w2);
        break;
    }
    case 9: {
        double s = std::sqrt(3.0 / 5.0);
        add(0.5, 0.25, 64.0 / 81.0 * 1.0 / 8.0);
        add((1 + s) / 2, (1 - s) * (1 + s) / 4, 100.0 / 324.0 * (1 - s) / 8.0);
        add((1 + s) / 2, (1 - s) * (1 - s) / 4, 100.0 / 324.0 * (1 - s) / 8.0);
        add((1 - s) / 2, (1 + s) * (1 + s) / 4, 100.0 / 324.0 * (1 + s) / 8.0);
        add((1 - s) / 2, (1 + s) * (1 - s) / 4, 100.0 / 324.0 * (1 + s) / 8.0);
        add(0.5, (1 + s) / 4, 40.0 / 81.0 * 1.0 / 8.0);
        add(0.5, (1 - s) / 4, 40.0 / 81.0 * 1.0 / 8.0);
        add((1 + s) / 2, (1 - s) / 4, 40.0 / 81.0 * (1 - s) / 8.0);
        add((1 - s) / 2, (1 + s) / 4, 40.0 / 81.0 * (1 + s) / 8.0);
        break;
    }
    case 12: {
        const double a = 0.5611400349004341, b = 0.2194299825497830, wa = 0.1713331241529811 * 0.5;
        const double c = 0.0397240717755698, d = 0.4801379641122151, wc = 0.0807310895930309 * 0.5;
        const double e = 0.0193717243612408, f = 0.1416190159239682, g = 0.8390092597147911,
                     we = 0.0406345597936607 * 0.5;
        add(a, b, wa);
        add(b, b, wa);
        add(b, a, wa);
        add(c, d, wc);
        add(d, d, wc);
        add(d, c, wc);
        add(e, f, we);
        add(f, g, we);
        add(g, e, we);
        add(f, e, we);
        add(e, g, we);
        add(g, f, we);
        break;
    }
    case 36: {
        auto g6 = gauss_legendre(6);
        for (int i = 0; i < 6; ++i)
            for (int j = 0; j < 6; ++j) {
                double u = (g6[2 * i] + 1) / 2, wa = g6[2 * i + 1] / 2, ub = (g6[2 * j] + 1) / 2, wb = g6[2 * j + 1] / 2;
                add(u, (1 - u) * ub, wa * wb * (1 - u));
            }
        break;
    }
    default: throw Error(VG_EINVAL, "triangle quadrature must be 1, 3, 4, 7, 9, 12 or 36");
    }
    return r;
}

}  // namespace

Solver::Solver(HostMesh&& mesh, const vg_geometry* geo, int k_, int nq_, int ng_, int device) : m(std::move(mesh)) {
    // option rules of vem/CurvedVEM_Darcy_gpu/src/solver_options.cpp:123-136
    if (k_ < 0 || k_ > 4) throw Error(VG_EINVAL, "polynomial degree k must be 0..4");
    if (nq_ != 1 && nq_ != 3 && nq_ != 4 && nq_ != 7 && nq_ != 9 && nq_ != 12 && nq_ != 36)
        throw Error(VG_EINVAL, "triangle quadrature must be 1, 3, 4, 7, 9, 12 or 36");
    if ((k_ >= 1 && nq_ == 1) || (k_ >= 2 && (nq_ == 3 || nq_ == 4)))
        throw Error(VG_EINVAL, "triangle quadrature under-integrates this degree");
    if ((k_ == 3 && nq_ < 12) || (k_ == 4 && nq_ != 36))
        throw Error(VG_EINVAL, "insufficient triangle quadrature for this degree");
    if (ng_ < k_ + 2 || ng_ > 10) throw Error(VG_EINVAL, "edge quadrature must be between k+2 and 10");
    k = k_;
    nq = nq_;
    ng = ng_;
    int ndev = 0;
    VG_CUDA(cudaGetDeviceCount(&ndev));
    if (ndev == 0) throw Error(VG_ECUDA, "no CUDA device");
    if (device >= 0) VG_CUDA(cudaSetDevice(device));
    VG_CUDA(cudaGetDevice(&device_));
    VG_CUDA(cudaDeviceGetAttribute(&sm_count_, cudaDevAttrMultiProcessorCount, device_));
    q = dimP(k);
    p = p_of(k);
    ngrad = ngrad_of(k);
    internal = internal_of(k);
    nf = m.ne * (k + 1) + m.nc * internal;
    np = m.nc * q;
    N = nf + np + 1;  // flux BC (reference default) until set_problem
    // geometry
    std::vector<int> edge_arc(m.ne, -1);
    std::vector<double> arcdata;
    if (geo) {
        geom_kind = geo->kind;
        eps = geo->eps;
        if (geom_kind < VG_GEOM_IDENTITY || geom_kind > VG_GEOM_ARCS) throw Error(VG_EINVAL, "unknown geometry kind");
        if (geom_kind == VG_GEOM_ARCS) {
            if (geo->num_arcs < 0 || (geo->num_arcs > 0 && (!geo->arc_nodes || !geo->arc_circles)))
                throw Error(VG_EINVAL, "arc geometry needs arc_nodes and arc_circles");
            std::unordered_map<unsigned long long, int> look;
            look.reserve(size_t(m.ne) * 2);
            for (int e = 0; e < m.ne; ++e)
                look[(static_cast<unsigned long long>(unsigned(m.eend[2 * e])) << 32) | unsigned(m.eend[2 * e + 1])] = e;
            arcdata.assign(3 * size_t(m.ne), 0.0);
            for (int a = 0; a < geo->num_arcs; ++a) {
                unsigned u = unsigned(geo->arc_nodes[2 * a]), v = unsigned(geo->arc_nodes[2 * a + 1]);
                auto it = look.find((static_cast<unsigned long long>(std::min(u, v)) << 32) | std::max(u, v));
                if (it == look.end()) throw Error(VG_EINVAL, "arc chord is not a mesh edge");
                if (m.eocc[it->second] != 1) throw Error(VG_EINVAL, "arc chord is not a boundary edge");
                if (!(geo->arc_circles[3 * a + 2] > 0)) throw Error(VG_EINVAL, "arc radius must be positive");
                edge_arc[it->second] = a;
                for (int c = 0; c < 3; ++c) arcdata[3 * size_t(it->second) + c] = geo->arc_circles[3 * a + c];
            }
        }
    }
    std::vector<char> curved(m.nc, 0);
    if (geom_kind == VG_GEOM_ARCS)
        for (int c = 0; c < m.nc; ++c)
            for (int j = m.cptr[c]; j < m.cptr[c + 1]; ++j)
                if (edge_arc[m.gedges[j]] >= 0) curved[c] = 1;
    std::vector<int> triptr;
    std::vector<TriIdx> tris;
    PhaseTimer pt;
    triangulate(m, curved, edge_arc, triptr, tris);
    pt.mark("triangulate");
    pack_layout();
    pt.mark("pack layout");
    // uploads
    ArenaScope scope(arena_);
    d_xy_.upload(m.xy);
    d_cptr_.upload(m.cptr);
    d_cnodes_.upload(m.cnodes);
    d_gedges_.upload(m.gedges);
    d_cx_.upload(m.cx);
    d_cy_.upload(m.cy);
    d_diam_.upload(m.diam);
    d_triptr_.upload(triptr);
    d_tris_.upload(tris);
    if (geom_kind == VG_GEOM_ARCS) d_arc_.upload(arcdata);
    d_slot_cell_.upload(slot_cell_);
    d_cell_slot_.upload(cell_slot_);
    d_pieces_.upload(pieces_);
    d_map_.upload(map_host_);
    plan_internal_order();
    pt.mark("uploads");
    plan_streams();
    pt.mark("record-stream plan");
    {
        std::vector<int> occ(m.eocc);
        DevBuf<int> tmp;
        tmp.upload(occ);
        d_eocc_ = std::move(tmp);
    }
    theta_.assign(m.nc, 0.0);
    d_theta_.upload(theta_);
    d_status_.resize(1);
    d_counter_.resize(1);
    d_counter_.zero();
    VG_CUDA(cudaEventCreate(&ev0_));
    VG_CUDA(cudaEventCreate(&ev1_));
    VG_CUDA(cudaEventCreateWithFlags(&ev_in_, cudaEventDisableTiming));
    VG_CUDA(cudaStreamCreateWithFlags(&stream_, cudaStreamNonBlocking));
    VG_CUDA(cudaStreamCreateWithFlags(&side_, cudaStreamNonBlocking));
    VG_CUDA(cudaEventCreateWithFlags(&ev_fork_, cudaEventDisableTiming));
    VG_CUDA(cudaEventCreateWithFlags(&ev_join_, cudaEventDisableTiming));
    d_loop_.resize(2);
}

Solver::~Solver() {
    arena_.close();
    destroy_graphs();
    destroy_minres_graphs();
    ms_destroy_graphs();
    if (h_err_) cudaFreeHost(h_err_);
    if (ev0_) cudaEventDestroy(ev0_);
    if (ev1_) cudaEventDestroy(ev1_);
    if (ev_in_) cudaEventDestroy(ev_in_);
    if (stream_) cudaStreamDestroy(stream_);
    if (side_) cudaStreamDestroy(side_);
    if (ev_fork_) cudaEventDestroy(ev_fork_);
    if (ev_join_) cudaEventDestroy(ev_join_);
}

void Solver::destroy_graphs() {
    for (int p = 0; p < 2; ++p) {
        if (gexec_[p]) cudaGraphExecDestroy(gexec_[p]);
        if (graph_[p]) cudaGraphDestroy(graph_[p]);
        gexec_[p] = nullptr;
        graph_[p] = nullptr;
    }
}

void Solver::plan_internal_order() {
    const long long NN = (long long)nf + np + 1;  // + the multiplier row, which keeps its index
    e2i_host_.assign(NN, -1);
    i2e_host_.assign(NN, -1);
    map_int_host_.assign(map_host_.size(), 0);
    prow_host_.assign(slot_cell_.size(), -1);
    int nextf = 0, nextp = 0;
    for (const auto& P : pieces_) {
        for (int i = 0; i < P.n; ++i)
            for (int j = 0; j < P.count; ++j) {
                const long long o = P.map_off + (long long)i * PIECE + j;
                const int g = map_host_[o], gg = g < 0 ? ~g : g;
                if (e2i_host_[gg] < 0) {
                    e2i_host_[gg] = nextf;
                    i2e_host_[nextf] = gg;
                    ++nextf;
                }
                const int gi = e2i_host_[gg];
                map_int_host_[o] = g < 0 ? ~gi : gi;
            }
        for (int j = 0; j < P.count; ++j) {
            const int c = slot_cell_[P.slot + j];
            prow_host_[P.slot + j] = nf + nextp * q;
            for (int r = 0; r < q; ++r) {
                e2i_host_[nf + (long long)c * q + r] = nf + nextp * q + r;
                i2e_host_[nf + (long long)nextp * q + r] = nf + c * q + r;
            }
            ++nextp;
        }
    }
    e2i_host_[NN - 1] = int(NN - 1);
    i2e_host_[NN - 1] = int(NN - 1);
    if (nextf != nf || nextp != m.nc) throw Error(VG_EMESH, "dof numbering does not cover every unknown");
    d_map_int_.upload(map_int_host_);
    d_prow_.upload(prow_host_);
    d_e2i_.upload(e2i_host_);
    d_i2e_.upload(i2e_host_);
}

void Solver::internal_copies() {
    d_mask_int_.resize(N);
    gather_launch<int>(d_mask_.data(), d_i2e_.data(), 0, d_mask_int_.data(), N, nullptr);
    d_Lint_.resize(size_t(np));
    d_Lint32_.resize(size_t(np));
    gather_launch<double>(d_L_.data(), d_i2e_.data(), nf, d_Lint_.data(), np, nullptr);
    gather_launch<float>(d_L32_.data(), d_i2e_.data(), nf, d_Lint32_.data(), np, nullptr);
    d_xi_.resize(N);
}

template <typename T>
void Solver::permute(const T* in, T* out, bool to_internal, cudaStream_t s) {
    gather_launch<T>(in, to_internal ? d_i2e_.data() : d_e2i_.data(), 0, out, N, s);
}
template void Solver::permute<double>(const double*, double*, bool, cudaStream_t);
template void Solver::permute<float>(const float*, float*, bool, cudaStream_t);

void Solver::pack_layout() {
    // chunks of CHUNK consecutive cells, grouped by edge count inside a chunk, split into pieces
    pieces_.clear();
    slot_cell_.clear();
    cell_slot_.assign(m.nc, -1);
    a_total_ = w_total_ = map_total_ = p_total_ = hw_total_ = e_total_ = s_total_ = 0;
    maxn = 0;
    int rank = 0;
    std::vector<std::vector<int>> byne(MAX_NE + 1), classes(MAX_NE + 1);
    for (int c0 = 0; c0 < m.nc; c0 += CHUNK) {
        int c1 = std::min(m.nc, c0 + CHUNK);
        for (auto& v : byne) v.clear();
        for (int c = c0; c < c1; ++c) byne[m.cptr[c + 1] - m.cptr[c]].push_back(c);
        for (int ne = 3; ne <= MAX_NE; ++ne)
            for (size_t s0 = 0; s0 < byne[ne].size(); s0 += PIECE) {
                Piece P{};
                P.ne = ne;
                P.n = (k + 1) * ne + internal;
                P.count = int(std::min<size_t>(PIECE, byne[ne].size() - s0));
                P.slot = (long long)pieces_.size() * PIECE;
                P.a_off = a_total_;
                P.w_off = w_total_;
                P.map_off = map_total_;
                P.p_off = p_total_;
                P.hw_off = hw_total_;
                P.e_off = e_total_;
                P.s_off = s_total_;
                P.rank0 = rank;
                rank += P.count;
                a_total_ += (long long)PIECE * (P.n * (P.n + 1) / 2);
                w_total_ += k >= 1 ? (long long)PIECE * q * P.n : 0;
                map_total_ += (long long)PIECE * P.n;
                p_total_ += (long long)PIECE * p * P.n;
                hw_total_ += (long long)PIECE * q * P.n;
                e_total_ += (long long)PIECE * ne;
                s_total_ += (long long)PIECE * ((k + 1) * ne * ((k + 1) * ne - 1) / 2);
                maxn = std::max(maxn, P.n);
                for (int l = 0; l < PIECE; ++l) {
                    int c = l < P.count ? byne[ne][s0 + l] : -1;
                    if (c >= 0) {
                        cell_slot_[c] = int(slot_cell_.size());
                        classes[ne].push_back(c);
                    }
                    slot_cell_.push_back(c);
                }
                pieces_.push_back(P);
            }
    }
    classes_.clear();
    class_cells_.clear();
    for (int ne = 3; ne <= MAX_NE; ++ne)
        if (!classes[ne].empty()) {
            class_cells_.emplace_back();
            class_cells_.back().upload(classes[ne]);
            classes_.push_back(CellClass{ne, (k + 1) * ne + internal, int(classes[ne].size()),
                                         class_cells_.back().data()});
        }
    // signed flux dof map (vem/CurvedVEM_Darcy_gpu/src/mesh_pack.cpp:209-225): edge moments degree-major,
    // sign -1 on even moments of an interior edge traversed against its (min, max) orientation
    map_host_.assign(map_total_, 0);
    for (const auto& P : pieces_) {
        for (int j = 0; j < P.count; ++j) {
            int c = slot_cell_[P.slot + j];
            int base = m.cptr[c];
            for (int r = 0; r <= k; ++r)
                for (int e = 0; e < P.ne; ++e) {
                    int ge = m.gedges[base + e];
                    int g = r * m.ne + ge;
                    bool rev = m.cnodes[base + e] != m.eend[2 * ge];
                    bool neg = m.eocc[ge] == 2 && rev && r % 2 == 0;
                    map_host_[P.map_off + (long long)(r * P.ne + e) * PIECE + j] = neg ? ~g : g;
                }
            for (int i = 0; i < internal; ++i)
                map_host_[P.map_off + (long long)((k + 1) * P.ne + i) * PIECE + j] = m.ne * (k + 1) + c * internal + i;
        }
    }
}

void Solver::set_problem(int problem_, int bc_) {
    if (problem_ < VG_PROBLEM_SINCOS || problem_ > VG_PROBLEM_ANNULUS) throw Error(VG_EINVAL, "unknown problem");
    if (bc_ != VG_BC_FLUX && bc_ != VG_BC_PRESSURE) throw Error(VG_EINVAL, "unknown boundary condition");
    problem = problem_;
    bc = bc_;
    N = nf + np + (bc == VG_BC_FLUX ? 1 : 0);
    built = false;
}

void Solver::set_theta(const double* theta, bool on_device) {
    if (!theta) throw Error(VG_EINVAL, "null theta");
    // a non-finite log permeability would turn the operator and every solve into NaN: rejected
    // before the handle's field changes
    long long bad = -1;
    if (on_device) {
        VG_CUDA(cudaDeviceSynchronize());  // theta may come from any stream
        bad = first_nonfinite(theta, m.nc, d_status_.data());
    } else {
        for (int c = 0; c < m.nc && bad < 0; ++c)
            if (!std::isfinite(theta[c])) bad = c;
    }
    if (bad >= 0) throw Error(VG_EINVAL, "non-finite log permeability in cell " + std::to_string(bad));
    if (on_device)
        VG_CUDA(cudaMemcpy(d_theta_.data(), theta, sizeof(double) * m.nc, cudaMemcpyDeviceToDevice));
    else
        VG_CUDA(cudaMemcpy(d_theta_.data(), theta, sizeof(double) * m.nc, cudaMemcpyHostToDevice));
    if (built) {
        PhaseTimer pt;
        rescale_ops(d_theta_.data(), d_slot_cell_.data(), d_pieces_.data(), int(pieces_.size()), d_A0_.data(),
                    d_A64_.data(), d_A32_.data(), nullptr);
        pack_streams(nullptr);
        pt.mark("rescale + record streams");
        if (minres_.ready) prepare_minres();
        if (hybrid_ready_) prepare_hybrid();
        lift_flux_rhs();
        VG_CUDA(cudaDeviceSynchronize());
    }
}

void Solver::check_status(const char* where) {
    unsigned long long st = 0;
    VG_CUDA(cudaMemcpy(&st, d_status_.data(), sizeof(st), cudaMemcpyDeviceToHost));
    if (!st) return;
    unsigned long long code = st >> 40;
    int cell = int(st & 0xffffffffull);
    if (code == ST_JACOBIAN)
        throw Error(VG_EGEOMETRY, std::string(where) + ": nonpositive Jacobian in cell " + std::to_string(cell));
    throw Error(VG_ESINGULAR, std::string(where) + ": singular local matrix in cell " + std::to_string(cell));
}

void Solver::build() {
    ArenaScope scope(arena_);
    upload_rules(triangle_rule(nq), gauss_legendre(ng));
    const int nqp = nq;
    d_A0_.resize(a_total_);
    d_A64_.resize(a_total_);
    d_A32_.resize(a_total_);
    d_W64_.resize(std::max<long long>(w_total_, 1));
    d_W32_.resize(std::max<long long>(w_total_, 1));
    d_P_.resize(p_total_);
    d_HW_.resize(hw_total_);
    d_L_.resize(size_t(m.nc) * q);
    d_L32_.resize(size_t(m.nc) * q);
    d_alpha_.resize(m.nc);
    d_rhs_.resize(N);
    d_bval_.resize(N);
    d_mask_.resize(N);
    d_rhs_.zero();
    d_bval_.zero();
    d_mask_.zero();
    d_status_.zero();
    SetupArgs a{};
    a.xy = d_xy_.data();
    a.cptr = d_cptr_.data();
    a.cnodes = d_cnodes_.data();
    a.gedges = d_gedges_.data();
    a.eocc = d_eocc_.data();
    a.cx = d_cx_.data();
    a.cy = d_cy_.data();
    a.diam = d_diam_.data();
    a.triptr = d_triptr_.data();
    a.tris = d_tris_.data();
    a.arc = geom_kind == VG_GEOM_ARCS ? d_arc_.data() : nullptr;
    a.slot_cell = d_slot_cell_.data();
    a.cell_slot = d_cell_slot_.data();
    a.pieces = d_pieces_.data();
    a.map = d_map_.data();
    a.theta = d_theta_.data();
    a.k = k;
    a.q = q;
    a.p = p;
    a.ngrad = ngrad;
    a.internal = internal;
    a.nqp = nqp;
    a.ng = ng;
    a.geom = geom_kind;
    a.problem = problem;
    a.bc = bc;
    a.nf = nf;
    a.eps = eps;
    a.A0 = d_A0_.data();
    a.A64 = d_A64_.data();
    a.A32 = d_A32_.data();
    a.W64 = d_W64_.data();
    a.W32 = d_W32_.data();
    a.P = d_P_.data();
    a.HW = d_HW_.data();
    a.L = d_L_.data();
    a.L32 = d_L32_.data();
    a.alpha = d_alpha_.data();
    a.rhs = d_rhs_.data();
    a.bval = d_bval_.data();
    a.mask = d_mask_.data();
    a.status = d_status_.data();
    setup_args_ = a;
    PhaseTimer pt;
    for (const auto& c : classes_) launch_setup(a, c, nqp, nullptr);
    VG_CUDA(cudaDeviceSynchronize());
    check_status("setup");
    internal_copies();
    pt.mark("device setup kernels");
    pack_streams(nullptr);
    pt.mark("pack record streams");
    // workspaces
    d_partials_.resize(2 * size_t(std::max(apply_blocks(int(pieces_.size())), VEC_BLOCKS)) + 16);
    d_red_.resize(8);
    d_out_.resize(sizeof(SolveOut) / sizeof(double));
    destroy_graphs();
    for (auto& b : sv64_) b.resize(N);
    // a build starts the condensed system and its multigrid from scratch (the operator or the boundary
    // condition may have changed). With the pressure condition they are made here; with the flux condition
    // by the first solve, since a Maxwell-Stefan handle never needs them.
    hybrid_condensed_ = hybrid_ready_ = use_amg = minres_.ready = false;
    if (bc == VG_BC_PRESSURE && !(minres_mesh() && prepare_minres())) prepare_hybrid();
    pt.mark("edge system (incl. multigrid)");
    // BC_FLUX: lifted right-hand side of MixedGpu::make_rhs (equation_gpu.cu:611-625):
    // free rows b - A g (unconstrained apply of the boundary values), boundary rows g
    d_rhs0_.resize(N);
    VG_CUDA(cudaMemcpy(d_rhs0_.data(), d_rhs_.data(), sizeof(double) * N, cudaMemcpyDeviceToDevice));
    lift_flux_rhs();
    VG_CUDA(cudaDeviceSynchronize());
    built = true;
}

// BC_FLUX: the lifted right-hand side depends on the operator (b - A g), so it is recomputed from
// the unlifted one whenever the permeability changes
void Solver::lift_flux_rhs() {
    if (bc != VG_BC_FLUX) return;
    VG_CUDA(cudaMemcpy(d_rhs_.data(), d_rhs0_.data(), sizeof(double) * N, cudaMemcpyDeviceToDevice));
    double* y = sv64_[0].data();
    sv64_[0].zero();
    apply64(d_bval_.data(), y, false, 1.0, nullptr);
    lift_rhs(d_mask_.data(), d_bval_.data(), y, d_rhs_.data(), N, nullptr);
}

template <typename T>
void Solver::apply_int(const T* x, T* y, bool constrained, T psign, cudaStream_t s, double* quad) {
    launch_apply(apply_args<T>(x, y, constrained, psign, quad, nullptr), s);
    n_launch += 1;
    ++n_apply;
}
template void Solver::apply_int<double>(const double*, double*, bool, double, cudaStream_t, double*);
template void Solver::apply_int<float>(const float*, float*, bool, float, cudaStream_t, double*);

// Reference order in and out, in one kernel: the same apply with the dof map, the pressure rows,
// the essential-BC mask and the multiplier vector in the reference's numbering, and (k <= 1) record
// streams packed with that map, built on the first call. The gathers and scatters are less
// coalesced than in the internal order, but no permutation pass runs.
void Solver::prepare_reference_order() {
    if (!d_prow_ref_.data()) {
        std::vector<int> prow(slot_cell_.size(), -1);
        for (size_t j = 0; j < slot_cell_.size(); ++j)
            if (slot_cell_[j] >= 0) prow[j] = nf + slot_cell_[j] * q;
        d_prow_ref_.upload(prow);
    }
    if (k <= 1 && !ref_streams_packed_) {
        d_rec64r_.resize(size_t(plan64_.bytes));
        d_rec32r_.resize(size_t(plan32_.bytes));
        pack_streams_reference(nullptr);
    }
}

void Solver::pack_streams_reference(cudaStream_t s) {
    const int np_ = int(pieces_.size());
    pack_stream<double>(d_pieces_.data(), np_, d_roff64_.data(), d_A64_.data(), d_W64_.data(), d_map_.data(),
                        d_prow_ref_.data(), k, d_rec64r_.data(), s);
    pack_stream<float>(d_pieces_.data(), np_, d_roff32_.data(), d_A32_.data(), d_W32_.data(), d_map_.data(),
                       d_prow_ref_.data(), k, d_rec32r_.data(), s);
    VG_CUDA(cudaStreamSynchronize(s));
    ref_streams_packed_ = true;
}

template <typename T>
void Solver::apply_ref(const T* x, T* y, bool constrained, T psign, cudaStream_t s, double* quad) {
    prepare_reference_order();
    ApplyArgs<T> a = apply_args<T>(x, y, constrained, psign, quad, nullptr);
    a.map = d_map_.data();
    a.prow = d_prow_ref_.data();
    a.mask = d_mask_.data();
    if constexpr (sizeof(T) == 8) {
        a.L = d_L_.data();
        if (a.rec) a.rec = d_rec64r_.data();
    } else {
        a.L = d_L32_.data();
        if (a.rec) a.rec = d_rec32r_.data();
    }
    launch_apply(a, s);
    n_launch += 1;
    ++n_apply;
}

void Solver::apply64(const double* x, double* y, bool constrained, double psign, cudaStream_t s, double* quad) {
    apply_ref<double>(x, y, constrained, psign, s, quad);
}

void Solver::apply32(const float* x, float* y, bool constrained, float psign, cudaStream_t s, double* quad) {
    apply_ref<float>(x, y, constrained, psign, s, quad);
}

void Solver::plan_streams() {
    // the kernels' error word: mapped pinned host memory, written by a kernel only when a bounded
    // wait gave up (a plain store) and read by the host with a plain load, no copy in any call
    if (!h_err_) {
        VG_CUDA(cudaHostAlloc(reinterpret_cast<void**>(&h_err_), sizeof(int), cudaHostAllocMapped));
        *h_err_ = 0;
        VG_CUDA(cudaHostGetDevicePointer(reinterpret_cast<void**>(&d_errp_), h_err_, 0));
    }
    if (k > 1) return;
    plan64_ = plan_stream(pieces_, k, 8, sm_count_);
    plan32_ = plan_stream(pieces_, k, 4, sm_count_);
    d_rec64_.resize(size_t(plan64_.bytes));
    d_rec32_.resize(size_t(plan32_.bytes));
    d_roff64_.upload(plan64_.rec_off);
    d_roff32_.upload(plan32_.rec_off);
    d_bat64_.upload(plan64_.batches);
    d_bat32_.upload(plan32_.batches);
    d_cta64_.upload(plan64_.cta_batch);
    d_cta32_.upload(plan32_.cta_batch);
    d_stall_.resize(1);
    d_stall_.zero();
    VG_CUDA(cudaDeviceSynchronize());
    prepare_stream_kernels();
}

void Solver::pack_streams(cudaStream_t s) {
    if (k > 1) return;
    const int np_ = int(pieces_.size());
    pack_stream<double>(d_pieces_.data(), np_, d_roff64_.data(), d_A64_.data(), d_W64_.data(), d_map_int_.data(),
                        d_prow_.data(), k, d_rec64_.data(), s);
    pack_stream<float>(d_pieces_.data(), np_, d_roff32_.data(), d_A32_.data(), d_W32_.data(), d_map_int_.data(),
                       d_prow_.data(), k, d_rec32_.data(), s);
    VG_CUDA(cudaStreamSynchronize(s));
    if (ref_streams_packed_) pack_streams_reference(s);  // new operator values (permeability update)
}

// Test hook of the failure path: in the next streamed apply one consumer's bounded wait runs out
// (a barrier nothing arrives on) and the apply reports its error word.
void Solver::inject_apply_stall() {
    if (k > 1 || !d_stall_.data()) throw Error(VG_ESTATE, "no streamed apply on this handle (k > 1)");
    const int one = 1;
    VG_CUDA(cudaMemcpy(d_stall_.data(), &one, sizeof(one), cudaMemcpyHostToDevice));
}

// vg_apply is asynchronous: a failed apply sets the mapped error word when its kernel gives up,
// and the next call on the handle that finds it set reports VG_ECUDA (the caller's stream never
// waits for a check)
void Solver::check_apply_probe() {
    if (h_err_ && *reinterpret_cast<volatile int*>(h_err_)) {
        VG_CUDA(cudaDeviceSynchronize());
        *reinterpret_cast<volatile int*>(h_err_) = 0;
        throw Error(VG_ECUDA, "an earlier vg_apply failed: apply pipeline wait timed out");
    }
}

// a kernel sets the error word when a pipeline or grid-barrier wait gave up (never in a correct run)
void Solver::check_pipeline() {
    if (h_err_ && *reinterpret_cast<volatile int*>(h_err_)) {
        VG_CUDA(cudaDeviceSynchronize());
        *reinterpret_cast<volatile int*>(h_err_) = 0;
        throw Error(VG_ECUDA, "a kernel's pipeline wait timed out");
    }
}

void Solver::rhs(double* b, cudaStream_t s) {
    VG_CUDA(cudaMemcpyAsync(b, d_rhs_.data(), sizeof(double) * N, cudaMemcpyDeviceToDevice, s));
}

template <typename T>
ApplyArgs<T> Solver::apply_args(const T* x, T* y, bool constrained, T psign, double* quad, const int* flags) {
    ApplyArgs<T> a{};
    a.x = x;
    a.y = y;
    if constexpr (sizeof(T) == 8) {
        a.A = d_A64_.data();
        a.W = d_W64_.data();
        a.L = d_Lint_.data();
    } else {
        a.A = d_A32_.data();
        a.W = d_W32_.data();
        a.L = d_Lint32_.data();
    }
    a.map = d_map_int_.data();
    a.prow = d_prow_.data();
    a.pieces = d_pieces_.data();
    a.npieces = int(pieces_.size());
    a.k = k;
    a.mask = d_mask_int_.data();
    a.flags = flags;
    a.nf = nf;
    a.N = N;
    a.psign = psign;
    a.constrained = (constrained && bc == VG_BC_FLUX) ? 1 : 0;
    a.mult = bc == VG_BC_FLUX ? 1 : 0;
    a.partials = d_partials_.data();
    a.counter = d_counter_.data();
    a.red = quad;
    if (k <= 1 && d_errp_) {
        const StreamPlan& pl = sizeof(T) == 8 ? plan64_ : plan32_;
        a.rec = sizeof(T) == 8 ? d_rec64_.data() : d_rec32_.data();
        a.batches = sizeof(T) == 8 ? d_bat64_.data() : d_bat32_.data();
        a.cta_batch = sizeof(T) == 8 ? d_cta64_.data() : d_cta32_.data();
        a.ncta = pl.ncta;
        a.stages = pl.stages;
        a.stage_bytes = pl.stage_bytes;
        a.err = d_errp_;
        a.stall = d_stall_.data();
    }
    return a;
}
template ApplyArgs<double> Solver::apply_args<double>(const double*, double*, bool, double, double*, const int*);
template ApplyArgs<float> Solver::apply_args<float>(const float*, float*, bool, float, double*, const int*);

void Solver::solve_host(const double* b_host, double* x_host, const vg_solve_opts& o, vg_solve_info& info) {
    if (!built) throw Error(VG_ESTATE, "vg_build must run before vg_solve_host");
    d_hb_.resize(N);
    d_hx_.resize(N);
    // copies on the solver stream: solve() orders its own work after the legacy stream, so the
    // inputs are enqueued there first
    VG_CUDA(cudaMemcpyAsync(d_hb_.data(), b_host, sizeof(double) * N, cudaMemcpyHostToDevice, nullptr));
    if (o.nonzero_guess)
        VG_CUDA(cudaMemcpyAsync(d_hx_.data(), x_host, sizeof(double) * N, cudaMemcpyHostToDevice, nullptr));
    solve(d_hb_.data(), d_hx_.data(), o, info, nullptr);
    VG_CUDA(cudaMemcpyAsync(x_host, d_hx_.data(), sizeof(double) * N, cudaMemcpyDeviceToHost, stream_));
    VG_CUDA(cudaStreamSynchronize(stream_));
}

// sparsity pattern of the assembled system (host, cached): row g of a flux dof holds the dofs of
// the cells around g, a pressure row the dofs of its cell, the multiplier row every pressure dof;
// every row holds its diagonal (the unit diagonal of masked rows)
void Solver::assembled_pattern() {
    if (!csr_ptr_.empty()) return;
    const bool mult = bc == VG_BC_FLUX;
    auto dofs_of = [&](int c, std::vector<int>& out) {
        const int slot = cell_slot_[c];
        const Piece& P = pieces_[slot / PIECE];
        const int lane = slot % PIECE;
        for (int i = 0; i < P.n; ++i) {
            int g = map_host_[P.map_off + (long long)i * PIECE + lane];
            out.push_back(g < 0 ? ~g : g);
        }
        for (int r = 0; r < q; ++r) out.push_back(nf + c * q + r);
        if (mult) out.push_back(N - 1);
    };
    // cells around every flux dof
    std::vector<int> cnt(nf + 1, 0), cells;
    std::vector<int> tmp;
    for (int c = 0; c < m.nc; ++c) {
        tmp.clear();
        dofs_of(c, tmp);
        for (int g : tmp)
            if (g < nf) cnt[g + 1]++;
    }
    for (int g = 0; g < nf; ++g) cnt[g + 1] += cnt[g];
    cells.assign(cnt[nf], 0);
    {
        std::vector<int> fill(cnt.begin(), cnt.end() - 1);
        for (int c = 0; c < m.nc; ++c) {
            tmp.clear();
            dofs_of(c, tmp);
            for (int g : tmp)
                if (g < nf) cells[fill[g]++] = c;
        }
    }
    csr_ptr_.assign(size_t(N) + 1, 0);
    csr_col_.clear();
    std::vector<int> row;
    auto emit = [&](long long r) {
        row.push_back(int(r));
        std::sort(row.begin(), row.end());
        row.erase(std::unique(row.begin(), row.end()), row.end());
        csr_col_.insert(csr_col_.end(), row.begin(), row.end());
        csr_ptr_[r + 1] = (long long)csr_col_.size();
    };
    for (int g = 0; g < nf; ++g) {
        row.clear();
        for (int t = cnt[g]; t < cnt[g + 1]; ++t) dofs_of(cells[t], row);
        emit(g);
    }
    for (int c = 0; c < m.nc; ++c)
        for (int r = 0; r < q; ++r) {
            row.clear();
            dofs_of(c, row);
            emit(nf + (long long)c * q + r);
        }
    if (mult) {
        row.clear();
        for (long long i = nf; i < nf + np; ++i) row.push_back(int(i));
        emit(N - 1);
    }
}

void Solver::assemble(int constrained, long long* nnz, long long* rp, int* ci, double* val) {
    if (!built) throw Error(VG_ESTATE, "vg_build must run before vg_assemble_csr");
    assembled_pattern();
    *nnz = (long long)csr_col_.size();
    if (!rp) return;
    if (!ci || !val) throw Error(VG_EINVAL, "vg_assemble_csr needs row_ptr, col_idx and values");
    VG_CUDA(cudaMemcpy(rp, csr_ptr_.data(), sizeof(long long) * csr_ptr_.size(), cudaMemcpyHostToDevice));
    VG_CUDA(cudaMemcpy(ci, csr_col_.data(), sizeof(int) * csr_col_.size(), cudaMemcpyHostToDevice));
    VG_CUDA(cudaMemset(val, 0, sizeof(double) * csr_col_.size()));
    DevBuf<int> bad(1);
    bad.zero();
    assemble_values(d_A64_.data(), d_W64_.data(), d_map_.data(), d_slot_cell_.data(), d_mask_.data(), d_L_.data(),
                    d_pieces_.data(), int(pieces_.size()), k, nf, N, (constrained && bc == VG_BC_FLUX) ? 1 : 0,
                    bc == VG_BC_FLUX ? 1 : 0, rp, ci, val, bad.data(), nullptr);
    int b = 0;
    VG_CUDA(cudaMemcpy(&b, bad.data(), sizeof(int), cudaMemcpyDeviceToHost));
    if (b) throw Error(VG_ESTATE, "assembled pattern does not hold an entry of a local block");
}

void Solver::axpy64(double* x, const double* d, double a, cudaStream_t s) {
    axpy64_kernel_launch(x, d, a, N, s);
}

void Solver::adjoint(const double* x, const double* dJdx, double* g, const vg_solve_opts& o, vg_solve_info& info,
                     cudaStream_t s) {
    if (!built) throw Error(VG_ESTATE, "vg_build must run before vg_adjoint_grad");
    // K_ref^T lambda = dJ/dx  <=>  K_sym mu = dJ/dx with mu = S lambda (S = diag(I, -I));
    // solve() takes a reference-sign right-hand side b and solves K_sym x = S b, so pass S dJ/dx
    d_adj_rhs_.resize(N);
    d_adj_mu_.resize(N);
    DevBuf<double>&rhs = d_adj_rhs_, &mu = d_adj_mu_;
    flip_pressure(dJdx, rhs.data(), nf, N, nullptr);  // legacy stream: solve() orders after it
    vg_solve_opts oo = o;
    oo.nonzero_guess = 0;
    solve(rhs.data(), mu.data(), oo, info, s);
    s = stream_;
    // dJ/dtheta_E = -lambda^T (dK/dtheta_E) x = mu_u,E^T A_E(theta) x_u,E  (dA_E/dtheta_E = -A_E)
    contract_adjoint(d_A64_.data(), d_map_.data(), d_slot_cell_.data(), d_mask_.data(), d_pieces_.data(),
                     int(pieces_.size()), k, x, mu.data(), bc == VG_BC_FLUX, g, s);
    VG_CUDA(cudaStreamSynchronize(s));
}

void Solver::errors(const double* x, double out[6], cudaStream_t s) {
    if (!built) throw Error(VG_ESTATE, "vg_build must run before vg_errors");
    DevBuf<double> per(6 * size_t(m.nc)), sum(6);
    for (const auto& c : classes_) launch_errors(setup_args_, c, nq, x, per.data(), s);
    launch_error_sum(per.data(), m.nc, sum.data(), s);
    VG_CUDA(cudaMemcpyAsync(out, sum.data(), 6 * sizeof(double), cudaMemcpyDeviceToHost, s));
    VG_CUDA(cudaStreamSynchronize(s));
}

namespace {
// Per-cell error figures (6 doubles a cell) and their sums for Solver::errors_static. Every word
// of the used part is overwritten by each call (error_kernel writes all six figures of every
// cell, error_sum_kernel all six sums), so nothing has to be cleared between calls. Shared by all
// handles of a device: calls that overlap on the GPU race on it.
constexpr long long kErrScratch = 6LL * VG_ERRORS_NOALLOC_MAX_CELLS + 8;
static __device__ __align__(256) double g_err_scratch[kErrScratch];

// device address of g_err_scratch on the current device. Looked up on every call (the lookup
// allocates nothing and is cheap): an address kept across calls would go stale when the device's
// primary context is reset and created again in the same process.
double* err_scratch() {
    void* p = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&p, g_err_scratch);
    if (e != cudaSuccess || !p) {
        cudaGetLastError();
        throw Error(VG_ECUDA, std::string("cudaGetSymbolAddress(error scratch): ") + cudaGetErrorString(e));
    }
    return static_cast<double*>(p);
}
}  // namespace

// The C ABI makes the handle's device current before this runs (DeviceScope in vg_capi.cu).
void Solver::errors_static(const double* x, double out[6]) {
    if (!built) throw Error(VG_ESTATE, "vg_build must run before vg_errors_noalloc");
    if (m.nc > VG_ERRORS_NOALLOC_MAX_CELLS)
        throw Error(VG_EINVAL, "vg_errors_noalloc: " + std::to_string(m.nc) +
                                   " cells exceed the static scratch limit VG_ERRORS_NOALLOC_MAX_CELLS = " +
                                   std::to_string(VG_ERRORS_NOALLOC_MAX_CELLS));
    double* per = err_scratch();
    double* sum = per + 6LL * VG_ERRORS_NOALLOC_MAX_CELLS;
    for (const auto& c : classes_) launch_errors(setup_args_, c, nq, x, per, nullptr);
    launch_error_sum(per, m.nc, sum, nullptr);
    VG_CUDA(cudaMemcpyAsync(out, sum, 6 * sizeof(double), cudaMemcpyDeviceToHost, nullptr));
    VG_CUDA(cudaStreamSynchronize(nullptr));
}

int Solver::local(int cell, int which, double* out) {
    if (!built) throw Error(VG_ESTATE, "vg_build must run before vg_local");
    if (cell < 0 || cell >= m.nc) throw Error(VG_EINVAL, "cell out of range");
    int slot = cell_slot_[cell];
    const Piece& b = pieces_[slot / PIECE];
    long long j = slot % PIECE, mcount = PIECE;
    int n = b.n;
    auto strided = [&](const double* base, long long off, int cnt, std::vector<double>& v) {
        v.resize(cnt);
        for (int e = 0; e < cnt; ++e)
            VG_CUDA(cudaMemcpy(&v[e], base + off + e * mcount + j, sizeof(double), cudaMemcpyDeviceToHost));
    };
    std::vector<double> v;
    switch (which) {
    case 0: {
        std::vector<double> pk;
        strided(d_A64_.data(), b.a_off, n * (n + 1) / 2, pk);
        v.assign(size_t(n) * n, 0.0);
        int e = 0;
        for (int i = 0; i < n; ++i)
            for (int c = i; c < n; ++c) {
                v[size_t(i) * n + c] = pk[e];
                v[size_t(c) * n + i] = pk[e];
                ++e;
            }
        break;
    }
    case 1:
        if (k == 0)
            v.assign(n, 1.0);
        else
            strided(d_W64_.data(), b.w_off, q * n, v);
        break;
    case 2: strided(d_P_.data(), b.p_off, p * n, v); break;
    case 3: {
        double a = 0;
        VG_CUDA(cudaMemcpy(&a, d_alpha_.data() + cell, sizeof(double), cudaMemcpyDeviceToHost));
        v.assign(1, a);
        break;
    }
    case 4: {
        v.resize(n);
        for (int i = 0; i < n; ++i) {
            int g = map_host_[b.map_off + i * mcount + j];
            v[i] = g < 0 ? -double(~g + 1) : double(g + 1);
        }
        break;
    }
    case 5: {
        v.resize(q);
        VG_CUDA(cudaMemcpy(v.data(), d_rhs_.data() + nf + (long long)cell * q, q * sizeof(double), cudaMemcpyDeviceToHost));
        break;
    }
    case 6: {
        v.assign(n, 0.0);
        if (bc == VG_BC_PRESSURE)
            for (int i = 0; i < (k + 1) * b.ne; ++i) {
                int g = map_host_[b.map_off + i * mcount + j];
                int e = m.gedges[m.cptr[cell] + i % b.ne];
                if (m.eocc[e] == 1)
                    VG_CUDA(cudaMemcpy(&v[i], d_rhs_.data() + g, sizeof(double), cudaMemcpyDeviceToHost));
            }
        break;
    }
    default: throw Error(VG_EINVAL, "unknown local quantity");
    }
    if (out) std::copy(v.begin(), v.end(), out);
    return int(v.size());
}

}  // namespace vg

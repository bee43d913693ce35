// wnlqg_b200.cu - C ABI of the B200 k-mesh response engine (declarations in include/wnlqg_b200.h).
//
// A model is copied to the device once; a plan compiles a task into Fourier channels, real-space
// tiles and response passes, and owns the batch workspaces.  Each batch runs
//   phase_kernel -> fourier_gemm -> jacobi_eigh -> response pass(es)
// on the plan's stream; mesh evaluation ends with one ordered reduction of the per-CTA partials.
#include "../../include/wnlqg_b200.h"

#include <cuda.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <limits>
#include <map>
#include <mutex>
#include <string>
#include <vector>

#include "common.cuh"
#include "eigh.cuh"
#include "regjacobi.cuh"
#include "onesided.cuh"
#include "fourier.cuh"
#include "response.cuh"
#include "shg.cuh"
#include "tc_fourier.cuh"
#include "nonorth.cuh"
#include "order.cuh"
#include "isolation.cuh"
#include "fdsea.cuh"
#include "bcd_analytic.cuh"
#include <cub/device/device_radix_sort.cuh>

namespace {

thread_local std::string g_error;

wnlqg_status fail(wnlqg_status st, const std::string &msg) {
    g_error = msg;
    return st;
}

#define WNLQG_CUDA(call)                                                                                  \
    do {                                                                                                  \
        cudaError_t err_ = (call);                                                                        \
        if (err_ != cudaSuccess)                                                                          \
            return fail(err_ == cudaErrorMemoryAllocation ? WNLQG_ERR_OUT_OF_MEMORY : WNLQG_ERR_CUDA,       \
                        std::string(#call) + ": " + cudaGetErrorString(err_));                            \
    } while (0)

// CH_DDA: d_c d_g A_p with d = 3 min(c, g) + max(c, g).
enum ChannelOp { CH_H = 0, CH_DH = 1, CH_DDH = 2, CH_A = 3, CH_DA = 4, CH_S = 5, CH_DS = 6, CH_DDS = 7, CH_DDA = 8 };

struct Channel {
    int op;
    int p;   // dH/ddH: first derivative axis; A/dA: position axis
    int d;   // ddH: second derivative axis; dA: derivative axis
};

}  // namespace

struct wnlqg_model {
    int device = 0;
    int nw = 0, nr = 0;
    double lattice[9];
    std::vector<int64_t> rvec, deg;
    std::vector<double2> H, A, S;
    bool has_position = false, has_overlap = false;
    int64_t *d_rvec = nullptr, *d_deg = nullptr;
};

struct Pass {
    RespParams params;   // template; batch-dependent fields set per launch
    bool global = false; // working set in global memory (does not fit shared memory)
    size_t smem = 0;
    int threads = 0;
    int grid = 0;
    int grid_wide = 0;   // grid of the 512-thread variant (FP64 orthogonal shared-memory passes), 0 = none
    bool fd = false;     // band-curvature pass of the finite-difference stencil (shifted points only)
};

struct wnlqg_plan {
    wnlqg_model *model = nullptr;
    wnlqg_task_desc task;
    std::vector<double> omegas, mus;
    std::vector<Channel> channels;
    int ch_H = 0, ch_S = -1;
    bool nonorth = false;
    int *d_status = nullptr;
    // Spectral isolation contract (isolation.cuh): -1 = none, else ISO_ALL_PAIRS or
    // ISO_SPECTRAL_BLOCKS with tolerance iso_tol; the first failing row and its record.
    int iso_mode = -1;
    double iso_tol = 0.0;
    unsigned long long *d_iso_key = nullptr;
    IsoRecord *d_iso_rec = nullptr;
    // Fermi-sea Berry dipole on the finite-difference geometry (fdsea.cuh): the derivative axes in
    // order of first use, their fractional steps, the (a, b) curvature pairs, the combine items,
    // and per batch the shifted k-points and band curvatures [entry][2 nd][npair][nw].
    int fd_nd = 0, fd_npair = 0;
    int fd_axis[3] = {0, 0, 0};
    int fd_pair[9][2];
    double fd_delta[3][3];
    double *d_fd_k = nullptr, *d_fd_curv = nullptr;
    SeaParams sea;
    // Mesh batches evaluate the shifted points k +- delta_j as the same mesh with tiles multiplied by
    // exp(+-2 pi i delta_j . R): 2 nd tile sets [set][NR][C][nw^2] for the staged contraction (exact,
    // like the centre's), when they fit the budget; else the stencil takes the arbitrary-k front.
    double2 *d_fd_tiles = nullptr;
    // Fermi-sea Berry dipole on the analytic geometry (bcd_analytic.cuh): items, channels, grid and
    // the per-CTA global working sets.
    BcdaParams bcda;
    int bcda_grid = 0;
    unsigned char *d_bcda_scratch = nullptr;
    int ch_dH[3], ch_A[3], ch_ddH[9], ch_dA[9];
    int nw = 0, nr = 0, C = 0;
    int64_t nn = 0, vc = 0, max_batch = 0;
    double2 *d_tiles = nullptr, *d_phase = nullptr, *d_xw = nullptr, *d_U = nullptr, *d_out = nullptr;
    double2 *d_points = nullptr;
    double *d_E = nullptr, *d_kpts = nullptr, *d_omegas = nullptr, *d_partials = nullptr, *d_weights = nullptr;
    double *d_mus = nullptr;
    int64_t *d_kidx = nullptr;
    int partial_slots = 0;                    // partial sums' slots: allocated, needed beside the second
    int other_slots = 0, call_slots = 0;      // harmonic's, and of the call in progress (begin_call)
    // Staged mesh Fourier: R grouping (device) and lazily sized Y/Z workspaces.
    int P12 = 0, P1 = 0;
    int *d_groups = nullptr;        // q12_start | q12_ridx | q12_r2 | q1_start | q1_q12 | q1_r1
    StagedGroups groups;
    double2 *d_stageY = nullptr, *d_stageZ = nullptr;
    size_t stageY_elems = 0, stageZ_elems = 0;
    bool use_staged_last = false;
    std::vector<Pass> passes;
    // Second-harmonic responses: one shg_kernel launch each, sharing one per-CTA scratch.
    std::vector<ShgParams> shg;
    size_t shg_smem = 0;
    int shg_grid = 0;
    int shg_grid_alloc = 0;   // CTAs the scratch is allocated for (the largest grid a launch may take)
    int shg_grid_l2 = 0;      // global working set: the grid whose sets stay L2-resident
    double2 *d_shg_scratch = nullptr;
    unsigned char *d_shg_gscratch = nullptr;
    bool shg_global = false;
    bool shg_pair = false;                    // two CTAs per SM fit (shg_takes_pairs says when they pay)
    bool shg_pair_now = false;                // and the call in progress takes them (begin_call)
    // Tensor-core Fourier for arbitrary k-points: Ozaki slices of the phases (A, per batch) and of
    // the channel tiles (B, built once), tcgen05 kind::i8 GEMM.  tc_slices == 0: FP64 CUDA cores.
    int tc_slices = 0;
    int64_t tc_kpad = 0, tc_npad = 0, tc_mpad = 0, tc_ncols = 0;
    int8_t *d_tcA = nullptr, *d_tcB = nullptr;
    double *d_tc_colscale = nullptr;
    int *d_tc_err = nullptr;
    bool tc_used = false;
    CUtensorMap tc_mapA, tc_mapB;
    int eigh_threads = 32;
    size_t eigh_smem = 0;
    bool warp_eigh = false;                   // orthogonal models, nw <= 32: team-per-matrix stages
    int eigh_team = 32;                       // threads per matrix of the FP64 refinement: 32, 64 or 128
    bool f32_team = false;                    // first stage in shared memory (mixed path)
    bool small_f64 = false;                   // FP64 path, nw <= 16: FP64 Jacobi in registers, no stages
    // Convention I: Cartesian and fractional Wannier centres (tau[a * nw + i]).
    bool conv1 = false;
    std::vector<double> tau_cart, tau_frac;
    bool cta_mixed = false;                   // orthogonal models above 32 orbitals: CTA FP32 + FP64 stages
    bool cta_gw1 = false, cta_gw2 = false;    // those stages' working sets in global memory
    int refine_cta_threads = 512;             // FP64 CTA refinement block size
    unsigned char *d_eigh_scratch = nullptr;  // per-CTA global working set of the CTA eigensolvers
    int64_t eigh_scratch_stride = 0;
    int eigh_grid = 0;
    int eigh_grid_alloc = 0;                  // CTAs the eigensolver working sets are allocated for
    int eigh_grid_l2 = 0;                     // the grid whose working sets stay L2-resident
    unsigned char *d_resp_scratch = nullptr;  // per-CTA global working set of the response passes
    int resp_gw_grid = 0;                     // grid of the global working-set passes; 0 = each pass's own
    int resp_gw_grid_alloc = 0;               // CTAs the response working sets are allocated for
    int64_t resp_scratch_stride = 0;
    // Nonorthogonal responses: metric geometry per batch (Berry connection, slopes, G pairs).
    NonorthParams ng;
    int ng_grid = 0;
    int ng_grid_alloc = 0;
    int ng_gidx[9];
    double2 *d_ng_r = nullptr, *d_ng_G = nullptr;
    double *d_ng_v = nullptr;
    unsigned char *d_ng_ws = nullptr;
    // Second harmonic generation of nonorthogonal models: metric inputs per batch point.
    bool metric_shg = false;
    MetricShgParams mshg;
    int mshg_grid = 0;
    int mshg_grid_alloc = 0;
    double2 *d_mshg_src = nullptr;
    double *d_mshg_diag = nullptr;
    unsigned char *d_mshg_ws = nullptr;
    int refine_threads = 32;
    int sm_count = 148;
    size_t refine_smem = 0;
    float2 *d_V32 = nullptr;
    // Morton ordering of arbitrary k-point batches (team eigensolver plans): keys and indices
    // (two halves each, radix-sort input and output), the ordered k-points and weights, and the
    // sort's temporary storage.
    bool order_points = false;
    // FP32 eigensolver stages warm-start along mesh runs and ordered batches (1) or always start
    // from the identity (0): WNLQG_B200_WARM_START at plan creation, then the autotuner.
    int warm_mode = 1;
    // FP64 response passes on the 512-thread variant (WNLQG_B200_RESPONSE_WIDE at plan creation,
    // then the autotuner).
    bool resp_wide = false;
    // Nonorthogonal models: FP64 Cholesky reduction C = L^-1 H L^-H (d_gC, with L in d_gL), the
    // orthogonal stages on C, back-substitution U = L^-H V.
    bool gen_mixed = false;
    double2 *d_gC = nullptr, *d_gL = nullptr;
    size_t gred_smem = 0;
    bool gred_gw = false;
    unsigned char *d_gred_scratch = nullptr;
    int64_t gred_stride = 0;
    int gred_grid = 0;
    uint32_t *d_okeys = nullptr;
    int *d_operm = nullptr;
    double *d_ok = nullptr, *d_ow = nullptr;
    void *d_osort_tmp = nullptr;
    size_t osort_bytes = 0;
    cudaStream_t stream = nullptr;
    std::vector<cudaEvent_t> events;
    size_t timing_batches = 0;
    int64_t launches = 0;
    bool timing_valid = false;
    // CUDA graphs that captured this plan's launches: while any exists, buffers that a later call
    // outgrows are retired (kept until the plan is destroyed) instead of freed, and the plan
    // cannot be destroyed.
    int graph_refs = 0;
    std::vector<void *> retired;
};

namespace {

int find_channel(const std::vector<Channel> &chs, int op, int p, int d) {
    for (size_t i = 0; i < chs.size(); ++i)
        if (chs[i].op == op && chs[i].p == p && chs[i].d == d) return (int)i;
    return -1;
}

int add_channel(std::vector<Channel> &chs, int op, int p, int d) {
    if ((op == CH_DDH || op == CH_DDS) && p > d) std::swap(p, d);   // symmetric second derivatives
    int idx = find_channel(chs, op, p, d);
    if (idx >= 0) return idx;
    chs.push_back(Channel{op, p, d});
    return (int)chs.size() - 1;
}

bool finite_array(const double *a, size_t n) {
    for (size_t i = 0; i < n; ++i)
        if (!std::isfinite(a[i])) return false;
    return true;
}

double lattice_det(const double *L) {
    auto e = [&](int i, int j) { return L[i + 3 * j]; };
    return e(0, 0) * (e(1, 1) * e(2, 2) - e(1, 2) * e(2, 1)) - e(0, 1) * (e(1, 0) * e(2, 2) - e(1, 2) * e(2, 0)) +
           e(0, 2) * (e(1, 0) * e(2, 1) - e(1, 1) * e(2, 0));
}

// CTAs whose working sets live in global memory: as many as the launch allows while the grid's
// working sets together stay within ~96 MB of the 126 MB L2 (at least half the SMs stay busy).
int l2_resident_grid(int grid, int64_t bytes_per_cta, int sm_count) {
    const int64_t cap = std::max<int64_t>(sm_count / 2, ((int64_t)96 << 20) / std::max<int64_t>(1, bytes_per_cta));
    return (int)std::max<int64_t>(1, std::min<int64_t>(grid, cap));
}

int eigh_block_threads(int nw) {
    int np = nw + (nw & 1);
    int blocks = (np / 2) * (np / 2);
    int t = ((blocks + 31) / 32) * 32;
    return std::max(32, std::min(256, t));
}

int response_threads(int nw) {
    int t = ((nw * nw / 4 + 31) / 32) * 32;
    return std::max(32, std::min(256, t));
}

// Raise a kernel's dynamic shared memory limit to everything the device allows beside the kernel's
// static shared memory.  The attribute belongs to the kernel, not to a plan: several plans of
// different sizes share it, so it is never lowered to one plan's need.
cudaError_t allow_dynamic_smem(const void *fn, int smem_optin) {
    cudaFuncAttributes a;
    cudaError_t e = cudaFuncGetAttributes(&a, fn);
    if (e != cudaSuccess) return e;
    return cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_optin - (int)a.sharedSizeBytes);
}

// The 512-thread FP64 response kernel (orthogonal models, working set in shared memory).
const void *response_wide_fn() { return (const void *)response_kernel<double, false, false, true>; }

// The response kernel instantiation for a precision, a geometry source and a working-set location.
const void *response_fn(bool mixed, bool nonorth, bool global, bool freq) {
    if (!freq && !nonorth) {
        if (mixed) return global ? (const void *)response_kernel<float, false, true, false, false> : (const void *)response_kernel<float, false, false, false, false>;
        return global ? (const void *)response_kernel<double, false, true, false, false> : (const void *)response_kernel<double, false, false, false, false>;
    }
    if (mixed) {
        if (nonorth) return global ? (const void *)response_kernel<float, true, true> : (const void *)response_kernel<float, true, false>;
        return global ? (const void *)response_kernel<float, false, true> : (const void *)response_kernel<float, false, false>;
    }
    if (nonorth) return global ? (const void *)response_kernel<double, true, true> : (const void *)response_kernel<double, true, false>;
    return global ? (const void *)response_kernel<double, false, true> : (const void *)response_kernel<double, false, false>;
}

// Build the response passes: group the requested components so that each pass fits the
// per-pass limits and the shared-memory budget.
wnlqg_status build_passes(wnlqg_plan *pl, int sm_count, size_t smem_limit) {
    const wnlqg_task_desc &t = pl->task;
    struct Item { int kind; int a, b, c, d; int64_t out; };
    // Band-curvature items of the finite-difference stencil: their own passes (shifted points only).
    const int ITEM_BANDCURV = -1;
    std::vector<Item> items;
    int64_t off = 0;
    for (int r = 0; r < t.num_responses; ++r) {
        const wnlqg_response_request &q = t.responses[r];
        if (q.kind == WNLQG_SECOND_HARMONIC) {   // its own kernel (build_shg)
            off += (int64_t)q.num_components * t.num_photon_energies * 14;
            continue;
        }
        if (q.kind == WNLQG_BERRY_DIPOLE_SEA) {   // sea_dipole_kernel (items set at plan creation)
            off += (int64_t)q.num_components * t.num_fermi_energies;
            continue;
        }
        for (int c = 0; c < q.num_components; ++c) {
            const int32_t *x = q.components[c];
            if (q.kind == WNLQG_SHIFT_CURRENT || q.kind == WNLQG_INJECTION_CURRENT || q.kind == WNLQG_JERK_CURRENT) {
                items.push_back({q.kind, x[0], x[1], x[2], x[3], off + (int64_t)c * t.num_photon_energies});
            } else if (q.kind == WNLQG_INTRINSIC_AHC || q.kind == WNLQG_BERRY_DIPOLE ||
                       q.kind == WNLQG_LINEAR_TRANSPORT_BERRY) {
                items.push_back({q.kind, x[0], x[1], x[2], 0, off + (int64_t)c * t.num_fermi_energies});
            } else {
                items.push_back({q.kind, x[0], x[1], 0, 0, off + c});
            }
        }
        if (q.kind == WNLQG_SHIFT_CURRENT || q.kind == WNLQG_INJECTION_CURRENT || q.kind == WNLQG_JERK_CURRENT)
            off += (int64_t)q.num_components * t.num_photon_energies;
        else if (q.kind == WNLQG_INTRINSIC_AHC || q.kind == WNLQG_BERRY_DIPOLE || q.kind == WNLQG_LINEAR_TRANSPORT_BERRY)
            off += (int64_t)q.num_components * t.num_fermi_energies;
        else
            off += q.num_components;
    }
    for (int pr = 0; pr < pl->fd_npair; ++pr) items.push_back({ITEM_BANDCURV, pl->fd_pair[pr][0], pl->fd_pair[pr][1], 0, 0, pr});
    const double vol = lattice_det(pl->model->lattice);
    const double e3 = WNLQG_ELEMENTARY_CHARGE_C * WNLQG_ELEMENTARY_CHARGE_C * WNLQG_ELEMENTARY_CHARGE_C;
    const double P_sc = WNLQG_HBAR_EV_S * WNLQG_PI * (-e3) / (2.0 * WNLQG_HBAR_J_S * WNLQG_HBAR_J_S * vol);
    const double P_ic = -WNLQG_PI * e3 / (WNLQG_HBAR_J_S * WNLQG_HBAR_J_S * vol);

    // Photon-energy window test: exact interval form when consecutive sorted energies are
    // closer than twice the half-width.
    std::vector<double> sorted = pl->omegas;
    std::sort(sorted.begin(), sorted.end());
    double max_gap = 0.0;
    for (size_t i = 1; i < sorted.size(); ++i) max_gap = std::max(max_gap, sorted[i] - sorted[i - 1]);
    const bool gaussian = t.broadening_type == WNLQG_GAUSSIAN;
    const double width = t.broadening;
    const double cutoff = width * std::sqrt(200.0);
    const double thr = t.transition_window_factor * width;
    const double half = gaussian ? cutoff : thr;
    const int interval_ok = !sorted.empty() && (sorted.size() == 1 || max_gap < 2.0 * half) ? 1 : 0;

    // The dynamic shared-memory ceiling is a per-function attribute: raise it once to the device
    // maximum so that passes of different sizes can all launch.
    const bool mixed = t.precision == WNLQG_PRECISION_MIXED;
    const int csize = mixed ? (int)sizeof(float2) : (int)sizeof(double2);
    {
        cudaError_t e = cudaSuccess;
        for (int v = 0; v < 8 && e == cudaSuccess; ++v)
            e = allow_dynamic_smem(response_fn(v & 1, v & 2, false, v & 4), (int)smem_limit);
        if (e == cudaSuccess) e = allow_dynamic_smem(response_wide_fn(), (int)smem_limit);
        if (e != cudaSuccess) return fail(WNLQG_ERR_CUDA, std::string("cudaFuncSetAttribute: ") + cudaGetErrorString(e));
    }
    // Orbital counts whose matrices do not fit shared memory keep each CTA's working set in global
    // memory (L1/L2-resident); passes are then limited only by the per-pass component limits.
    const bool global_mode = RespSmem::layout(pl->nw, 4, 1, 1, csize).total > smem_limit;
    size_t i = 0;
    while (i < items.size()) {
        Pass ps;
        RespParams &p = ps.params;
        std::memset(&p, 0, sizeof(p));
        p.nw = pl->nw;
        p.ld = pl->nw + 1;
        for (int a = 0; a < 3; ++a) {
            p.slot_dH[a] = -1; p.slot_A[a] = -1; p.slot_D[a] = -1;
            p.ch_dH[a] = pl->ch_dH[a]; p.ch_A[a] = pl->ch_A[a];
        }
        for (int a = 0; a < 9; ++a) { p.ch_ddH[a] = pl->ch_ddH[a]; p.ch_dA[a] = pl->ch_dA[a]; }
        bool needH[3] = {false, false, false}, needA[3] = {false, false, false}, needD[3] = {false, false, false};
        std::vector<std::pair<int, int>> gl, hl;
        auto hindex = [&](int aa, int dd, bool commit) {
            for (size_t h = 0; h < hl.size(); ++h)
                if (hl[h].first == aa && hl[h].second == dd) return (int)h;
            if (!commit) return (int)hl.size();
            hl.push_back({aa, dd});
            return (int)hl.size() - 1;
        };
        auto gindex = [&](int pp, int dd, bool commit) {
            for (size_t g = 0; g < gl.size(); ++g)
                if (gl[g].first == pp && gl[g].second == dd) return (int)g;
            if (!commit) return (int)gl.size();
            gl.push_back({pp, dd});
            return (int)gl.size() - 1;
        };
        size_t start = i;
        bool pass_global = global_mode;   // a pass whose first component alone exceeds shared memory
        const bool pass_fd = items[start].kind == ITEM_BANDCURV;
        while (i < items.size()) {
            const Item &it = items[i];
            if ((it.kind == ITEM_BANDCURV) != pass_fd) break;   // stencil passes hold only curvature items
            // Tentatively add the item and check limits.
            bool tH[3], tA[3], tD[3];
            std::copy(needH, needH + 3, tH);
            std::copy(needA, needA + 3, tA);
            std::copy(needD, needD + 3, tD);
            int newg = 0, newh = 0;
            auto need_r = [&](int a) { tH[a] = true; tA[a] = true; };
            const bool freq = it.kind == WNLQG_SHIFT_CURRENT || it.kind == WNLQG_INJECTION_CURRENT ||
                              it.kind == WNLQG_JERK_CURRENT;
            const bool muaxis = it.kind == WNLQG_INTRINSIC_AHC || it.kind == WNLQG_BERRY_DIPOLE ||
                                it.kind == WNLQG_LINEAR_TRANSPORT_BERRY || it.kind == ITEM_BANDCURV;
            const int mode = it.kind == WNLQG_JERK_CURRENT ? 1 : 0;
            if (freq && p.n_fc > 0 && p.pair_mode != mode) break;   // one pair family per pass
            if (it.kind == WNLQG_SHIFT_CURRENT) {
                need_r(it.a); need_r(it.b); need_r(it.c);
                tD[it.a] = true;
                if (gindex(it.c, it.a, false) == (int)gl.size()) ++newg;
                if (!(it.b == it.c) && gindex(it.b, it.a, false) == (int)gl.size()) ++newg;
            } else if (it.kind == WNLQG_INJECTION_CURRENT) {
                tH[it.a] = true; need_r(it.b); need_r(it.c);
            } else if (it.kind == WNLQG_JERK_CURRENT) {
                tH[it.a] = true; tH[it.d] = true; need_r(it.b); need_r(it.c);
                if (hindex(it.a, it.d, false) == (int)hl.size()) ++newh;
            } else {
                need_r(it.a); need_r(it.b);
                if (it.kind == WNLQG_BERRY_DIPOLE) tH[it.c] = true;
            }
            int nslots = (int)gl.size() + newg;
            for (int a = 0; a < 3; ++a) nslots += (tH[a] ? 1 : 0) + (tA[a] ? 1 : 0) + (tD[a] ? 1 : 0);
            int nfc = p.n_fc + (freq ? 1 : 0);
            int nsc = p.n_sc + ((!freq && !muaxis) ? 1 : 0);
            int nmi = p.n_mu + (muaxis ? 1 : 0);
            size_t smem = RespSmem::layout(pl->nw, nslots, nfc, 1, csize).total;
            bool fits = nfc <= RS_MAX_FREQ && nsc <= RS_MAX_SCALAR && nmi <= RS_MAX_SCALAR &&
                        (int)gl.size() + newg <= RS_MAX_G && (int)hl.size() + newh <= RS_MAX_HESS &&
                        (pass_global || smem <= smem_limit);
            if (!fits) {
                if (i == start) {
                    if (!pass_global) {
                        pass_global = true;   // runs from the per-CTA global working set
                        continue;
                    }
                    return fail(WNLQG_ERR_UNSUPPORTED, "one response component exceeds the per-pass limits");
                }
                break;
            }
            std::copy(tH, tH + 3, needH);
            std::copy(tA, tA + 3, needA);
            std::copy(tD, tD + 3, needD);
            if (it.kind == WNLQG_SHIFT_CURRENT) {
                int g1 = gindex(it.c, it.a, true);
                int g2 = gindex(it.b, it.a, true);
                int c = p.n_fc++;
                p.fc_kind[c] = RS_FC_SHIFT; p.fc_a[c] = it.a; p.fc_b[c] = it.b; p.fc_c[c] = it.c;
                p.fc_g1[c] = g1; p.fc_g2[c] = g2; p.fc_pref[c] = P_sc; p.fc_out[c] = it.out;
                p.pair_mode = 0;
            } else if (it.kind == WNLQG_INJECTION_CURRENT) {
                int c = p.n_fc++;
                p.fc_kind[c] = RS_FC_INJECTION; p.fc_a[c] = it.a; p.fc_b[c] = it.b; p.fc_c[c] = it.c;
                p.fc_g1[c] = 0; p.fc_g2[c] = 0; p.fc_pref[c] = P_ic; p.fc_out[c] = it.out;
                p.pair_mode = 0;
            } else if (it.kind == WNLQG_JERK_CURRENT) {
                int c = p.n_fc++;
                p.fc_kind[c] = RS_FC_JERK; p.fc_a[c] = it.a; p.fc_b[c] = it.b; p.fc_c[c] = it.c;
                p.fc_g1[c] = 0; p.fc_g2[c] = 0; p.fc_pref[c] = 1.0; p.fc_out[c] = it.out;
                p.fc_hess[c] = hindex(it.a, it.d, true);
                p.pair_mode = 1;
            } else if (muaxis) {
                int m = p.n_mu++;
                p.mu_kind[m] = it.kind == WNLQG_INTRINSIC_AHC ? RS_MU_AHC
                               : it.kind == WNLQG_BERRY_DIPOLE ? RS_MU_DIPOLE
                               : it.kind == ITEM_BANDCURV ? RS_MU_BANDCURV : RS_MU_LT;
                p.mu_a[m] = it.a; p.mu_b[m] = it.b; p.mu_c[m] = it.c; p.mu_out[m] = it.out;
            } else {
                int s = p.n_sc++;
                p.sc_kind[s] = it.kind == WNLQG_BERRY_CURVATURE ? RS_SC_BERRY : RS_SC_METRIC;
                p.sc_a[s] = it.a; p.sc_b[s] = it.b; p.sc_out[s] = it.out;
            }
            ++i;
        }
        int slot = 0;
        for (int a = 0; a < 3; ++a) if (needH[a]) p.slot_dH[a] = slot++;
        for (int a = 0; a < 3; ++a) if (needA[a]) p.slot_A[a] = slot++;
        for (int a = 0; a < 3; ++a) if (needD[a]) p.slot_D[a] = slot++;
        p.n_g = (int)gl.size();
        for (int g = 0; g < p.n_g; ++g) { p.g_p[g] = gl[g].first; p.g_d[g] = gl[g].second; p.g_slot[g] = slot++; }
        p.n_slots = slot;
        p.n_hess = (int)hl.size();
        for (int h = 0; h < p.n_hess; ++h) { p.hess_a[h] = hl[h].first; p.hess_d[h] = hl[h].second; }
        p.nmu = (int)t.num_fermi_energies;
        p.mus = pl->d_mus;
        p.temperature = t.temperature;
        p.fs_width = t.fermi_surface_broadening;
        p.lt_gamma = t.linear_transport_gamma_inter;
        // factor = e^2 / hbar * 1e-20 of _linear_transport_response (LinearTransportKernels.jl:116).
        p.lt_factor = WNLQG_ELEMENTARY_CHARGE_C * WNLQG_ELEMENTARY_CHARGE_C / WNLQG_HBAR_J_S * 1e-20;
        p.nom = (int)t.num_photon_energies;
        p.omegas = pl->d_omegas;
        p.mu = t.fermi_energy;
        p.kT = WNLQG_KB_EV_K * t.temperature;
        p.gaussian = gaussian ? 1 : 0;
        p.width = width;
        p.cutoff = cutoff;
        p.gscale = gaussian ? 1.0 / (std::sqrt(WNLQG_PI) * width) : 0.0;
        p.thr = thr;
        p.window_interval = interval_ok;
        p.om_lo = sorted.empty() ? 0.0 : sorted.front();
        p.om_hi = sorted.empty() ? 0.0 : sorted.back();
        p.eta_reg = t.denominator_regularization;
        p.band_window = t.band_window_size;
        p.use_sel = t.use_band_selection ? 1 : 0;
        for (int w = 0; w < 4; ++w) { p.vsel[w] = t.valence_bands[w]; p.csel[w] = t.conduction_bands[w]; }
        p.degeneracy_threshold = t.degeneracy_threshold;
        p.vc = pl->vc;
        p.xw_stride = (int64_t)pl->C * pl->nn;
        p.curv_stride = (int64_t)2 * pl->fd_nd * pl->fd_npair * pl->nw;
        ps.smem = RespSmem::layout(pl->nw, p.n_slots, p.n_fc, 1, csize).total;
        ps.global = pass_global;
        ps.fd = pass_fd;
        ps.threads = response_threads(pl->nw);
        int per_sm = 0;
        const size_t launch_smem = pass_global ? 0 : ps.smem;
        cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, response_fn(mixed, pl->nonorth, pass_global, p.n_fc > 0),
                                                                      ps.threads, launch_smem);
        if (e != cudaSuccess) return fail(WNLQG_ERR_CUDA, std::string("occupancy query: ") + cudaGetErrorString(e));
        if (per_sm < 1) return fail(WNLQG_ERR_UNSUPPORTED, "response kernel cannot be resident with its shared memory");
        ps.grid = sm_count * per_sm;
        if (pass_global) ps.grid = l2_resident_grid(ps.grid, (int64_t)ps.smem, sm_count);
        if (!mixed && !pl->nonorth && !pass_global && p.n_fc > 0 && ps.threads == 256) {
            int per_sm_w = 0;
            e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm_w, response_wide_fn(), 512, ps.smem);
            if (e != cudaSuccess) return fail(WNLQG_ERR_CUDA, std::string("occupancy query: ") + cudaGetErrorString(e));
            ps.grid_wide = per_sm_w >= 1 ? sm_count * per_sm_w : 0;
        }
        pl->passes.push_back(ps);
    }
    bool any_global = false;
    for (const Pass &ps : pl->passes) any_global |= ps.global;
    // Global working-set passes default to two CTAs per SM (measured at 96 and 128 orbitals: 1.8-2.9x
    // faster than the L2-resident grids); the autotuner may pick another grid.
    if (any_global) pl->resp_gw_grid = 2 * sm_count;
    if (any_global) {
        int64_t grid = 0;
        size_t bytes = 0;
        for (const Pass &ps : pl->passes) {
            if (!ps.global) continue;
            grid = std::max<int64_t>(grid, std::max(ps.grid, 2 * sm_count));   // up to two CTAs per SM
            bytes = std::max(bytes, ps.smem);
        }
        pl->resp_scratch_stride = (int64_t)((bytes + 255) & ~(size_t)255);
        pl->resp_gw_grid_alloc = (int)grid;
        cudaError_t e = cudaMalloc(&pl->d_resp_scratch, (size_t)grid * pl->resp_scratch_stride);
        if (e != cudaSuccess) {
            cudaGetLastError();
            return fail(WNLQG_ERR_OUT_OF_MEMORY, "cudaMalloc of the response working set failed");
        }
    }
    return WNLQG_OK;
}

// Second-harmonic launches: parameters per SHG response, shared-memory size, grid and the per-CTA
// global scratch (G matrices, pair coefficients, pair data).
// The second-harmonic kernel's instantiation.
const void *shg_function(bool global, bool pair) {
    if (global) return (const void *)shg_kernel<true, false>;
    return pair ? (const void *)shg_kernel<false, true> : (const void *)shg_kernel<false, false>;
}

// Whether a launch takes the form with two CTAs per SM, where shared memory allows it.  Two conditions.
//   - The contraction, in passes of 256 threads over the energies and component chunks: the narrower
//     chunks of that form may need more passes, and each evaluates the resonances again.  1184 points
//     of 22 orbitals, one CTA -> two: 3.76 -> 3.11 ms (3 components, 48 energies: 1 pass either way),
//     11.48 -> 10.95 (6, 400: 4 and 5), 7.56 -> 7.85 (6, 256: 2 and 3), 4.29 -> 4.56 (3, 256: 1 and 2; 5.16 ->
//     6.12 with the Gaussian's exponentials).  Up to 8 orbitals the other steps outweigh that: 0.72 -> 0.63
//     at 4 (3, 256).
//   - Rounds of points over the SMs: a round of two points takes 1.4 to 1.7 times one of one point, least
//     for few orbitals and energies.  300 points, 3 rounds -> 2: 16 orbitals 0.86 -> 1.08 ms (2 components,
//     256 energies), 4 orbitals 0.29 -> 0.25 (1, 48).
bool shg_takes_pairs(const ShgParams &p, int64_t nb, int sm_count) {
    auto passes = [&](bool pair) {
        const int cb = shg_components(pair);
        return ((int64_t)p.nom * ((p.nc + cb - 1) / cb) + 255) / 256;
    };
    const int64_t ones = (nb + sm_count - 1) / sm_count, pairs = (nb + 2 * sm_count - 1) / (2 * sm_count);
    const bool light = p.nw <= 12 && (int64_t)p.nc * p.nom <= 256;
    return (p.nw <= 8 || 5 * passes(true) <= 7 * passes(false)) && (light ? 15 : 17) * pairs <= 10 * ones;
}

wnlqg_status build_shg(wnlqg_plan *pl, int sm_count, size_t smem_limit) {
    const wnlqg_task_desc &t = pl->task;
    int64_t off = 0;
    int max_nc = 0;
    for (int r = 0; r < t.num_responses; ++r) {
        const wnlqg_response_request &q = t.responses[r];
        int64_t width;
        if (q.kind == WNLQG_SHIFT_CURRENT || q.kind == WNLQG_INJECTION_CURRENT || q.kind == WNLQG_JERK_CURRENT)
            width = (int64_t)q.num_components * t.num_photon_energies;
        else if (q.kind == WNLQG_SECOND_HARMONIC)
            width = (int64_t)q.num_components * t.num_photon_energies * 14;
        else if (q.kind == WNLQG_INTRINSIC_AHC || q.kind == WNLQG_BERRY_DIPOLE)
            width = (int64_t)q.num_components * t.num_fermi_energies;
        else
            width = q.num_components;
        if (q.kind == WNLQG_SECOND_HARMONIC) {
            ShgParams p;
            std::memset(&p, 0, sizeof(p));
            p.nw = pl->nw;
            p.ld = pl->nw + 1;
            p.xw_stride = (int64_t)pl->C * pl->nn;
            for (int a = 0; a < 3; ++a) { p.ch_dH[a] = pl->ch_dH[a]; p.ch_A[a] = pl->ch_A[a]; }
            for (int a = 0; a < 9; ++a) { p.ch_ddH[a] = pl->ch_ddH[a]; p.ch_dA[a] = pl->ch_dA[a]; }
            p.nc = q.num_components;
            for (int c = 0; c < q.num_components; ++c)
                for (int j = 0; j < 3; ++j) p.comp[c][j] = q.components[c][j];
            p.out = off;
            p.nom = (int)t.num_photon_energies;
            p.omegas = pl->d_omegas;
            p.mu = t.fermi_energy;
            p.T = t.temperature;
            p.width = t.broadening;
            p.low_width = t.shg_low_frequency_broadening;
            p.eta = t.shg_intermediate_regularization > 0 ? t.shg_intermediate_regularization : t.denominator_regularization;
            p.degeneracy = t.degeneracy_threshold;
            p.gaussian = t.broadening_type == WNLQG_GAUSSIAN ? 1 : 0;
            p.eta_correction = t.shg_eta_correction ? 1 : 0;
            p.vc = pl->vc;
            pl->shg.push_back(p);
            max_nc = std::max(max_nc, q.num_components);
        }
        off += width;
    }
    if (pl->shg.empty()) return WNLQG_OK;
    const size_t shg_bytes = ShgSmem::layout(pl->nw, max_nc).total;
    const bool shg_global = shg_bytes > smem_limit;   // large nw: matrices in a per-CTA global working set
    pl->shg_smem = shg_global ? 0 : shg_bytes;
    pl->shg_global = shg_global;
    const void *shg_fn = shg_function(shg_global, false);
    cudaError_t e = allow_dynamic_smem(shg_fn, (int)smem_limit);
    if (e == cudaSuccess && !shg_global) e = allow_dynamic_smem(shg_function(false, true), (int)smem_limit);
    if (e != cudaSuccess) return fail(WNLQG_ERR_CUDA, std::string("cudaFuncSetAttribute: ") + cudaGetErrorString(e));
    int per_sm = 0, pair_per_sm = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, shg_fn, 256, pl->shg_smem);
    if (e == cudaSuccess && !shg_global)
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&pair_per_sm, shg_function(false, true), 256, pl->shg_smem);
    if (e != cudaSuccess) return fail(WNLQG_ERR_CUDA, std::string("occupancy query: ") + cudaGetErrorString(e));
    if (per_sm < 1) return fail(WNLQG_ERR_UNSUPPORTED, "second-harmonic kernel cannot be resident with its shared memory");
    pl->shg_grid = sm_count * per_sm;
    pl->shg_pair = pair_per_sm >= 2;
    // A global working set is allocated for up to two CTAs per SM; one CTA per SM is the default
    // (measured at 64 orbitals: the L2-resident half grid is slower), the autotuner may change it.
    pl->shg_grid_alloc = shg_global || pl->shg_pair ? std::max(pl->shg_grid, 2 * sm_count) : pl->shg_grid;
    if (shg_global) {
        pl->shg_grid_l2 = l2_resident_grid(pl->shg_grid, (int64_t)shg_bytes, sm_count);
        pl->shg_grid = sm_count;
    }
    if (const char *g = std::getenv("WNLQG_B200_SHG_GRID")) {
        pl->shg_grid = std::max(1, std::min(pl->shg_grid_alloc, std::atoi(g)));
        pl->shg_pair = false;
    }
    const int64_t stride = ShgSmem::scratch_entries(pl->nw, max_nc);
    for (ShgParams &p : pl->shg) p.scratch_stride = stride;
    e = cudaMalloc(&pl->d_shg_scratch, (size_t)pl->shg_grid_alloc * stride * sizeof(double2));
    if (e != cudaSuccess) {
        cudaGetLastError();
        return fail(WNLQG_ERR_OUT_OF_MEMORY, "cudaMalloc of the second-harmonic scratch failed");
    }
    if (shg_global) {
        const int64_t gstride = (int64_t)((shg_bytes + 255) & ~(size_t)255);
        e = cudaMalloc(&pl->d_shg_gscratch, (size_t)pl->shg_grid_alloc * gstride);
        if (e != cudaSuccess) {
            cudaGetLastError();
            return fail(WNLQG_ERR_OUT_OF_MEMORY, "cudaMalloc of the second-harmonic working set failed");
        }
        for (ShgParams &p : pl->shg) p.gscratch_stride = gstride;
    }
    return WNLQG_OK;
}

wnlqg_status record_event(wnlqg_plan *pl, size_t idx) {
    while (pl->events.size() <= idx) {
        cudaEvent_t ev;
        WNLQG_CUDA(cudaEventCreate(&ev));
        pl->events.push_back(ev);
    }
    WNLQG_CUDA(cudaEventRecord(pl->events[idx], pl->stream));
    return WNLQG_OK;
}

// Tensor-core Fourier of one batch: phase slices, then the persistent tcgen05 GEMM writing the
// FP64 channels.
template <int S>
wnlqg_status launch_tc_fourier(wnlqg_plan *pl, int64_t nb, int64_t k_begin, const int64_t *mesh,
                               const double *kpts_device, const int64_t *kidx_device) {
    typedef tcf::Layout<S> L;
    const int64_t total = nb * (pl->tc_kpad / 2);
    const int blocks = (int)std::min<int64_t>((total + 255) / 256, (int64_t)pl->sm_count * 32);
    tcf::phase_slices_kernel<S><<<blocks, 256, 0, pl->stream>>>(
        pl->d_tcA, pl->tc_mpad, pl->tc_kpad, pl->model->d_rvec, pl->model->d_deg, pl->nr, nb, k_begin,
        mesh ? mesh[0] : 1, mesh ? mesh[1] : 1, mesh ? mesh[2] : 1, kpts_device, kidx_device);
    tcf::TcArgs a;
    a.colscale = pl->d_tc_colscale;
    a.xw = pl->d_xw;
    a.nb = nb;
    a.ncols = pl->tc_ncols;
    a.kblocks = (int)(pl->tc_kpad / tcf::BK);
    a.mtiles = (int)((nb + tcf::BM - 1) / tcf::BM);
    a.ntiles = (int)(pl->tc_npad / L::NT);
    a.err = pl->d_tc_err;
    const int tiles = a.mtiles * a.ntiles;
    const int grid = std::min(tiles, pl->sm_count);
    tcf::tc_fourier_kernel<S><<<grid, tcf::THREADS, L::SMEM_BYTES, pl->stream>>>(pl->tc_mapA, pl->tc_mapB, a);
    pl->launches += 1;
    pl->tc_used = true;
    WNLQG_CUDA(cudaGetLastError());
    return WNLQG_OK;
}

wnlqg_status run_tc_fourier(wnlqg_plan *pl, int64_t nb, int64_t k_begin, const int64_t *mesh, const double *kpts_device,
                            const int64_t *kidx_device) {
    switch (pl->tc_slices) {
    case 7: return launch_tc_fourier<7>(pl, nb, k_begin, mesh, kpts_device, kidx_device);
    case 4: return launch_tc_fourier<4>(pl, nb, k_begin, mesh, kpts_device, kidx_device);
    default: return fail(WNLQG_ERR_UNSUPPORTED, "tensor-core Fourier slice count");
    }
}

// Reports (and clears) a bounded-wait failure of the tensor-core Fourier after a synchronised call.
wnlqg_status tc_check(wnlqg_plan *pl) {
    if (!pl->tc_used || !pl->d_tc_err) return WNLQG_OK;
    pl->tc_used = false;
    int h = 0;
    WNLQG_CUDA(cudaMemcpy(&h, pl->d_tc_err, sizeof(int), cudaMemcpyDeviceToHost));
    if (h) {
        cudaMemset(pl->d_tc_err, 0, sizeof(int));
        return fail(WNLQG_ERR_DEVICE_TIMEOUT, "tensor-core Fourier: a bounded device wait gave up");
    }
    return WNLQG_OK;
}

// The isolation contract on one batch's energies (after the eigensolve): rows are row_base + the
// batch entry, or row_base + perm[entry] for Morton-ordered batches.
wnlqg_status run_isolation(wnlqg_plan *pl, int64_t nb, int64_t row_base, const int *perm, int prio = 0) {
    if (pl->iso_mode < 0 || nb <= 0) return WNLQG_OK;
    isolation_check_kernel<<<(unsigned)((nb + 127) / 128), 128, 0, pl->stream>>>(pl->d_E, nb, pl->nw, pl->iso_tol,
                                                                               pl->iso_mode, row_base, perm,
                                                                               pl->d_iso_key);
    isolation_record_kernel<<<1, 1, 0, pl->stream>>>(pl->d_E, nb, pl->nw, pl->iso_tol, pl->iso_mode, row_base,
                                                      pl->d_iso_key, pl->d_iso_rec, prio);
    pl->launches += 2;
    WNLQG_CUDA(cudaGetLastError());
    return WNLQG_OK;
}

// Reports (and clears) an isolation failure after a synchronised call, with the reference's
// message (geometry_isolated_spectrum_minimum_gap, OrthogonalBandDerivatives.jl:66-82;
// spectral_subspace_blocks, SubspacePositionMatrixElements.jl:5-22; bands 1-based).
wnlqg_status iso_check(wnlqg_plan *pl) {
    if (pl->iso_mode < 0 || !pl->d_iso_key) return WNLQG_OK;
    unsigned long long key = ISO_NONE;
    WNLQG_CUDA(cudaMemcpy(&key, pl->d_iso_key, sizeof(key), cudaMemcpyDeviceToHost));
    if (key == ISO_NONE) return WNLQG_OK;
    IsoRecord rec;
    WNLQG_CUDA(cudaMemcpy(&rec, pl->d_iso_rec, sizeof(rec), cudaMemcpyDeviceToHost));
    WNLQG_CUDA(cudaMemset(pl->d_iso_key, 0xFF, sizeof(unsigned long long)));
    WNLQG_CUDA(cudaMemset(pl->d_iso_rec, 0xFF, sizeof(IsoRecord)));
    char buf[256];
    const long long row = (long long)(key >> ISO_LOCAL_BITS);
    if (!std::isfinite(rec.gap))
        std::snprintf(buf, sizeof(buf), "empty/nonfinite geometry spectrum (k-point row %lld)", row);
    else if (pl->iso_mode == ISO_ALL_PAIRS)
        std::snprintf(buf, sizeof(buf),
                      "GEOMETRY_SINGLE_BAND_SPECTRUM_NOT_ISOLATED: bands=(%d,%d), gap_ev=%.17g, threshold_ev=%.17g "
                      "(k-point row %lld)",
                      rec.l + 1, rec.m + 1, rec.gap, pl->iso_tol, row);
    else
        std::snprintf(buf, sizeof(buf), "SPECTRAL_CROSS_BLOCK_GAP_UNRESOLVED: gap=%.17g eV (k-point row %lld)", rec.gap,
                      row);
    return fail(WNLQG_ERR_INVALID_ARGUMENT, buf);
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                  const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// 3D int8 tensor map [slices][rows][kpad] with a box of (64 bytes, box_rows, slices), 64-byte swizzle.
wnlqg_status encode_slices_map(EncodeTiledFn enc, CUtensorMap *map, int8_t *ptr, int64_t kpad, int64_t rows, int slices,
                               int box_rows) {
    cuuint64_t dims[3] = {(cuuint64_t)kpad, (cuuint64_t)rows, (cuuint64_t)slices};
    cuuint64_t strides[2] = {(cuuint64_t)kpad, (cuuint64_t)(kpad * rows)};
    cuuint32_t box[3] = {(cuuint32_t)tcf::BK, (cuuint32_t)box_rows, (cuuint32_t)slices};
    cuuint32_t estr[3] = {1, 1, 1};
    CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, ptr, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                     CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return fail(WNLQG_ERR_CUDA, "cuTensorMapEncodeTiled failed (" + std::to_string((int)r) + ")");
    return WNLQG_OK;
}

// Builds the B slices of the channel tiles (host, once per plan), the phase-slice buffer and both
// tensor maps.  tiles: [NR][C][nw^2] complex.
template <int S>
wnlqg_status setup_tc_fourier(wnlqg_plan *pl, const std::vector<double2> &tiles) {
    typedef tcf::Layout<S> L;
    const int64_t nr = pl->nr, nn = pl->nn, C = pl->C;
    const int64_t ncols = 2 * C * nn;
    const int64_t kpad = ((2 * nr + tcf::BK - 1) / tcf::BK) * tcf::BK;
    const int64_t npad = ((ncols + L::NT - 1) / L::NT) * L::NT;
    const int64_t mpad = ((pl->max_batch + tcf::BM - 1) / tcf::BM) * tcf::BM;
    std::vector<int8_t> Bq((size_t)S * npad * kpad, 0);
    std::vector<double> colscale((size_t)npad, 0.0);
    const int64_t row_stride = C * nn;
    for (int64_t n = 0; n < C * nn; ++n) {
        double mx = 0.0;
        for (int64_t r = 0; r < nr; ++r) {
            const double2 t = tiles[(size_t)(r * row_stride + n)];
            mx = std::max(mx, std::max(std::fabs(t.x), std::fabs(t.y)));
        }
        int e = 0;
        if (mx > 0.0) std::frexp(mx, &e);
        for (int sidx = 0; sidx < 2; ++sidx) {
            const int64_t row = 2 * n + sidx;
            colscale[(size_t)row] = std::ldexp(1.0, e - 12);
            for (int64_t r = 0; r < nr; ++r) {
                const double2 t = tiles[(size_t)(r * row_stride + n)];
                const double v0 = sidx == 0 ? t.x : t.y;    // multiplies Re F
                const double v1 = sidx == 0 ? -t.y : t.x;   // multiplies Im F
                int8_t s0[S], s1[S];
                tcf::slice_value<S>(std::ldexp(v0, -e), s0);
                tcf::slice_value<S>(std::ldexp(v1, -e), s1);
                for (int i = 0; i < S; ++i) {
                    Bq[(size_t)((i * npad + row) * kpad + 2 * r)] = s0[i];
                    Bq[(size_t)((i * npad + row) * kpad + 2 * r + 1)] = s1[i];
                }
            }
        }
    }
    auto alloc = [&](void **ptr, size_t bytes) -> wnlqg_status {
        cudaError_t ce = cudaMalloc(ptr, std::max<size_t>(bytes, 16));
        if (ce != cudaSuccess) {
            cudaGetLastError();
            return fail(WNLQG_ERR_OUT_OF_MEMORY, "cudaMalloc of " + std::to_string(bytes) + " bytes failed");
        }
        return WNLQG_OK;
    };
    wnlqg_status st;
    if ((st = alloc((void **)&pl->d_tcB, Bq.size())) != WNLQG_OK) return st;
    if ((st = alloc((void **)&pl->d_tcA, (size_t)S * mpad * kpad)) != WNLQG_OK) return st;
    if ((st = alloc((void **)&pl->d_tc_colscale, colscale.size() * sizeof(double))) != WNLQG_OK) return st;
    if ((st = alloc((void **)&pl->d_tc_err, sizeof(int))) != WNLQG_OK) return st;
    WNLQG_CUDA(cudaMemcpy(pl->d_tcB, Bq.data(), Bq.size(), cudaMemcpyHostToDevice));
    WNLQG_CUDA(cudaMemcpy(pl->d_tc_colscale, colscale.data(), colscale.size() * sizeof(double), cudaMemcpyHostToDevice));
    WNLQG_CUDA(cudaMemset(pl->d_tc_err, 0, sizeof(int)));
    WNLQG_CUDA(cudaMemset(pl->d_tcA, 0, (size_t)S * mpad * kpad));
    void *fn = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fn, 12000, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess || !fn)
        return fail(WNLQG_ERR_CUDA, "cuTensorMapEncodeTiled is not available from the driver");
    EncodeTiledFn enc = reinterpret_cast<EncodeTiledFn>(fn);
    if ((st = encode_slices_map(enc, &pl->tc_mapA, pl->d_tcA, kpad, mpad, S, tcf::BM)) != WNLQG_OK) return st;
    if ((st = encode_slices_map(enc, &pl->tc_mapB, pl->d_tcB, kpad, npad, S, L::NT)) != WNLQG_OK) return st;
    WNLQG_CUDA(cudaFuncSetAttribute(tcf::tc_fourier_kernel<S>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)L::SMEM_BYTES));
    pl->tc_kpad = kpad;
    pl->tc_npad = npad;
    pl->tc_mpad = mpad;
    pl->tc_ncols = ncols;
    pl->tc_slices = S;
    return WNLQG_OK;
}

// One batch: phases, Fourier GEMM, eigensolve.  kpts_device == nullptr selects mesh mode.
// The orthogonal eigensolver stages on Hermitian matrices hk + b * stride_in (nw x nw, upper
// triangle read): the team stages up to 32 orbitals, the CTA mixed-precision stages above;
// eigenvalues into d_E, canonical eigenvectors into d_U.  warm_in: warm-start along the batch.
wnlqg_status run_orth_eigen(wnlqg_plan *pl, const double2 *hk, int64_t stride_in, int64_t nb, int warm_in) {
    if (pl->warp_eigh) {
        const int np = pl->nw + (pl->nw & 1);
        if (pl->small_f64) {
            const RegKernel rk = reg_f64_kernel(np);
            const int per_block = 128 / rk.lanes;
            const size_t smem = rk.group_smem * per_block;
            int per_sm = 1;
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, rk.fn, 128, smem);
            const int64_t grid = std::min<int64_t>((nb + per_block - 1) / per_block, (int64_t)std::max(1, per_sm) * pl->sm_count);
            int64_t stride = stride_in, nb_arg = nb;
            int nw_arg = pl->nw;
            double *E = pl->d_E;
            double2 *U = pl->d_U;
            void *args[] = {(void *)&hk, &stride, &nb_arg, &nw_arg, &E, &U};
            WNLQG_CUDA(cudaLaunchKernel(rk.fn, dim3((unsigned)grid), dim3(128), args, smem, pl->stream));
            WNLQG_CUDA(cudaGetLastError());
            return WNLQG_OK;
        }
        // Stage 1, FP64 path (17 to 32 orbitals): one-sided Jacobi, one warp per chain of neighbouring
        // points, twelve chains per SM (what the kernel's registers hold).  The mixed path keeps the
        // two-sided stage in shared memory: its one first-order completion leaves errors of second
        // order in what stage 1 leaves, so another stage 1 would show in its sums (2e-8 relative).
        // Stage 2: 64-thread blocks holding two one-warp teams or one 64-thread team.
        const int tm = pl->eigh_team;
        const void *ref_fn = tm == 128 ? (const void *)eigh_refine_f64_team_kernel<128>
                             : tm == 64 ? (const void *)eigh_refine_f64_team_kernel<64> : (const void *)eigh_refine_f64_team_kernel<32>;
        const int ref_threads = tm == 128 ? 128 : 64, ref_teams = tm == 32 ? 2 : 1;
        int warm = warm_in;
        if (pl->f32_team) {
            const void *f32_fn = tm == 128 ? (const void *)jacobi_f32_team_kernel<128>
                                 : tm == 64 ? (const void *)jacobi_f32_team_kernel<64> : (const void *)jacobi_f32_team_kernel<32>;
            const int f32_threads = tm == 32 ? 128 : tm, f32_teams = tm == 32 ? 4 : 1;
            int per_sm = 1;
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, f32_fn, f32_threads, pl->eigh_smem);
            const int64_t f32_grid = std::min<int64_t>((nb + f32_teams - 1) / f32_teams, (int64_t)std::max(1, per_sm) * pl->sm_count);
            int64_t nb_arg = nb;
            int nw_arg = pl->nw;
            float2 *v32 = pl->d_V32;
            int64_t stride = stride_in;
            void *args[] = {(void *)&hk, &stride, &nb_arg, &nw_arg, &v32, &warm};
            WNLQG_CUDA(cudaLaunchKernel(f32_fn, dim3((unsigned)f32_grid), dim3(f32_threads), args, pl->eigh_smem, pl->stream));
        } else {
            const RegKernel rk = onesided_kernel(np);
            const int per_block = 128 / rk.lanes;
            int64_t chains = std::min<int64_t>(nb, (int64_t)12 * pl->sm_count);
            int64_t nb_arg = nb;
            int nw_arg = pl->nw;
            float2 *v32 = pl->d_V32;
            int64_t stride = stride_in;
            void *args[] = {(void *)&hk, &stride, &nb_arg, &nw_arg, &v32, &chains, &warm};
            WNLQG_CUDA(cudaLaunchKernel(rk.fn, dim3((unsigned)((chains + per_block - 1) / per_block)), dim3(128), args,
                                        rk.group_smem * per_block, pl->stream));
        }
        int per_sm_r = 1;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm_r, ref_fn, ref_threads, pl->refine_smem);
        const int64_t r_grid = std::min<int64_t>((nb + ref_teams - 1) / ref_teams, (int64_t)std::max(1, per_sm_r) * pl->sm_count);
        {
            int64_t stride = stride_in, nb_arg = nb;
            int nw_arg = pl->nw;
            const float2 *v32 = pl->d_V32;
            double *E = pl->d_E;
            double2 *U = pl->d_U;
            int converge = pl->task.precision == WNLQG_PRECISION_MIXED ? 0 : 1;
            void *args[] = {(void *)&hk, &stride, (void *)&v32, &nb_arg, &nw_arg, &E, &U, &converge};
            WNLQG_CUDA(cudaLaunchKernel(ref_fn, dim3((unsigned)r_grid), dim3(ref_threads), args, pl->refine_smem, pl->stream));
        }
        pl->launches += 1;
    } else if (pl->cta_mixed) {
        const int converge = pl->task.precision == WNLQG_PRECISION_MIXED ? 0 : 1;
        const int warm = warm_in;
        const int64_t N = stride_in;
        if (converge) {
            const void *fn = onesided_cta_fn(pl->nw + (pl->nw & 1));
            const int threads = OsCtaSmem::threads(pl->nw + (pl->nw & 1));
            int per_sm = 1;
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, threads, pl->eigh_smem);
            const int64_t grid = std::min<int64_t>(nb, (int64_t)std::max(1, per_sm) * pl->sm_count);
            int64_t stride = N, nb_arg = nb;
            int nw_arg = pl->nw, warm_arg = warm;
            float2 *v32 = pl->d_V32;
            void *args[] = {(void *)&hk, &stride, &nb_arg, &nw_arg, &v32, &warm_arg};
            WNLQG_CUDA(cudaLaunchKernel(fn, dim3((unsigned)grid), dim3(threads), args, pl->eigh_smem, pl->stream));
        } else if (pl->cta_gw1) {
            jacobi_f32_cta_kernel<true><<<(unsigned)std::min<int64_t>(nb, pl->eigh_grid), 256, 0, pl->stream>>>(
                hk, N, nb, pl->nw, pl->d_V32, pl->d_eigh_scratch, pl->eigh_scratch_stride, warm);
        } else {
            int per_sm = 1;
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, jacobi_f32_cta_kernel<false>, 256, pl->eigh_smem);
            const int64_t grid = std::min<int64_t>(nb, (int64_t)std::max(1, per_sm) * pl->sm_count);
            jacobi_f32_cta_kernel<false><<<(unsigned)grid, 256, pl->eigh_smem, pl->stream>>>(hk, N, nb, pl->nw, pl->d_V32,
                                                                                            nullptr, 0, warm);
        }
        if (pl->cta_gw2) {
            eigh_refine_f64_cta_kernel<true><<<(unsigned)std::min<int64_t>(nb, pl->eigh_grid), pl->refine_cta_threads, 0, pl->stream>>>(
                hk, N, pl->d_V32, nb, pl->nw, pl->d_E, pl->d_U, converge, pl->d_eigh_scratch, pl->eigh_scratch_stride);
        } else {
            int per_sm = 1;
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, eigh_refine_f64_cta_kernel<false>, pl->refine_cta_threads,
                                                          pl->refine_smem);
            const int64_t grid = std::min<int64_t>(nb, (int64_t)std::max(1, per_sm) * pl->sm_count);
            eigh_refine_f64_cta_kernel<false><<<(unsigned)grid, pl->refine_cta_threads, pl->refine_smem, pl->stream>>>(
                hk, N, pl->d_V32, nb, pl->nw, pl->d_E, pl->d_U, converge, nullptr, 0);
        }
        pl->launches += 1;
    }
    WNLQG_CUDA(cudaGetLastError());
    return WNLQG_OK;
}

wnlqg_status run_front(wnlqg_plan *pl, int64_t nb, int64_t k_begin, const int64_t *mesh, const double *kpts_device,
                       size_t ev_base, const int64_t *kidx_device = nullptr, bool ordered = false,
                       const double2 *staged_tiles = nullptr) {
    const int nr = pl->nr;
    int64_t N = (int64_t)pl->C * pl->nn;
    const bool staged = mesh != nullptr && kpts_device == nullptr && kidx_device == nullptr && pl->P1 <= STAGED_MAX_P1 &&
                        mesh[0] >= pl->P1;
    pl->use_staged_last = staged;
    if (staged) {
        const int64_t n1 = mesh[0], n2 = mesh[1], n3 = mesh[2];
        const int64_t line_first = k_begin / n1, line_last = (k_begin + nb - 1) / n1;
        const int64_t nlines = line_last - line_first + 1;
        const int64_t i3_first = line_first / n2, i3_last = line_last / n2;
        const int64_t n3t = i3_last - i3_first + 1;
        const size_t needY = (size_t)n3t * pl->P12 * N, needZ = (size_t)nlines * pl->P1 * N;
        if (needY > pl->stageY_elems) {
            if (pl->d_stageY && pl->graph_refs > 0) pl->retired.push_back(pl->d_stageY);
            else if (pl->d_stageY) WNLQG_CUDA(cudaFree(pl->d_stageY));
            pl->d_stageY = nullptr;
            pl->stageY_elems = 0;
            WNLQG_CUDA(cudaMalloc(&pl->d_stageY, needY * sizeof(double2)));
            pl->stageY_elems = needY;
        }
        if (needZ > pl->stageZ_elems) {
            if (pl->d_stageZ && pl->graph_refs > 0) pl->retired.push_back(pl->d_stageZ);
            else if (pl->d_stageZ) WNLQG_CUDA(cudaFree(pl->d_stageZ));
            pl->d_stageZ = nullptr;
            pl->stageZ_elems = 0;
            WNLQG_CUDA(cudaMalloc(&pl->d_stageZ, needZ * sizeof(double2)));
            pl->stageZ_elems = needZ;
        }
        const unsigned cb = (unsigned)((N + 255) / 256);
        staged_r3_kernel<<<dim3(cb, pl->P12, (unsigned)n3t), 256, 0, pl->stream>>>(
            staged_tiles ? staged_tiles : pl->d_tiles, N, pl->groups, pl->model->d_rvec, pl->model->d_deg, i3_first, n3, pl->d_stageY);
        staged_r2_kernel<<<dim3(cb, pl->P1, (unsigned)nlines), 256, 0, pl->stream>>>(pl->d_stageY, N, pl->groups,
                                                                                       line_first, n2, i3_first,
                                                                                       pl->d_stageZ);
        staged_r1_kernel<<<dim3(cb, (unsigned)((nb + STAGED_BT - 1) / STAGED_BT)), 256, 0, pl->stream>>>(
            pl->d_stageZ, N, pl->groups, k_begin, nb, n1, line_first, pl->d_xw);
    } else if (pl->tc_slices > 0) {
        wnlqg_status tst = run_tc_fourier(pl, nb, k_begin, mesh, kpts_device, kidx_device);
        if (tst != WNLQG_OK) return tst;
    } else {
        int64_t total = nb * nr;
        int blocks = (int)std::min<int64_t>((total + 255) / 256, 148 * 32);
        phase_kernel<<<blocks, 256, 0, pl->stream>>>(pl->d_phase, pl->model->d_rvec, pl->model->d_deg, nr, nb,
                                                     k_begin, mesh ? mesh[0] : 1, mesh ? mesh[1] : 1,
                                                     mesh ? mesh[2] : 1, kpts_device, kidx_device);
        dim3 grid((unsigned)((N + FG_BN - 1) / FG_BN), (unsigned)((nb + FG_BM - 1) / FG_BM));
        fourier_gemm_f64<<<grid, 256, 0, pl->stream>>>(pl->d_phase, pl->d_tiles, pl->d_xw, nb, N, nr);
    }
    wnlqg_status st = record_event(pl, ev_base + 1);
    if (st != WNLQG_OK) return st;
    const unsigned eigh_grid = (unsigned)(pl->d_eigh_scratch ? std::min<int64_t>(nb, pl->eigh_grid) : nb);
    if (pl->nonorth && pl->gen_mixed) {
        // FP64 Cholesky reduction, the orthogonal stages of the plan's precision on C, U = L^-H V.
        const double2 *hk = pl->d_xw + (int64_t)pl->ch_H * pl->nn, *sk = pl->d_xw + (int64_t)pl->ch_S * pl->nn;
        if (pl->gred_gw) {
            cholesky_reduce_kernel<true><<<(unsigned)std::min<int64_t>(nb, pl->gred_grid), 256, 0, pl->stream>>>(
                hk, sk, N, nb, pl->nw, pl->d_gC, pl->d_gL, pl->d_status, pl->d_gred_scratch, pl->gred_stride);
        } else {
            int per_sm = 1;
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, cholesky_reduce_kernel<false>, 256, pl->gred_smem);
            const int64_t grid = std::min<int64_t>(nb, (int64_t)std::max(1, per_sm) * pl->sm_count);
            cholesky_reduce_kernel<false><<<(unsigned)grid, 256, pl->gred_smem, pl->stream>>>(
                hk, sk, N, nb, pl->nw, pl->d_gC, pl->d_gL, pl->d_status, nullptr, 0);
        }
        const bool contiguous = mesh != nullptr && kpts_device == nullptr && kidx_device == nullptr;
        const int warm = pl->warm_mode && (contiguous || ordered) ? 1 : 0;
        if ((st = run_orth_eigen(pl, pl->d_gC, pl->nn, nb, warm)) != WNLQG_OK) return st;
        gen_back_substitute_kernel<<<(unsigned)std::min<int64_t>(nb, (int64_t)pl->sm_count * 16), 128, 0, pl->stream>>>(
            pl->d_gL, pl->d_U, nb, pl->nw);
        pl->launches += 2;
    } else if (pl->nonorth) {
        if (pl->d_eigh_scratch)
            generalized_eigh_kernel<true><<<eigh_grid, pl->eigh_threads, 0, pl->stream>>>(
                pl->d_xw + (int64_t)pl->ch_H * pl->nn, pl->d_xw + (int64_t)pl->ch_S * pl->nn, N, nb, pl->nw, pl->d_E,
                pl->d_U, pl->d_status, pl->d_eigh_scratch, pl->eigh_scratch_stride);
        else
            generalized_eigh_kernel<false><<<eigh_grid, pl->eigh_threads, pl->eigh_smem, pl->stream>>>(
                pl->d_xw + (int64_t)pl->ch_H * pl->nn, pl->d_xw + (int64_t)pl->ch_S * pl->nn, N, nb, pl->nw, pl->d_E,
                pl->d_U, pl->d_status);
    } else if (pl->warp_eigh || pl->cta_mixed) {
        const bool contiguous = mesh != nullptr && kpts_device == nullptr && kidx_device == nullptr;
        // Mesh runs and Morton-ordered point batches warm-start the FP32 stage along the run.
        const int warm = pl->warm_mode && (contiguous || ordered) ? 1 : 0;
        if ((st = run_orth_eigen(pl, pl->d_xw + (int64_t)pl->ch_H * pl->nn, N, nb, warm)) != WNLQG_OK) return st;
    } else
        if (pl->d_eigh_scratch)
            jacobi_eigh_kernel<double, true><<<eigh_grid, pl->eigh_threads, 0, pl->stream>>>(
                pl->d_xw + (int64_t)pl->ch_H * pl->nn, N, nb, pl->nw, pl->d_E, pl->d_U, 8.673617379884035e-19,
                pl->d_eigh_scratch, pl->eigh_scratch_stride);
        else
            jacobi_eigh_kernel<double, false><<<eigh_grid, pl->eigh_threads, pl->eigh_smem, pl->stream>>>(
                pl->d_xw + (int64_t)pl->ch_H * pl->nn, N, nb, pl->nw, pl->d_E, pl->d_U, 8.673617379884035e-19);
    st = record_event(pl, ev_base + 2);
    if (st != WNLQG_OK) return st;
    pl->launches += staged ? 4 : 3;
    WNLQG_CUDA(cudaGetLastError());
    return WNLQG_OK;
}

// One response-kernel pass over the current batch (curv_out: the stencil slot of band-curvature passes).
wnlqg_status launch_pass(wnlqg_plan *pl, const Pass &ps, int64_t nb, int mode, double scale, int64_t point_offset,
                         const double *weights, const int *out_perm, double *curv_out) {
    RespParams p = ps.params;
    if (pl->nonorth) {
        p.ng_r = pl->d_ng_r;
        p.ng_v = pl->d_ng_v;
        p.ng_G = pl->d_ng_G;
        p.ng_pairs = pl->ng.npairs;
        for (int g = 0; g < p.n_g; ++g) p.g_ng[g] = pl->ng_gidx[p.g_p[g] * 3 + p.g_d[g]];
    }
    p.batch = nb;
    p.xw = pl->d_xw;
    p.E = pl->d_E;
    p.U = pl->d_U;
    p.mode = mode;
    p.scale = scale;
    p.weights = weights;
    p.partials = pl->d_partials;
    p.out_points = pl->d_points;
    p.point_offset = point_offset;
    p.out_perm = out_perm;
    p.curv_out = curv_out;
    p.gscratch = ps.global ? pl->d_resp_scratch : nullptr;
    p.gscratch_stride = pl->resp_scratch_stride;
    const size_t launch_smem = ps.global ? 0 : ps.smem;
    void *args[] = {&p};
    if (pl->resp_wide && ps.grid_wide > 0)
        WNLQG_CUDA(cudaLaunchKernel(response_wide_fn(), dim3(ps.grid_wide), dim3(512), args, launch_smem, pl->stream));
    else
        WNLQG_CUDA(cudaLaunchKernel(response_fn(pl->task.precision == WNLQG_PRECISION_MIXED, pl->nonorth, ps.global, p.n_fc > 0),
                                    dim3(ps.global && pl->resp_gw_grid > 0 ? pl->resp_gw_grid : ps.grid),
                                    dim3(ps.threads), args, launch_smem, pl->stream));
    pl->launches += 1;
    return WNLQG_OK;
}

wnlqg_status run_passes(wnlqg_plan *pl, int64_t nb, int mode, double scale, int64_t point_offset,
                        const double *weights = nullptr, const int *out_perm = nullptr) {
    if (pl->nonorth && !pl->passes.empty()) {
        NonorthParams q = pl->ng;
        q.batch = nb;
        q.xw = pl->d_xw;
        q.E = pl->d_E;
        q.U = pl->d_U;
        nonorth_geometry_kernel<<<(unsigned)std::min<int64_t>(nb, pl->ng_grid), 256, 0, pl->stream>>>(q);
        pl->launches += 1;
    }
    for (const Pass &ps : pl->passes) {
        if (ps.fd) continue;
        wnlqg_status st = launch_pass(pl, ps, nb, mode, scale, point_offset, weights, out_perm, nullptr);
        if (st != WNLQG_OK) return st;
    }
    if (pl->fd_nd > 0 && nb > 0) {
        // Fermi-sea dipole: centre occupations times the stencil's curvature differences.
        SeaParams q = pl->sea;
        q.batch = nb;
        q.E = pl->d_E;
        q.mus = pl->d_mus;
        q.scale = scale;
        q.weights = weights;
        q.mode = mode;
        q.partials = pl->d_partials;
        q.out_points = pl->d_points;
        q.point_offset = point_offset;
        q.out_perm = out_perm;
        const int grid = (int)std::max<int64_t>(1, std::min<int64_t>(nb, std::min(pl->sm_count, pl->partial_slots)));
        sea_dipole_kernel<<<grid, 128, 0, pl->stream>>>(q);
        pl->launches += 1;
    }
    if (pl->bcda.n_items > 0 && nb > 0) {
        // Fermi-sea dipole, analytic geometry: the local dipole of every band from the centre.
        BcdaParams q = pl->bcda;
        q.batch = nb;
        q.xw = pl->d_xw;
        q.E = pl->d_E;
        q.U = pl->d_U;
        q.mus = pl->d_mus;
        q.scale = scale;
        q.weights = weights;
        q.mode = mode;
        q.partials = pl->d_partials;
        q.out_points = pl->d_points;
        q.point_offset = point_offset;
        q.out_perm = out_perm;
        bcd_analytic_kernel<<<(unsigned)pl->bcda_grid, 256, 0, pl->stream>>>(q);
        pl->launches += 1;
    }
    if (pl->metric_shg && !pl->shg.empty()) {
        MetricShgParams q = pl->mshg;
        q.batch = nb;
        q.xw = pl->d_xw;
        q.E = pl->d_E;
        q.U = pl->d_U;
        metric_shg_kernel<<<(unsigned)std::min<int64_t>(nb, pl->mshg_grid), 256, 0, pl->stream>>>(q);
        pl->launches += 1;
    }
    for (const ShgParams &tmpl : pl->shg) {
        ShgParams p = tmpl;
        p.batch = nb;
        if (pl->metric_shg) {
            p.metric = 1;
            p.vertex_eta = pl->task.denominator_regularization;
            p.m_src = pl->d_mshg_src;
            p.m_diag = pl->d_mshg_diag;
        }
        p.xw = pl->d_xw;
        p.E = pl->d_E;
        p.U = pl->d_U;
        p.mode = mode;
        p.scale = scale;
        p.weights = weights;
        p.partials = pl->d_partials;
        p.out_points = pl->d_points;
        p.point_offset = point_offset;
        p.out_perm = out_perm;
        p.scratch = pl->d_shg_scratch;
        p.gscratch = pl->d_shg_gscratch;
        void *args[] = {(void *)&p};
        WNLQG_CUDA(cudaLaunchKernel(shg_function(pl->shg_global, pl->shg_pair_now),
                                    dim3(pl->shg_pair_now ? 2 * pl->sm_count : pl->shg_grid), dim3(256), args,
                                    pl->shg_smem, pl->stream));
        pl->launches += 1;
    }
    WNLQG_CUDA(cudaGetLastError());
    return WNLQG_OK;
}

// The finite-difference stencil of the Fermi-sea Berry dipole for one batch (its k-points from
// the same source as the centre's front): for each derivative axis j and sign, the shifted points
// k +- delta_j go through the arbitrary-k front, the isolation contract (priority 1 + 2 j + sign,
// after the centre's 0, the reference's order) and the band-curvature passes into stencil slot
// 2 j + sign.  Runs before the centre's front, which then leaves the centre's energies in place.
wnlqg_status run_fd_stencil(wnlqg_plan *pl, int64_t nb, int64_t k_begin, const int64_t *mesh, const double *kpts_device,
                            const int64_t *kidx_device, bool ordered, size_t ev_base, int64_t row_base, const int *perm) {
    if (pl->fd_nd == 0 || nb <= 0) return WNLQG_OK;
    // Shifted runs follow the centre's order: mesh runs and ordered batches warm-start the eigensolver.
    const bool run = ordered || (mesh != nullptr && kpts_device == nullptr && kidx_device == nullptr);
    const int64_t slot = (int64_t)pl->fd_npair * pl->nw;
    // A run of mesh points shifted by +-delta is the same run with the shifted tile sets.
    const bool staged = pl->d_fd_tiles && mesh != nullptr && kpts_device == nullptr && kidx_device == nullptr &&
                        mesh[0] >= pl->P1;
    const size_t per = (size_t)pl->nr * pl->C * pl->nn;
    for (int j = 0; j < pl->fd_nd; ++j)
        for (int sgn = 0; sgn < 2; ++sgn) {
            wnlqg_status st;
            if (staged) {
                st = run_front(pl, nb, k_begin, mesh, nullptr, ev_base, nullptr, false, pl->d_fd_tiles + (2 * j + sgn) * per);
            } else {
                const double s = sgn == 0 ? 1.0 : -1.0;
                const double *dl = pl->fd_delta[j];
                fd_shift_kernel<<<(unsigned)((nb + 255) / 256), 256, 0, pl->stream>>>(
                    kpts_device, kidx_device, k_begin, mesh ? mesh[0] : 1, mesh ? mesh[1] : 1, mesh ? mesh[2] : 1, nb,
                    s * dl[0], s * dl[1], s * dl[2], pl->d_fd_k);
                pl->launches += 1;
                st = run_front(pl, nb, 0, nullptr, pl->d_fd_k, ev_base, nullptr, run);
            }
            if (st != WNLQG_OK) return st;
            if ((st = run_isolation(pl, nb, row_base, perm, 1 + 2 * j + sgn)) != WNLQG_OK) return st;
            for (const Pass &ps : pl->passes) {
                if (!ps.fd) continue;
                if ((st = launch_pass(pl, ps, nb, 1, 1.0, 0, nullptr, nullptr, pl->d_fd_curv + (2 * j + sgn) * slot)) != WNLQG_OK)
                    return st;
            }
        }
    WNLQG_CUDA(cudaGetLastError());
    return WNLQG_OK;
}

wnlqg_status check_plan(const wnlqg_plan *pl) {
    if (!pl) return fail(WNLQG_ERR_INVALID_ARGUMENT, "plan is NULL");
    return WNLQG_OK;
}

}  // namespace

extern "C" {

const char *wnlqg_b200_version(void) { return "wnlqg-b200 0.1.0 (sm_100a)"; }

wnlqg_status wnlqg_b200_last_error(char *buffer, size_t capacity) {
    if (!buffer || capacity == 0) return WNLQG_ERR_INVALID_ARGUMENT;
    size_t n = std::min(capacity - 1, g_error.size());
    std::memcpy(buffer, g_error.data(), n);
    buffer[n] = '\0';
    return WNLQG_OK;
}

int32_t wnlqg_b200_device_count(void) {
    int n = 0;
    if (cudaGetDeviceCount(&n) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return n;
}

wnlqg_status wnlqg_b200_model_create(const wnlqg_model_desc *desc, int32_t device, wnlqg_model **out_model) {
    if (!desc || !out_model) return fail(WNLQG_ERR_INVALID_ARGUMENT, "NULL argument");
    *out_model = nullptr;
    if (desc->num_orbitals <= 0 || desc->num_r_vectors <= 0)
        return fail(WNLQG_ERR_DIMENSION_MISMATCH, "num_orbitals and num_r_vectors must be positive");
    if (desc->num_orbitals > 128)
        return fail(WNLQG_ERR_UNSUPPORTED, "this build supports num_orbitals <= 128");
    if (!desc->lattice || !desc->r_vectors || !desc->r_degeneracies || !desc->hamiltonian_r)
        return fail(WNLQG_ERR_INVALID_ARGUMENT, "lattice, r_vectors, r_degeneracies and hamiltonian_r are required");
    const int nw = (int)desc->num_orbitals, nr = (int)desc->num_r_vectors;
    const size_t nn = (size_t)nw * nw;
    if (!finite_array(desc->lattice, 9)) return fail(WNLQG_ERR_NONFINITE, "lattice contains non-finite values");
    if (!finite_array(desc->hamiltonian_r, 2 * nn * nr)) return fail(WNLQG_ERR_NONFINITE, "hamiltonian_r contains non-finite values");
    if (desc->position_r && !finite_array(desc->position_r, 2 * nn * 3 * nr))
        return fail(WNLQG_ERR_NONFINITE, "position_r contains non-finite values");
    if (desc->overlap_r && !finite_array(desc->overlap_r, 2 * nn * nr))
        return fail(WNLQG_ERR_NONFINITE, "overlap_r contains non-finite values");
    for (int r = 0; r < nr; ++r)
        if (desc->r_degeneracies[r] <= 0) return fail(WNLQG_ERR_INVALID_ARGUMENT, "r_degeneracies must be positive");
    int ndev = 0;
    WNLQG_CUDA(cudaGetDeviceCount(&ndev));
    if (device < 0 || device >= ndev) return fail(WNLQG_ERR_INVALID_ARGUMENT, "device index out of range");
    WNLQG_CUDA(cudaSetDevice(device));
    wnlqg_model *m = new wnlqg_model();
    m->device = device;
    m->nw = nw;
    m->nr = nr;
    std::memcpy(m->lattice, desc->lattice, sizeof(m->lattice));
    m->rvec.assign(desc->r_vectors, desc->r_vectors + 3 * (size_t)nr);
    m->deg.assign(desc->r_degeneracies, desc->r_degeneracies + nr);
    m->H.resize(nn * nr);
    std::memcpy(m->H.data(), desc->hamiltonian_r, sizeof(double2) * nn * nr);
    m->has_overlap = desc->overlap_r != nullptr;
    if (m->has_overlap) {
        m->S.resize(nn * nr);
        std::memcpy(m->S.data(), desc->overlap_r, sizeof(double2) * nn * nr);
    }
    m->has_position = desc->position_r != nullptr;
    if (m->has_position) {
        m->A.resize(nn * 3 * nr);
        std::memcpy(m->A.data(), desc->position_r, sizeof(double2) * nn * 3 * nr);
    }
    cudaError_t e1 = cudaMalloc(&m->d_rvec, sizeof(int64_t) * 3 * nr);
    cudaError_t e2 = cudaMalloc(&m->d_deg, sizeof(int64_t) * nr);
    if (e1 != cudaSuccess || e2 != cudaSuccess) {
        cudaFree(m->d_rvec);
        cudaFree(m->d_deg);
        delete m;
        return fail(WNLQG_ERR_OUT_OF_MEMORY, "cudaMalloc failed for the model");
    }
    WNLQG_CUDA(cudaMemcpy(m->d_rvec, m->rvec.data(), sizeof(int64_t) * 3 * nr, cudaMemcpyHostToDevice));
    WNLQG_CUDA(cudaMemcpy(m->d_deg, m->deg.data(), sizeof(int64_t) * nr, cudaMemcpyHostToDevice));
    *out_model = m;
    return WNLQG_OK;
}

wnlqg_status wnlqg_b200_model_destroy(wnlqg_model *model) {
    if (!model) return WNLQG_OK;
    cudaSetDevice(model->device);
    cudaFree(model->d_rvec);
    cudaFree(model->d_deg);
    delete model;
    return WNLQG_OK;
}

wnlqg_status wnlqg_b200_plan_destroy(wnlqg_plan *pl) {
    if (!pl) return WNLQG_OK;
    if (pl->graph_refs > 0)
        return fail(WNLQG_ERR_INVALID_ARGUMENT, "plan is captured in a CUDA graph: destroy the graph first");
    cudaSetDevice(pl->model->device);
    for (void *ptr : pl->retired) cudaFree(ptr);
    if (pl->stream) cudaStreamSynchronize(pl->stream);
    for (void *ptr : {(void *)pl->d_tiles, (void *)pl->d_phase, (void *)pl->d_xw, (void *)pl->d_U, (void *)pl->d_out,
                      (void *)pl->d_points, (void *)pl->d_E, (void *)pl->d_kpts, (void *)pl->d_omegas,
                      (void *)pl->d_partials, (void *)pl->d_weights, (void *)pl->d_groups, (void *)pl->d_stageY,
                      (void *)pl->d_stageZ, (void *)pl->d_V32, (void *)pl->d_kidx, (void *)pl->d_mus, (void *)pl->d_status,
                      (void *)pl->d_shg_scratch, (void *)pl->d_tcA, (void *)pl->d_tcB, (void *)pl->d_tc_colscale,
                      (void *)pl->d_tc_err, (void *)pl->d_shg_gscratch, (void *)pl->d_eigh_scratch,
                      (void *)pl->d_resp_scratch, (void *)pl->d_ng_r, (void *)pl->d_ng_v, (void *)pl->d_ng_G,
                      (void *)pl->d_ng_ws, (void *)pl->d_mshg_src, (void *)pl->d_mshg_diag, (void *)pl->d_mshg_ws,
                      (void *)pl->d_okeys, (void *)pl->d_operm, (void *)pl->d_ok, (void *)pl->d_ow, pl->d_osort_tmp,
                      (void *)pl->d_gC, (void *)pl->d_gL, (void *)pl->d_gred_scratch, (void *)pl->d_iso_key,
                      (void *)pl->d_iso_rec, (void *)pl->d_fd_k, (void *)pl->d_fd_curv, (void *)pl->d_bcda_scratch,
                      (void *)pl->d_fd_tiles})
        if (ptr) cudaFree(ptr);
    for (cudaEvent_t ev : pl->events) cudaEventDestroy(ev);
    if (pl->stream) cudaStreamDestroy(pl->stream);
    delete pl;
    return WNLQG_OK;
}

wnlqg_status wnlqg_b200_plan_create(wnlqg_model *model, const wnlqg_task_desc *task, int64_t max_batch,
                                    wnlqg_plan **out_plan) {
    if (!model || !task || !out_plan) return fail(WNLQG_ERR_INVALID_ARGUMENT, "NULL argument");
    *out_plan = nullptr;
    const wnlqg_task_desc &t = *task;
    if (t.num_responses < 1 || t.num_responses > WNLQG_MAX_RESPONSES)
        return fail(WNLQG_ERR_INVALID_ARGUMENT, "num_responses must be in 1..8");
    if (!(t.broadening > 0) || !std::isfinite(t.broadening))
        return fail(WNLQG_ERR_INVALID_ARGUMENT, "broadening must be finite and positive");
    if (t.broadening_type != WNLQG_GAUSSIAN && t.broadening_type != WNLQG_LORENTZIAN)
        return fail(WNLQG_ERR_INVALID_ARGUMENT, "Unknown smearing type");
    if (!(t.denominator_regularization >= 0) || !std::isfinite(t.denominator_regularization))
        return fail(WNLQG_ERR_INVALID_ARGUMENT, "denominator_regularization must be finite and >= 0");
    if (!std::isfinite(t.fermi_energy) || !(t.temperature >= 0) || !std::isfinite(t.temperature))
        return fail(WNLQG_ERR_INVALID_ARGUMENT, "fermi_energy and temperature must be finite (temperature >= 0)");
    if (t.num_photon_energies < 0 || (t.num_photon_energies > 0 && !t.photon_energies))
        return fail(WNLQG_ERR_INVALID_ARGUMENT, "photon energies missing");
    if (t.num_photon_energies > 0 && !finite_array(t.photon_energies, (size_t)t.num_photon_energies))
        return fail(WNLQG_ERR_NONFINITE, "photon energies must be finite");
    if (t.precision != WNLQG_PRECISION_FP64 && t.precision != WNLQG_PRECISION_MIXED)
        return fail(WNLQG_ERR_INVALID_ARGUMENT, "unknown precision");
    if (t.band_window_size < -1 || t.band_window_size == 0)
        return fail(WNLQG_ERR_INVALID_ARGUMENT, "band_window_size must be -1 or positive");
    if (t.wannier_center_convention != 0 && t.wannier_center_convention != 1)
        return fail(WNLQG_ERR_INVALID_ARGUMENT, "wannier_center_convention must be 0 (II) or 1 (I)");
    if (t.wannier_center_convention == 1 && model->has_overlap)
        return fail(WNLQG_ERR_UNSUPPORTED, "Convention I with an overlap is not built");
    if (!(std::isfinite(t.spectral_gap_tolerance) && t.spectral_gap_tolerance >= 0))
        return fail(WNLQG_ERR_INVALID_ARGUMENT, "invalid spectral isolation threshold");
    if (t.use_band_selection) {
        // validate_interband_band_selection (CalculationUtils.jl:501-522): two nonempty, disjoint
        // groups inside the orbitals.
        bool any_v = false, any_c = false, overlap = false, outside = false;
        for (int w = 0; w < 4; ++w) {
            any_v |= t.valence_bands[w] != 0;
            any_c |= t.conduction_bands[w] != 0;
            overlap |= (t.valence_bands[w] & t.conduction_bands[w]) != 0;
            for (int bit = 0; bit < 32; ++bit)
                if (32 * w + bit >= model->nw && (((t.valence_bands[w] | t.conduction_bands[w]) >> bit) & 1u)) outside = true;
        }
        if (!any_v || !any_c || outside)
            return fail(WNLQG_ERR_INVALID_ARGUMENT, "band_selection groups must be nonempty and inside the orbitals");
        if (overlap) return fail(WNLQG_ERR_INVALID_ARGUMENT, "band_selection groups must not overlap");
        if (t.band_window_size != -1)
            return fail(WNLQG_ERR_UNSUPPORTED, "band_selection together with a band window is not built");
    }
    WNLQG_CUDA(cudaSetDevice(model->device));

    wnlqg_plan *pl = new wnlqg_plan();
    pl->model = model;
    pl->task = t;
    pl->omegas.assign(t.photon_energies, t.photon_energies + t.num_photon_energies);
    if (t.num_fermi_energies > 0 && t.fermi_energies) pl->mus.assign(t.fermi_energies, t.fermi_energies + t.num_fermi_energies);
    pl->task.photon_energies = pl->omegas.data();
    pl->task.fermi_energies = pl->mus.data();
    pl->nw = model->nw;
    pl->nr = model->nr;
    pl->nn = (int64_t)pl->nw * pl->nw;
    std::memset(&pl->sea, 0, sizeof(pl->sea));
    std::memset(&pl->bcda, 0, sizeof(pl->bcda));
    auto bail = [&](wnlqg_status st) { wnlqg_b200_plan_destroy(pl); return st; };

    // Channels required by the requested components.
    for (int a = 0; a < 3; ++a) { pl->ch_dH[a] = -1; pl->ch_A[a] = -1; }
    for (int a = 0; a < 9; ++a) { pl->ch_ddH[a] = -1; pl->ch_dA[a] = -1; }
    std::vector<Channel> &ch = pl->channels;
    pl->ch_H = add_channel(ch, CH_H, 0, 0);
    auto need_r = [&](int a) { pl->ch_dH[a] = add_channel(ch, CH_DH, a, 0); pl->ch_A[a] = add_channel(ch, CH_A, a, 0); };
    int64_t vc = 0;
    for (int r = 0; r < t.num_responses; ++r) {
        const wnlqg_response_request &q = t.responses[r];
        if (q.num_components < 1 || q.num_components > WNLQG_MAX_COMPONENTS)
            return bail(fail(WNLQG_ERR_INVALID_ARGUMENT, "num_components must be in 1..81"));
        for (int c = 0; c < q.num_components; ++c) {
            const int32_t *x = q.components[c];
            for (int i = 0; i < 4; ++i)
                if (x[i] < 0 || x[i] > 2) return bail(fail(WNLQG_ERR_INVALID_ARGUMENT, "component axis out of range"));
            int a = x[0], b = x[1], cc = x[2];
            if (model->has_overlap && q.kind != WNLQG_SHIFT_CURRENT && q.kind != WNLQG_INJECTION_CURRENT &&
                q.kind != WNLQG_SECOND_HARMONIC)
                return bail(fail(WNLQG_ERR_UNSUPPORTED,
                                 "nonorthogonal models: shift current, injection current and second harmonic generation "
                                 "are built; other responses are not"));
            if (model->has_overlap && q.kind == WNLQG_SECOND_HARMONIC) {
                // Metric SHG preconditions (NonorthogonalMatrixElements.jl:1088-1110).
                if (t.shg_eta_correction)
                    return bail(fail(WNLQG_ERR_INVALID_ARGUMENT, "NONORTHOGONAL_SHG_ETA_CORRECTION_UNSUPPORTED"));
                if (!(std::isfinite(t.denominator_regularization) && t.denominator_regularization > 0))
                    return bail(fail(WNLQG_ERR_INVALID_ARGUMENT, "NONORTHOGONAL_SHG_POSITIVE_GEOMETRY_REQUIRED"));
                pl->metric_shg = true;
            }
            switch (q.kind) {
            case WNLQG_SHIFT_CURRENT: {
                need_r(a); need_r(b); need_r(cc);
                for (auto pd : {std::make_pair(cc, a), std::make_pair(b, a)}) {
                    int pp = pd.first, dd = pd.second;
                    pl->ch_dA[pp * 3 + dd] = add_channel(ch, CH_DA, pp, dd);
                    int hidx = add_channel(ch, CH_DDH, pp, dd);
                    pl->ch_ddH[pp * 3 + dd] = hidx;
                    pl->ch_ddH[dd * 3 + pp] = hidx;
                }
                break;
            }
            case WNLQG_INJECTION_CURRENT:
                pl->ch_dH[a] = add_channel(ch, CH_DH, a, 0);
                need_r(b); need_r(cc);
                break;
            case WNLQG_BERRY_CURVATURE:
                need_r(a); need_r(b);
                pl->ch_dA[b * 3 + a] = add_channel(ch, CH_DA, b, a);
                pl->ch_dA[a * 3 + b] = add_channel(ch, CH_DA, a, b);
                break;
            case WNLQG_QUANTUM_METRIC:
                need_r(a); need_r(b);
                break;
            case WNLQG_INTRINSIC_AHC:
            case WNLQG_BERRY_DIPOLE:
            case WNLQG_LINEAR_TRANSPORT_BERRY:
            case WNLQG_BERRY_DIPOLE_SEA:
                need_r(a); need_r(b);
                pl->ch_dA[b * 3 + a] = add_channel(ch, CH_DA, b, a);
                pl->ch_dA[a * 3 + b] = add_channel(ch, CH_DA, a, b);
                if (q.kind == WNLQG_BERRY_DIPOLE) pl->ch_dH[cc] = add_channel(ch, CH_DH, cc, 0);
                if (q.kind == WNLQG_BERRY_DIPOLE_SEA && t.derivative_backend == 1) {
                    // Jets of orthogonal_bcd_partition_matrices! and of the band derivatives D_a, D_c,
                    // D_ac, D_bc (OrthogonalGeometryDerivatives.jl:24-102, OrthogonalBandDerivatives.jl:123-245).
                    need_r(cc);
                    for (int x : {a, b}) {
                        const int hidx = add_channel(ch, CH_DDH, x, cc);
                        pl->ch_ddH[x * 3 + cc] = pl->ch_ddH[cc * 3 + x] = hidx;
                        pl->ch_dA[x * 3 + cc] = add_channel(ch, CH_DA, x, cc);
                        pl->ch_dA[cc * 3 + x] = add_channel(ch, CH_DA, cc, x);
                    }
                    add_channel(ch, CH_DDA, b, std::min(a, cc) * 3 + std::max(a, cc));
                    add_channel(ch, CH_DDA, a, std::min(b, cc) * 3 + std::max(b, cc));
                }
                break;
            case WNLQG_SECOND_HARMONIC:
                // Every Cartesian channel: the nine cutoff derivatives G^{ab} and both one-band terms.
                for (int u = 0; u < 3; ++u) {
                    need_r(u);
                    for (int v = 0; v < 3; ++v) {
                        pl->ch_dA[u * 3 + v] = add_channel(ch, CH_DA, u, v);
                        const int hidx = add_channel(ch, CH_DDH, u, v);
                        pl->ch_ddH[u * 3 + v] = hidx;
                        pl->ch_ddH[v * 3 + u] = hidx;
                    }
                }
                break;
            case WNLQG_JERK_CURRENT: {
                const int dd = x[3];
                need_r(b); need_r(cc);
                pl->ch_dH[a] = add_channel(ch, CH_DH, a, 0);
                pl->ch_dH[dd] = add_channel(ch, CH_DH, dd, 0);
                const int hidx = add_channel(ch, CH_DDH, a, dd);
                pl->ch_ddH[a * 3 + dd] = hidx;
                pl->ch_ddH[dd * 3 + a] = hidx;
                break;
            }
            default:
                return bail(fail(WNLQG_ERR_UNSUPPORTED, "response kind not supported by this build"));
            }
        }
        if (q.kind == WNLQG_SHIFT_CURRENT || q.kind == WNLQG_INJECTION_CURRENT || q.kind == WNLQG_JERK_CURRENT) {
            if (t.num_photon_energies < 1) return bail(fail(WNLQG_ERR_INVALID_ARGUMENT, "photon energies required"));
            if (q.kind == WNLQG_JERK_CURRENT && !(t.denominator_regularization > 0))
                return bail(fail(WNLQG_ERR_INVALID_ARGUMENT, "third-order matrix width must be finite and positive"));
            vc += (int64_t)q.num_components * t.num_photon_energies;
        } else if (q.kind == WNLQG_SECOND_HARMONIC) {
            // second_harmonic_response! argument checks (SecondHarmonicKernels.jl:129-138).
            if (t.num_photon_energies < 1) return bail(fail(WNLQG_ERR_INVALID_ARGUMENT, "photon energies required"));
            const double eta = t.shg_intermediate_regularization > 0 ? t.shg_intermediate_regularization
                                                                      : t.denominator_regularization;
            if (!(std::isfinite(t.shg_low_frequency_broadening) && t.shg_low_frequency_broadening > 0 &&
                  std::isfinite(eta) && eta > 0))
                return bail(fail(WNLQG_ERR_INVALID_ARGUMENT,
                                 "SHG optical widths and intermediate_regularization must be finite and positive in eV"));
            if (!(std::isfinite(t.degeneracy_threshold) && t.degeneracy_threshold >= 0))
                return bail(fail(WNLQG_ERR_INVALID_ARGUMENT, "SHG degeneracy_threshold must be finite and nonnegative in eV"));
            vc += (int64_t)q.num_components * t.num_photon_energies * 14;
        } else if (q.kind == WNLQG_INTRINSIC_AHC || q.kind == WNLQG_BERRY_DIPOLE ||
                   q.kind == WNLQG_LINEAR_TRANSPORT_BERRY || q.kind == WNLQG_BERRY_DIPOLE_SEA) {
            // intrinsic_hall_fermi_sea is zero-temperature only (IntrinsicHallOccupations.jl:15-16);
            // the finite-temperature Berry channel is the linear transport kind.
            if (q.kind == WNLQG_INTRINSIC_AHC && t.temperature != 0.0)
                return bail(fail(WNLQG_ERR_INVALID_ARGUMENT, "INTRINSIC_HALL_REQUIRES_ZERO_TEMPERATURE"));
            if (q.kind == WNLQG_LINEAR_TRANSPORT_BERRY) {
                // spectral_response_geometry(data) (SpectralResponseGeometry.jl:61-66) and the
                // interband rate of _linear_transport_response (LinearTransportKernels.jl:100-163).
                if (!(std::isfinite(t.denominator_regularization) && t.denominator_regularization > 0))
                    return bail(fail(WNLQG_ERR_INVALID_ARGUMENT,
                                     "spectral position regularization must be finite and positive"));
                if (!(std::isfinite(t.linear_transport_gamma_inter) && t.linear_transport_gamma_inter >= 0))
                    return bail(fail(WNLQG_ERR_INVALID_ARGUMENT, "gamma_inter_ev must be finite and nonnegative"));
            }
            if (t.num_fermi_energies < 1 || !t.fermi_energies)
                return bail(fail(WNLQG_ERR_INVALID_ARGUMENT, "finite nonempty Fermi energy axis required"));
            if (!finite_array(t.fermi_energies, (size_t)t.num_fermi_energies))
                return bail(fail(WNLQG_ERR_INVALID_ARGUMENT, "finite nonempty Fermi energy axis required"));
            if (q.kind == WNLQG_BERRY_DIPOLE && t.temperature == 0.0 && !(t.fermi_surface_broadening > 0))
                return bail(fail(WNLQG_ERR_INVALID_ARGUMENT, "T=0 requires positive eta_fs_ev"));
            if (q.kind == WNLQG_BERRY_DIPOLE_SEA && t.derivative_backend != 0 && t.derivative_backend != 1)
                return bail(fail(WNLQG_ERR_INVALID_ARGUMENT, "derivative_backend must be 0 (finite difference) or 1 (analytic)"));
            if (q.kind == WNLQG_BERRY_DIPOLE_SEA && t.derivative_backend == 1) {
                for (int c = 0; c < q.num_components; ++c) {
                    if (pl->bcda.n_items >= BCDA_MAX_ITEMS)
                        return bail(fail(WNLQG_ERR_UNSUPPORTED, "more than 32 analytic Fermi-sea dipole components in one task"));
                    const int it = pl->bcda.n_items++;
                    pl->bcda.item_a[it] = q.components[c][0];
                    pl->bcda.item_b[it] = q.components[c][1];
                    pl->bcda.item_c[it] = q.components[c][2];
                    pl->bcda.item_out[it] = vc + (int64_t)c * t.num_fermi_energies;
                }
            } else if (q.kind == WNLQG_BERRY_DIPOLE_SEA) {
                if (!(std::isfinite(t.finite_difference_step) && t.finite_difference_step > 0))
                    return bail(fail(WNLQG_ERR_INVALID_ARGUMENT, "finite_difference_step must be finite and positive"));
                // Derivative axes in order of first use and the distinct (a, b) curvature pairs.
                for (int c = 0; c < q.num_components; ++c) {
                    const int32_t *x = q.components[c];
                    int j = 0, pr = 0;
                    while (j < pl->fd_nd && pl->fd_axis[j] != x[2]) ++j;
                    if (j == pl->fd_nd) pl->fd_axis[pl->fd_nd++] = x[2];
                    while (pr < pl->fd_npair && !(pl->fd_pair[pr][0] == x[0] && pl->fd_pair[pr][1] == x[1])) ++pr;
                    if (pr == pl->fd_npair) {
                        pl->fd_pair[pr][0] = x[0];
                        pl->fd_pair[pr][1] = x[1];
                        ++pl->fd_npair;
                    }
                    if (pl->sea.n_items >= SEA_MAX_ITEMS)
                        return bail(fail(WNLQG_ERR_UNSUPPORTED, "more than 96 Fermi-sea dipole components in one task"));
                    const int it = pl->sea.n_items++;
                    pl->sea.item_dir[it] = j;
                    pl->sea.item_pair[it] = pr;
                    pl->sea.item_out[it] = vc + (int64_t)c * t.num_fermi_energies;
                }
            }
            vc += (int64_t)q.num_components * t.num_fermi_energies;
        } else {
            vc += q.num_components;
        }
    }
    pl->vc = vc;
    for (int g = 0; g < 9; ++g) pl->ng_gidx[g] = -1;
    if (model->has_overlap) {
        // Nonorthogonal model: the spectrum uses S(k); the conventional currents take the metric
        // geometry (dH, dS, r on all axes; d2H, d2S, dr per generalized-derivative pair).
        pl->nonorth = true;
        pl->ch_S = add_channel(ch, CH_S, 0, 0);
        if (vc > 0) {
            NonorthParams &q = pl->ng;
            std::memset(&q, 0, sizeof(q));
            for (int a = 0; a < 3; ++a) {
                q.ch_dH[a] = pl->ch_dH[a] = add_channel(ch, CH_DH, a, 0);
                q.ch_dS[a] = add_channel(ch, CH_DS, a, 0);
                q.ch_A[a] = pl->ch_A[a] = add_channel(ch, CH_A, a, 0);
            }
            for (int pd = 0; pd < 9; ++pd) {
                if (pl->ch_dA[pd] < 0) continue;
                const int pp = pd / 3, dd = pd % 3, g = q.npairs++;
                q.pair_p[g] = pp;
                q.pair_d[g] = dd;
                q.ch_dA[g] = pl->ch_dA[pd];
                q.ch_ddH[g] = pl->ch_ddH[pd];
                q.ch_ddS[g] = add_channel(ch, CH_DDS, pp, dd);
                pl->ng_gidx[pd] = g;
            }
            q.eta = t.denominator_regularization;
        }
        if (pl->metric_shg) {
            // Metric SHG: dH, dS, r on every axis and d2H, d2S, dr for every (axis, derivative).
            MetricShgParams &ms = pl->mshg;
            std::memset(&ms, 0, sizeof(ms));
            for (int a = 0; a < 3; ++a) {
                ms.ch_dH[a] = add_channel(ch, CH_DH, a, 0);
                ms.ch_dS[a] = add_channel(ch, CH_DS, a, 0);
                ms.ch_A[a] = add_channel(ch, CH_A, a, 0);
                for (int bb = 0; bb < 3; ++bb) {
                    ms.ch_ddH[a * 3 + bb] = add_channel(ch, CH_DDH, a, bb);
                    ms.ch_ddS[a * 3 + bb] = add_channel(ch, CH_DDS, a, bb);
                    ms.ch_dA[a * 3 + bb] = add_channel(ch, CH_DA, a, bb);
                }
            }
            ms.eta = t.denominator_regularization;
        }
    }
    pl->C = (int)ch.size();

    // Convention I centres (_initialize_wannier_center_scratch!, WannierCenterConventionTransforms.jl:15-56):
    // tau = Re diag A(R = 0), fractional coordinates from the lattice rows.
    int home = -1;
    if (t.wannier_center_convention == 1) {
        for (int r = 0; r < pl->nr; ++r) {
            const int64_t *rv = &model->rvec[3 * (size_t)r];
            if (rv[0] == 0 && rv[1] == 0 && rv[2] == 0) {
                if (home >= 0) return bail(fail(WNLQG_ERR_INVALID_ARGUMENT, "TB model contains more than one R=(0,0,0) block."));
                home = r;
            }
        }
        if (home < 0)
            return bail(fail(WNLQG_ERR_INVALID_ARGUMENT, "Convention_I requires one R=(0,0,0) position block in the TB model."));
        const int nwc = pl->nw;
        pl->tau_cart.assign(3 * (size_t)nwc, 0.0);
        pl->tau_frac.assign(3 * (size_t)nwc, 0.0);
        if (model->has_position)
            for (int i = 0; i < nwc; ++i)
                for (int a = 0; a < 3; ++a) {
                    const double2 v = model->A[((size_t)home * 3 + a) * pl->nn + i + (size_t)nwc * i];
                    if (!std::isfinite(v.x) || !std::isfinite(v.y))
                        return bail(fail(WNLQG_ERR_NONFINITE, "Convention_I Wannier center is non-finite"));
                    if (std::fabs(v.y) > 1.0e-10)
                        return bail(fail(WNLQG_ERR_INVALID_ARGUMENT, "Convention_I Wannier center has an imaginary part"));
                    pl->tau_cart[a * nwc + i] = v.x;
                }
        // tau_cart[j] = sum_i tau_frac_i lattice[i + 3 j]: solve the 3 x 3 system (Cramer).
        const double *L = model->lattice;
        auto M = [&](int i, int j) { return L[i + 3 * j]; };   // row i = lattice vector i
        const double det = M(0, 0) * (M(1, 1) * M(2, 2) - M(2, 1) * M(1, 2)) - M(1, 0) * (M(0, 1) * M(2, 2) - M(2, 1) * M(0, 2)) +
                           M(2, 0) * (M(0, 1) * M(1, 2) - M(1, 1) * M(0, 2));
        if (!(std::fabs(det) > 0)) return bail(fail(WNLQG_ERR_INVALID_ARGUMENT, "singular lattice"));
        for (int i = 0; i < nwc; ++i) {
            const double b[3] = {pl->tau_cart[i], pl->tau_cart[nwc + i], pl->tau_cart[2 * nwc + i]};
            // Unknown x with sum_r x_r M(r, j) = b_j: columns of the system matrix are M(r, :).
            auto solve_col = [&](int c) {
                double A3[3][3];
                for (int j = 0; j < 3; ++j)
                    for (int r = 0; r < 3; ++r) A3[j][r] = r == c ? b[j] : M(r, j);
                return (A3[0][0] * (A3[1][1] * A3[2][2] - A3[1][2] * A3[2][1]) -
                        A3[0][1] * (A3[1][0] * A3[2][2] - A3[1][2] * A3[2][0]) +
                        A3[0][2] * (A3[1][0] * A3[2][1] - A3[1][1] * A3[2][0])) / det;
            };
            for (int c = 0; c < 3; ++c) pl->tau_frac[c * nwc + i] = solve_col(c);
        }
        pl->conv1 = true;
    }

    // Real-space tiles T[R][c][i + nw j] (prepare_hamiltonian_real_space!,
    // HamiltonianMatrixElements.jl:92-177; prepare_position_real_space!, PositionMatrixElements.jl:8-84;
    // Convention II displacements).
    const int nw = pl->nw, nr = pl->nr;
    const int64_t nn = pl->nn;
    std::vector<double2> tiles((size_t)nr * pl->C * nn);
    for (int r = 0; r < nr; ++r) {
        double rc[3];
        const int64_t *rv = &model->rvec[3 * (size_t)r];
        for (int j = 0; j < 3; ++j)
            rc[j] = (double)rv[0] * model->lattice[0 + 3 * j] + (double)rv[1] * model->lattice[1 + 3 * j] +
                    (double)rv[2] * model->lattice[2 + 3 * j];
        for (int c = 0; c < pl->C; ++c) {
            const Channel &cc = ch[c];
            double2 *dst = &tiles[((size_t)r * pl->C + c) * nn];
            for (int64_t e = 0; e < nn; ++e) {
                double2 h = model->H[(size_t)r * nn + e];
                double2 v = make_double2(0.0, 0.0);
                // Convention I: displacement R + tau_j - tau_i (_convention_displacement_component,
                // WannierCenterConventionTransforms.jl:85-96) and the centred home-cell connection
                // A - tau (_convention_position_value, :99-113).
                const int ei = (int)(e % nw), ej = (int)(e / nw);
                double dsp[3] = {rc[0], rc[1], rc[2]};
                if (pl->conv1)
                    for (int x = 0; x < 3; ++x) dsp[x] += pl->tau_cart[x * nw + ej] - pl->tau_cart[x * nw + ei];
                auto position = [&](int p) {
                    double2 a = model->A[((size_t)r * 3 + p) * nn + e];
                    if (pl->conv1 && r == home && ei == ej) a.x -= pl->tau_cart[p * nw + ei];
                    return a;
                };
                switch (cc.op) {
                case CH_H: v = h; break;
                case CH_DH: v = cmuli(cscale(h, dsp[cc.p])); break;
                case CH_DDH: v = cscale(h, -dsp[cc.p] * dsp[cc.d]); break;
                case CH_A:
                    if (model->has_position) v = position(cc.p);
                    break;
                case CH_DA:
                    if (model->has_position) v = cmuli(cscale(position(cc.p), dsp[cc.d]));
                    break;
                case CH_S:
                    v = model->S[(size_t)r * nn + e];
                    break;
                case CH_DS:
                    v = cmuli(cscale(model->S[(size_t)r * nn + e], rc[cc.p]));
                    break;
                case CH_DDS:
                    v = cscale(model->S[(size_t)r * nn + e], -rc[cc.p] * rc[cc.d]);
                    break;
                case CH_DDA:
                    if (model->has_position) v = cscale(position(cc.p), -dsp[cc.d / 3] * dsp[cc.d % 3]);
                    break;
                }
                dst[e] = v;
            }
        }
    }

    int sm_count = 148;
    int dev = model->device;
    cudaDeviceGetAttribute(&sm_count, cudaDevAttrMultiProcessorCount, dev);
    pl->sm_count = sm_count;
    int smem_optin = 0;
    cudaDeviceGetAttribute(&smem_optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    if (smem_optin <= 0) smem_optin = 48 * 1024;

    if (max_batch <= 0) {
        int64_t per_k = (int64_t)pl->C * nn * 16 + (int64_t)nr * 16 + nn * 16 + nw * 8 + vc * 16;
        if (pl->metric_shg) per_k += MetricShgWs::src_entries(nw) * 16 + MetricShgWs::diag_entries(nw) * 8;
        if (pl->nonorth) per_k += 2 * nn * 16 + nn * 8;
        per_k += (int64_t)2 * pl->fd_nd * pl->fd_npair * nw * 8 + (pl->fd_nd > 0 ? 24 : 0);
        // About 4 GiB of batch workspace (HBM is 180 GB): long runs of neighbouring k-points per
        // CTA for the warm-started eigensolver and few batches per call.
        max_batch = std::max<int64_t>(256, std::min<int64_t>(1 << 20, ((int64_t)1 << 32) / per_k));
        max_batch = (max_batch / 64) * 64;
    }
    pl->max_batch = max_batch;
    WNLQG_CUDA(cudaStreamCreateWithFlags(&pl->stream, cudaStreamNonBlocking));
    auto alloc = [&](void **ptr, size_t bytes) -> wnlqg_status {
        cudaError_t e = cudaMalloc(ptr, std::max<size_t>(bytes, 16));
        if (e != cudaSuccess) {
            cudaGetLastError();
            return fail(WNLQG_ERR_OUT_OF_MEMORY, std::string("cudaMalloc of ") + std::to_string(bytes) + " bytes failed");
        }
        return WNLQG_OK;
    };
    wnlqg_status st;
    if ((st = alloc((void **)&pl->d_tiles, tiles.size() * sizeof(double2))) != WNLQG_OK) return bail(st);
    if ((st = alloc((void **)&pl->d_phase, (size_t)max_batch * nr * sizeof(double2))) != WNLQG_OK) return bail(st);
    if ((st = alloc((void **)&pl->d_xw, (size_t)max_batch * pl->C * nn * sizeof(double2))) != WNLQG_OK) return bail(st);
    if ((st = alloc((void **)&pl->d_U, (size_t)max_batch * nn * sizeof(double2))) != WNLQG_OK) return bail(st);
    if ((st = alloc((void **)&pl->d_E, (size_t)max_batch * nw * sizeof(double))) != WNLQG_OK) return bail(st);
    if ((st = alloc((void **)&pl->d_kpts, (size_t)max_batch * 3 * sizeof(double))) != WNLQG_OK) return bail(st);
    if ((st = alloc((void **)&pl->d_weights, (size_t)max_batch * sizeof(double))) != WNLQG_OK) return bail(st);
    if ((st = alloc((void **)&pl->d_kidx, (size_t)max_batch * sizeof(int64_t))) != WNLQG_OK) return bail(st);
    if ((st = alloc((void **)&pl->d_status, (size_t)max_batch * sizeof(int))) != WNLQG_OK) return bail(st);
    if (pl->bcda.n_items > 0) {
        // Analytic Fermi-sea dipole: channel indices, two CTAs per SM, BCDA_SLOTS matrices per CTA.
        BcdaParams &q = pl->bcda;
        q.nw = nw;
        q.ld = nw + 1;
        q.xw_stride = (int64_t)pl->C * nn;
        for (int x = 0; x < 3; ++x) {
            q.ch_dH[x] = find_channel(ch, CH_DH, x, 0);
            q.ch_A[x] = find_channel(ch, CH_A, x, 0);
            for (int y = 0; y < 3; ++y) {
                q.ch_ddH[x * 3 + y] = find_channel(ch, CH_DDH, std::min(x, y), std::max(x, y));
                q.ch_dA[x * 3 + y] = find_channel(ch, CH_DA, x, y);
                for (int z = 0; z < 3; ++z) q.ch_ddA[x * 9 + y * 3 + z] = find_channel(ch, CH_DDA, x, std::min(y, z) * 3 + std::max(y, z));
            }
        }
        q.nmu = (int)t.num_fermi_energies;
        q.temperature = t.temperature;
        q.vc = vc;
        q.gscratch_stride = (int64_t)(((size_t)BCDA_SLOTS * nw * (nw + 1) * sizeof(double2) + 255) & ~(size_t)255);
        pl->bcda_grid = 2 * sm_count;
        if ((st = alloc((void **)&pl->d_bcda_scratch, (size_t)pl->bcda_grid * q.gscratch_stride)) != WNLQG_OK) return bail(st);
        q.gscratch = pl->d_bcda_scratch;
    }
    if (pl->fd_nd > 0) {
        // Fractional image lattice * (h e_c) / 2 pi of each Cartesian step (finite_difference_step_matrix,
        // Core/Coordinates.jl:33-44; lattice element (i, c) at i + 3 c).
        for (int j = 0; j < pl->fd_nd; ++j)
            for (int i = 0; i < 3; ++i)
                pl->fd_delta[j][i] = model->lattice[i + 3 * pl->fd_axis[j]] * t.finite_difference_step / (2.0 * WNLQG_PI);
        if ((st = alloc((void **)&pl->d_fd_k, (size_t)max_batch * 3 * sizeof(double))) != WNLQG_OK) return bail(st);
        if ((st = alloc((void **)&pl->d_fd_curv, (size_t)max_batch * 2 * pl->fd_nd * pl->fd_npair * nw * sizeof(double))) !=
            WNLQG_OK)
            return bail(st);
        SeaParams &q = pl->sea;
        q.nw = nw;
        q.curv = pl->d_fd_curv;
        q.nd = pl->fd_nd;
        q.npair = pl->fd_npair;
        q.nmu = (int)t.num_fermi_energies;
        q.temperature = t.temperature;
        q.two_h = 2.0 * t.finite_difference_step;
        q.vc = vc;
    }
    {
        // Isolation contract: the Berry dipole needs every pair split by more than
        // degeneracy_threshold (BerryMultipoleGeometry.jl:81); eta = 0 geometry by more than
        // spectral_gap_tolerance (PositionMatrixElements.jl:447-452); the linear transport Berry
        // channel resolves its spectral blocks with spectral_gap_tolerance.
        bool dipole = false, exact = false, blocks = false;
        for (int r = 0; r < t.num_responses; ++r) {
            const int kind = t.responses[r].kind;
            dipole |= kind == WNLQG_BERRY_DIPOLE || kind == WNLQG_BERRY_DIPOLE_SEA;
            exact |= t.denominator_regularization == 0.0 &&
                     (kind == WNLQG_SHIFT_CURRENT || kind == WNLQG_INJECTION_CURRENT || kind == WNLQG_BERRY_CURVATURE ||
                      kind == WNLQG_QUANTUM_METRIC || kind == WNLQG_BERRY_DIPOLE || kind == WNLQG_BERRY_DIPOLE_SEA);
            blocks |= kind == WNLQG_LINEAR_TRANSPORT_BERRY;
        }
        if (dipole && !(std::isfinite(t.degeneracy_threshold) && t.degeneracy_threshold >= 0))
            return bail(fail(WNLQG_ERR_INVALID_ARGUMENT, "invalid spectral isolation threshold"));
        if (dipole || exact) {
            pl->iso_mode = ISO_ALL_PAIRS;
            pl->iso_tol = std::max(dipole ? t.degeneracy_threshold : 0.0, exact ? t.spectral_gap_tolerance : 0.0);
        } else if (blocks) {
            pl->iso_mode = ISO_SPECTRAL_BLOCKS;
            pl->iso_tol = t.spectral_gap_tolerance;
        }
        if (pl->iso_mode >= 0) {
            if (max_batch > ((int64_t)1 << ISO_LOCAL_BITS))
                return bail(fail(WNLQG_ERR_UNSUPPORTED, "max_batch above 2^24 with a spectral isolation check"));
            if ((st = alloc((void **)&pl->d_iso_key, sizeof(unsigned long long))) != WNLQG_OK) return bail(st);
            if ((st = alloc((void **)&pl->d_iso_rec, sizeof(IsoRecord))) != WNLQG_OK) return bail(st);
            WNLQG_CUDA(cudaMemset(pl->d_iso_key, 0xFF, sizeof(unsigned long long)));
            WNLQG_CUDA(cudaMemset(pl->d_iso_rec, 0xFF, sizeof(IsoRecord)));   // row -1: no record
        }
    }
    if (pl->nonorth && vc > 0) {
        NonorthParams &q = pl->ng;
        q.nw = nw;
        q.ld = nw + 1;
        q.xw_stride = (int64_t)pl->C * nn;
        q.ws_stride = (NonorthWs::bytes(nw) + 255) & ~(int64_t)255;
        // Two CTAs per SM over the per-CTA global working sets (measured at 64 orbitals: the
        // L2-resident grid takes twice as long).
        pl->ng_grid_alloc = 2 * sm_count;
        pl->ng_grid = 2 * sm_count;
        if (const char *g = std::getenv("WNLQG_B200_NG_GRID"))
            pl->ng_grid = std::max(1, std::min(pl->ng_grid_alloc, std::atoi(g)));
        if ((st = alloc((void **)&pl->d_ng_r, (size_t)max_batch * 3 * nn * sizeof(double2))) != WNLQG_OK) return bail(st);
        if ((st = alloc((void **)&pl->d_ng_v, (size_t)max_batch * 3 * nw * sizeof(double))) != WNLQG_OK) return bail(st);
        if ((st = alloc((void **)&pl->d_ng_G, (size_t)max_batch * std::max(1, q.npairs) * nn * sizeof(double2))) != WNLQG_OK)
            return bail(st);
        if ((st = alloc((void **)&pl->d_ng_ws, (size_t)std::max(pl->ng_grid, pl->ng_grid_alloc) * q.ws_stride)) != WNLQG_OK)
            return bail(st);
        q.r_out = pl->d_ng_r;
        q.v_out = pl->d_ng_v;
        q.g_out = pl->d_ng_G;
        q.ws = pl->d_ng_ws;
    }
    if (pl->metric_shg) {
        MetricShgParams &ms = pl->mshg;
        ms.nw = nw;
        ms.ld = nw + 1;
        ms.xw_stride = (int64_t)pl->C * nn;
        ms.ws_stride = (MetricShgWs::bytes(nw) + 255) & ~(int64_t)255;
        // Metric inputs: up to four CTAs per SM over the per-CTA global working sets; two by default
        // (measured at 64 orbitals), the autotuner may change it.
        pl->mshg_grid_alloc = 4 * sm_count;
        pl->mshg_grid = 2 * sm_count;
        if (const char *g = std::getenv("WNLQG_B200_MSHG_GRID"))
            pl->mshg_grid = std::max(1, std::min(pl->mshg_grid_alloc, std::atoi(g)));
        if ((st = alloc((void **)&pl->d_mshg_src, (size_t)max_batch * MetricShgWs::src_entries(nw) * sizeof(double2))) != WNLQG_OK)
            return bail(st);
        if ((st = alloc((void **)&pl->d_mshg_diag, (size_t)max_batch * MetricShgWs::diag_entries(nw) * sizeof(double))) != WNLQG_OK)
            return bail(st);
        if ((st = alloc((void **)&pl->d_mshg_ws, (size_t)pl->mshg_grid_alloc * ms.ws_stride)) != WNLQG_OK) return bail(st);
        ms.src = pl->d_mshg_src;
        ms.diag = pl->d_mshg_diag;
        ms.ws = pl->d_mshg_ws;
    }
    if ((st = alloc((void **)&pl->d_points, (size_t)max_batch * vc * sizeof(double2))) != WNLQG_OK) return bail(st);
    if ((st = alloc((void **)&pl->d_out, (size_t)vc * sizeof(double2))) != WNLQG_OK) return bail(st);
    if ((st = alloc((void **)&pl->d_omegas, std::max<size_t>(1, pl->omegas.size()) * sizeof(double))) != WNLQG_OK) return bail(st);
    if ((st = alloc((void **)&pl->d_mus, std::max<size_t>(1, pl->mus.size()) * sizeof(double))) != WNLQG_OK) return bail(st);
    if (!pl->mus.empty())
        WNLQG_CUDA(cudaMemcpy(pl->d_mus, pl->mus.data(), pl->mus.size() * sizeof(double), cudaMemcpyHostToDevice));
    WNLQG_CUDA(cudaMemcpy(pl->d_tiles, tiles.data(), tiles.size() * sizeof(double2), cudaMemcpyHostToDevice));
    if (!pl->omegas.empty())
        WNLQG_CUDA(cudaMemcpy(pl->d_omegas, pl->omegas.data(), pl->omegas.size() * sizeof(double), cudaMemcpyHostToDevice));

    // Group the R-vectors for the staged mesh contraction.
    {
        std::vector<std::pair<std::pair<int64_t, int64_t>, int>> keyed;
        for (int r = 0; r < nr; ++r) keyed.push_back({{model->rvec[3 * r], model->rvec[3 * r + 1]}, r});
        std::stable_sort(keyed.begin(), keyed.end(),
                         [](const auto &x, const auto &y) { return x.first < y.first; });
        std::vector<int> q12_start, q12_ridx, q12_r2, q12_r1;
        for (size_t i = 0; i < keyed.size(); ++i) {
            if (i == 0 || keyed[i].first != keyed[i - 1].first) {
                q12_start.push_back((int)i);
                q12_r1.push_back((int)keyed[i].first.first);
                q12_r2.push_back((int)keyed[i].first.second);
            }
            q12_ridx.push_back(keyed[i].second);
        }
        const int P12 = (int)q12_r2.size();
        q12_start.push_back(nr);
        std::vector<int> q1_start, q1_q12, q1_r1;
        for (int q = 0; q < P12; ++q) {   // q12 are sorted by (r1, r2): r1 groups are contiguous
            if (q == 0 || q12_r1[q] != q12_r1[q - 1]) {
                q1_start.push_back(q);
                q1_r1.push_back(q12_r1[q]);
            }
            q1_q12.push_back(q);
        }
        const int P1 = (int)q1_r1.size();
        q1_start.push_back(P12);
        std::vector<int> packed;
        packed.insert(packed.end(), q12_start.begin(), q12_start.end());
        packed.insert(packed.end(), q12_ridx.begin(), q12_ridx.end());
        packed.insert(packed.end(), q12_r2.begin(), q12_r2.end());
        packed.insert(packed.end(), q1_start.begin(), q1_start.end());
        packed.insert(packed.end(), q1_q12.begin(), q1_q12.end());
        packed.insert(packed.end(), q1_r1.begin(), q1_r1.end());
        if ((st = alloc((void **)&pl->d_groups, packed.size() * sizeof(int))) != WNLQG_OK) return bail(st);
        WNLQG_CUDA(cudaMemcpy(pl->d_groups, packed.data(), packed.size() * sizeof(int), cudaMemcpyHostToDevice));
        pl->P12 = P12;
        pl->P1 = P1;
        int *base = pl->d_groups;
        pl->groups.P12 = P12;
        pl->groups.P1 = P1;
        pl->groups.q12_start = base; base += P12 + 1;
        pl->groups.q12_ridx = base; base += nr;
        pl->groups.q12_r2 = base; base += P12;
        pl->groups.q1_start = base; base += P1 + 1;
        pl->groups.q1_q12 = base; base += P12;
        pl->groups.q1_r1 = base;
    }
    if (pl->fd_nd > 0 && pl->P1 <= STAGED_MAX_P1 &&
        2 * (size_t)pl->fd_nd * tiles.size() * sizeof(double2) <= ((size_t)4 << 30)) {
        // Shifted tile sets of the finite-difference stencil on meshes: T_R exp(2 pi i s delta_j . R).
        const size_t per = tiles.size();
        if ((st = alloc((void **)&pl->d_fd_tiles, 2 * (size_t)pl->fd_nd * per * sizeof(double2))) != WNLQG_OK) return bail(st);
        std::vector<double2> shifted(per);
        const size_t per_r = (size_t)pl->C * nn;
        for (int j = 0; j < pl->fd_nd; ++j)
            for (int sgn = 0; sgn < 2; ++sgn) {
                const double s = sgn == 0 ? 1.0 : -1.0;
                for (int r = 0; r < nr; ++r) {
                    const int64_t *rv = &model->rvec[3 * (size_t)r];
                    const double phase = 2.0 * WNLQG_PI * s *
                                         (pl->fd_delta[j][0] * (double)rv[0] + pl->fd_delta[j][1] * (double)rv[1] +
                                          pl->fd_delta[j][2] * (double)rv[2]);
                    const double2 f = make_double2(std::cos(phase), std::sin(phase));
                    for (size_t e = 0; e < per_r; ++e) shifted[r * per_r + e] = cmul(tiles[r * per_r + e], f);
                }
                WNLQG_CUDA(cudaMemcpy(pl->d_fd_tiles + (size_t)(2 * j + sgn) * per, shifted.data(), per * sizeof(double2),
                                      cudaMemcpyHostToDevice));
            }
    }

    // Arbitrary k-point batches are put in Morton order so that the FP32 eigensolver stage can
    // warm-start along them (WNLQG_B200_POINT_ORDER=0 keeps the caller's order and cold starts).
    {
        const char *wm = std::getenv("WNLQG_B200_WARM_START");
        pl->warm_mode = (wm && wm[0] == '0') ? 0 : 1;
        const char *rw = std::getenv("WNLQG_B200_RESPONSE_WIDE");
        pl->resp_wide = rw && rw[0] == '1';
    }
    auto alloc_ordering = [&]() -> wnlqg_status {
        const char *ord = std::getenv("WNLQG_B200_POINT_ORDER");
        if ((ord && ord[0] == '0') || max_batch >= ((int64_t)1 << 31)) return WNLQG_OK;
        size_t tmp = 0;
        cudaError_t ce = cub::DeviceRadixSort::SortPairs(nullptr, tmp, (const uint32_t *)nullptr, (uint32_t *)nullptr,
                                                         (const int *)nullptr, (int *)nullptr, (int)max_batch, 0, 30);
        if (ce != cudaSuccess) return fail(WNLQG_ERR_CUDA, std::string("radix sort sizing: ") + cudaGetErrorString(ce));
        wnlqg_status s2;
        if ((s2 = alloc((void **)&pl->d_okeys, 2 * (size_t)max_batch * sizeof(uint32_t))) != WNLQG_OK) return s2;
        if ((s2 = alloc((void **)&pl->d_operm, 2 * (size_t)max_batch * sizeof(int))) != WNLQG_OK) return s2;
        if ((s2 = alloc((void **)&pl->d_ok, (size_t)max_batch * 3 * sizeof(double))) != WNLQG_OK) return s2;
        if ((s2 = alloc((void **)&pl->d_ow, (size_t)max_batch * sizeof(double))) != WNLQG_OK) return s2;
        if ((s2 = alloc(&pl->d_osort_tmp, tmp)) != WNLQG_OK) return s2;
        pl->osort_bytes = std::max<size_t>(tmp, 16);
        pl->order_points = true;
        return WNLQG_OK;
    };
    pl->eigh_threads = eigh_block_threads(nw);
    // Up to 32 orbitals the warp eigensolvers: on the FP64 path one FP64 kernel up to 16 orbitals and
    // the one-sided FP32 stage with the FP64 refinement above, on the mixed path the two-sided FP32
    // stage with its refinement.  WNLQG_B200_CTA_EIGH=1 keeps the FP64 CTA Jacobi on the FP64 path.
    {
        const char *cta = std::getenv("WNLQG_B200_CTA_EIGH");
        const bool cta_fp64 = cta && cta[0] == '1' && t.precision != WNLQG_PRECISION_MIXED;
        // Nonorthogonal models reduce to C = L^-1 H L^-H in FP64 and then take the orthogonal stages of
        // their precision (WNLQG_B200_GEN_MIXED=0, and WNLQG_B200_CTA_EIGH=1 on the FP64 path, keep the
        // FP64 generalised Jacobi: 64 orbitals, 1024 points, 14.0 ms against 4.8 for
        // the four kernels).
        const char *gm = std::getenv("WNLQG_B200_GEN_MIXED");
        pl->gen_mixed = pl->nonorth && !cta_fp64 && !(gm && gm[0] == '0');
        const bool orth_stages = !pl->nonorth || pl->gen_mixed;
        pl->warp_eigh = orth_stages && nw <= 32 && !cta_fp64;
        pl->f32_team = pl->warp_eigh && t.precision == WNLQG_PRECISION_MIXED;
        pl->small_f64 = pl->warp_eigh && nw <= 16 && t.precision != WNLQG_PRECISION_MIXED;
        // Above 32 orbitals the CTA stages: FP32 one-sided (mixed path: two-sided) and FP64 refinement.
        pl->cta_mixed = orth_stages && nw > 32 && !cta_fp64;
    }
    if (pl->nonorth && !pl->gen_mixed) {
        pl->eigh_threads = std::max(pl->eigh_threads, ((nw + (nw & 1)) / 2 + 31) / 32 * 32);
        pl->eigh_smem = GenEighSmem::bytes(nw);
    } else if (pl->warp_eigh) {
        const int np = nw + (nw & 1);
        // Above 16 orbitals four warps share a matrix (128-thread teams); WNLQG_B200_EIGH_TEAM=32,
        // 64 or 128 overrides the choice.
        pl->eigh_team = nw > 16 ? 128 : 32;
        if (const char *tm = std::getenv("WNLQG_B200_EIGH_TEAM")) {
            if (std::string(tm) == "32") pl->eigh_team = 32;
            else if (std::string(tm) == "64") pl->eigh_team = 64;
            else if (std::string(tm) == "128") pl->eigh_team = 128;
        }
        pl->eigh_smem = (pl->eigh_team == 32 ? 4 : 1) * WarpJacobiSmem::per_team(nw);
        pl->refine_smem = (pl->eigh_team == 32 ? 2 : 1) * WarpRefineSmem::per_team(nw);
        {
            // Off-diagonal pair blocks of the team Jacobi: w = k2 (k2 - 1) / 2 + k1, k1 < k2 < 16.
            unsigned char off[120][2];
            for (int k2 = 1, w = 0; k2 < 16; ++k2)
                for (int k1 = 0; k1 < k2; ++k1, ++w) { off[w][0] = (unsigned char)k1; off[w][1] = (unsigned char)k2; }
            cudaError_t et = cudaMemcpyToSymbol(c_jacobi_offdiag, off, sizeof(off));
            if (et != cudaSuccess) return bail(fail(WNLQG_ERR_CUDA, std::string("cudaMemcpyToSymbol: ") + cudaGetErrorString(et)));
            cudaError_t ea = cudaSuccess;
            if (pl->small_f64) ea = allow_dynamic_smem(reg_f64_kernel(np).fn, smem_optin);
            else if (!pl->f32_team) ea = allow_dynamic_smem(onesided_kernel(np).fn, smem_optin);
            if (ea == cudaSuccess) ea = allow_dynamic_smem((const void *)jacobi_f32_team_kernel<32>, smem_optin);
            if (ea == cudaSuccess) ea = allow_dynamic_smem((const void *)jacobi_f32_team_kernel<64>, smem_optin);
            if (ea == cudaSuccess) ea = allow_dynamic_smem((const void *)jacobi_f32_team_kernel<128>, smem_optin);
            if (ea != cudaSuccess) return bail(fail(WNLQG_ERR_CUDA, std::string("cudaFuncSetAttribute: ") + cudaGetErrorString(ea)));
        }
        // Both stages need blockDim >= np/2 (pairs) and 8 * blockDim >= np^2 (register-staged products).
        pl->refine_threads = std::max(32, std::min(256, ((np * np / 8 + 31) / 32) * 32));
        pl->refine_threads = std::max(pl->refine_threads, ((np / 2 + 31) / 32) * 32);
        pl->eigh_threads = pl->refine_threads;
        // Point ordering and the FP32 vectors serve the warm-started first stage.
        if (!pl->small_f64) {
            if ((st = alloc((void **)&pl->d_V32, (size_t)max_batch * np * np * sizeof(float2))) != WNLQG_OK) return bail(st);
            if ((st = alloc_ordering()) != WNLQG_OK) return bail(st);
        }
        cudaError_t e = allow_dynamic_smem((const void *)eigh_refine_f64_team_kernel<32>, smem_optin);
        if (e == cudaSuccess) e = allow_dynamic_smem((const void *)eigh_refine_f64_team_kernel<64>, smem_optin);
        if (e == cudaSuccess) e = allow_dynamic_smem((const void *)eigh_refine_f64_team_kernel<128>, smem_optin);
        if (e != cudaSuccess) return bail(fail(WNLQG_ERR_CUDA, std::string("cudaFuncSetAttribute: ") + cudaGetErrorString(e)));
    } else if (pl->cta_mixed) {
        // Above 32 orbitals: FP32 CTA Jacobi (256 threads) and FP64 CTA refinement (512 threads),
        // each in shared memory when it fits beside the kernel's static shared memory, else in a
        // per-CTA global working set (one scratch, one grid, the larger stride).
        const int np = nw + (nw & 1);
        pl->eigh_smem = EighSmem::bytes(nw, sizeof(float2));
        pl->refine_smem = RefineCtaSmem::bytes(nw);
        cudaFuncAttributes fa1, fa2;
        cudaError_t fe = cudaFuncGetAttributes(&fa1, (const void *)jacobi_f32_cta_kernel<false>);
        if (fe == cudaSuccess) fe = cudaFuncGetAttributes(&fa2, (const void *)eigh_refine_f64_cta_kernel<false>);
        if (fe != cudaSuccess) return bail(fail(WNLQG_ERR_CUDA, std::string("cudaFuncGetAttributes: ") + cudaGetErrorString(fe)));
        pl->cta_gw1 = pl->eigh_smem + fa1.sharedSizeBytes > (size_t)smem_optin;
        if (t.precision != WNLQG_PRECISION_MIXED) {
            pl->cta_gw1 = false;   // the one-sided stage always fits shared memory
            pl->eigh_smem = OsCtaSmem::bytes(np);
        }
        pl->cta_gw2 = pl->refine_smem + fa2.sharedSizeBytes > (size_t)smem_optin;
        // 256-thread refinement blocks when two fit an SM (shared memory and registers), else 512.
        pl->refine_cta_threads =
            (!pl->cta_gw2 && 2 * (pl->refine_smem + fa2.sharedSizeBytes) <= (size_t)smem_optin) ? 256 : 512;
        if ((st = alloc((void **)&pl->d_V32, (size_t)max_batch * np * np * sizeof(float2))) != WNLQG_OK) return bail(st);
        if ((st = alloc_ordering()) != WNLQG_OK) return bail(st);
        if (pl->cta_gw1 || pl->cta_gw2) {
            const size_t need = std::max(pl->cta_gw1 ? pl->eigh_smem : 0, pl->cta_gw2 ? pl->refine_smem : 0);
            pl->eigh_scratch_stride = (int64_t)((need + 255) & ~(size_t)255);
            pl->eigh_grid = l2_resident_grid(4 * sm_count, pl->eigh_scratch_stride, sm_count);
            pl->eigh_grid_l2 = pl->eigh_grid;
            pl->eigh_grid_alloc = std::max(pl->eigh_grid, 2 * sm_count);
            pl->eigh_grid = 2 * sm_count;   // measured faster than the L2-resident grid; tunable
            if ((st = alloc((void **)&pl->d_eigh_scratch, (size_t)pl->eigh_grid_alloc * pl->eigh_scratch_stride)) != WNLQG_OK)
                return bail(st);
        }
        cudaError_t e = cudaSuccess;
        if (t.precision != WNLQG_PRECISION_MIXED) e = allow_dynamic_smem(onesided_cta_fn(np), smem_optin);
        else if (!pl->cta_gw1) e = allow_dynamic_smem((const void *)jacobi_f32_cta_kernel<false>, smem_optin);
        if (e == cudaSuccess && !pl->cta_gw2) e = allow_dynamic_smem((const void *)eigh_refine_f64_cta_kernel<false>, smem_optin);
        if (e != cudaSuccess) return bail(fail(WNLQG_ERR_CUDA, std::string("cudaFuncSetAttribute: ") + cudaGetErrorString(e)));
    } else {
        // FP64 CTA Jacobi (WNLQG_B200_CTA_EIGH=1 on the FP64 path).
        pl->eigh_smem = EighSmem::bytes(nw, sizeof(double2));
    }
    if (!pl->warp_eigh && !pl->cta_mixed) {
        // CTA eigensolvers keep A, V (and the Cholesky factor) in shared memory when they fit
        // beside the kernel's static shared memory, else in a per-CTA global working set (large nw).
        const void *cta_fn = pl->nonorth ? (const void *)generalized_eigh_kernel<false> : (const void *)jacobi_eigh_kernel<double, false>;
        cudaFuncAttributes fa;
        cudaError_t fe = cudaFuncGetAttributes(&fa, cta_fn);
        if (fe != cudaSuccess) return bail(fail(WNLQG_ERR_CUDA, std::string("cudaFuncGetAttributes: ") + cudaGetErrorString(fe)));
        if (pl->eigh_smem + fa.sharedSizeBytes > (size_t)smem_optin) {
            pl->eigh_scratch_stride = (int64_t)((pl->eigh_smem + 255) & ~(size_t)255);
            pl->eigh_grid = l2_resident_grid(4 * sm_count, pl->eigh_scratch_stride, sm_count);
            pl->eigh_grid_l2 = pl->eigh_grid;
            pl->eigh_grid_alloc = std::max(pl->eigh_grid, 2 * sm_count);
            pl->eigh_grid = 2 * sm_count;   // measured faster than the L2-resident grid; tunable
            if ((st = alloc((void **)&pl->d_eigh_scratch, (size_t)pl->eigh_grid_alloc * pl->eigh_scratch_stride)) != WNLQG_OK)
                return bail(st);
            pl->eigh_smem = 0;
        } else {
            cudaError_t e = allow_dynamic_smem(cta_fn, smem_optin);
            if (e != cudaSuccess) return bail(fail(WNLQG_ERR_CUDA, std::string("cudaFuncSetAttribute: ") + cudaGetErrorString(e)));
        }
    }
    if (pl->gen_mixed) {
        if ((st = alloc((void **)&pl->d_gC, (size_t)max_batch * nn * sizeof(double2))) != WNLQG_OK) return bail(st);
        if ((st = alloc((void **)&pl->d_gL, (size_t)max_batch * nn * sizeof(double2))) != WNLQG_OK) return bail(st);
        pl->gred_smem = GenReduceSmem::bytes(nw);
        cudaFuncAttributes fa;
        cudaError_t fe = cudaFuncGetAttributes(&fa, (const void *)cholesky_reduce_kernel<false>);
        if (fe != cudaSuccess) return bail(fail(WNLQG_ERR_CUDA, std::string("cudaFuncGetAttributes: ") + cudaGetErrorString(fe)));
        if (pl->gred_smem + fa.sharedSizeBytes > (size_t)smem_optin) {
            pl->gred_gw = true;
            pl->gred_stride = (int64_t)((pl->gred_smem + 255) & ~(size_t)255);
            pl->gred_grid = l2_resident_grid(4 * sm_count, pl->gred_stride, sm_count);
            if ((st = alloc((void **)&pl->d_gred_scratch, (size_t)pl->gred_grid * pl->gred_stride)) != WNLQG_OK)
                return bail(st);
        } else {
            cudaError_t e = allow_dynamic_smem((const void *)cholesky_reduce_kernel<false>, smem_optin);
            if (e != cudaSuccess) return bail(fail(WNLQG_ERR_CUDA, std::string("cudaFuncSetAttribute: ") + cudaGetErrorString(e)));
        }
    }
    // Arbitrary-point Fourier on the tcgen05 tensor cores (sm_100): 7 slices (FP64 path) or 4
    // (mixed path).  WNLQG_B200_DIRECT_FOURIER=1 keeps the FP64 CUDA-core GEMM instead.
    {
        int major = 0;
        cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, dev);
        const char *direct = std::getenv("WNLQG_B200_DIRECT_FOURIER");
        if (major == 10 && !(direct && direct[0] == '1')) {
            st = t.precision == WNLQG_PRECISION_MIXED ? setup_tc_fourier<4>(pl, tiles) : setup_tc_fourier<7>(pl, tiles);
            if (st != WNLQG_OK) return bail(st);
        }
    }
    if ((st = build_passes(pl, sm_count, (size_t)smem_optin)) != WNLQG_OK) return bail(st);
    if ((st = build_shg(pl, sm_count, (size_t)smem_optin)) != WNLQG_OK) return bail(st);
    for (const Pass &ps : pl->passes)
        pl->partial_slots = std::max(pl->partial_slots, std::max(ps.global ? std::max(ps.grid, 2 * sm_count) : ps.grid,
                                                                   ps.grid_wide));
    pl->partial_slots = std::max(pl->partial_slots, pl->bcda_grid);
    pl->other_slots = std::max(pl->partial_slots, sm_count);   // the Fermi-sea dipole's grid is at most sm_count
    pl->partial_slots = std::max(pl->partial_slots, pl->shg_grid_alloc);
    if ((st = alloc((void **)&pl->d_partials, (size_t)pl->partial_slots * vc * 4 * sizeof(double))) != WNLQG_OK)
        return bail(st);
    *out_plan = pl;
    return WNLQG_OK;
}

int64_t wnlqg_b200_plan_value_count(const wnlqg_plan *plan) { return plan ? plan->vc : -1; }

}  // extern "C"

namespace {

// Morton order of nb device k-points (and weights, when given): afterwards pl->d_ok (and d_ow)
// hold them in that order and pl->d_operm + max_batch the original row of each ordered entry.
wnlqg_status order_batch(wnlqg_plan *pl, const double *k, const double *w, int64_t nb) {
    if (nb <= 0) return WNLQG_OK;
    uint32_t *keys_in = pl->d_okeys, *keys_out = pl->d_okeys + pl->max_batch;
    int *idx_in = pl->d_operm, *idx_out = pl->d_operm + pl->max_batch;
    const unsigned blocks = (unsigned)((nb + 255) / 256);
    morton_keys_kernel<<<blocks, 256, 0, pl->stream>>>(k, nb, keys_in, idx_in);
    size_t tmp = pl->osort_bytes;
    WNLQG_CUDA(cub::DeviceRadixSort::SortPairs(pl->d_osort_tmp, tmp, keys_in, keys_out, idx_in, idx_out, (int)nb, 0, 30,
                                               pl->stream));
    gather_points_kernel<<<blocks, 256, 0, pl->stream>>>(k, w, idx_out, nb, pl->d_ok, pl->d_ow);
    pl->launches += 2;
    WNLQG_CUDA(cudaGetLastError());
    return WNLQG_OK;
}

// The form of the second-harmonic kernel and the partial sums' slots for a call over n points.
void begin_call(wnlqg_plan *pl, int64_t n) {
    pl->shg_pair_now = false;
    if (pl->shg_pair)
        for (const ShgParams &p : pl->shg)
            pl->shg_pair_now |= shg_takes_pairs(p, std::min(n, pl->max_batch), pl->sm_count);
    const int shg_slots = pl->shg.empty() ? 0 : (pl->shg_pair_now ? 2 * pl->sm_count : pl->shg_grid);
    pl->call_slots = std::min(pl->partial_slots, std::max(pl->other_slots, shg_slots));
}

// The same for a call that sums: the slots it uses, zeroed.
wnlqg_status begin_sums(wnlqg_plan *pl, int64_t n) {
    begin_call(pl, n);
    WNLQG_CUDA(cudaMemsetAsync(pl->d_partials, 0, (size_t)pl->call_slots * pl->vc * 4 * sizeof(double), pl->stream));
    return WNLQG_OK;
}

// The plan's partial sums, summed over their slots into out (device, value-count complex values).
wnlqg_status launch_reduce(wnlqg_plan *pl, double2 *out) {
    const int64_t vx = reduce_values_per_block(pl->vc);
    reduce_partials_kernel<<<(unsigned)std::max<int64_t>(1, (pl->vc + vx - 1) / vx), REDUCE_THREADS, 0, pl->stream>>>(
        pl->d_partials, pl->call_slots, pl->vc, out);
    pl->launches += 1;
    WNLQG_CUDA(cudaGetLastError());
    return WNLQG_OK;
}

wnlqg_status check_mesh_args(wnlqg_plan *pl, const int64_t mesh[3], int64_t k_begin, int64_t k_end, const double *out) {
    wnlqg_status st = check_plan(pl);
    if (st != WNLQG_OK) return st;
    if (!mesh || !out) return fail(WNLQG_ERR_INVALID_ARGUMENT, "NULL argument");
    if (mesh[0] <= 0 || mesh[1] <= 0 || mesh[2] <= 0) return fail(WNLQG_ERR_INVALID_ARGUMENT, "mesh counts must be positive");
    const int64_t nk = mesh[0] * mesh[1] * mesh[2];
    if (k_begin < 0 || k_end > nk || k_begin > k_end) return fail(WNLQG_ERR_INVALID_ARGUMENT, "k range outside the mesh");
    return WNLQG_OK;
}

// Stream a's subsequent work waits for everything queued on stream b so far.
wnlqg_status stream_after(cudaStream_t a, cudaStream_t b) {
    cudaEvent_t ev;
    WNLQG_CUDA(cudaEventCreateWithFlags(&ev, cudaEventDisableTiming));
    WNLQG_CUDA(cudaEventRecord(ev, b));
    WNLQG_CUDA(cudaStreamWaitEvent(a, ev, 0));
    cudaEventDestroy(ev);
    return WNLQG_OK;
}

// The mesh sum on the plan's own stream (ordering with other streams is the caller's).
wnlqg_status enqueue_mesh(wnlqg_plan *pl, const int64_t mesh[3], int64_t k_begin, int64_t k_end, double *out_device) {
    wnlqg_status st;
    const int64_t nk = mesh[0] * mesh[1] * mesh[2];
    if ((st = record_event(pl, 0)) != WNLQG_OK) return st;
    pl->launches = 0;
    if ((st = begin_sums(pl, k_end - k_begin)) != WNLQG_OK) return st;
    const double scale = 1.0 / (double)nk;
    size_t nbatch = 0;
    for (int64_t s = k_begin; s < k_end; s += pl->max_batch, ++nbatch) {
        int64_t nb = std::min(pl->max_batch, k_end - s);
        size_t base = 1 + 3 * nbatch;
        if ((st = record_event(pl, base)) != WNLQG_OK) return st;
        if ((st = run_fd_stencil(pl, nb, s, mesh, nullptr, nullptr, false, base, s, nullptr)) != WNLQG_OK) return st;
        if ((st = run_front(pl, nb, s, mesh, nullptr, base)) != WNLQG_OK) return st;
        if ((st = run_isolation(pl, nb, s, nullptr)) != WNLQG_OK) return st;
        if ((st = run_passes(pl, nb, 0, scale, 0)) != WNLQG_OK) return st;
    }
    // Events: [0] start, per batch b: [1+3b] batch start, [2+3b] after Fourier, [3+3b] after eigh,
    // next batch start (or the final event) closes the response stage.
    size_t final_ev = 1 + 3 * nbatch;
    if ((st = record_event(pl, final_ev)) != WNLQG_OK) return st;
    if ((st = launch_reduce(pl, reinterpret_cast<double2 *>(out_device))) != WNLQG_OK) return st;
    if ((st = record_event(pl, final_ev + 1)) != WNLQG_OK) return st;
    pl->timing_valid = true;
    pl->timing_batches = nbatch;
    return WNLQG_OK;
}

// Events that order streams: destroyed at once in direct calls, kept alive until the end of a
// stream capture (the capture records their dependencies).
struct EventKeeper {
    std::vector<cudaEvent_t> *keep = nullptr;
    void done(cudaEvent_t ev) {
        if (keep) keep->push_back(ev);
        else cudaEventDestroy(ev);
    }
};

wnlqg_status order_after(cudaStream_t a, cudaStream_t b, EventKeeper &ek) {
    cudaEvent_t ev;
    WNLQG_CUDA(cudaEventCreateWithFlags(&ev, cudaEventDisableTiming));
    cudaError_t e = cudaEventRecord(ev, b);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(a, ev, 0);
    ek.done(ev);
    if (e != cudaSuccess) return fail(WNLQG_ERR_CUDA, std::string("stream ordering: ") + cudaGetErrorString(e));
    return WNLQG_OK;
}

// Several plans' mesh sums forked from `origin` and joined back into it.
wnlqg_status enqueue_many(wnlqg_plan *const *plans, int32_t count, const int64_t *meshes, const int64_t *k_begin,
                          const int64_t *k_end, double *const *outs_device, cudaStream_t origin, EventKeeper &ek) {
    cudaEvent_t fork;
    WNLQG_CUDA(cudaEventCreateWithFlags(&fork, cudaEventDisableTiming));
    cudaError_t e = cudaEventRecord(fork, origin);
    for (int32_t i = 0; i < count && e == cudaSuccess; ++i) {
        plans[i]->timing_valid = false;
        e = cudaStreamWaitEvent(plans[i]->stream, fork, 0);
    }
    ek.done(fork);
    if (e != cudaSuccess) return fail(WNLQG_ERR_CUDA, std::string("stream fork: ") + cudaGetErrorString(e));
    for (int32_t i = 0; i < count; ++i) {
        wnlqg_status st = enqueue_mesh(plans[i], meshes + 3 * i, k_begin[i], k_end[i], outs_device[i]);
        if (st != WNLQG_OK) return st;
    }
    for (int32_t i = 0; i < count; ++i) {
        wnlqg_status st = order_after(origin, plans[i]->stream, ek);
        if (st != WNLQG_OK) return st;
    }
    return WNLQG_OK;
}

// Weighted point sum on the plan's stream: out = sum_i w_i value(k_i), k-points and weights on
// the device.
wnlqg_status enqueue_points_weighted(wnlqg_plan *pl, const double *kpoints_device, const double *weights_device,
                                     int64_t n, double *out_device) {
    wnlqg_status st;
    if ((st = record_event(pl, 0)) != WNLQG_OK) return st;
    pl->launches = 0;
    if ((st = begin_sums(pl, n)) != WNLQG_OK) return st;
    size_t nbatch = 0;
    for (int64_t s = 0; s < n; s += pl->max_batch, ++nbatch) {
        const int64_t nb = std::min(pl->max_batch, n - s);
        const size_t base = 1 + 3 * nbatch;
        if ((st = record_event(pl, base)) != WNLQG_OK) return st;
        const double *kb = kpoints_device + 3 * s, *wb = weights_device + s;
        const bool ord = pl->order_points && nb > 1;
        if (ord) {
            if ((st = order_batch(pl, kb, wb, nb)) != WNLQG_OK) return st;
            kb = pl->d_ok;
            wb = pl->d_ow;
        }
        const int *perm = ord ? pl->d_operm + pl->max_batch : nullptr;
        if ((st = run_fd_stencil(pl, nb, 0, nullptr, kb, nullptr, ord, base, s, perm)) != WNLQG_OK) return st;
        if ((st = run_front(pl, nb, 0, nullptr, kb, base, nullptr, ord)) != WNLQG_OK) return st;
        if ((st = run_isolation(pl, nb, s, perm)) != WNLQG_OK) return st;
        if ((st = run_passes(pl, nb, 0, 1.0, 0, wb)) != WNLQG_OK) return st;
    }
    const size_t final_ev = 1 + 3 * nbatch;
    if ((st = record_event(pl, final_ev)) != WNLQG_OK) return st;
    if ((st = launch_reduce(pl, reinterpret_cast<double2 *>(out_device))) != WNLQG_OK) return st;
    if ((st = record_event(pl, final_ev + 1)) != WNLQG_OK) return st;
    pl->timing_valid = true;
    pl->timing_batches = nbatch;
    return WNLQG_OK;
}

wnlqg_status check_points_args(wnlqg_plan *pl, const double *kpoints_device, const double *weights_device, int64_t n,
                               const double *out_device) {
    wnlqg_status st = check_plan(pl);
    if (st != WNLQG_OK) return st;
    if (n < 0 || (n > 0 && (!kpoints_device || !weights_device)) || !out_device)
        return fail(WNLQG_ERR_INVALID_ARGUMENT, "invalid points");
    return WNLQG_OK;
}

wnlqg_status check_many_args(wnlqg_plan *const *plans, int32_t count, const int64_t *meshes, const int64_t *k_begin,
                             const int64_t *k_end, double *const *outs_device) {
    if (count < 0 || (count > 0 && (!plans || !meshes || !k_begin || !k_end || !outs_device)))
        return fail(WNLQG_ERR_INVALID_ARGUMENT, "invalid plan list");
    for (int32_t i = 0; i < count; ++i) {
        wnlqg_status st = check_plan(plans[i]);
        if (st != WNLQG_OK) return st;
        if (i > 0 && plans[i]->model->device != plans[0]->model->device)
            return fail(WNLQG_ERR_INVALID_ARGUMENT, "all plans of one call must live on one device");
    }
    for (int32_t i = 0; i < count; ++i) {
        wnlqg_status st = check_mesh_args(plans[i], meshes + 3 * i, k_begin[i], k_end[i], outs_device[i]);
        if (st != WNLQG_OK) return st;
    }
    return WNLQG_OK;
}

}  // namespace

extern "C" {

wnlqg_status wnlqg_b200_eval_mesh_device(wnlqg_plan *pl, const int64_t mesh[3], int64_t k_begin, int64_t k_end,
                                         double *out_device, void *stream) {
    wnlqg_status st = check_mesh_args(pl, mesh, k_begin, k_end, out_device);
    if (st != WNLQG_OK) return st;
    WNLQG_CUDA(cudaSetDevice(pl->model->device));
    // The caller's stream (NULL = the legacy default stream) and the plan's non-blocking stream
    // are ordered both ways with events: the work starts after everything queued on the caller's
    // stream and the caller's stream resumes after the result is written.
    cudaStream_t user = static_cast<cudaStream_t>(stream);
    pl->timing_valid = false;
    if ((st = stream_after(pl->stream, user)) != WNLQG_OK) return st;
    if ((st = enqueue_mesh(pl, mesh, k_begin, k_end, out_device)) != WNLQG_OK) return st;
    return stream_after(user, pl->stream);
}

wnlqg_status wnlqg_b200_eval_points_weighted_device(wnlqg_plan *pl, const double *kpoints_device,
                                                    const double *weights_device, int64_t n, double *out_device,
                                                    void *stream) {
    wnlqg_status st = check_points_args(pl, kpoints_device, weights_device, n, out_device);
    if (st != WNLQG_OK) return st;
    WNLQG_CUDA(cudaSetDevice(pl->model->device));
    cudaStream_t user = static_cast<cudaStream_t>(stream);
    EventKeeper ek;
    if ((st = order_after(pl->stream, user, ek)) != WNLQG_OK) return st;
    if ((st = enqueue_points_weighted(pl, kpoints_device, weights_device, n, out_device)) != WNLQG_OK) return st;
    return order_after(user, pl->stream, ek);
}

wnlqg_status wnlqg_b200_eval_mesh_many(wnlqg_plan *const *plans, int32_t count, const int64_t *meshes,
                                       const int64_t *k_begin, const int64_t *k_end, double *const *outs_device,
                                       void *stream) {
    wnlqg_status st = check_many_args(plans, count, meshes, k_begin, k_end, outs_device);
    if (st != WNLQG_OK) return st;
    if (count == 0) return WNLQG_OK;
    WNLQG_CUDA(cudaSetDevice(plans[0]->model->device));
    // Every plan's stream forks from the caller's stream before any plan is enqueued and joins back
    // after all are, so the models' kernels overlap on the device.
    EventKeeper ek;
    return enqueue_many(plans, count, meshes, k_begin, k_end, outs_device, static_cast<cudaStream_t>(stream), ek);
}

wnlqg_status wnlqg_b200_eval_mesh(wnlqg_plan *pl, const int64_t mesh[3], int64_t k_begin, int64_t k_end, double *out) {
    wnlqg_status st = check_plan(pl);
    if (st != WNLQG_OK) return st;
    if (!out) return fail(WNLQG_ERR_INVALID_ARGUMENT, "NULL output");
    if ((st = wnlqg_b200_eval_mesh_device(pl, mesh, k_begin, k_end, reinterpret_cast<double *>(pl->d_out), nullptr)) != WNLQG_OK)
        return st;
    WNLQG_CUDA(cudaMemcpyAsync(out, pl->d_out, (size_t)pl->vc * sizeof(double2), cudaMemcpyDeviceToHost, pl->stream));
    WNLQG_CUDA(cudaStreamSynchronize(pl->stream));
    if ((st = tc_check(pl)) != WNLQG_OK) return st;
    if ((st = iso_check(pl)) != WNLQG_OK) return st;
    for (int64_t v = 0; v < 2 * pl->vc; ++v)
        if (!std::isfinite(out[v])) return fail(WNLQG_ERR_NONFINITE, "response contains non-finite values");
    return WNLQG_OK;
}

wnlqg_status wnlqg_b200_eval_points(wnlqg_plan *pl, const double *kpoints, int64_t n, double *out) {
    wnlqg_status st = check_plan(pl);
    if (st != WNLQG_OK) return st;
    if (n < 0 || (n > 0 && (!kpoints || !out))) return fail(WNLQG_ERR_INVALID_ARGUMENT, "invalid points");
    if (!finite_array(kpoints, 3 * (size_t)n)) return fail(WNLQG_ERR_NONFINITE, "k-points must be finite");
    WNLQG_CUDA(cudaSetDevice(pl->model->device));
    pl->launches = 0;
    begin_call(pl, n);
    for (int64_t s = 0; s < n; s += pl->max_batch) {
        int64_t nb = std::min(pl->max_batch, n - s);
        WNLQG_CUDA(cudaMemcpyAsync(pl->d_kpts, kpoints + 3 * s, (size_t)nb * 3 * sizeof(double), cudaMemcpyHostToDevice,
                                   pl->stream));
        const bool ord = pl->order_points && nb > 1;
        if (ord && (st = order_batch(pl, pl->d_kpts, nullptr, nb)) != WNLQG_OK) return st;
        const int *perm = ord ? pl->d_operm + pl->max_batch : nullptr;
        if ((st = run_fd_stencil(pl, nb, 0, nullptr, ord ? pl->d_ok : pl->d_kpts, nullptr, ord, 1, s, perm)) != WNLQG_OK)
            return st;
        if ((st = run_front(pl, nb, 0, nullptr, ord ? pl->d_ok : pl->d_kpts, 1, nullptr, ord)) != WNLQG_OK) return st;
        if ((st = run_isolation(pl, nb, s, perm)) != WNLQG_OK) return st;
        if ((st = run_passes(pl, nb, 1, 1.0, 0, nullptr, ord ? pl->d_operm + pl->max_batch : nullptr)) != WNLQG_OK)
            return st;
        WNLQG_CUDA(cudaMemcpyAsync(out + 2 * s * pl->vc, pl->d_points, (size_t)nb * pl->vc * sizeof(double2),
                                   cudaMemcpyDeviceToHost, pl->stream));
    }
    WNLQG_CUDA(cudaStreamSynchronize(pl->stream));
    pl->timing_valid = false;
    if ((st = tc_check(pl)) != WNLQG_OK) return st;
    if ((st = iso_check(pl)) != WNLQG_OK) return st;
    for (int64_t v = 0; v < 2 * n * pl->vc; ++v)
        if (!std::isfinite(out[v])) return fail(WNLQG_ERR_NONFINITE, "response contains non-finite values");
    return WNLQG_OK;
}

wnlqg_status wnlqg_b200_eval_points_weighted(wnlqg_plan *pl, const double *kpoints, const double *weights,
                                             int64_t n, double *out) {
    wnlqg_status st = check_plan(pl);
    if (st != WNLQG_OK) return st;
    if (n < 0 || (n > 0 && (!kpoints || !weights)) || !out) return fail(WNLQG_ERR_INVALID_ARGUMENT, "invalid points");
    if (!finite_array(kpoints, 3 * (size_t)n) || !finite_array(weights, (size_t)n))
        return fail(WNLQG_ERR_NONFINITE, "k-points and weights must be finite");
    WNLQG_CUDA(cudaSetDevice(pl->model->device));
    pl->launches = 0;
    if ((st = begin_sums(pl, n)) != WNLQG_OK) return st;
    for (int64_t s = 0; s < n; s += pl->max_batch) {
        int64_t nb = std::min(pl->max_batch, n - s);
        WNLQG_CUDA(cudaMemcpyAsync(pl->d_kpts, kpoints + 3 * s, (size_t)nb * 3 * sizeof(double), cudaMemcpyHostToDevice,
                                   pl->stream));
        WNLQG_CUDA(cudaMemcpyAsync(pl->d_weights, weights + s, (size_t)nb * sizeof(double), cudaMemcpyHostToDevice,
                                   pl->stream));
        const bool ord = pl->order_points && nb > 1;
        if (ord && (st = order_batch(pl, pl->d_kpts, pl->d_weights, nb)) != WNLQG_OK) return st;
        const int *perm = ord ? pl->d_operm + pl->max_batch : nullptr;
        if ((st = run_fd_stencil(pl, nb, 0, nullptr, ord ? pl->d_ok : pl->d_kpts, nullptr, ord, 1, s, perm)) != WNLQG_OK)
            return st;
        if ((st = run_front(pl, nb, 0, nullptr, ord ? pl->d_ok : pl->d_kpts, 1, nullptr, ord)) != WNLQG_OK) return st;
        if ((st = run_isolation(pl, nb, s, perm)) != WNLQG_OK) return st;
        if ((st = run_passes(pl, nb, 0, 1.0, 0, ord ? pl->d_ow : pl->d_weights)) != WNLQG_OK) return st;
    }
    if ((st = launch_reduce(pl, pl->d_out)) != WNLQG_OK) return st;
    WNLQG_CUDA(cudaMemcpyAsync(out, pl->d_out, (size_t)pl->vc * sizeof(double2), cudaMemcpyDeviceToHost, pl->stream));
    WNLQG_CUDA(cudaStreamSynchronize(pl->stream));
    pl->timing_valid = false;
    if ((st = tc_check(pl)) != WNLQG_OK) return st;
    if ((st = iso_check(pl)) != WNLQG_OK) return st;
    for (int64_t v = 0; v < 2 * pl->vc; ++v)
        if (!std::isfinite(out[v])) return fail(WNLQG_ERR_NONFINITE, "response contains non-finite values");
    return WNLQG_OK;
}

wnlqg_status wnlqg_b200_eval_mesh_weighted(wnlqg_plan *pl, const int64_t mesh[3], const int64_t *indices,
                                           const double *weights, int64_t n, double *out) {
    wnlqg_status st = check_plan(pl);
    if (st != WNLQG_OK) return st;
    if (!mesh || !out || n < 0 || (n > 0 && (!indices || !weights))) return fail(WNLQG_ERR_INVALID_ARGUMENT, "invalid arguments");
    if (mesh[0] <= 0 || mesh[1] <= 0 || mesh[2] <= 0) return fail(WNLQG_ERR_INVALID_ARGUMENT, "mesh counts must be positive");
    const int64_t nk = mesh[0] * mesh[1] * mesh[2];
    for (int64_t i = 0; i < n; ++i)
        if (indices[i] < 0 || indices[i] >= nk) return fail(WNLQG_ERR_INVALID_ARGUMENT, "mesh index out of range");
    if (!finite_array(weights, (size_t)n)) return fail(WNLQG_ERR_NONFINITE, "weights must be finite");
    WNLQG_CUDA(cudaSetDevice(pl->model->device));
    pl->launches = 0;
    if ((st = begin_sums(pl, n)) != WNLQG_OK) return st;
    for (int64_t s = 0; s < n; s += pl->max_batch) {
        const int64_t nb = std::min(pl->max_batch, n - s);
        bool contiguous = true;
        for (int64_t i = 1; i < nb && contiguous; ++i) contiguous = indices[s + i] == indices[s] + i;
        WNLQG_CUDA(cudaMemcpyAsync(pl->d_weights, weights + s, (size_t)nb * sizeof(double), cudaMemcpyHostToDevice,
                                   pl->stream));
        if (contiguous) {
            // A run of consecutive mesh indices takes the staged mesh contraction.
            if ((st = run_fd_stencil(pl, nb, indices[s], mesh, nullptr, nullptr, false, 1, s, nullptr)) != WNLQG_OK) return st;
            if ((st = run_front(pl, nb, indices[s], mesh, nullptr, 1)) != WNLQG_OK) return st;
        } else {
            WNLQG_CUDA(cudaMemcpyAsync(pl->d_kidx, indices + s, (size_t)nb * sizeof(int64_t), cudaMemcpyHostToDevice,
                                       pl->stream));
            if ((st = run_fd_stencil(pl, nb, 0, mesh, nullptr, pl->d_kidx, false, 1, s, nullptr)) != WNLQG_OK) return st;
            if ((st = run_front(pl, nb, 0, mesh, nullptr, 1, pl->d_kidx)) != WNLQG_OK) return st;
        }
        if ((st = run_isolation(pl, nb, s, nullptr)) != WNLQG_OK) return st;
        if ((st = run_passes(pl, nb, 0, 1.0, 0, pl->d_weights)) != WNLQG_OK) return st;
    }
    if ((st = launch_reduce(pl, pl->d_out)) != WNLQG_OK) return st;
    WNLQG_CUDA(cudaMemcpyAsync(out, pl->d_out, (size_t)pl->vc * sizeof(double2), cudaMemcpyDeviceToHost, pl->stream));
    WNLQG_CUDA(cudaStreamSynchronize(pl->stream));
    pl->timing_valid = false;
    if ((st = tc_check(pl)) != WNLQG_OK) return st;
    if ((st = iso_check(pl)) != WNLQG_OK) return st;
    for (int64_t v = 0; v < 2 * pl->vc; ++v)
        if (!std::isfinite(out[v])) return fail(WNLQG_ERR_NONFINITE, "response contains non-finite values");
    return WNLQG_OK;
}

}  // extern "C"

namespace {

// out[b][row][col] = U[b][col][row].
__global__ void transpose_vectors_kernel(const double2 *__restrict__ U, int64_t nb, int nw, double2 *__restrict__ out) {
    const int64_t nn = (int64_t)nw * nw, e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (e >= nb * nn) return;
    const int64_t b = e / nn;
    const int r = (int)(e - b * nn);
    out[b * nn + (int64_t)(r % nw) * nw + r / nw] = U[e];
}

wnlqg_status eval_spectrum(wnlqg_plan *pl, const double *kpoints, int64_t n, double *energies, double *eigenvectors,
                           bool rows) {
    wnlqg_status st = check_plan(pl);
    if (st != WNLQG_OK) return st;
    if (n < 0 || (n > 0 && (!kpoints || !energies))) return fail(WNLQG_ERR_INVALID_ARGUMENT, "invalid points");
    if (!finite_array(kpoints, 3 * (size_t)n)) return fail(WNLQG_ERR_NONFINITE, "k-points must be finite");
    WNLQG_CUDA(cudaSetDevice(pl->model->device));
    std::vector<int> stat(pl->nonorth ? (size_t)n : 0);
    for (int64_t s = 0; s < n; s += pl->max_batch) {
        int64_t nb = std::min(pl->max_batch, n - s);
        WNLQG_CUDA(cudaMemcpyAsync(pl->d_kpts, kpoints + 3 * s, (size_t)nb * 3 * sizeof(double), cudaMemcpyHostToDevice,
                                   pl->stream));
        if ((st = run_front(pl, nb, 0, nullptr, pl->d_kpts, 1)) != WNLQG_OK) return st;
        if (pl->nonorth)
            WNLQG_CUDA(cudaMemcpyAsync(stat.data() + s, pl->d_status, (size_t)nb * sizeof(int), cudaMemcpyDeviceToHost,
                                       pl->stream));
        WNLQG_CUDA(cudaMemcpyAsync(energies + s * pl->nw, pl->d_E, (size_t)nb * pl->nw * sizeof(double),
                                   cudaMemcpyDeviceToHost, pl->stream));
        if (eigenvectors) {
            const double2 *src = pl->d_U;
            if (rows) {
                // The channels are spent once the vectors exist: their buffer takes the transposes.  601 points
                // of 31 orbitals, row-major vectors: 2.9 ms with the transposition on the host, 1.2 with this.
                // The copy is the plain one: pinned halves with the host copying a chunk out while the next
                // is on its way took 1.3, and their allocation 1.4 to 3 ms more in a plan's first call.
                transpose_vectors_kernel<<<(unsigned)((nb * pl->nn + 255) / 256), 256, 0, pl->stream>>>(pl->d_U, nb, pl->nw,
                                                                                                     pl->d_xw);
                WNLQG_CUDA(cudaGetLastError());
                src = pl->d_xw;
            }
            WNLQG_CUDA(cudaMemcpyAsync(eigenvectors + 2 * s * pl->nn, src, (size_t)nb * pl->nn * sizeof(double2),
                                       cudaMemcpyDeviceToHost, pl->stream));
        }
    }
    WNLQG_CUDA(cudaStreamSynchronize(pl->stream));
    pl->timing_valid = false;
    if ((st = tc_check(pl)) != WNLQG_OK) return st;
    if (pl->nonorth)
        for (int v : stat)
            if (v) return fail(WNLQG_ERR_INVALID_ARGUMENT, "effective S(k) is not positive definite");
    return WNLQG_OK;
}

}  // namespace

extern "C" {

wnlqg_status wnlqg_b200_eval_spectrum_rows(wnlqg_plan *pl, const double *kpoints, int64_t n, double *energies,
                                           double *eigenvectors) {
    wnlqg_status st = check_plan(pl);
    if (st != WNLQG_OK) return st;
    if (pl->conv1) return fail(WNLQG_ERR_UNSUPPORTED, "row-major vectors in Convention I are not built");
    return eval_spectrum(pl, kpoints, n, energies, eigenvectors, true);
}

wnlqg_status wnlqg_b200_eval_spectrum(wnlqg_plan *pl, const double *kpoints, int64_t n, double *energies,
                                      double *eigenvectors) {
    wnlqg_status st = eval_spectrum(pl, kpoints, n, energies, eigenvectors, false);
    if (st != WNLQG_OK) return st;
    if (pl->conv1 && eigenvectors) {
        // Convention I eigenvectors: D(k)^H U, D = diag(exp(2 pi i k.tau_frac)) (the similarity of
        // _apply_wannier_center_similarity!), then the canonical phase rule again
        // (canonicalize_eigenvectors!, HamiltonianMatrixElements.jl:6-25); energies are unchanged.
        const int nw = pl->nw;
        std::vector<double2> ph(nw);
        for (int64_t s = 0; s < n; ++s) {
            const double *k = kpoints + 3 * s;
            for (int i = 0; i < nw; ++i) {
                const double x = 2.0 * WNLQG_PI * (k[0] * pl->tau_frac[i] + k[1] * pl->tau_frac[nw + i] + k[2] * pl->tau_frac[2 * nw + i]);
                ph[i] = make_double2(std::cos(x), -std::sin(x));   // conj(phi_i)
            }
            double2 *u = reinterpret_cast<double2 *>(eigenvectors) + s * pl->nn;
            for (int c = 0; c < nw; ++c) {
                double2 *col = u + (size_t)nw * c;
                int pivot = 0;
                double pm = -1.0;
                for (int i = 0; i < nw; ++i) {
                    col[i] = cmul(ph[i], col[i]);
                    const double mg = std::hypot(col[i].x, col[i].y);
                    if (mg > pm) { pm = mg; pivot = i; }
                }
                if (pm > 0.0) {
                    const double2 q = make_double2(col[pivot].x / pm, -col[pivot].y / pm);
                    for (int i = 0; i < nw; ++i) col[i] = cmul(col[i], q);
                }
            }
        }
    }
    return WNLQG_OK;
}

wnlqg_status wnlqg_b200_plan_last_timing(const wnlqg_plan *pl_const, double *fourier_ms, double *eigen_ms,
                                         double *response_ms, double *total_ms) {
    wnlqg_plan *pl = const_cast<wnlqg_plan *>(pl_const);
    wnlqg_status st = check_plan(pl);
    if (st != WNLQG_OK) return st;
    if (!pl->timing_valid) return fail(WNLQG_ERR_INVALID_ARGUMENT, "no mesh evaluation to report");
    WNLQG_CUDA(cudaSetDevice(pl->model->device));
    WNLQG_CUDA(cudaStreamSynchronize(pl->stream));
    size_t nbatch = pl->timing_batches;
    double f = 0, e = 0, r = 0;
    for (size_t b = 0; b < nbatch; ++b) {
        float ms = 0;
        size_t base = 1 + 3 * b;
        WNLQG_CUDA(cudaEventElapsedTime(&ms, pl->events[base], pl->events[base + 1]));
        f += ms;
        WNLQG_CUDA(cudaEventElapsedTime(&ms, pl->events[base + 1], pl->events[base + 2]));
        e += ms;
        WNLQG_CUDA(cudaEventElapsedTime(&ms, pl->events[base + 2], pl->events[base + 3]));
        r += ms;
    }
    float tot = 0;
    WNLQG_CUDA(cudaEventElapsedTime(&tot, pl->events[0], pl->events[1 + 3 * nbatch + 1]));
    if (fourier_ms) *fourier_ms = f;
    if (eigen_ms) *eigen_ms = e;
    if (response_ms) *response_ms = r;
    if (total_ms) *total_ms = tot;
    return WNLQG_OK;
}

int64_t wnlqg_b200_plan_last_launch_count(const wnlqg_plan *plan) { return plan ? plan->launches : -1; }

wnlqg_status wnlqg_b200_plan_status(wnlqg_plan *pl) {
    wnlqg_status st = check_plan(pl);
    if (st != WNLQG_OK) return st;
    WNLQG_CUDA(cudaSetDevice(pl->model->device));
    pl->tc_used = true;   // read the flag even if the last direct call did not use the tensor cores
    if ((st = tc_check(pl)) != WNLQG_OK) return st;
    return iso_check(pl);
}

}  // extern "C"

// ---------------------------------------------------------------------------------------------
// CUDA graphs: the whole interpolate -> eigensolve -> integrand -> reduce chain of one call (one
// plan, or several plans on their own streams forked from one origin), captured once and replayed
// with one cudaGraphLaunch.  The graph bakes in the call's arguments and the plans' buffers.
// ---------------------------------------------------------------------------------------------
struct wnlqg_graph {
    std::vector<wnlqg_plan *> plans;
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    cudaStream_t origin = nullptr;
    int device = 0;
    int64_t kernels = 0;
};

namespace {

void graph_release(wnlqg_graph *g) {
    if (!g) return;
    if (g->exec) cudaGraphExecDestroy(g->exec);
    if (g->graph) cudaGraphDestroy(g->graph);
    if (g->origin) cudaStreamDestroy(g->origin);
    for (wnlqg_plan *pl : g->plans) pl->graph_refs -= 1;
    delete g;
}

// Runs `body(origin, keeper)` once directly (so that every lazily sized buffer exists), then under
// stream capture of a private origin stream, and instantiates the captured graph.
template <typename Body>
wnlqg_status capture_graph(const std::vector<wnlqg_plan *> &plans, Body body, wnlqg_graph **out) {
    if (!out) return fail(WNLQG_ERR_INVALID_ARGUMENT, "NULL graph handle");
    *out = nullptr;
    wnlqg_graph *g = new wnlqg_graph();
    g->device = plans[0]->model->device;
    WNLQG_CUDA(cudaSetDevice(g->device));
    cudaError_t e = cudaStreamCreateWithFlags(&g->origin, cudaStreamNonBlocking);
    if (e != cudaSuccess) {
        delete g;
        return fail(WNLQG_ERR_CUDA, std::string("cudaStreamCreate: ") + cudaGetErrorString(e));
    }
    // Plans join the graph's reference count first: buffers a later call outgrows are retired.
    g->plans = plans;
    for (wnlqg_plan *pl : plans) pl->graph_refs += 1;
    {
        EventKeeper direct;
        wnlqg_status st = body(g->origin, direct);
        if (st == WNLQG_OK && (e = cudaStreamSynchronize(g->origin)) != cudaSuccess)
            st = fail(WNLQG_ERR_CUDA, std::string("graph warm-up: ") + cudaGetErrorString(e));
        if (st != WNLQG_OK) {
            graph_release(g);
            return st;
        }
    }
    std::vector<cudaEvent_t> kept;
    EventKeeper keeper;
    keeper.keep = &kept;
    e = cudaStreamBeginCapture(g->origin, cudaStreamCaptureModeRelaxed);
    if (e != cudaSuccess) {
        graph_release(g);
        return fail(WNLQG_ERR_CUDA, std::string("cudaStreamBeginCapture: ") + cudaGetErrorString(e));
    }
    wnlqg_status st = body(g->origin, keeper);
    cudaGraph_t graph = nullptr;
    e = cudaStreamEndCapture(g->origin, &graph);
    for (cudaEvent_t ev : kept) cudaEventDestroy(ev);
    for (wnlqg_plan *pl : plans) pl->timing_valid = false;   // the captured event records time nothing
    if (st == WNLQG_OK && e != cudaSuccess)
        st = fail(WNLQG_ERR_CUDA, std::string("cudaStreamEndCapture: ") + cudaGetErrorString(e));
    if (st != WNLQG_OK) {
        if (graph) cudaGraphDestroy(graph);
        cudaGetLastError();
        graph_release(g);
        return st;
    }
    g->graph = graph;
    e = cudaGraphInstantiate(&g->exec, g->graph, 0);
    if (e != cudaSuccess) {
        graph_release(g);
        return fail(WNLQG_ERR_CUDA, std::string("cudaGraphInstantiate: ") + cudaGetErrorString(e));
    }
    for (wnlqg_plan *pl : plans) g->kernels += pl->launches;
    *out = g;
    return WNLQG_OK;
}

}  // namespace

extern "C" {

wnlqg_status wnlqg_b200_graph_capture_mesh_many(wnlqg_plan *const *plans, int32_t count, const int64_t *meshes,
                                                const int64_t *k_begin, const int64_t *k_end,
                                                double *const *outs_device, wnlqg_graph **out_graph) {
    wnlqg_status st = check_many_args(plans, count, meshes, k_begin, k_end, outs_device);
    if (st != WNLQG_OK) return st;
    if (count == 0) return fail(WNLQG_ERR_INVALID_ARGUMENT, "a graph needs at least one plan");
    std::vector<wnlqg_plan *> list(plans, plans + count);
    for (size_t i = 0; i < list.size(); ++i)
        for (size_t j = 0; j < i; ++j)
            if (list[i] == list[j]) return fail(WNLQG_ERR_INVALID_ARGUMENT, "a plan appears twice in one graph");
    std::vector<int64_t> m(meshes, meshes + 3 * (size_t)count), kb(k_begin, k_begin + count), ke(k_end, k_end + count);
    std::vector<double *> outs(outs_device, outs_device + count);
    return capture_graph(list, [&](cudaStream_t origin, EventKeeper &ek) {
        return enqueue_many(list.data(), count, m.data(), kb.data(), ke.data(), outs.data(), origin, ek);
    }, out_graph);
}

wnlqg_status wnlqg_b200_graph_capture_points_weighted(wnlqg_plan *plan, const double *kpoints_device,
                                                      const double *weights_device, int64_t n, double *out_device,
                                                      wnlqg_graph **out_graph) {
    wnlqg_status st = check_points_args(plan, kpoints_device, weights_device, n, out_device);
    if (st != WNLQG_OK) return st;
    std::vector<wnlqg_plan *> list{plan};
    return capture_graph(list, [&](cudaStream_t origin, EventKeeper &ek) {
        wnlqg_status s2 = order_after(plan->stream, origin, ek);
        if (s2 == WNLQG_OK) s2 = enqueue_points_weighted(plan, kpoints_device, weights_device, n, out_device);
        if (s2 == WNLQG_OK) s2 = order_after(origin, plan->stream, ek);
        return s2;
    }, out_graph);
}

wnlqg_status wnlqg_b200_graph_launch(wnlqg_graph *graph, void *stream) {
    if (!graph || !graph->exec) return fail(WNLQG_ERR_INVALID_ARGUMENT, "invalid graph");
    WNLQG_CUDA(cudaSetDevice(graph->device));
    WNLQG_CUDA(cudaGraphLaunch(graph->exec, static_cast<cudaStream_t>(stream)));
    return WNLQG_OK;
}

wnlqg_status wnlqg_b200_graph_status(wnlqg_graph *graph) {
    if (!graph) return fail(WNLQG_ERR_INVALID_ARGUMENT, "invalid graph");
    WNLQG_CUDA(cudaSetDevice(graph->device));
    for (wnlqg_plan *pl : graph->plans) {
        if (!pl->d_tc_err) continue;
        int h = 0;
        WNLQG_CUDA(cudaMemcpy(&h, pl->d_tc_err, sizeof(int), cudaMemcpyDeviceToHost));
        if (h) {
            cudaMemset(pl->d_tc_err, 0, sizeof(int));
            return fail(WNLQG_ERR_DEVICE_TIMEOUT, "tensor-core Fourier: a bounded device wait gave up");
        }
    }
    for (wnlqg_plan *pl : graph->plans) {
        wnlqg_status st = iso_check(pl);
        if (st != WNLQG_OK) return st;
    }
    return WNLQG_OK;
}

int64_t wnlqg_b200_graph_kernel_count(const wnlqg_graph *graph) { return graph ? graph->kernels : -1; }

wnlqg_status wnlqg_b200_graph_destroy(wnlqg_graph *graph) {
    if (!graph) return WNLQG_OK;
    cudaSetDevice(graph->device);
    cudaDeviceSynchronize();
    graph_release(graph);
    return WNLQG_OK;
}

}  // extern "C"

// ---------------------------------------------------------------------------------------------
// Autotuner: per orbital count, the eigensolver team (threads per matrix of the FP64 refinement and,
// on the mixed path, the FP32 Jacobi; up to 32 orbitals) and the contraction tile (photon
// energies per thread) measured on the caller's own mesh block; the fastest of each is kept in
// the plan and remembered for the process (device, orbitals, precision, geometry, energies,
// values).  Every candidate is a configuration the library runs anyway.
// ---------------------------------------------------------------------------------------------
namespace {

struct TuneChoice {
    int team, omb, warm, wide, mshg_grid, shg_grid, resp_grid, eigh_grid;
    wnlqg_autotune_report report;
};
std::map<std::tuple<int, int, int, int, int64_t, int64_t>, TuneChoice> g_tune_cache;
std::mutex g_tune_mutex;

void apply_team(wnlqg_plan *pl, int team) {
    pl->eigh_team = team;
    pl->eigh_smem = (team == 32 ? 4 : 1) * WarpJacobiSmem::per_team(pl->nw);
    pl->refine_smem = (team == 32 ? 2 : 1) * WarpRefineSmem::per_team(pl->nw);
}

void apply_omb(wnlqg_plan *pl, int omb) {
    for (Pass &ps : pl->passes) ps.params.omb_force = omb;
}

// Two timed mesh sums (the first warms caches); the second's eigensolve and response times.
wnlqg_status tune_measure(wnlqg_plan *pl, const int64_t mesh[3], int64_t kb, int64_t ke, double *eig, double *resp) {
    *eig = *resp = std::numeric_limits<double>::infinity();
    for (int rep = 0; rep < 2; ++rep) {
        wnlqg_status st = enqueue_mesh(pl, mesh, kb, ke, reinterpret_cast<double *>(pl->d_out));
        if (st != WNLQG_OK) return st;
        double f = 0, e = 0, r = 0, t = 0;
        if ((st = wnlqg_b200_plan_last_timing(pl, &f, &e, &r, &t)) != WNLQG_OK) return st;
        if (rep == 1) {
            *eig = e;
            *resp = r;
        }
    }
    return WNLQG_OK;
}

}  // namespace

extern "C" wnlqg_status wnlqg_b200_plan_autotune(wnlqg_plan *pl, const int64_t mesh[3], int64_t k_begin,
                                                 int64_t k_end, wnlqg_autotune_report *report) {
    wnlqg_status st = check_mesh_args(pl, mesh, k_begin, k_end, reinterpret_cast<const double *>(pl ? pl->d_out : nullptr));
    if (st != WNLQG_OK) return st;
    if (pl->graph_refs > 0)
        return fail(WNLQG_ERR_INVALID_ARGUMENT, "plan is captured in a CUDA graph: tune it before capturing");
    WNLQG_CUDA(cudaSetDevice(pl->model->device));
    const auto key = std::make_tuple(pl->model->device, pl->nw, (int)pl->task.precision, pl->nonorth ? 1 : 0,
                                     (int64_t)pl->task.num_photon_energies, pl->vc);
    {
        std::lock_guard<std::mutex> lock(g_tune_mutex);
        auto it = g_tune_cache.find(key);
        if (it != g_tune_cache.end()) {
            if (pl->warp_eigh && it->second.team) apply_team(pl, it->second.team);
            if (it->second.warm >= 0) pl->warm_mode = it->second.warm;
            if (it->second.wide >= 0) pl->resp_wide = it->second.wide == 1;
            // Grids are clamped to what this plan's working sets and partial slots were sized for:
            // the cache key leaves out the solver choices (environment switches at plan creation)
            // that decide those sizes.
            if (it->second.mshg_grid > 0 && pl->d_mshg_ws)
                pl->mshg_grid = std::min(it->second.mshg_grid, pl->mshg_grid_alloc);
            if (it->second.shg_grid > 0 && pl->shg_grid_alloc > 0)
                pl->shg_grid = std::min(it->second.shg_grid, pl->shg_grid_alloc);
            if (it->second.resp_grid >= 0 && pl->d_resp_scratch)
                pl->resp_gw_grid = std::min(it->second.resp_grid, pl->resp_gw_grid_alloc);
            if (it->second.eigh_grid > 0 && pl->d_eigh_scratch)
                pl->eigh_grid = std::min(it->second.eigh_grid, pl->eigh_grid_alloc);
            apply_omb(pl, it->second.omb);
            if (report) {
                *report = it->second.report;
                report->from_cache = 1;
            }
            return WNLQG_OK;
        }
    }
    wnlqg_autotune_report rep;
    std::memset(&rep, 0, sizeof(rep));
    for (int i = 0; i < 3; ++i) rep.eigh_ms[i] = rep.response_ms[i] = -1.0;
    rep.warm_start = -1;
    rep.start_ms[0] = rep.start_ms[1] = -1.0;
    rep.response_threads = -1;
    rep.width_ms[0] = rep.width_ms[1] = -1.0;
    rep.metric_shg_grid = rep.shg_grid = -1;
    for (int i = 0; i < 3; ++i) rep.metric_shg_grid_ms[i] = rep.shg_grid_ms[i] = -1.0;
    rep.response_grid = rep.eigh_grid = -1;
    for (int i = 0; i < 3; ++i) rep.response_grid_ms[i] = rep.eigh_grid_ms[i] = -1.0;
    if (pl->d_eigh_scratch && pl->eigh_grid_alloc > 0) {
        // Eigensolver stages with per-CTA global working sets: the L2-resident grid, 1 or 2 CTAs per SM.
        const int start = pl->eigh_grid;
        const int cand[3] = {pl->eigh_grid_l2, pl->sm_count, 2 * pl->sm_count};
        double best = std::numeric_limits<double>::infinity(), r = 0;
        for (int i = 0; i < 3; ++i) {
            pl->eigh_grid = std::max(1, std::min(cand[i], pl->eigh_grid_alloc));
            if ((st = tune_measure(pl, mesh, k_begin, k_end, &rep.eigh_grid_ms[i], &r)) != WNLQG_OK) {
                pl->eigh_grid = start;
                return st;
            }
            if (rep.eigh_grid_ms[i] < best) { best = rep.eigh_grid_ms[i]; rep.eigh_grid = pl->eigh_grid; }
        }
        pl->eigh_grid = rep.eigh_grid;
    }
    const int teams[3] = {32, 64, 128}, ombs[3] = {1, 2, 4};
    if (pl->small_f64) {
        // One kernel reads neither the team nor the start: one time stands for every candidate, and the
        // plan keeps its settings.
        double r = 0;
        if ((st = tune_measure(pl, mesh, k_begin, k_end, &rep.eigh_ms[0], &r)) != WNLQG_OK) return st;
        rep.eigh_ms[1] = rep.eigh_ms[2] = rep.start_ms[0] = rep.start_ms[1] = rep.eigh_ms[0];
        rep.eigh_team = pl->eigh_team;
        rep.warm_start = pl->warm_mode;
    } else if (pl->warp_eigh) {
        const int start = pl->eigh_team;
        int best = start;
        double best_ms = std::numeric_limits<double>::infinity(), r = 0;
        for (int i = 0; i < 3; ++i) {
            apply_team(pl, teams[i]);
            if ((st = tune_measure(pl, mesh, k_begin, k_end, &rep.eigh_ms[i], &r)) != WNLQG_OK) {
                apply_team(pl, start);
                return st;
            }
            if (rep.eigh_ms[i] < best_ms) { best_ms = rep.eigh_ms[i]; best = teams[i]; }
        }
        apply_team(pl, best);
        rep.eigh_team = best;
    }
    if ((pl->warp_eigh && !pl->small_f64) || pl->cta_mixed) {
        const int start = pl->warm_mode;
        double r = 0;
        for (int w = 0; w < 2; ++w) {
            pl->warm_mode = w;
            if ((st = tune_measure(pl, mesh, k_begin, k_end, &rep.start_ms[w], &r)) != WNLQG_OK) {
                pl->warm_mode = start;
                return st;
            }
        }
        pl->warm_mode = rep.start_ms[1] <= rep.start_ms[0] ? 1 : 0;
        rep.warm_start = pl->warm_mode;
    }
    bool freq = false;
    for (const Pass &ps : pl->passes) freq |= ps.params.n_fc > 0 && ps.params.nom > 0;
    if (freq) {
        int best = 0;
        double best_ms = std::numeric_limits<double>::infinity(), e = 0;
        for (int i = 0; i < 3; ++i) {
            apply_omb(pl, ombs[i]);
            if ((st = tune_measure(pl, mesh, k_begin, k_end, &e, &rep.response_ms[i])) != WNLQG_OK) {
                apply_omb(pl, 0);
                return st;
            }
            if (rep.response_ms[i] < best_ms) { best_ms = rep.response_ms[i]; best = ombs[i]; }
        }
        apply_omb(pl, best);
        rep.energies_per_thread = best;
    }
    bool widen = false;
    for (const Pass &ps : pl->passes) widen |= ps.grid_wide > 0;
    if (widen) {
        const bool start = pl->resp_wide;
        double e = 0;
        for (int w = 0; w < 2; ++w) {
            pl->resp_wide = w == 1;
            if ((st = tune_measure(pl, mesh, k_begin, k_end, &e, &rep.width_ms[w])) != WNLQG_OK) {
                pl->resp_wide = start;
                return st;
            }
        }
        pl->resp_wide = rep.width_ms[1] < rep.width_ms[0];
        rep.response_threads = pl->resp_wide ? 512 : 256;
    }
    bool gw_pass = false;
    for (const Pass &ps : pl->passes) gw_pass |= ps.global;
    if (gw_pass) {
        // Response passes with per-CTA global working sets: their L2-resident grids, 1 or 2 CTAs per SM.
        const int cand[3] = {0, pl->sm_count, 2 * pl->sm_count};
        double best = std::numeric_limits<double>::infinity(), e = 0;
        for (int i = 0; i < 3; ++i) {
            pl->resp_gw_grid = cand[i];
            if ((st = tune_measure(pl, mesh, k_begin, k_end, &e, &rep.response_grid_ms[i])) != WNLQG_OK) {
                pl->resp_gw_grid = 0;
                return st;
            }
            if (rep.response_grid_ms[i] < best) { best = rep.response_grid_ms[i]; rep.response_grid = cand[i]; }
        }
        pl->resp_gw_grid = rep.response_grid;
    }
    if (pl->metric_shg && !pl->shg.empty()) {
        const int start = pl->mshg_grid;
        const int cand[3] = {pl->sm_count, 2 * pl->sm_count, 4 * pl->sm_count};
        double best = std::numeric_limits<double>::infinity(), e = 0;
        for (int i = 0; i < 3; ++i) {
            pl->mshg_grid = std::min(cand[i], pl->mshg_grid_alloc);
            if ((st = tune_measure(pl, mesh, k_begin, k_end, &e, &rep.metric_shg_grid_ms[i])) != WNLQG_OK) {
                pl->mshg_grid = start;
                return st;
            }
            if (rep.metric_shg_grid_ms[i] < best) { best = rep.metric_shg_grid_ms[i]; rep.metric_shg_grid = pl->mshg_grid; }
        }
        pl->mshg_grid = rep.metric_shg_grid;
    }
    if (pl->shg_global && !pl->shg.empty()) {
        const int start = pl->shg_grid;
        const int cand[3] = {pl->shg_grid_l2, pl->sm_count, 2 * pl->sm_count};
        double best = std::numeric_limits<double>::infinity(), e = 0;
        for (int i = 0; i < 3; ++i) {
            pl->shg_grid = std::max(1, std::min(cand[i], pl->shg_grid_alloc));
            if ((st = tune_measure(pl, mesh, k_begin, k_end, &e, &rep.shg_grid_ms[i])) != WNLQG_OK) {
                pl->shg_grid = start;
                return st;
            }
            if (rep.shg_grid_ms[i] < best) { best = rep.shg_grid_ms[i]; rep.shg_grid = pl->shg_grid; }
        }
        pl->shg_grid = rep.shg_grid;
    }
    {
        std::lock_guard<std::mutex> lock(g_tune_mutex);
        g_tune_cache[key] = TuneChoice{rep.eigh_team, rep.energies_per_thread, rep.warm_start,
                                       rep.response_threads < 0 ? -1 : (rep.response_threads == 512 ? 1 : 0),
                                       rep.metric_shg_grid, rep.shg_grid, rep.response_grid, rep.eigh_grid, rep};
    }
    if (report) *report = rep;
    return WNLQG_OK;
}

// ---------------------------------------------------------------------------------------------
// Allocation-free spectrum entry point.
//
// Some callers cannot let this library call cudaMalloc: applications whose device memory is
// owned by another pool allocator under a hard budget (a Julia CUDA.jl pool, PyTorch's caching
// allocator, a serving process that reserves all HBM up front), where an allocation behind the
// pool's back fails or evicts the pool's own buffers.  wnlqg_b200_spectrum_noalloc serves them:
// the caller passes device inputs and outputs, and the only scratch (phase table and H(k)) lives
// in the fixed file-scope array below, which every GPU that loads the library keeps until exit.
// ---------------------------------------------------------------------------------------------
#define WNLQG_NOALLOC_SCRATCH_BYTES ((size_t)8 << 20)   // 8 MiB per device

static __device__ __align__(256) unsigned char g_noalloc_scratch[WNLQG_NOALLOC_SCRATCH_BYTES];

namespace {
constexpr int kNoallocMaxDevices = 64;
void *g_noalloc_ptr[kNoallocMaxDevices] = {nullptr};
std::mutex g_noalloc_mutex;

// Device address of the scratch array on the current device, looked up once per device.  In
// host code the array's name is only a host-side stand-in, never a device address.
wnlqg_status noalloc_scratch(int device, void **out) {
    if (device < 0 || device >= kNoallocMaxDevices) return fail(WNLQG_ERR_UNSUPPORTED, "device index too large");
    std::lock_guard<std::mutex> lock(g_noalloc_mutex);
    if (!g_noalloc_ptr[device]) {
        void *ptr = nullptr;
        cudaError_t e = cudaGetSymbolAddress(&ptr, g_noalloc_scratch);
        if (e != cudaSuccess || !ptr)
            return fail(WNLQG_ERR_CUDA, std::string("cudaGetSymbolAddress(scratch): ") + cudaGetErrorString(e));
        g_noalloc_ptr[device] = ptr;
    }
    *out = g_noalloc_ptr[device];
    return WNLQG_OK;
}
}  // namespace

extern "C" wnlqg_status wnlqg_b200_spectrum_noalloc(int64_t num_orbitals, int64_t num_r_vectors,
                                                    const double *hamiltonian_r, const int64_t *r_vectors,
                                                    const int64_t *r_degeneracies, const double *kpoints,
                                                    int64_t n, double *energies, double *eigenvectors,
                                                    void *stream) {
    if (num_orbitals <= 0 || num_orbitals > 32 || num_r_vectors <= 0)
        return fail(WNLQG_ERR_UNSUPPORTED, "spectrum_noalloc supports 1 <= num_orbitals <= 32 and num_r_vectors >= 1");
    if (n < 0) return fail(WNLQG_ERR_INVALID_ARGUMENT, "negative point count");
    if (n == 0) return WNLQG_OK;
    if (!hamiltonian_r || !r_vectors || !r_degeneracies || !kpoints || !energies || !eigenvectors)
        return fail(WNLQG_ERR_INVALID_ARGUMENT, "NULL device pointer");
    const int nw = (int)num_orbitals, nr = (int)num_r_vectors;
    const int64_t nn = (int64_t)nw * nw;
    // Scratch: phase table [n][NR] then H(k) [n][nw*nw], complex double, 256-byte aligned parts.
    // The point count is bounded by a division first, so no product below can wrap around.
    const size_t per_point = (size_t)(nr + nn) * sizeof(double2);
    const size_t max_points = (WNLQG_NOALLOC_SCRATCH_BYTES - 256) / per_point;
    const std::string too_many = "spectrum_noalloc: n*(NR + nw^2)*16 bytes exceeds the 8 MiB scratch; pass fewer points "
                                 "per call (at most " + std::to_string(max_points) + ")";
    if ((uint64_t)n > (uint64_t)max_points) return fail(WNLQG_ERR_INVALID_ARGUMENT, too_many);
    const size_t phase_bytes = (((size_t)n * nr * sizeof(double2)) + 255) & ~(size_t)255;
    const size_t hk_bytes = (size_t)n * nn * sizeof(double2);
    if (phase_bytes + hk_bytes > WNLQG_NOALLOC_SCRATCH_BYTES) return fail(WNLQG_ERR_INVALID_ARGUMENT, too_many);
    int device = 0;
    WNLQG_CUDA(cudaGetDevice(&device));
    void *scratch = nullptr;
    wnlqg_status st = noalloc_scratch(device, &scratch);
    if (st != WNLQG_OK) return st;
    double2 *phases = reinterpret_cast<double2 *>(scratch);
    double2 *hk = reinterpret_cast<double2 *>(static_cast<unsigned char *>(scratch) + phase_bytes);
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const int64_t total = n * nr;
    const int blocks = (int)std::min<int64_t>((total + 255) / 256, 148 * 32);
    // Every scratch element is overwritten before it is read, so nothing needs clearing.
    phase_kernel<<<blocks, 256, 0, s>>>(phases, r_vectors, r_degeneracies, nr, n, 0, 1, 1, 1, kpoints);
    dim3 grid((unsigned)((nn + FG_BN - 1) / FG_BN), (unsigned)((n + FG_BM - 1) / FG_BM));
    fourier_gemm_f64<<<grid, 256, 0, s>>>(phases, reinterpret_cast<const double2 *>(hamiltonian_r), hk, n, nn, nr);
    jacobi_eigh_kernel<double><<<(unsigned)n, eigh_block_threads(nw), EighSmem::bytes(nw, sizeof(double2)), s>>>(
        hk, nn, n, nw, energies, reinterpret_cast<double2 *>(eigenvectors), 8.673617379884035e-19);
    WNLQG_CUDA(cudaGetLastError());
    return WNLQG_OK;
}

// ---------------------------------------------------------------------------------------------
// Refinement-proposer MLP (no counterpart in the reference; it only ranks cells for refinement).
// ---------------------------------------------------------------------------------------------
#include "mlp.cuh"

struct wnlqg_mlp {
    int device = 0;
    float *d_master = nullptr, *d_m = nullptr, *d_v = nullptr, *d_grad = nullptr, *d_partial = nullptr;
    __nv_bfloat16 *d_wb = nullptr;
    float *d_x = nullptr, *d_y = nullptr, *d_out = nullptr;
    int64_t cap = 0;
    int slots = 0;
    int64_t step = 0;
    cudaStream_t stream = nullptr;
};

namespace {
wnlqg_status mlp_reserve(wnlqg_mlp *m, int64_t n) {
    if (n <= m->cap) return WNLQG_OK;
    cudaFree(m->d_x);
    cudaFree(m->d_y);
    cudaFree(m->d_out);
    m->d_x = m->d_y = m->d_out = nullptr;
    m->cap = 0;
    WNLQG_CUDA(cudaMalloc(&m->d_x, (size_t)n * MLP_F * sizeof(float)));
    WNLQG_CUDA(cudaMalloc(&m->d_y, (size_t)n * sizeof(float)));
    WNLQG_CUDA(cudaMalloc(&m->d_out, (size_t)n * sizeof(float)));
    m->cap = n;
    return WNLQG_OK;
}

int mlp_grid(int64_t n, int maxslots) {
    return (int)std::max<int64_t>(1, std::min<int64_t>((n + MLP_TILE - 1) / MLP_TILE, maxslots));
}

wnlqg_status mlp_loss_grad_device(wnlqg_mlp *m, int64_t n) {
    const int grid = mlp_grid(n, m->slots);
    mlp_backward_kernel<<<grid, MLP_H, 0, m->stream>>>(m->d_wb, m->d_master, m->d_x, m->d_y, n, m->d_partial);
    mlp_reduce_kernel<<<(MlpLayout::COUNT + 256) / 256, 256, 0, m->stream>>>(m->d_partial, grid, m->d_grad);
    WNLQG_CUDA(cudaGetLastError());
    return WNLQG_OK;
}
}  // namespace

extern "C" int64_t wnlqg_b200_mlp_param_count(void) { return MlpLayout::COUNT; }

extern "C" wnlqg_status wnlqg_b200_mlp_create(int32_t device, uint64_t seed, wnlqg_mlp **out) {
    if (!out) return fail(WNLQG_ERR_INVALID_ARGUMENT, "NULL argument");
    *out = nullptr;
    WNLQG_CUDA(cudaSetDevice(device));
    wnlqg_mlp *m = new wnlqg_mlp();
    m->device = device;
    m->slots = 148 * 4;
    // Glorot-uniform weights from a seeded 64-bit LCG, zero biases.
    std::vector<float> p(MlpLayout::COUNT, 0.0f);
    uint64_t state = seed * 6364136223846793005ULL + 1442695040888963407ULL;
    auto uni = [&]() {
        state = state * 6364136223846793005ULL + 1442695040888963407ULL;
        return (double)(state >> 11) * (1.0 / 9007199254740992.0);
    };
    auto fill = [&](int off, int fan_out, int fan_in) {
        const double lim = std::sqrt(6.0 / (fan_in + fan_out));
        for (int i = 0; i < fan_out * fan_in; ++i) p[off + i] = (float)((2.0 * uni() - 1.0) * lim);
    };
    fill(MlpLayout::W1, MLP_H, MLP_F);
    fill(MlpLayout::W2, MLP_H, MLP_H);
    fill(MlpLayout::W3, MLP_H, MLP_H);
    fill(MlpLayout::W4, 1, MLP_H);
    auto cleanup = [&]() {
        cudaFree(m->d_master); cudaFree(m->d_m); cudaFree(m->d_v); cudaFree(m->d_grad);
        cudaFree(m->d_partial); cudaFree(m->d_wb);
        delete m;
    };
    const size_t pb = (size_t)MlpLayout::COUNT * sizeof(float);
    if (cudaMalloc(&m->d_master, pb) != cudaSuccess || cudaMalloc(&m->d_m, pb) != cudaSuccess ||
        cudaMalloc(&m->d_v, pb) != cudaSuccess || cudaMalloc(&m->d_grad, pb + sizeof(float)) != cudaSuccess ||
        cudaMalloc(&m->d_partial, (size_t)m->slots * (MlpLayout::COUNT + 1) * sizeof(float)) != cudaSuccess ||
        cudaMalloc(&m->d_wb, (size_t)MlpLayout::COUNT * sizeof(__nv_bfloat16)) != cudaSuccess) {
        cudaGetLastError();
        cleanup();
        return fail(WNLQG_ERR_OUT_OF_MEMORY, "cudaMalloc failed for the MLP");
    }
    if (cudaStreamCreateWithFlags(&m->stream, cudaStreamNonBlocking) != cudaSuccess) {
        cleanup();
        return fail(WNLQG_ERR_CUDA, "cudaStreamCreate failed");
    }
    WNLQG_CUDA(cudaMemcpy(m->d_master, p.data(), pb, cudaMemcpyHostToDevice));
    WNLQG_CUDA(cudaMemset(m->d_m, 0, pb));
    WNLQG_CUDA(cudaMemset(m->d_v, 0, pb));
    mlp_to_bf16_kernel<<<(MlpLayout::COUNT + 255) / 256, 256, 0, m->stream>>>(m->d_master, m->d_wb, MlpLayout::COUNT);
    WNLQG_CUDA(cudaStreamSynchronize(m->stream));
    *out = m;
    return WNLQG_OK;
}

extern "C" wnlqg_status wnlqg_b200_mlp_destroy(wnlqg_mlp *m) {
    if (!m) return WNLQG_OK;
    cudaSetDevice(m->device);
    if (m->stream) cudaStreamSynchronize(m->stream);
    for (void *ptr : {(void *)m->d_master, (void *)m->d_m, (void *)m->d_v, (void *)m->d_grad, (void *)m->d_partial,
                      (void *)m->d_wb, (void *)m->d_x, (void *)m->d_y, (void *)m->d_out})
        if (ptr) cudaFree(ptr);
    if (m->stream) cudaStreamDestroy(m->stream);
    delete m;
    return WNLQG_OK;
}

extern "C" wnlqg_status wnlqg_b200_mlp_get_params(wnlqg_mlp *m, float *params) {
    if (!m || !params) return fail(WNLQG_ERR_INVALID_ARGUMENT, "NULL argument");
    WNLQG_CUDA(cudaSetDevice(m->device));
    WNLQG_CUDA(cudaMemcpyAsync(params, m->d_master, (size_t)MlpLayout::COUNT * sizeof(float), cudaMemcpyDeviceToHost,
                               m->stream));
    WNLQG_CUDA(cudaStreamSynchronize(m->stream));
    return WNLQG_OK;
}

extern "C" wnlqg_status wnlqg_b200_mlp_set_params(wnlqg_mlp *m, const float *params) {
    if (!m || !params) return fail(WNLQG_ERR_INVALID_ARGUMENT, "NULL argument");
    for (int i = 0; i < MlpLayout::COUNT; ++i)
        if (!std::isfinite(params[i])) return fail(WNLQG_ERR_NONFINITE, "parameters must be finite");
    WNLQG_CUDA(cudaSetDevice(m->device));
    WNLQG_CUDA(cudaMemcpyAsync(m->d_master, params, (size_t)MlpLayout::COUNT * sizeof(float), cudaMemcpyHostToDevice,
                               m->stream));
    mlp_to_bf16_kernel<<<(MlpLayout::COUNT + 255) / 256, 256, 0, m->stream>>>(m->d_master, m->d_wb, MlpLayout::COUNT);
    WNLQG_CUDA(cudaStreamSynchronize(m->stream));
    return WNLQG_OK;
}

extern "C" wnlqg_status wnlqg_b200_mlp_forward(wnlqg_mlp *m, const float *x, int64_t n, float *y) {
    if (!m || n < 0 || (n > 0 && (!x || !y))) return fail(WNLQG_ERR_INVALID_ARGUMENT, "invalid arguments");
    if (n == 0) return WNLQG_OK;
    WNLQG_CUDA(cudaSetDevice(m->device));
    wnlqg_status st = mlp_reserve(m, n);
    if (st != WNLQG_OK) return st;
    WNLQG_CUDA(cudaMemcpyAsync(m->d_x, x, (size_t)n * MLP_F * sizeof(float), cudaMemcpyHostToDevice, m->stream));
    mlp_forward_kernel<<<mlp_grid(n, 148 * 8), MLP_H, 0, m->stream>>>(m->d_wb, m->d_master, m->d_x, n, m->d_out);
    WNLQG_CUDA(cudaGetLastError());
    WNLQG_CUDA(cudaMemcpyAsync(y, m->d_out, (size_t)n * sizeof(float), cudaMemcpyDeviceToHost, m->stream));
    WNLQG_CUDA(cudaStreamSynchronize(m->stream));
    return WNLQG_OK;
}

extern "C" wnlqg_status wnlqg_b200_mlp_loss_grad(wnlqg_mlp *m, const float *x, const float *target, int64_t n,
                                                 float *loss, float *grad) {
    if (!m || n <= 0 || !x || !target) return fail(WNLQG_ERR_INVALID_ARGUMENT, "invalid arguments");
    WNLQG_CUDA(cudaSetDevice(m->device));
    wnlqg_status st = mlp_reserve(m, n);
    if (st != WNLQG_OK) return st;
    WNLQG_CUDA(cudaMemcpyAsync(m->d_x, x, (size_t)n * MLP_F * sizeof(float), cudaMemcpyHostToDevice, m->stream));
    WNLQG_CUDA(cudaMemcpyAsync(m->d_y, target, (size_t)n * sizeof(float), cudaMemcpyHostToDevice, m->stream));
    if ((st = mlp_loss_grad_device(m, n)) != WNLQG_OK) return st;
    std::vector<float> g(MlpLayout::COUNT + 1);
    WNLQG_CUDA(cudaMemcpyAsync(g.data(), m->d_grad, g.size() * sizeof(float), cudaMemcpyDeviceToHost, m->stream));
    WNLQG_CUDA(cudaStreamSynchronize(m->stream));
    if (loss) *loss = g[MlpLayout::COUNT];
    if (grad) std::memcpy(grad, g.data(), (size_t)MlpLayout::COUNT * sizeof(float));
    return WNLQG_OK;
}

extern "C" wnlqg_status wnlqg_b200_mlp_train(wnlqg_mlp *m, const float *x, const float *target, int64_t n,
                                             int32_t steps, float lr, float *final_loss) {
    if (!m || n <= 0 || !x || !target || steps < 0 || !(lr > 0))
        return fail(WNLQG_ERR_INVALID_ARGUMENT, "invalid arguments");
    WNLQG_CUDA(cudaSetDevice(m->device));
    wnlqg_status st = mlp_reserve(m, n);
    if (st != WNLQG_OK) return st;
    WNLQG_CUDA(cudaMemcpyAsync(m->d_x, x, (size_t)n * MLP_F * sizeof(float), cudaMemcpyHostToDevice, m->stream));
    WNLQG_CUDA(cudaMemcpyAsync(m->d_y, target, (size_t)n * sizeof(float), cudaMemcpyHostToDevice, m->stream));
    const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
    for (int s = 0; s < steps; ++s) {
        if ((st = mlp_loss_grad_device(m, n)) != WNLQG_OK) return st;
        m->step += 1;
        const float bc1 = 1.0f - std::pow(b1, (float)m->step), bc2 = 1.0f - std::pow(b2, (float)m->step);
        mlp_adam_kernel<<<(MlpLayout::COUNT + 255) / 256, 256, 0, m->stream>>>(m->d_master, m->d_grad, m->d_m, m->d_v,
                                                                               m->d_wb, lr, b1, b2, eps, bc1, bc2);
    }
    WNLQG_CUDA(cudaGetLastError());
    if (final_loss) {
        if ((st = mlp_loss_grad_device(m, n)) != WNLQG_OK) return st;
        float l = 0.f;
        WNLQG_CUDA(cudaMemcpyAsync(&l, m->d_grad + MlpLayout::COUNT, sizeof(float), cudaMemcpyDeviceToHost, m->stream));
        WNLQG_CUDA(cudaStreamSynchronize(m->stream));
        *final_loss = l;
    }
    WNLQG_CUDA(cudaStreamSynchronize(m->stream));
    return WNLQG_OK;
}

// ---- measured arithmetic peaks ----------------------------------------------------------------
namespace {

// Each warp keeps 8 independent DMMA accumulator pairs; every iteration issues one m8n8k4 per
// pair (512 FLOP per warp each).  The operands drift with the accumulators so nothing is hoisted.
__global__ void __launch_bounds__(256) peak_dmma_kernel(int iters, double *out) {
    double acc[8][2];
#pragma unroll
    for (int q = 0; q < 8; ++q) { acc[q][0] = 1e-3 * q; acc[q][1] = 2e-3 * q; }
    double a = 1.0 + 1e-9 * threadIdx.x, b = 1.0 - 1e-9 * blockIdx.x;
    for (int it = 0; it < iters; ++it) {
#pragma unroll
        for (int q = 0; q < 8; ++q) dmma_m8n8k4(acc[q][0], acc[q][1], a, b);
        a = a * 0.999999999 + 1e-12;
    }
    double s = 0.0;
#pragma unroll
    for (int q = 0; q < 8; ++q) s += acc[q][0] + acc[q][1];
    if (s == 123.456) out[0] = s;   // keeps the chains live; never true for these inputs
}

template <typename T>
__global__ void __launch_bounds__(256) peak_fma_kernel(int iters, T *out) {
    T acc[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) acc[q] = (T)(1e-3 * (q + threadIdx.x));
    const T a = (T)(1.0 - 1e-7 * blockIdx.x), b = (T)1e-7;
    for (int it = 0; it < iters; ++it) {
#pragma unroll
        for (int q = 0; q < 8; ++q) acc[q] = fma(acc[q], a, b);
    }
    T s = 0;
#pragma unroll
    for (int q = 0; q < 8; ++q) s += acc[q];
    if (s == (T)123.456) out[0] = s;
}

}  // namespace

extern "C" wnlqg_status wnlqg_b200_measure_peaks(int32_t device, double *fp64_dmma_tflops, double *fp64_fma_tflops,
                                                 double *fp32_fma_tflops) {
    if (!fp64_dmma_tflops || !fp64_fma_tflops || !fp32_fma_tflops) return fail(WNLQG_ERR_INVALID_ARGUMENT, "NULL argument");
    WNLQG_CUDA(cudaSetDevice(device));
    int sms = 148;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    double *scratch = nullptr;
    WNLQG_CUDA(cudaMalloc(&scratch, 64));
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    const int blocks = sms * 8, threads = 256;
    auto time_ms = [&](auto launch) {
        launch();   // warm-up
        cudaEventRecord(e0);
        launch();
        cudaEventRecord(e1);
        cudaEventSynchronize(e1);
        float ms = 0.0f;
        cudaEventElapsedTime(&ms, e0, e1);
        return (double)ms;
    };
    const int it_dmma = 4096, it_fma = 16384;
    const double t_dmma = time_ms([&] { peak_dmma_kernel<<<blocks, threads>>>(it_dmma, scratch); });
    const double t_f64 = time_ms([&] { peak_fma_kernel<double><<<blocks, threads>>>(it_fma, scratch); });
    const double t_f32 = time_ms([&] { peak_fma_kernel<float><<<blocks, threads>>>(it_fma, reinterpret_cast<float *>(scratch)); });
    cudaError_t err = cudaGetLastError();
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    cudaFree(scratch);
    if (err != cudaSuccess) return fail(WNLQG_ERR_CUDA, std::string("peak probe: ") + cudaGetErrorString(err));
    const double warps = (double)blocks * threads / 32.0, thr = (double)blocks * threads;
    *fp64_dmma_tflops = warps * it_dmma * 8.0 * 512.0 / (t_dmma * 1e-3) / 1e12;
    *fp64_fma_tflops = thr * it_fma * 8.0 * 2.0 / (t_f64 * 1e-3) / 1e12;
    *fp32_fma_tflops = thr * it_fma * 8.0 * 2.0 / (t_f32 * 1e-3) / 1e12;
    return WNLQG_OK;
}

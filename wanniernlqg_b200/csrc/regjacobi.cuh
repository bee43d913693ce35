// regjacobi.cuh - FP64 Hermitian Jacobi with the matrix in registers, for orders up to 16: one group of
// lanes per matrix, lane i holding row i of A and of the eigenvectors V.
//
// The rounds are those of the shared-memory sweeps (eigh.cuh): the circle method pairs the np indices
// (np even), and A <- J^H A J, V <- V J per round.  Columns are kept in slots: slot 0 holds index 0,
// slot s >= 1 index ((s - 1 + round) mod (np - 1)) + 1, and the pair k of a round is slots k and
// np - 1 - k, so that every register index is static; after each round the contents of slots
// 1 .. np - 1 move down by one.  A round is
//   - the rotation of each pair, computed by the two lanes that own its rows (the diagonal is kept in
//     one register per lane, the pair's element is selected from the row by its slot) and passed to the
//     other lanes through shared memory (np / 2 broadcast reads);
//   - the column rotations of A and V, lane-local;
//   - the row rotations of A: each lane exchanges its row with its partner's by shuffles.
// There is no barrier beyond __syncwarp, and shared memory carries the np / 2 rotations only; the
// shared-memory form moved both matrices through it twice per round, with two block barriers.
// A warp holds two groups of 16 lanes (np <= 8: four of 8, np <= 4: eight of 4).
#pragma once
#include "common.cuh"

template <int NP> struct RegGroup {
    static_assert(NP >= 2 && NP <= 32 && NP % 2 == 0, "even orders up to 32");
    static constexpr int LANES = NP <= 4 ? 4 : (NP <= 8 ? 8 : (NP <= 16 ? 16 : 32));
    static constexpr int PER_WARP = 32 / LANES;
    static WNLQG_D int lane() { return threadIdx.x & (LANES - 1); }
    static WNLQG_D int group() { return (threadIdx.x & 31) / LANES; }
    template <typename T> static WNLQG_D T from(T v, int src) { return __shfl_sync(0xffffffffu, v, src, LANES); }
    template <typename T> static WNLQG_D T sum(T v) {
#pragma unroll
        for (int o = LANES / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o, LANES);
        return v;
    }
    // Whether v holds in any lane of this lane's group.
    static WNLQG_D bool any(bool v) {
        const unsigned m = __ballot_sync(0xffffffffu, v);
        return ((m >> (group() * LANES)) & (LANES == 32 ? 0xffffffffu : (1u << (LANES & 31)) - 1u)) != 0;
    }
};

struct alignas(16) RegRot { double c, sx, sy, pad; };

// out = a[sel], 0 <= sel < N, by a tree of selects (static register indices).
template <int N> WNLQG_D double2 reg_select(const double2 *a, int sel) {
    double2 t[N];
#pragma unroll
    for (int j = 0; j < N; ++j) t[j] = a[j];
    int n = N;
#pragma unroll
    for (int bit = 1; bit < N; bit <<= 1) {
        const bool odd = sel & bit;
        const int m = (n + 1) / 2;
#pragma unroll
        for (int j = 0; j < m; ++j) {
            if (2 * j + 1 < n) {
                t[j].x = odd ? t[2 * j + 1].x : t[2 * j].x;
                t[j].y = odd ? t[2 * j + 1].y : t[2 * j].y;
            } else {
                t[j] = t[2 * j];
            }
        }
        n = m;
    }
    return t[0];
}

// One sweep (NP - 1 rounds) of the group's matrix: a, v rows of A and V, d the diagonal element of
// this lane's index.  Elements with |a_pq| <= tol are left.  rot: 2 x NP / 2 rotations of the group's
// shared memory.  Slot s holds index s at entry and exit.  Returns whether the group rotated.
template <int NP>
WNLQG_D bool reg_jacobi_sweep(double2 (&a)[NP], double2 (&v)[NP], double &d, double tol, RegRot *rot) {
    typedef RegGroup<NP> G;
    constexpr int H = NP / 2;
    const int i = G::lane();
    const bool active = i < NP;
    int pos = active ? i : 0;   // slot of this lane's index
    bool rotated = false;
#pragma unroll 1
    for (int round = 0; round < NP - 1; ++round) {
        const int ps = NP - 1 - pos;   // the partner's slot and index
        int partner = ps - 1 + round;
        if (partner >= NP - 1) partner -= NP - 1;
        partner = ps == 0 ? 0 : partner + 1;
        if (!active) partner = i;
        const bool upper = pos >= H;
        // beta = A[upper index, lower index] from the upper lane's row.
        const double2 own = reg_select<H>(a, upper ? ps : 0);
        double2 beta;
        beta.x = G::from(own.x, partner);
        beta.y = G::from(own.y, partner);
        if (upper) beta = own;
        const double dp = G::from(d, partner);
        const double g2 = beta.x * beta.x + beta.y * beta.y;
        double c = 1.0;
        double2 s = make_double2(0.0, 0.0);   // x' = c x - conj(s) y, y' = s x + c y for the lower slot x and the upper y
        if (active && g2 > tol * tol) {
            const double ginv = rsqrt(g2);
            const double theta = (upper ? d - dp : dp - d) * (0.5 * ginv);
            const double tt = copysign(1.0 / (fabs(theta) + sqrt(theta * theta + 1.0)), theta);
            c = rsqrt(tt * tt + 1.0);
            const double sg = tt * c * ginv;
            s.x = sg * beta.x;
            s.y = -sg * beta.y;
            const double shift = tt * (g2 * ginv);
            d += upper ? shift : -shift;
            rotated = true;
        }
        RegRot *r = rot + (round & 1) * H;
        if (active && !upper) {
            RegRot q;
            q.c = c; q.sx = s.x; q.sy = s.y; q.pad = 0.0;
            r[pos] = q;
        }
        __syncwarp();
        auto columns = [&](double2 &x, double2 &y, const RegRot &q) {
            const double2 x0 = x, y0 = y;
            x.x = fma(-q.sy, y0.y, fma(-q.sx, y0.x, q.c * x0.x));
            x.y = fma(q.sy, y0.x, fma(-q.sx, y0.y, q.c * x0.y));
            y.x = fma(-q.sy, x0.y, fma(q.sx, x0.x, q.c * y0.x));
            y.y = fma(q.sy, x0.x, fma(q.sx, x0.y, q.c * y0.y));
        };
#pragma unroll
        for (int k = 0; k < H; ++k) {
            const RegRot q = r[k];
            columns(a[k], a[NP - 1 - k], q);
            columns(v[k], v[NP - 1 - k], q);
        }
        // Row rotation: lower row <- c own - s partner, upper row <- c own + conj(s) partner.
        const double wx = upper ? s.x : -s.x, wy = -s.y;
#pragma unroll
        for (int j = 0; j < NP; ++j) {
            const double px = G::from(a[j].x, partner), py = G::from(a[j].y, partner);
            a[j].x = fma(-wy, py, fma(wx, px, c * a[j].x));
            a[j].y = fma(wy, px, fma(wx, py, c * a[j].y));
        }
        if constexpr (NP > 2) {
            const double2 a1 = a[1], v1 = v[1];
#pragma unroll
            for (int j = 1; j < NP - 1; ++j) { a[j] = a[j + 1]; v[j] = v[j + 1]; }
            a[NP - 1] = a1;
            v[NP - 1] = v1;
            if (active && i > 0) pos = pos == 1 ? NP - 1 : pos - 1;
        }
    }
    return G::any(rotated);
}

// Squared off-diagonal norm of the group's matrix (slot s holding index s).
template <int NP> WNLQG_D double reg_offdiag2(const double2 (&a)[NP]) {
    const int i = RegGroup<NP>::lane();
    double s = 0.0;
#pragma unroll
    for (int j = 0; j < NP; ++j) s += j == i ? 0.0 : a[j].x * a[j].x + a[j].y * a[j].y;
    return RegGroup<NP>::sum(i < NP ? s : 0.0);
}

// Shared memory of one group: a matrix of NP rows of LD complex entries (16-byte rows), rotations.
template <int NP> struct RegSmem {
    static constexpr int LD = NP + 2;
    double2 m[NP * LD];
    RegRot rot[NP];
};

// Upper triangle of a stored Hermitian matrix into shared rows S[i * LD + j] (lower = conjugate, real
// diagonal, zeros beyond nw), here in FP64 and in FP32 for the one-sided stage (onesided.cuh); valid = 0
// stores zeros.  Closes with __syncwarp.
template <typename T, int NP>
WNLQG_D void reg_stage_hermitian(typename cplx_of<T>::type *S, const double2 *__restrict__ h, int nw, bool valid) {
    typedef typename cplx_of<T>::type C;
    constexpr int LD = NP + 2;
    const int i = RegGroup<NP>::lane();
    if (i < NP)
#pragma unroll 4
        for (int j = 0; j < NP; ++j) {
            if (j < i) continue;
            double2 x = make_double2(0.0, 0.0);
            if (valid && i < nw && j < nw) x = h[i + (int64_t)nw * j];
            if (i == j) x.y = 0.0;
            const C z = from_c64<C>(x);
            S[i * LD + j] = z;
            if (i != j) S[j * LD + i] = cconj(z);
        }
    __syncwarp();
}

// FP64 spectrum of orthogonal models up to 16 orbitals, FP64 Jacobi from the identity to the FP64 CTA
// Jacobi's stopping rule (off-diagonal norm <= np 2^-60 ||H||, or a sweep with every |a_pq| <=
// 2^-60 ||H||), ascending order and canonical phases (jacobi_eigh_kernel).  Group g of the grid takes
// the points g, g + groups, ...; no point depends on another, so nothing is gained by ordering them.
// Blocks of 128 threads.  One kernel in place of an FP32 stage and an FP64 refinement of one warp per
// matrix: 4 orbitals on a 32^3 mesh, the whole call 1.66 -> 0.56 ms (1.15 of it the two stages);
// 33 points, 187 -> 140 us with the ordering that is no longer needed.
template <int NP>
__global__ void __launch_bounds__(128, NP > 8 ? 2 : 3) jacobi_f64_reg_kernel(
    const double2 *__restrict__ h_in, int64_t h_stride, int64_t batch, int nw, double *__restrict__ E_out,
    double2 *__restrict__ U_out) {
    typedef RegGroup<NP> G;
    typedef RegSmem<NP> Smem;
    constexpr int LD = Smem::LD;
    extern __shared__ __align__(16) unsigned char reg_smem_raw[];
    Smem &sm = reinterpret_cast<Smem *>(reg_smem_raw)[threadIdx.x / G::LANES];
    double2 *S = sm.m;
    const int i = G::lane(), ic = min(i, NP - 1);
    const int64_t groups = (int64_t)gridDim.x * blockDim.x / G::LANES;
    const int64_t g = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / G::LANES;
    double2 a[NP], v[NP];
    for (int64_t b0 = g - G::group(); b0 < batch; b0 += groups) {   // uniform over the warp
        const int64_t b = b0 + G::group();
        const bool valid = b < batch;
        reg_stage_hermitian<double, NP>(S, h_in + (valid ? b : 0) * h_stride, nw, valid);
        double f2 = 0.0, d = 0.0;
#pragma unroll
        for (int j = 0; j < NP; ++j) {
            a[j] = S[ic * LD + j];
            f2 += a[j].x * a[j].x + a[j].y * a[j].y;
            if (j == i) d = a[j].x;
            v[j] = make_double2(j == i ? 1.0 : 0.0, 0.0);
        }
        const double fro = sqrt(G::sum(i < NP ? f2 : 0.0));
        double tol = fro * 8.673617379884035e-19;
        const double stop = tol * NP;
        bool done = !valid;
        for (int sweep = 0; sweep < 30; ++sweep) {
            const double off = sqrt(reg_offdiag2<NP>(a));   // every lane takes the shuffles
            done = done || off <= stop;
            if (__all_sync(0xffffffffu, done)) break;
            if (done) tol = 1.0e150;   // nothing rotates
            const bool any = reg_jacobi_sweep<NP>(a, v, d, tol, sm.rot);
            done = done || !any;
        }
        // Lane i: rank of eigenvalue i (ascending, ties in index order), pivot and phase of its column.
        int rank = 0;
#pragma unroll
        for (int j = 0; j < NP; ++j) {
            const double dj = G::from(d, j);
            if (j < nw) rank += (dj < d) || (dj == d && j < i);
        }
        __syncwarp();
        if (i < NP)
#pragma unroll
            for (int j = 0; j < NP; ++j) S[i * LD + j] = v[j];
        __syncwarp();
        double2 phase = make_double2(1.0, 0.0);
        {
            int pivot = 0;
            double pm = hypot(S[ic].x, S[ic].y);
            for (int r = 1; r < nw; ++r) {
                const double mg = hypot(S[r * LD + ic].x, S[r * LD + ic].y);
                if (mg > pm) { pm = mg; pivot = r; }
            }
            if (pm > 0.0) phase = make_double2(S[pivot * LD + ic].x / pm, -S[pivot * LD + ic].y / pm);
        }
        if (valid && i < nw) E_out[b * nw + rank] = d;
        double2 *u = U_out + (valid ? b : 0) * (int64_t)nw * nw;
#pragma unroll
        for (int j = 0; j < NP; ++j) {
            const int rj = G::from(rank, j);
            const double2 pj = make_double2(G::from(phase.x, j), G::from(phase.y, j));
            if (valid && i < nw && j < nw) u[i + (int64_t)nw * rj] = cmul(v[j], pj);
        }
        __syncwarp();
    }
}

// Kernel and group shared memory of an even order np.
struct RegKernel {
    const void *fn;
    size_t group_smem;
    int lanes;
};
template <int NP> RegKernel reg_f64_entry() {
    return {(const void *)jacobi_f64_reg_kernel<NP>, sizeof(RegSmem<NP>), RegGroup<NP>::LANES};
}
inline RegKernel reg_f64_kernel(int np) {
    static const RegKernel k[8] = {reg_f64_entry<2>(),  reg_f64_entry<4>(),  reg_f64_entry<6>(),  reg_f64_entry<8>(),
                                   reg_f64_entry<10>(), reg_f64_entry<12>(), reg_f64_entry<14>(), reg_f64_entry<16>()};
    return k[np / 2 - 1];
}

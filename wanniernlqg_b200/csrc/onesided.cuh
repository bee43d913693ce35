// onesided.cuh - FP32 first stage of the FP64 path's eigensolver above 16 orbitals: one-sided Jacobi.
//
// For a Hermitian H and a shift c > ||H||, the columns of G = (H + c I) V are rotated in pairs until they
// are orthogonal; then G = U S with S = diag(lambda + c) > 0, so the normalised columns are H's
// eigenvectors (the method of Hestenes, applied to a definite shift of H).  A pair (x, y) is
// orthogonalised by the rotation that diagonalises its Gram matrix [n_x, a; conj(a), n_y],
// a = x^H y: x' = c x - conj(s) y, y' = s x + c y.  Only G is read, rotated and written: against the
// two-sided sweeps (rows and columns of A, columns of V) that is a quarter of the traffic, and the
// start from a neighbouring point's V takes one product instead of four.
//   - H is scaled by a power of two to a Frobenius norm in [1/2, 1), so no square leaves the FP32 range.
//   - A sweep is the last when no pair above the rounding level (cosine 2^-20) turned by more than
//     an angle: convergence is quadratic, but what the last sweep leaves adds up over the columns.
//     With every pair just below 2^-10, as between neighbours of a dense mesh, ||V^H V - 1|| came to
//     3e-5 (32 orbitals) and 9e-5 (128), of which the FP64 stage's second-order orthonormalisation
//     leaves 1e-14 and 1e-13, and ratios a_ij / (d_i - d_j) to 3e-4 and 1e-3, which its first completion
//     refuses.  2^-11 up to 32 orbitals and 2^-12 above leave at most 8e-6 (3e-16 after the FP64 stage)
//     and ratios below 1e-4.
//   - The angle left by rounding is about 2^-24 (lambda + c) / (difference of two levels), so a tighter
//     c is a more accurate start.  A cold start takes c = 1.1 ||H||_F, a warm one 1.3 max |lambda| of
//     the columns it starts from (in the present point's scaling); above 32 orbitals a start with a
//     loose c (a cold one, or max |lambda| fell along the chain) is followed by one from its own vectors.
//   - The start V has to be orthonormal (G G^H = (H + c I)^2): it always is a converged one.
//   - H + c I has to be definite: of an indefinite one the lengths are |lambda + c|, and two levels of
//     equal length mix.  H may have moved beyond the shift along a chain, so a warm point is accepted
//     only if no column is shorter than 0.05 c and the lengths sum to tr(H + c I) within 0.05 c (a
//     level below -c would add twice its length); else it is started cold.
// On random spectra the vectors are otherwise orthonormal to 4e-7 (18 orbitals) to 1.2e-6 (128), ratios
// 3e-6 to 7e-5: below the 2^-13 that the FP64 stage's first completion asks for.
// Measured against the two-sided stage: 32 orbitals, 32768 points of a 256^3 mesh, 6.9 -> 2.5 ms; 96
// orbitals, 2048 points, 44.4 -> 6.1 ms (and the FP64 stage, which no longer needs a sweep before its
// completion, 32.5 -> 10.2 ms).
#pragma once
#include "common.cuh"
#include "regjacobi.cuh"

#define OS_ANGLE_WARP 4.8828125e-04f      // 2^-11
#define OS_ANGLE_CTA 2.44140625e-04f      // 2^-12
#define OS_MAX_SWEEPS 20

// The rotation of a pair with Gram matrix [nx, a; conj(a), ny]; a at or below the rounding level of the
// two norms is left (c = 1, s = 0).  Returns whether the pair turned by more than `angle`; shift =
// t |a| is what ny gains and nx loses.
WNLQG_D bool os_rotation(float2 a, float nx, float ny, float angle, float &c, float2 &s, float &shift) {
    const float a2 = a.x * a.x + a.y * a.y;
    c = 1.0f;
    s = make_float2(0.0f, 0.0f);
    shift = 0.0f;
    if (!(a2 > 2.2737368e-13f * 0.0625f * (nx * ny))) return false;   // cosine 2^-23
    const float inv = rsqrtf(a2);
    const float theta = (ny - nx) * (0.5f * inv);
    const float t = copysignf(__frcp_rn(fabsf(theta) + sqrtf(theta * theta + 1.0f)), theta);
    c = rsqrtf(t * t + 1.0f);
    const float sg = t * c * inv;
    s = make_float2(sg * a.x, sg * a.y);
    shift = t * (a2 * inv);
    return a2 > 9.0949470e-13f * (nx * ny) && fabsf(t) > angle;    // cosine 2^-20
}

WNLQG_D void os_rotate(float2 &x, float2 &y, float c, float2 s) {
    const float2 x0 = x, y0 = y;
    x.x = fmaf(-s.y, y0.y, fmaf(-s.x, y0.x, c * x0.x));
    x.y = fmaf(s.y, y0.x, fmaf(-s.x, y0.y, c * x0.y));
    y.x = fmaf(-s.y, x0.y, fmaf(s.x, x0.x, c * y0.x));
    y.y = fmaf(s.y, x0.x, fmaf(s.x, x0.y, c * y0.y));
}

// The power of two that scales norm `fro` into [1/2, 1); 1 for zero and non-finite norms.
WNLQG_D float os_scale(double fro) {
    if (!(fro > 0.0) || !isfinite(fro)) return 1.0f;
    int e;
    frexp(fro, &e);
    e = max(-120, min(120, e));
    return ldexpf(1.0f, -e);
}

// The shift of a point that starts cold, and of one that starts from vectors with max |lambda| = lmax in
// the present scaling.
WNLQG_D float os_cold_shift(double fro, float sc) { return 1.1f * (float)fmax(fro * (double)sc, 0.5); }
WNLQG_D float os_warm_shift(float lmax) { return fmaxf(1.3f * lmax, 0.01f); }

// Whether H + c I is definite, from the smallest and the sum of its columns' lengths and its trace.
WNLQG_D bool os_definite(float smallest, float sum, float trace, float shift) {
    return smallest >= 0.05f * shift && fabsf(sum - trace) <= 0.05f * shift;
}

// Sum over the warp of the complex v[0 .. 15], scattered: lanes 2m and 2m + 1 get v[m].
WNLQG_D float2 os_scatter16(float2 (&v)[16]) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int w = 8; w > 0; w >>= 1) {
        const bool up = lane & (2 * w);
#pragma unroll
        for (int j = 0; j < w; ++j) {
            const float2 keep = up ? v[j + w] : v[j], send = up ? v[j] : v[j + w];
            v[j].x = keep.x + __shfl_xor_sync(0xffffffffu, send.x, 2 * w);
            v[j].y = keep.y + __shfl_xor_sync(0xffffffffu, send.y, 2 * w);
        }
    }
    v[0].x += __shfl_xor_sync(0xffffffffu, v[0].x, 1);
    v[0].y += __shfl_xor_sync(0xffffffffu, v[0].y, 1);
    return v[0];
}

// ---- up to 32 orbitals: one warp per matrix, lane i holds row i of G --------------------------------
// Slots and pairs as in regjacobi.cuh (slot 0 fixed, the others move down by one after each round);
// lane 2m keeps the squared norm of slot m, lane 2m + 1 that of slot NP - 1 - m.
template <int NP> struct alignas(16) OsSmem {
    static constexpr int LD = NP + 2;
    float2 S1[NP * LD], S2[NP * LD];
    float4 rot[2][16];
    float inv[32];
};

// Squared norms of the columns, each in its lane (slot s holding index s).
template <int NP> WNLQG_D float os_norms(const float2 (&g)[NP]) {
    float2 v[16];
#pragma unroll
    for (int k = 0; k < 16; ++k)
        v[k] = k < NP / 2 ? make_float2(g[k].x * g[k].x + g[k].y * g[k].y,
                                        g[NP - 1 - k].x * g[NP - 1 - k].x + g[NP - 1 - k].y * g[NP - 1 - k].y)
                          : make_float2(0.0f, 0.0f);
    const float2 n = os_scatter16(v);
    return (threadIdx.x & 1) ? n.y : n.x;
}

// One sweep; returns whether a pair turned by more than OS_ANGLE_WARP.
template <int NP> WNLQG_D bool os_sweep(float2 (&g)[NP], float4 (*rot)[16]) {
    constexpr int H = NP / 2;
    const int lane = threadIdx.x & 31, m = lane >> 1;
    float n = os_norms<NP>(g);
    // The lane that holds the norm which moves into this lane's slot after a round.
    int src = lane;
    if (m < H) {
        const int slot = (lane & 1) ? NP - 1 - m : m;
        const int next = slot == 0 ? 0 : (slot == NP - 1 ? 1 : slot + 1);
        src = next < H ? 2 * next : 2 * (NP - 1 - next) + 1;
    }
    bool big = false;
#pragma unroll 1
    for (int round = 0; round < NP - 1; ++round) {
        float2 v[16];
#pragma unroll
        for (int k = 0; k < 16; ++k) {
            if (k < H) {
                const float2 x = g[k], y = g[NP - 1 - k];
                v[k] = make_float2(fmaf(x.y, y.y, x.x * y.x), fmaf(-x.y, y.x, x.x * y.y));
            } else {
                v[k] = make_float2(0.0f, 0.0f);
            }
        }
        const float2 a = os_scatter16(v);
        const float other = __shfl_xor_sync(0xffffffffu, n, 1);
        float c, shift;
        float2 s;
        const bool turned = os_rotation(a, (lane & 1) ? other : n, (lane & 1) ? n : other, OS_ANGLE_WARP, c, s, shift);
        big = big || turned;
        n += (lane & 1) ? shift : -shift;
        float4 *r = rot[round & 1];
        if (!(lane & 1)) r[m] = make_float4(c, s.x, s.y, 0.0f);
        __syncwarp();
#pragma unroll
        for (int k = 0; k < H; ++k) {
            const float4 q = r[k];
            os_rotate(g[k], g[NP - 1 - k], q.x, make_float2(q.y, q.z));
        }
        n = __shfl_sync(0xffffffffu, n, src);
        const float2 g1 = g[1];
#pragma unroll
        for (int j = 1; j < NP - 1; ++j) g[j] = g[j + 1];
        g[NP - 1] = g1;
    }
    return __any_sync(0xffffffffu, big);
}

// Chain w of `chains` takes the points [batch w / chains, batch (w + 1) / chains), each warm-started from
// the one before it; V_out gets the vectors (column-major np x np, unsorted).  Blocks of 128 threads,
// one warp per chain.  Bound by instruction issue, about 16 np per lane and round; 168 registers (three
// blocks per SM) because 128 spill a row's third.
template <int NP>
__global__ void __launch_bounds__(128, 3) onesided_warp_kernel(const double2 *__restrict__ h_in, int64_t h_stride,
                                                               int64_t batch, int nw, float2 *__restrict__ V_out,
                                                               int64_t chains, int warm_start) {
    extern __shared__ __align__(16) unsigned char os_smem_raw[];
    constexpr int LD = OsSmem<NP>::LD;
    OsSmem<NP> &sm = reinterpret_cast<OsSmem<NP> *>(os_smem_raw)[threadIdx.x >> 5];
    const int i = threadIdx.x & 31, ic = min(i, NP - 1);
    const int64_t w = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (w >= chains) return;   // whole warps
    const int64_t kb = (batch * w) / chains, ke = (batch * (w + 1)) / chains;
    float2 g[NP];
    float shift = 0.0f, lmax = 0.0f, sc_before = 1.0f;
    // g <- its normalised columns, lmax their largest |lambda|; returns whether H + c I is definite
    // (h_trace: tr H).
    auto normalise = [&](float h_trace) -> bool {
        const float n2 = os_norms<NP>(g);
        const int m = i >> 1;
        const bool held = m < NP / 2;
        const float len = sqrtf(n2);
        float smin = held ? len : 3.0e38f, sum = held ? len : 0.0f;
        lmax = held ? fabsf(len - shift) : 0.0f;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            lmax = fmaxf(lmax, __shfl_xor_sync(0xffffffffu, lmax, o));
            smin = fminf(smin, __shfl_xor_sync(0xffffffffu, smin, o));
            sum += __shfl_xor_sync(0xffffffffu, sum, o);
        }
        __syncwarp();
        if (held) sm.inv[(i & 1) ? NP - 1 - m : m] = n2 > 0.0f ? rsqrtf(n2) : 0.0f;
        __syncwarp();
#pragma unroll
        for (int j = 0; j < NP; ++j) {
            const float f = sm.inv[j];
            g[j] = make_float2(g[j].x * f, g[j].y * f);
        }
        return __all_sync(0xffffffffu, os_definite(smin, sum, h_trace + NP * shift, shift));
    };
    for (int64_t b = kb; b < ke; ++b) {
        __syncwarp();
        reg_stage_hermitian<float, NP>(sm.S2, h_in + b * h_stride, nw, true);
        double f2 = 0.0, trace = 0.0;
        for (int j = 0; j < NP; ++j) {
            const float2 z = sm.S2[j * LD + ic];
            f2 += (double)z.x * z.x + (double)z.y * z.y;
            if (j == i) trace = z.x;
        }
        if (i >= NP) f2 = 0.0;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            f2 += __shfl_xor_sync(0xffffffffu, f2, o);
            trace += __shfl_xor_sync(0xffffffffu, trace, o);
        }
        const double fro = sqrt(f2);
        const float sc = os_scale(fro), cold_shift = os_cold_shift(fro, sc);
        bool cold = b == kb || !warm_start;
        for (;;) {
            if (cold) {
                shift = cold_shift;
#pragma unroll
                for (int j = 0; j < NP; ++j) {
                    const float2 z = sm.S2[j * LD + ic];   // H[i][j] = conj(H[j][i])
                    g[j] = make_float2(sc * z.x + (j == i ? shift : 0.0f), -sc * z.y);
                    if (i >= NP) g[j] = make_float2(0.0f, 0.0f);
                }
            } else {
                // g <- (H + c I) V.
                shift = fminf(os_warm_shift(lmax * (sc / sc_before)), cold_shift);
                if (i < NP)
#pragma unroll
                    for (int j = 0; j < NP; j += 2)
                        *reinterpret_cast<float4 *>(sm.S1 + i * LD + j) = make_float4(g[j].x, g[j].y, g[j + 1].x, g[j + 1].y);
                __syncwarp();
#pragma unroll
                for (int j = 0; j < NP; ++j) g[j] = make_float2(shift * g[j].x, shift * g[j].y);
#pragma unroll 1
                for (int l = 0; l < NP; ++l) {
                    const float2 z = sm.S2[l * LD + ic];
                    const float2 h = i < NP ? make_float2(sc * z.x, -sc * z.y) : make_float2(0.0f, 0.0f);
#pragma unroll
                    for (int j = 0; j < NP; j += 2) {
                        const float4 y = *reinterpret_cast<const float4 *>(sm.S1 + l * LD + j);
                        g[j] = cfma(h, make_float2(y.x, y.y), g[j]);
                        g[j + 1] = cfma(h, make_float2(y.z, y.w), g[j + 1]);
                    }
                }
                __syncwarp();
            }
            for (int sweep = 0; sweep < OS_MAX_SWEEPS; ++sweep)
                if (!os_sweep<NP>(g, sm.rot)) break;
            if (normalise((float)(trace * (double)sc)) || cold) break;
            cold = true;
        }
        sc_before = sc;
        if (i < NP) {
            float2 *vo = V_out + b * (int64_t)NP * NP;
#pragma unroll
            for (int j = 0; j < NP; ++j) vo[i + (int64_t)NP * j] = g[j];
        }
    }
}

// ---- above 32 orbitals: one CTA per matrix, G in shared memory ---------------------------------------
// Columns go in blocks of four.  A warp takes a pair of blocks (the circle method over the blocks, one
// barrier per block round) into registers, lane l holding rows l, l + 32, ... of the eight columns,
// turns every pair between the two blocks (and, in a sweep's first round, inside them) in rounds of
// four disjoint pairs, and writes them back: eight columns are read and written once for 16 pairs.
// H is kept beside G as its packed upper triangle (element (i, j), i <= j, at j (j + 1) / 2 + i).
#define OS_ROWS(RP) (32 * (RP))
struct OsCtaSmem {
    static __host__ __device__ int blocks(int np) { int n = (np + 3) / 4; return n + (n & 1); }
    static __host__ __device__ int rows_per_lane(int np) { return (np + 31) / 32; }
    static __host__ __device__ size_t bytes(int np) {
        return ((size_t)4 * blocks(np) * 32 * rows_per_lane(np) + (size_t)np * (np + 1) / 2 + 2) * sizeof(float2);
    }
    static __host__ __device__ int threads(int np) { return 32 * (blocks(np) / 2); }   // at most 16 warps
};

// Sums over the warp of the complex v[0 .. 3]; lane group q = lane / 8 gets v[q].
WNLQG_D float2 os_scatter4(float2 (&v)[4]) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int w = 2; w > 0; w >>= 1) {
        const bool up = lane & (8 * w);
#pragma unroll
        for (int j = 0; j < w; ++j) {
            const float2 keep = up ? v[j + w] : v[j], send = up ? v[j] : v[j + w];
            v[j].x = keep.x + __shfl_xor_sync(0xffffffffu, send.x, 8 * w);
            v[j].y = keep.y + __shfl_xor_sync(0xffffffffu, send.y, 8 * w);
        }
    }
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) {
        v[0].x += __shfl_xor_sync(0xffffffffu, v[0].x, o);
        v[0].y += __shfl_xor_sync(0xffffffffu, v[0].y, o);
    }
    return v[0];
}

// Squared norms of the warp's eight columns, the same in every lane.
template <int RP> WNLQG_D void os_norms8(const float2 (&g)[8][RP], float (&n)[8]) {
    float2 v[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        v[q] = make_float2(0.0f, 0.0f);
#pragma unroll
        for (int r = 0; r < RP; ++r) {
            v[q].x += g[q][r].x * g[q][r].x + g[q][r].y * g[q][r].y;
            v[q].y += g[q + 4][r].x * g[q + 4][r].x + g[q + 4][r].y * g[q + 4][r].y;
        }
    }
    const float2 s = os_scatter4(v);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        n[q] = __shfl_sync(0xffffffffu, s.x, 8 * q);
        n[q + 4] = __shfl_sync(0xffffffffu, s.y, 8 * q);
    }
}

// One round of four disjoint pairs (X[k], Y[k]) of the warp's eight columns.
template <int RP, int X0, int Y0, int X1, int Y1, int X2, int Y2, int X3, int Y3>
WNLQG_D bool os_round4(float2 (&g)[8][RP], float (&n)[8]) {
    constexpr int X[4] = {X0, X1, X2, X3}, Y[4] = {Y0, Y1, Y2, Y3};
    const int q = (threadIdx.x & 31) >> 3;
    float2 v[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        v[k] = make_float2(0.0f, 0.0f);
#pragma unroll
        for (int r = 0; r < RP; ++r) v[k] = cfmaconj(g[X[k]][r], g[Y[k]][r], v[k]);
    }
    const float2 a = os_scatter4(v);
    const float nx = q < 2 ? (q == 0 ? n[X0] : n[X1]) : (q == 2 ? n[X2] : n[X3]);
    const float ny = q < 2 ? (q == 0 ? n[Y0] : n[Y1]) : (q == 2 ? n[Y2] : n[Y3]);
    float c, shift;
    float2 s;
    const bool turned = os_rotation(a, nx, ny, OS_ANGLE_CTA, c, s, shift);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const float ck = __shfl_sync(0xffffffffu, c, 8 * k), hk = __shfl_sync(0xffffffffu, shift, 8 * k);
        const float2 sk = make_float2(__shfl_sync(0xffffffffu, s.x, 8 * k), __shfl_sync(0xffffffffu, s.y, 8 * k));
        n[X[k]] -= hk;
        n[Y[k]] += hk;
#pragma unroll
        for (int r = 0; r < RP; ++r) os_rotate(g[X[k]][r], g[Y[k]][r], ck, sk);
    }
    return turned;
}

// Block b of the grid takes the points [batch b / grid, batch (b + 1) / grid).  Bound by instruction
// issue: a round of four pairs is 64 RP FMAs and about 100 others per lane.  One warp per pair of
// blocks; the register budget (128 at two and four rows per lane, 168 at three) is what spills little.
template <int RP>
__global__ void __launch_bounds__(RP == 2 ? 256 : (RP == 3 ? 384 : 512), RP == 2 ? 2 : 1)
    onesided_cta_kernel(const double2 *__restrict__ h_in, int64_t h_stride, int64_t batch, int nw,
                        float2 *__restrict__ V_out, int warm_start) {
    extern __shared__ __align__(16) unsigned char os_smem_raw[];
    __shared__ float red[3][16];
    __shared__ double dred[16];
    constexpr int LR = OS_ROWS(RP);
    const int np = nw + (nw & 1);
    const int nblk = OsCtaSmem::blocks(np), ncol = 4 * nblk;
    float2 *G = reinterpret_cast<float2 *>(os_smem_raw);   // column j at G + j LR
    float2 *Hp = G + (size_t)ncol * LR;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    const int64_t kb = (batch * (int64_t)blockIdx.x) / gridDim.x, ke = (batch * ((int64_t)blockIdx.x + 1)) / gridDim.x;
    float shift = 0.0f, lmax = 0.0f, sc_before = 1.0f;
    float2 g[8][RP];
    float n[8];
    auto load8 = [&](int cI, int cJ) {
#pragma unroll
        for (int q = 0; q < 8; ++q)
#pragma unroll
            for (int r = 0; r < RP; ++r) g[q][r] = G[(size_t)((q < 4 ? cI + q : cJ + q - 4)) * LR + lane + 32 * r];
    };
    auto store8 = [&](int cI, int cJ) {
#pragma unroll
        for (int q = 0; q < 8; ++q)
#pragma unroll
            for (int r = 0; r < RP; ++r) G[(size_t)((q < 4 ? cI + q : cJ + q - 4)) * LR + lane + 32 * r] = g[q][r];
    };
    // One sweep; returns (in every thread) whether a pair turned by more than OS_ANGLE_CTA.
    auto sweep = [&]() -> bool {
        bool big = false;
#pragma unroll 1
        for (int round = 0; round < nblk - 1; ++round) {
            for (int k = warp; k < nblk / 2; k += nwarps) {
                const int s2 = nblk - 1 - k;
                int I = k == 0 ? 0 : k - 1 + round, J = s2 - 1 + round;
                if (k > 0) I = (I >= nblk - 1 ? I - (nblk - 1) : I) + 1;
                J = (J >= nblk - 1 ? J - (nblk - 1) : J) + 1;
                load8(4 * I, 4 * J);
                os_norms8<RP>(g, n);
                if (round == 0) {
                    big |= os_round4<RP, 0, 1, 2, 3, 4, 5, 6, 7>(g, n);
                    big |= os_round4<RP, 0, 2, 1, 3, 4, 6, 5, 7>(g, n);
                    big |= os_round4<RP, 0, 3, 1, 2, 4, 7, 5, 6>(g, n);
                }
                big |= os_round4<RP, 0, 4, 1, 5, 2, 6, 3, 7>(g, n);
                big |= os_round4<RP, 0, 5, 1, 6, 2, 7, 3, 4>(g, n);
                big |= os_round4<RP, 0, 6, 1, 7, 2, 4, 3, 5>(g, n);
                big |= os_round4<RP, 0, 7, 1, 4, 2, 5, 3, 6>(g, n);
                store8(4 * I, 4 * J);
            }
            __syncthreads();
        }
        return __syncthreads_or(big ? 1 : 0) != 0;
    };
    // Columns normalised in place, lmax their largest |lambda|; returns whether H + c I is definite
    // (h_trace: tr H), all over the np columns and in every thread.
    auto normalise = [&](float h_trace) -> bool {
        float lm = 0.0f, smin = 3.0e38f, sum = 0.0f;
        for (int k = warp; k < nblk / 2; k += nwarps) {
            load8(8 * k, 8 * k + 4);
            os_norms8<RP>(g, n);
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                if (8 * k + q < np) {
                    const float len = sqrtf(n[q]);
                    lm = fmaxf(lm, fabsf(len - shift));
                    smin = fminf(smin, len);
                    sum += len;
                }
                const float f = n[q] > 0.0f ? rsqrtf(n[q]) : 0.0f;
#pragma unroll
                for (int r = 0; r < RP; ++r) g[q][r] = make_float2(g[q][r].x * f, g[q][r].y * f);
            }
            store8(8 * k, 8 * k + 4);
        }
        if (lane == 0) { red[0][warp] = lm; red[1][warp] = smin; red[2][warp] = sum; }
        __syncthreads();
        lmax = 0.0f;
        smin = 3.0e38f;
        sum = 0.0f;
        for (int w = 0; w < nwarps; ++w) {
            lmax = fmaxf(lmax, red[0][w]);
            smin = fminf(smin, red[1][w]);
            sum += red[2][w];
        }
        __syncthreads();
        return os_definite(smin, sum, h_trace + np * shift, shift);
    };
    bool redo = false;
    for (int64_t b = kb; b < ke; ++b) {
        const double2 *h = h_in + b * h_stride;
        double f2 = 0.0;
        for (int j = warp; j < np; j += nwarps)
            for (int i = lane; i <= j; i += 32) {
                double2 x = make_double2(0.0, 0.0);
                if (j < nw) x = h[i + (int64_t)nw * j];
                if (i == j) x.y = 0.0;
                const float2 z = make_float2((float)x.x, (float)x.y);
                f2 += (i == j ? 1.0 : 2.0) * ((double)z.x * z.x + (double)z.y * z.y);
                Hp[(size_t)j * (j + 1) / 2 + i] = z;
            }
        for (int o = 16; o > 0; o >>= 1) f2 += __shfl_xor_sync(0xffffffffu, f2, o);
        if (lane == 0) dred[warp] = f2;
        __syncthreads();
        double fro = 0.0;
        for (int w = 0; w < nwarps; ++w) fro += dred[w];
        fro = sqrt(fro);
        const float sc = os_scale(fro), cold_shift = os_cold_shift(fro, sc);
        float h_trace = 0.0f;
        for (int j = lane; j < np; j += 32) h_trace += sc * Hp[(size_t)j * (j + 1) / 2 + j].x;
        for (int o = 16; o > 0; o >>= 1) h_trace += __shfl_xor_sync(0xffffffffu, h_trace, o);
        auto h_elem = [&](int r, int l) -> float2 {   // scaled H[r][l]
            if (r >= np) return make_float2(0.0f, 0.0f);
            const float2 z = r <= l ? Hp[(size_t)l * (l + 1) / 2 + r] : Hp[(size_t)r * (r + 1) / 2 + l];
            return make_float2(sc * z.x, r <= l ? sc * z.y : -sc * z.y);
        };
        lmax *= sc / sc_before;
        sc_before = sc;
        // Also cold where max |lambda| fell so far that the warm shift would be the looser one.
        const bool cold = b == kb || !warm_start || redo || !(lmax <= cold_shift);
        redo = false;
        if (cold) {
            shift = cold_shift;
            for (int e = threadIdx.x; e < ncol * LR; e += blockDim.x) {
                const int j = e / LR, r = e % LR;
                float2 z = make_float2(0.0f, 0.0f);
                if (j < np) {
                    z = h_elem(r, j);
                    if (r == j) z.x += shift;
                }
                G[e] = z;
            }
            __syncthreads();
            for (int s = 0; s < OS_MAX_SWEEPS; ++s)
                if (!sweep()) break;
            normalise(h_trace);
        }
        bool definite = true;
        for (int start = 0; start < 2; ++start) {
            // G <- (H + c I) V: a warp needs its own eight columns of V only.
            shift = os_warm_shift(lmax);
            for (int k = warp; k < nblk / 2; k += nwarps) {
                load8(8 * k, 8 * k + 4);
#pragma unroll
                for (int q = 0; q < 8; ++q)
#pragma unroll
                    for (int r = 0; r < RP; ++r) g[q][r] = make_float2(shift * g[q][r].x, shift * g[q][r].y);
                const float2 *Vc = G + (size_t)8 * k * LR;
#pragma unroll 1
                for (int l = 0; l < np; ++l) {
                    float2 hr[RP];
#pragma unroll
                    for (int r = 0; r < RP; ++r) hr[r] = h_elem(lane + 32 * r, l);
#pragma unroll
                    for (int q = 0; q < 8; ++q) {
                        const float2 y = Vc[q * LR + l];
#pragma unroll
                        for (int r = 0; r < RP; ++r) g[q][r] = cfma(hr[r], y, g[q][r]);
                    }
                }
                __syncwarp();
                store8(8 * k, 8 * k + 4);
            }
            __syncthreads();
            for (int s = 0; s < OS_MAX_SWEEPS; ++s)
                if (!sweep()) break;
            definite = normalise(h_trace);
            if (!definite || shift <= 1.5f * lmax) break;
        }
        if (!definite && !cold) {   // again from a cold start
            redo = true;
            --b;
            continue;
        }
        float2 *vo = V_out + b * (int64_t)np * np;
        for (int j = warp; j < np; j += nwarps)
            for (int i = lane; i < np; i += 32) vo[i + (int64_t)np * j] = G[(size_t)j * LR + i];
        __syncthreads();
    }
}

// Kernel, group shared memory and lanes of the warp form for an even order 18 <= np <= 32.
template <int NP> RegKernel onesided_entry() { return {(const void *)onesided_warp_kernel<NP>, sizeof(OsSmem<NP>), 32}; }
inline RegKernel onesided_kernel(int np) {
    static const RegKernel k[8] = {onesided_entry<18>(), onesided_entry<20>(), onesided_entry<22>(), onesided_entry<24>(),
                                   onesided_entry<26>(), onesided_entry<28>(), onesided_entry<30>(), onesided_entry<32>()};
    return k[(np - 18) / 2];
}
inline const void *onesided_cta_fn(int np) {
    const int rp = OsCtaSmem::rows_per_lane(np);
    return rp == 2 ? (const void *)onesided_cta_kernel<2>
                   : (rp == 3 ? (const void *)onesided_cta_kernel<3> : (const void *)onesided_cta_kernel<4>);
}

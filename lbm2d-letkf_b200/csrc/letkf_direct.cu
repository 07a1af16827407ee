// letkf_direct.cu -- the LETKF local analysis without an eigensolver, for sm_100a: the solver of
// the allocation-free entry point (noalloc.cu), 9 to 32 members.  The contexts' analyses keep the Jacobi
// kernels (letkf_kernels.cu): a run of cycles amplifies last-bit differences, and theirs must go on
// reproducing earlier runs; the two solvers' analyses agree to half an ulp of a population (2e-5 of an
// increment of 1.5e-3).
//
// The analysis applies W = sqrt(M-1) Q^-1/2 + Q^-1 c 1^T, Q = (M-1)/beta I + dY^T R^-1 dY
// (letkf_solver.h:243-316), to nine rows dX only, so the eigenvectors of Q are never needed.
// With a = (M-1)/beta, C = (R^-1/2 / sqrt(a)) dY (one row per observation) and d the innovations
// scaled likewise, every grid point is one symmetric positive definite matrix of order n,
//
//     primal (n = M)      B = I + C^T C,   rows R = dX,        g = C^T d,
//     dual   (n = obs)    B = I + C C^T,   rows R = dX C^T,    g = d,
//
// whose spectrum starts at 1.  The dual form serves windows of up to 16 observations, fewer than
// there are members (3 in the reference's default window, 12 at DA_XYPRUNE 2):
//   1. Householder reduction B = H T H^T, with the nine rows of R and g carried along as extra
//      rows of the same matrix (R' = R H, g' = g H): a group of LPP lanes holds one point,
//      a matrix row and a carried row per lane in registers, and each step needs two small broadcasts
//      through shared memory, the pivot column and B v.
//   2. T^-1/2 as a sum of N shifted inverses, t^-1/2 = sum_j w_j / (t + s_j) on [1, kappa]:
//      Zolotarev's best rational approximation (relative error below 2e-8 up to kappa = 1e12;
//      shifts from Jacobi elliptic functions, computed on the host).  kappa is bounded
//      per point by Gershgorin's circles of T, and picks one of the tables at powers of 4.
//      Every shifted T is solved by one tridiagonal elimination; T^-1 g' likewise.
//   3. the rows go back through the reflections, Z = R' T^-1/2 H^T, and
//      primal  Xa = xbar + s + sqrt(beta) Z,
//      dual    Xa = xbar + s + sqrt(beta) (dX + Z C)   with t^-1/2 - 1 over t - 1 in place of
//              t^-1/2: the same shifts, weights -w_j / (1 + s_j), no cancellation;
//      s = R' T^-1 g', the update of the mean.
// A point costs 4/3 n^3 + O(n^2) operations against 9 n^3 per Jacobi sweep, and has no
// iteration to converge.  In FP32 the reduction keeps the small eigenvalues less well than the iteration
// on columns does: a tile with a point above the limit of its form (trace_limit) is marked and left to
// the Jacobi kernel, launched behind this one.
#include <algorithm>
#include <cmath>

#include "lbl_internal.h"

namespace lbl {
namespace {

__host__ __device__ constexpr int exq(int q) { return (q % 3) - 1; }
__host__ __device__ constexpr int eyq(int q) { return (q / 3) - 1; }

using u64 = unsigned long long;  // a pair of floats for the packed FP32 instructions

__device__ __forceinline__ u64 pk(float lo, float hi) {
    u64 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ float lo_of(u64 a) {
    float l, h;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(l), "=f"(h) : "l"(a));
    return l;
}
__device__ __forceinline__ float hi_of(u64 a) {
    float l, h;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(l), "=f"(h) : "l"(a));
    return h;
}
__device__ __forceinline__ u64 fma2(u64 a, u64 b, u64 c) {
    u64 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ u64 add2(u64 a, u64 b) {
    u64 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
// a shared read the compiler may not merge with an earlier one of the same address
__device__ __forceinline__ ulonglong2 lds_again(const float* p) {
    ulonglong2 r;
    asm volatile("ld.shared.v2.u64 {%0, %1}, [%2];" : "=l"(r.x), "=l"(r.y) : "r"(uint32_t(__cvta_generic_to_shared(p))));
    return r;
}
__device__ __forceinline__ float sum2(u64 a) { return lo_of(a) + hi_of(a); }
__device__ __forceinline__ float rcp_approx(float x) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

__device__ __forceinline__ float sqrt_approx(float x) {  // within an ulp: the reflections stay orthogonal to working precision
    float r;
    asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// x as the sum of two TF32 values, and D += A (16 x 8) B (8 x 8) on the tensor cores with FP32 sums
__device__ __forceinline__ void split_tf32(float x, uint32_t& hi, uint32_t& lo) {
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(hi) : "f"(x));
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(lo) : "f"(x - __uint_as_float(hi)));
}
__device__ __forceinline__ void mma_tf32(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                         uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// s / m correctly rounded but for rare cases, from the rounded reciprocal of m
__device__ __forceinline__ float mean_of(float s, float m, float inv_m) {
    const float q = s * inv_m;
    return fmaf(fmaf(-q, m, s), inv_m, q);
}

constexpr int kB = 10;          // carried rows: nine of R, then g
constexpr int kMaxPoles = 30;   // shifts of one table
constexpr int kTables = 20;     // kappa <= 4^1 .. 4^20
constexpr int kMaxRounds = 6;   // of a CTA
constexpr float kKappaMax = 1e8f;  // a point of order 16 above it counts as not converged: its mean update is good to 1e-3

// the shifts and weights, one table per kappa = 4^(b+1)
struct PoleTables {
    int n[kTables];
    float s[kTables][kMaxPoles], w[kTables][kMaxPoles];
};

struct DirParams {
    const float *fin, *dY, *dyo;
    float *fout, *mac;
    const int4* wtab;       // {slot, variable, sqrt(w), w} per pattern (i mod p, j mod p)
    const int* wcnt;
    int* stats;
    int nx, ny, nxy, M;
    int p, nsx, nsy, nsites, nobs, nox, nl_off;
    int nbx, nby;           // p x p observation blocks per tile
    int rounds;             // rounds of points of a CTA (blockIdx.y counts the shares of a tile)
    int ms;                 // floats per slot of the staged window (at least N in the primal form): 4 (mod 8),
                            // so that eight lanes reading 16 bytes of consecutive slots hit different banks
    float inv_sqrt_a, sqrt_beta, c, inv_m;
    float limit;            // the largest bound of a tile's traces of C^T C solved here
    int write_v;
};

template <int N, int LPP, bool DUAL>
struct Shape {
    static constexpr int GPW = 32 / LPP;  // points per warp
    // shared floats per point: pivot column and B v (each with N floats of room below and above), diagonal,
    // off-diagonal, tau, R' [N][12], reflections, partial sums, xbar + s (24), observations
    static constexpr int VSZ = LPP == 32 ? N * N / 2 : N * N;
    static constexpr int BUF = LPP == 32 ? 0 : 16 * (N + 4);  // partial sums of the shifted solves
    static constexpr int FIXED = 9 * N + 12 * N + VSZ + BUF + 24 + 2 * N;
};
// Warps of a CTA.  The kernel's code is larger than the instruction caches near the schedulers, so an
// SM's warps walk it together: one CTA of twelve warps (168 registers) per SM above order 16, two of
// eight (128 registers) below (one where shared memory holds no second: the dual order 16 from 21 members
// on, 117 kB), with a barrier between the stages of a point.  Independent CTAs of four warps spent half of
// their cycles waiting for instructions.
__host__ __device__ constexpr int warps_of(int n) { return n > 16 ? 12 : 8; }
// floats of a point's shared region; mx = members rounded up to 4.  Dual: dX as [member][12], then the point's
// weighted window [member][N]; primal: the rows on their way in, [12][N]
__host__ __device__ constexpr int region_floats(int fixed, int n, bool dual, int mx) {
    return fixed + (dual ? (12 + n) * mx : 12 * n);
}

// ---------------------------------------------------------------------------
// The Householder reduction.  A lane holds two rows in registers: matrix row `lane` (slot 0) and a carried row
// (slot 1).  r[t][m] holds columns k0 + 2m, k0 + 2m + 1 of row t; the second reflection of a pair (PAR = 1)
// moves the columns down by one register pair as it updates them, so no register is indexed at run
// time.  Rows of the pivot column and of B v go through sx / sp at their distance from k0; finished
// rows write below the arrays' start (they begin at their owner's lane), the last two rows clear the
// entries that shifting uncovers.  Per reflection on W columns: 3 W packed multiply-adds and W / 2
// 16-byte shared reads (3 W / 4 above 16 columns).
// ---------------------------------------------------------------------------
struct Rows {
    int n;                  // unknowns (even)
    int row0;               // matrix row of slot 0 (2^20 when it is none: never a pivot)
    bool carry;             // slot 1 holds a carried row
    bool last0;             // one of the last two matrix rows
    bool entry;             // the lane has an entry of whole-row reflections
    // offsets into the CTA's shared memory:
    int px0;                // sx + row, less k0 (moves down two per pair)
    int pR;                 // R' entry of the carried row, [column][12]
    int pV0;                // reflections: entry of the row in the current one
    int pT;                 // diagonal of T at k (off-diagonal N, tau 2 N further)
};

template <int PAR, int W, int N>
__device__ __forceinline__ void reflect(u64 (&r)[2][N / 2], Rows& R, const int k0, float* smem, const float* sx, const float* sp) {
    constexpr int SP = 3 * N;  // sp - sx
    const int k = k0 + PAR;
    const float el0 = PAR ? hi_of(r[0][0]) : lo_of(r[0][0]), el1 = PAR ? hi_of(r[1][0]) : lo_of(r[1][0]);
    const bool below0 = R.row0 > k;
    smem[R.px0] = below0 ? el0 : 0.f;
    if (R.carry) smem[R.pR] = el1;
    if (PAR == 0 && R.last0) smem[R.px0 + 2] = 0.f;
    R.pR += 12;
    __syncwarp();
    u64 v[W / 2];
#pragma unroll
    for (int m = 0; m < W / 2; m += 2) {
        const ulonglong2 x = *reinterpret_cast<const ulonglong2*>(sx + 2 * m);
        v[m] = x.x;
        v[m + 1] = x.y;
    }
    u64 q0 = 0, q1 = 0;
#pragma unroll
    for (int m = PAR; m < W / 2; m += 2) q0 = fma2(v[m], v[m], q0);
#pragma unroll
    for (int m = PAR + 1; m < W / 2; m += 2) q1 = fma2(v[m], v[m], q1);
    q0 = add2(q0, q1);
    const float sq = sum2(q0);
    const float x0 = PAR ? lo_of(v[1]) : hi_of(v[0]);
    // a column this small (the diagonal is at least 1) is zero to working precision
    const bool turn = !(sq <= 1e-24f);
    const float mu = copysignf(sqrt_approx(sq), x0);
    const float v0 = x0 + mu;
    const float tau = turn ? rcp_approx(fmaf(x0, mu, sq)) : 0.f;
    if (PAR) v[1] = pk(v0, hi_of(v[1]));
    else v[0] = pk(0.f, v0);
    if (R.row0 == k) {
        smem[R.pT] = 1.f + el0;
        smem[R.pT + N] = turn ? -mu : 0.f;
        smem[R.pT + 2 * N] = tau;
    }
    R.pT++;
    const float vr0 = R.row0 == k + 1 ? v0 : (below0 ? el0 : 0.f);
    u64 a0 = 0, a1 = 0, b0 = 0, b1 = 0;
#pragma unroll
    for (int m = PAR; m < W / 2; m += 2) {
        a0 = fma2(r[0][m], v[m], a0);
        b0 = fma2(r[1][m], v[m], b0);
    }
#pragma unroll
    for (int m = PAR + 1; m < W / 2; m += 2) {
        a1 = fma2(r[0][m], v[m], a1);
        b1 = fma2(r[1][m], v[m], b1);
    }
    const float p0 = tau * sum2(add2(a0, a1)), p1 = tau * sum2(add2(b0, b1));
    smem[R.px0 + SP] = below0 ? p0 : 0.f;
    if (PAR == 0 && R.last0) smem[R.px0 + SP + 2] = 0.f;
    if (N == 32) {  // packed: the n - 1 - k entries below the pivot
        if (below0 && R.row0 < R.n) smem[R.pV0] = vr0;
        R.pV0 += R.n - 2 - k;
    } else {                // whole rows, zero at and above the pivot
        // (at order 8 sixteen lanes hold a point: the eight without an entry would store zeros over the others')
        if (N == 16 || R.entry) smem[R.pV0] = vr0;
        R.pV0 += N;
    }
    __syncwarp();
    u64 p[W / 2];
    u64 c0 = 0, c1 = 0;
#pragma unroll
    for (int m = 0; m < W / 2; m += 2) {
        const ulonglong2 x = *reinterpret_cast<const ulonglong2*>(sp + 2 * m);
        c0 = fma2(x.x, v[m], c0);
        c1 = fma2(x.y, v[m + 1], c1);
        if (W <= 16) {
            p[m] = x.x;
            p[m + 1] = x.y;
        }
    }
    const float kh = -0.5f * tau * sum2(add2(c0, c1));
    const u64 nkh = pk(kh, kh);
    const float w0 = fmaf(kh, vr0, p0);
    const u64 nv0 = pk(-vr0, -vr0), nw0 = pk(-w0, -w0), nw1 = pk(-p1, -p1);  // (a carried row has no v)
#pragma unroll
    for (int m = 0; m < W / 2; m += 2) {
        u64 pa, pb;
        if (W <= 16) {
            pa = p[m];
            pb = p[m + 1];
        } else {  // once more rather than W more registers
            const ulonglong2 x = lds_again(sp + 2 * m);
            pa = x.x;
            pb = x.y;
        }
        const u64 wa = fma2(nkh, v[m], pa), wb = fma2(nkh, v[m + 1], pb);
        if (m >= PAR) {
            r[0][m - PAR] = fma2(nv0, wa, fma2(nw0, v[m], r[0][m]));
            r[1][m - PAR] = fma2(nw1, v[m], r[1][m]);
        }
        r[0][m + 1 - PAR] = fma2(nv0, wb, fma2(nw0, v[m + 1], r[0][m + 1]));
        r[1][m + 1 - PAR] = fma2(nw1, v[m + 1], r[1][m + 1]);
    }
    if (PAR) {
        r[0][W / 2 - 1] = 0;
        r[1][W / 2 - 1] = 0;
        R.px0 -= 2;
    }
}

// pairs of reflections on W columns while more than `below` remain
template <int W, int N>
__device__ __forceinline__ void reduce_while(u64 (&r)[2][N / 2], Rows& R, int& k0, const int below, float* smem,
                                             const float* sx, const float* sp) {
#pragma unroll 1
    while (k0 <= R.n - 4 && R.n - k0 > below) {
        reflect<0, W, N>(r, R, k0, smem, sx, sp);
        reflect<1, W, N>(r, R, k0, smem, sx, sp);
        k0 += 2;
    }
}

// ---------------------------------------------------------------------------
// The local analysis of one CTA's tile of nbx x nby observation blocks (p x p points each).
//   N the most unknowns (a multiple of 8), LPP lanes per point, DUAL the form above
// ---------------------------------------------------------------------------
template <int N, int LPP, bool DUAL>
__global__ void __launch_bounds__(32 * warps_of(N), N > 16 ? 1 : 2) analysis_direct_kernel(const DirParams A, const __grid_constant__ PoleTables T) {
    using S = Shape<N, LPP, DUAL>;
    constexpr int kWarps = warps_of(N);
    constexpr bool LIMITED = !DUAL;  // see trace_limit
    extern __shared__ __align__(16) float smem[];
    const int tid = threadIdx.x, wl = tid & 31, warp = tid >> 5;
    const int lane = wl % LPP, grp = wl / LPP;
    const int M = A.M, mx = (M + 3) & ~3, ms = A.ms;
    const float fM = float(M);
    const int ux = A.nbx + A.nox - 1, uy = A.nby + A.nox - 1, us = ux * uy, slots = 3 * us;

    // ---- the tile's window: every slot's dY row (unweighted), zero beyond M, and its innovation
    float* sY = smem;                                   // [slots][ms]
    float* sDyo = sY + size_t(slots) * ms;              // [slots]
    int* sOff = reinterpret_cast<int*>(sDyo + ((slots + 3) & ~3));  // [nobs] window slot -> tile slot of block (0, 0)
    float* region = reinterpret_cast<float*>(sOff + ((A.nobs + 3) & ~3));
    const int tiles_x = (A.nsx + A.nbx - 1) / A.nbx;
    const int bx0 = (blockIdx.x % tiles_x) * A.nbx, by0 = (blockIdx.x / tiles_x) * A.nby;
#pragma unroll 1
    for (int o = tid; o < A.nobs; o += 32 * kWarps) {
        const int n2 = A.nox * A.nox, var = o / n2, ab = o - var * n2, b = ab / A.nox, a = ab - b * A.nox;
        sOff[o] = a + ux * b + var * us;
    }
    int top[3] = {0, 0, 0};  // the lane's member: the largest dY^2 of each variable
    if constexpr (LIMITED) {
        if (tid < 96) region[tid] = 0.f;
        __syncthreads();
    }
#pragma unroll 2
    for (int sl = warp; sl < slots; sl += kWarps) {
        const int var = sl / us, s2 = sl - var * us, b = s2 / ux, a = s2 - b * ux;
        int sj = (by0 + b - A.nl_off) % A.nsy, si = (bx0 + a - A.nl_off) % A.nsx;
        sj += sj < 0 ? A.nsy : 0;
        si += si < 0 ? A.nsx : 0;
        const size_t site = size_t(var) * A.nsites + si + size_t(A.nsx) * sj;
#pragma unroll 1
        for (int m = wl; m < ms; m += 32) {
            const float y = m < M ? __ldg(A.dY + site * M + m) : 0.f;
            sY[sl * ms + m] = y;
            if (LIMITED && m < 32) {  // (a NaN stays one: its square, as an integer, is above every number's)
                const int y2 = __float_as_int(y * y);
                top[0] = var == 0 ? max(top[0], y2) : top[0];
                top[1] = var == 1 ? max(top[1], y2) : top[1];
                top[2] = var == 2 ? max(top[2], y2) : top[2];
            }
        }
        if (wl == 0) sDyo[sl] = __ldg(A.dyo + site);
    }
    if constexpr (LIMITED) {
#pragma unroll
        for (int var = 0; var < 3; var++) atomicMax(reinterpret_cast<int*>(region) + 32 * var + wl, top[var]);
    }
    __syncthreads();
    const int tw = A.nbx * A.p, npts = tw * A.nby * A.p;
    constexpr int kPerRound = kWarps * S::GPW;
    const int round0 = blockIdx.y * A.rounds, round1 = min(round0 + A.rounds, (npts + kPerRound - 1) / kPerRound);
    // ---- a tile that may hold a point above the limit is left to the Jacobi kernel, before it costs a solve.
    // The trace of C^T C, sum of w |dY|^2 / a, is at least kappa - 1; every member's largest dY of the window
    // and the weights of the pattern (0, 0) bound it to within a factor of a few.
    if constexpr (LIMITED) {
        float t = 0.f;
#pragma unroll
        for (int var = 0; var < 3; var++) t = fmaf(__int_as_float(__ldg(A.stats + 5 + var)), region[32 * var + wl], t);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
        if (!(t * (A.inv_sqrt_a * A.inv_sqrt_a) <= A.limit)) {  // (all warps see the same sum)
#pragma unroll 1
            for (int pt = round0 * kPerRound + tid; pt < min(round1 * kPerRound, npts); pt += 32 * kWarps) {
                const int i = bx0 * A.p + pt % tw, j = by0 * A.p + pt / tw;
                if (i < A.nx && j < A.ny) A.mac[i + A.nx * j] = __uint_as_float(kLeftPoint);
            }
            if (tid == 0) A.stats[4] = 1;
            return;
        }
        __syncthreads();  // the region is the points' from here on
    }
    // ---- the point's shared region
    constexpr int VSTRIDE = LPP == 32 ? 0 : N;
    float* base = region + size_t(warp * S::GPW + grp) *
                               size_t(region_floats(S::FIXED, N, DUAL, mx));
    float* sx = base + N;          // [N]
    float* sp = sx + 3 * N;        // [N]
    float* sd = sp + 2 * N;        // [N] diagonal of T
    float* se = sd + N;            // [N] off-diagonal of T
    float* st = se + N;            // [N] tau
    float* sR = st + N;            // [N][12] R' and g', then the rows of Z
    float* sV = sR + 12 * N;       // reflections
    float* buf = sV + S::VSZ;      // [16][N + 4] partial sums (LPP = 16)
    float* sXs = buf + S::BUF;     // [12] xbar, [12] s
    float* sS = sXs + 24;          // [N] (slot bits, sqrt(w / a)) of the point's observations
    float* sX = sS + 2 * N;        // DUAL: dX [mx][12]; else the rows on their way in: [12][N]
    float* sC = sX + 12 * mx;      // DUAL: C [mx][N]

    bool bad = false;
    int noconv = 0;
#pragma unroll 1
    for (int round = round0; round < round1; round++) {
        __syncthreads();  // the stages' barriers keep the warps on the same instructions
        const int pt0 = (round * kWarps + warp) * S::GPW;
        // ---- the point; an idle group (a tile's edge) repeats the tile's first point and writes nothing
        int pt = pt0 + grp;
        bool active = pt < npts;
        int i = bx0 * A.p + pt % tw, j = by0 * A.p + pt / tw;
        active = active && i < A.nx && j < A.ny;
        if (!active) {
            pt = 0;
            i = bx0 * A.p;
            j = by0 * A.p;
        }
        const int point = i + A.nx * j;
        const int bx = i / A.p - bx0, by = j / A.p - by0;
        const int blk = bx + ux * by;                   // tile slot offset of the point's block
        const int pat = (i - (bx0 + bx) * A.p) + A.p * (j - (by0 + by) * A.p);
        const int cnt = __ldg(A.wcnt + pat);
        const int4* ent = A.wtab + size_t(pat) * A.nobs;
        int n = DUAL ? cnt : M;
        if (DUAL && LPP == 16) n = max(n, __shfl_xor_sync(0xffffffffu, n, 16));
        n = max(4, (n + 1) & ~1);
        const int own_n = DUAL ? cnt : M;               // unknowns of this point; the rest are identity rows
        // the lane's rows: matrix row `lane`, and a carried row
        const bool mat0 = lane < n, carry = lane < kB;
        const int crow = lane;
        __syncwarp();  // the previous point's region is no longer read
#pragma unroll 1
        for (int e = lane; e < N; e += LPP) {
            sx[e] = sx[e + N] = 0.f;
            sp[e] = sp[e + N] = 0.f;
            sd[e] = 1.f;
            se[e] = 0.f;
            if (e >= n)
#pragma unroll
                for (int q = 0; q < 12; q++) sR[e * 12 + q] = 0.f;
        }

        // ---- forecast ensemble at the point: X, xbar, dX (letkf_solver.h:278-280)
        u64 r[2][N / 2];
#pragma unroll
        for (int m = 0; m < N / 2; m++) r[0][m] = r[1][m] = 0;
        if constexpr (DUAL) {
            float sum[kQ];
#pragma unroll
            for (int q = 0; q < kQ; q++) sum[q] = 0.f;
#pragma unroll 1
            for (int m = lane; m < mx; m += LPP) {
                float x[kQ];
#pragma unroll
                for (int q = 0; q < kQ; q++) x[q] = m < M ? __ldg(A.fin + (size_t(m) * kQ + q) * A.nxy + point) : 0.f;
#pragma unroll
                for (int q = 0; q < kQ; q++) sum[q] += x[q];
                float4* d = reinterpret_cast<float4*>(sX + 12 * m);
                d[0] = make_float4(x[0], x[1], x[2], x[3]);
                d[1] = make_float4(x[4], x[5], x[6], x[7]);
                d[2] = make_float4(x[8], 0.f, 0.f, 0.f);
            }
#pragma unroll
            for (int q = 0; q < kQ; q++) {
#pragma unroll
                for (int o = LPP / 2; o > 0; o >>= 1) sum[q] += __shfl_xor_sync(0xffffffffu, sum[q], o);
                sum[q] = mean_of(sum[q], fM, A.inv_m);
            }
            if (lane == 0)
#pragma unroll
                for (int q = 0; q < kQ; q++) sXs[q] = sum[q];
#pragma unroll 1
            for (int m = lane; m < M; m += LPP) {  // members past M stay zero
                float* d = sX + 12 * m;
#pragma unroll
                for (int q = 0; q < kQ; q++) d[q] -= sum[q];
            }
            // the point's observations, (slot, scaled weight).  The rows past them are rows of the identity, zeros
            // whatever the window holds (their slot is the block's first, never multiplied); a pattern whose
            // weights all round to zero has only such rows, and no table entry to read
#pragma unroll 1
            for (int e = lane; e < N; e += LPP) {
                float2 ow = make_float2(__int_as_float(blk), 0.f);
                if (e < cnt) {
                    const int4 w = __ldg(ent + e);
                    ow = make_float2(__int_as_float(sOff[w.x] + blk), __int_as_float(w.z) * A.inv_sqrt_a);
                }
                *reinterpret_cast<float2*>(sS + 2 * e) = ow;
            }
            __syncwarp();
            // rows R = dX C^T (and g = d): lane = observation, then to the carried rows' lanes
            u64 acc[5];
            const int o1 = min(lane, N - 1);
            const bool observed = o1 < cnt;
            const float sw = sS[2 * o1 + 1];
            const float* yrow = sY + __float_as_int(sS[2 * o1]) * ms;
#pragma unroll
            for (int q = 0; q < 5; q++) acc[q] = 0;
#pragma unroll 1
            for (int m = 0; m < mx; m += 4) {
                // the weighted window by members, for the products and the update
                float4 y = *reinterpret_cast<const float4*>(yrow + m);
                y = observed ? make_float4(y.x * sw, y.y * sw, y.z * sw, y.w * sw) : make_float4(0.f, 0.f, 0.f, 0.f);
                if (lane < N) {
                    sC[(m + 0) * N + lane] = y.x;
                    sC[(m + 1) * N + lane] = y.y;
                    sC[(m + 2) * N + lane] = y.z;
                    sC[(m + 3) * N + lane] = y.w;
                }
#pragma unroll
                for (int h = 0; h < 4; h++) {
                    const ulonglong2 d0 = *reinterpret_cast<const ulonglong2*>(sX + 12 * (m + h));
                    const ulonglong2 d1 = *reinterpret_cast<const ulonglong2*>(sX + 12 * (m + h) + 4);
                    const u64 d2 = *reinterpret_cast<const u64*>(sX + 12 * (m + h) + 8);
                    const float yv = h == 0 ? y.x : h == 1 ? y.y : h == 2 ? y.z : y.w;
                    const u64 yy = pk(yv, yv);
                    acc[0] = fma2(yy, d0.x, acc[0]);
                    acc[1] = fma2(yy, d0.y, acc[1]);
                    acc[2] = fma2(yy, d1.x, acc[2]);
                    acc[3] = fma2(yy, d1.y, acc[3]);
                    acc[4] = fma2(yy, d2, acc[4]);
                }
            }
            float* rows = buf;  // [10][N], 10 N <= 16 (N + 4)
            if (lane < N) {
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    rows[(2 * q) * N + lane] = lo_of(acc[q]);
                    rows[(2 * q + 1) * N + lane] = hi_of(acc[q]);
                }
                rows[8 * N + lane] = lo_of(acc[4]);
                rows[9 * N + lane] = observed ? sw * sDyo[__float_as_int(sS[2 * o1])] : 0.f;
            }
            __syncwarp();
            if (carry)
#pragma unroll
                for (int m = 0; m < N / 2; m += 2) {
                    const ulonglong2 x2 = *reinterpret_cast<const ulonglong2*>(rows + crow * N + 2 * m);
                    r[1][m] = x2.x;
                    r[1][m + 1] = x2.y;
                }
            // matrix rows: I + C C^T
            {
                // lane's own column of C against every column; idle lanes accumulate column N - 1 and drop it
                const int own = min(lane, N - 1);
#pragma unroll 2
                for (int m = 0; m < M; m++) {
                    const float y = sC[m * N + own];
                    const u64 yy = pk(y, y);
#pragma unroll
                    for (int h = 0; h < N / 2; h += 2) {
                        const ulonglong2 x2 = *reinterpret_cast<const ulonglong2*>(sC + m * N + 2 * h);
                        r[0][h] = fma2(yy, x2.x, r[0][h]);
                        r[0][h + 1] = fma2(yy, x2.y, r[0][h + 1]);
                    }
                }
#pragma unroll
                for (int m = 0; m < N / 2; m++)
                    if (!mat0) r[0][m] = 0;
            }
        } else {
            // lane = member: X into rows [q][member]; every carried row then centres itself
            if (lane < N)
#pragma unroll
                for (int q = 0; q < kQ; q++)
                    sX[q * N + lane] = lane < M ? __ldg(A.fin + (size_t(lane) * kQ + q) * A.nxy + point) : 0.f;
            // Gram: row `lane` of C^T C, and g = C^T d (letkf_solver.h:252-254)
            {
                // On the tensor cores, the whole warp for one point after the other, eight observations at a
                // time: lane (g, c) brings members g, g + 8, ... of observations c and c + 4 of C, which are both
                // its share of A = C^T and of B.  Every entry is split into two TF32 terms (2^-23 relative) and all
                // four products are summed in FP32, the smallest first.  As (w dY)^T dY, whose factors are rounded and
                // split apart, in three products, the error against FP64 was 1.3 to 2 times as large (64 x 32 points of 16 and
                // 32 members, 27 and 42 observations, kappa 1e3 to 1e6) and above the Jacobi kernel's from kappa 1e3 on.
                // Now it is that of multiply-adds, which read the window row of every observation in every lane: 390 against
                // 348 us at 256^2 x 16 (42 observations), 1708 / 1674 at 256^2 x 32.
                constexpr int MT = N / 16, YT = N / 8;
                const int g8 = wl >> 2, c4 = wl & 3;
#pragma unroll 1
                for (int pg = 0; pg < S::GPW; pg++) {
                    const int pcnt = __shfl_sync(0xffffffffu, cnt, pg * LPP), pblk = __shfl_sync(0xffffffffu, blk, pg * LPP);
                    const int4* pent = A.wtab + size_t(__shfl_sync(0xffffffffu, pat, pg * LPP)) * A.nobs;
                    float acc[MT][YT][4], gs[YT];
#pragma unroll
                    for (int i1 = 0; i1 < MT; i1++)
#pragma unroll
                        for (int i2 = 0; i2 < YT; i2++) acc[i1][i2][0] = acc[i1][i2][1] = acc[i1][i2][2] = acc[i1][i2][3] = 0.f;
#pragma unroll
                    for (int i2 = 0; i2 < YT; i2++) gs[i2] = 0.f;
#pragma unroll 1
                    for (int o0 = 0; o0 < pcnt; o0 += 8) {
                        uint32_t bh[2][YT], bl[2][YT];
#pragma unroll
                        for (int h = 0; h < 2; h++) {
                            const int o = o0 + c4 + 4 * h;  // past the end: the first observation with weight 0
                            const int4 e = __ldg(pent + (o < pcnt ? o : 0));
                            const int slot = sOff[e.x] + pblk;
                            const float sw = o < pcnt ? __int_as_float(e.z) * A.inv_sqrt_a : 0.f;
                            const float d = sw * sDyo[slot];
#pragma unroll
                            for (int i2 = 0; i2 < YT; i2++) {
                                const float y = sw * sY[slot * ms + g8 + 8 * i2];
                                split_tf32(y, bh[h][i2], bl[h][i2]);
                                gs[i2] = fmaf(y, d, gs[i2]);
                            }
                        }
#pragma unroll
                        for (int i1 = 0; i1 < MT; i1++)
#pragma unroll
                            for (int i2 = 0; i2 < YT; i2++) {
                                mma_tf32(acc[i1][i2], bl[0][2 * i1], bl[0][2 * i1 + 1], bl[1][2 * i1], bl[1][2 * i1 + 1], bl[0][i2], bl[1][i2]);
                                mma_tf32(acc[i1][i2], bl[0][2 * i1], bl[0][2 * i1 + 1], bl[1][2 * i1], bl[1][2 * i1 + 1], bh[0][i2], bh[1][i2]);
                                mma_tf32(acc[i1][i2], bh[0][2 * i1], bh[0][2 * i1 + 1], bh[1][2 * i1], bh[1][2 * i1 + 1], bl[0][i2], bl[1][i2]);
                                mma_tf32(acc[i1][i2], bh[0][2 * i1], bh[0][2 * i1 + 1], bh[1][2 * i1], bh[1][2 * i1 + 1], bh[0][i2], bh[1][i2]);
                            }
                    }
                    float* pbase = base + (pg - grp) * (region_floats(S::FIXED, N, DUAL, mx));
#pragma unroll
                    for (int i2 = 0; i2 < YT; i2++) {
                        gs[i2] += __shfl_xor_sync(0xffffffffu, gs[i2], 1);
                        gs[i2] += __shfl_xor_sync(0xffffffffu, gs[i2], 2);
                        if (c4 == 0) pbase[S::FIXED + 9 * N + g8 + 8 * i2] = gs[i2];
                    }
                    // the rows to their lanes, 16 at a time, through R' and the reflections' space
                    float* stage = pbase + 9 * N;
#pragma unroll
                    for (int i1 = 0; i1 < MT; i1++) {
#pragma unroll
                        for (int i2 = 0; i2 < YT; i2++) {
                            *reinterpret_cast<float2*>(stage + g8 * (N + 4) + 8 * i2 + 2 * c4) = make_float2(acc[i1][i2][0], acc[i1][i2][1]);
                            *reinterpret_cast<float2*>(stage + (g8 + 8) * (N + 4) + 8 * i2 + 2 * c4) = make_float2(acc[i1][i2][2], acc[i1][i2][3]);
                        }
                        __syncwarp();
                        if (grp == pg && (lane >> 4) == i1)
#pragma unroll
                            for (int m = 0; m < N / 2; m += 2) {
                                const ulonglong2 x2 = *reinterpret_cast<const ulonglong2*>(stage + (lane & 15) * (N + 4) + 2 * m);
                                r[0][m] = x2.x;
                                r[0][m + 1] = x2.y;
                            }
                        __syncwarp();
                    }
                }
                // R' past n is read as zero rows of T
                for (int e = n + lane; e < N; e += LPP)
#pragma unroll
                    for (int q = 0; q < 12; q++) sR[e * 12 + q] = 0.f;
            }
            __syncwarp();
            if (carry) {
                float s0 = 0.f;
#pragma unroll
                for (int m = 0; m < N / 2; m += 2) {
                    const ulonglong2 x2 = *reinterpret_cast<const ulonglong2*>(sX + crow * N + 2 * m);
                    r[1][m] = x2.x;
                    r[1][m + 1] = x2.y;
                    s0 += (lo_of(x2.x) + hi_of(x2.x)) + (lo_of(x2.y) + hi_of(x2.y));
                }
                if (crow < kQ) {
                    const float mean = mean_of(s0, fM, A.inv_m);
                    sXs[crow] = mean;
#pragma unroll
                    for (int m = 0; m < N / 2; m++)
                        r[1][m] = pk(2 * m < M ? lo_of(r[1][m]) - mean : 0.f, 2 * m + 1 < M ? hi_of(r[1][m]) - mean : 0.f);
                }
            }
        }
        __syncwarp();

        __syncthreads();
        // ---- 1. the reduction to tridiagonal form
        // two column counts: more would save multiply-adds but outgrow the instruction cache
        constexpr int HALF = N / 2 + 3 & ~3;
        Rows R;
        R.n = n;
        R.row0 = mat0 ? lane : 1 << 20;  // a lane without a row is never a pivot and writes beside the arrays
        R.carry = carry;
        R.last0 = mat0 && lane >= n - 2;
        R.entry = lane < N;
        const int at = int(base - smem);
        R.px0 = at + N + (mat0 ? lane : N + lane % N);
        R.pT = at + 6 * N;
        R.pR = at + 9 * N + min(crow, 11);
        R.pV0 = at + 21 * N + (VSTRIDE ? lane % N : lane - 1);
        int k0 = 0;
        reduce_while<N, N>(r, R, k0, N > 8 ? HALF : 0, smem, sx, sp);
        if constexpr (N > 8) reduce_while<HALF, N>(r, R, k0, 0, smem, sx, sp);
        // the last 2 x 2 block
        if (R.row0 == n - 2) {
            sd[n - 2] = 1.f + lo_of(r[0][0]);
            se[n - 2] = hi_of(r[0][0]);
        }
        if (R.row0 == n - 1) {
            sd[n - 1] = 1.f + hi_of(r[0][0]);
            se[n - 1] = 0.f;
        }
        if (carry) {
            smem[R.pR] = lo_of(r[1][0]);
            smem[R.pR + 12] = hi_of(r[1][0]);
        }
        __syncthreads();

        // ---- 2. shifts for this spectrum: Gershgorin's bound of the largest eigenvalue
        float kap = 0.f;
#pragma unroll 1
        for (int e = lane; e < n; e += LPP) kap = fmaxf(kap, sd[e] + fabsf(se[e]) + (e > 0 ? fabsf(se[e - 1]) : 0.f));
#pragma unroll
        for (int o = LPP / 2; o > 0; o >>= 1) kap = fmaxf(kap, __shfl_xor_sync(0xffffffffu, kap, o));
        int tab = 0;
        for (float lim = 4.f; tab < kTables - 1 && kap > lim; lim *= 4.f) tab++;
        const int np = T.n[tab];
        if (DUAL && N > 8 && active && lane == 0) noconv += kap <= kKappaMax ? 0 : 1;

        if constexpr (LPP == 16) {
            // lane = (shift j of 8, half h of the carried rows); the eighth shift is 0, for g alone
            const int j = lane & 7, h = lane >> 3;
            u64 z[5];
#pragma unroll
            for (int v = 0; v < 5; v++) z[v] = 0;
            // batches of seven shifts; both points of the warp take the larger number
            int nb = (np + 6) / 7;
            nb = max(nb, __shfl_xor_sync(0xffffffffu, nb, 16));
#pragma unroll 1
            for (int b = 0; b < nb; b++) {
                const int pj = 7 * b + j;
                const bool real = j < 7 && pj < np;
                const float s = real ? T.s[tab][pj] : (j == 7 ? 0.f : 1.f);
                float w = real ? T.w[tab][pj] : 0.f;
                if (DUAL) w = -w * rcp_approx(1.f + s);
                float inv[N], l[N];
                {
                    float piv = sd[0] + s;
#pragma unroll
                    for (int i2 = 0; i2 < N; i2++) {
                        inv[i2] = rcp_approx(piv);
                        const float e = se[i2];
                        l[i2] = e * inv[i2];
                        if (i2 + 1 < N) piv = fmaf(-e, l[i2], sd[i2 + 1] + s);
                    }
                }
#pragma unroll 1
                for (int v = 0; v < 5; v++) {
                    const int q = 5 * h + v;
                    float x[N];
                    x[0] = sR[q];
#pragma unroll
                    for (int i2 = 1; i2 < N; i2++) x[i2] = fmaf(-l[i2 - 1], x[i2 - 1], sR[i2 * 12 + q]);
                    x[N - 1] *= inv[N - 1];
#pragma unroll
                    for (int i2 = N - 2; i2 >= 0; i2--) x[i2] = fmaf(-l[i2], x[i2 + 1], x[i2] * inv[i2]);
                    if (q == 9 && j == 7 && b == 0) {  // T^-1 g'
#pragma unroll
                        for (int i2 = 0; i2 < N; i2++) sx[i2] = x[i2];
                    }
                    float* out = buf + (2 * j + h) * (N + 4);
#pragma unroll
                    for (int i2 = 0; i2 < N; i2 += 4)
                        *reinterpret_cast<float4*>(out + i2) = make_float4(w * x[i2], w * x[i2 + 1], w * x[i2 + 2], w * x[i2 + 3]);
                    __syncwarp();
                    if (2 * j < N) {
                        u64 a = z[0];  // rotated below, so that z needs no register index
                        const u64 one = pk(1.f, 1.f);
#pragma unroll
                        for (int jj = 0; jj < 8; jj++)
                            a = fma2(one, *reinterpret_cast<const u64*>(buf + (2 * jj + h) * (N + 4) + 2 * j), a);
                        z[0] = z[1]; z[1] = z[2]; z[2] = z[3]; z[3] = z[4]; z[4] = a;
                    }
                    __syncwarp();
                }
            }
            // s_q = R'_q . T^-1 g'; the rows of f(T) R' into buf [9][N + 4]
            if (lane < kQ) {
                float s = 0.f;
#pragma unroll
                for (int i2 = 0; i2 < N; i2++) s = fmaf(sR[i2 * 12 + lane], sx[i2], s);
                sXs[12 + lane] = s;
            }
            if (2 * j < N)
#pragma unroll
                for (int v = 0; v < 5; v++)
                    if (5 * h + v < kQ) *reinterpret_cast<u64*>(buf + (5 * h + v) * (N + 4) + 2 * j) = z[v];
            __syncwarp();
            // ---- 3. back through the reflections: lane = row
            u64 y[N / 2];
            const int q = min(lane, kQ - 1);
#pragma unroll
            for (int m = 0; m < N / 2; m += 2) {
                const ulonglong2 x2 = *reinterpret_cast<const ulonglong2*>(buf + q * (N + 4) + 2 * m);
                y[m] = x2.x;
                y[m + 1] = x2.y;
            }
            __syncwarp();
#pragma unroll 1
            for (int k = (n & ~1) - 3; k >= 0; k--) {
                u64 v[N / 2];
                u64 a0 = 0, a1 = 0;
#pragma unroll
                for (int m = 0; m < N / 2; m += 2) {
                    const ulonglong2 x2 = *reinterpret_cast<const ulonglong2*>(sV + k * N + 2 * m);
                    v[m] = x2.x;
                    v[m + 1] = x2.y;
                    a0 = fma2(v[m], y[m], a0);
                    a1 = fma2(v[m + 1], y[m + 1], a1);
                }
                const float f = -st[k] * (sum2(a0) + sum2(a1));
                const u64 ff = pk(f, f);
#pragma unroll
                for (int m = 0; m < N / 2; m++) y[m] = fma2(ff, v[m], y[m]);
            }
            if (lane < kQ)
#pragma unroll
                for (int m = 0; m < N / 2; m++) {
                    sR[(2 * m) * 12 + lane] = lo_of(y[m]);
                    sR[(2 * m + 1) * 12 + lane] = hi_of(y[m]);
                }
            __syncwarp();
        } else {
            // lane = (carried row q of 10, third g of the shifts); lanes 30, 31 repeat row 0 and are dropped
            const int g = min(lane / 10, 2), q = lane < 30 ? lane - 10 * g : 0;
            float acc[N];
#pragma unroll
            for (int i2 = 0; i2 < N; i2++) acc[i2] = 0.f;
            const int batches = (np + 2) / 3;
#pragma unroll 1
            for (int b = 0; b < batches; b++) {
                const int pj = 3 * b + g;
                float s = 1.f, w = 0.f;
                if (q == 9) {
                    s = 0.f;  // T^-1 g', once
                    w = pj == 0 ? 1.f : 0.f;
                } else if (pj < np) {
                    s = T.s[tab][pj];
                    w = T.w[tab][pj];
                    if (DUAL) w = -w * rcp_approx(1.f + s);
                }
                float x[N];
                float piv = sd[0] + s, y = sR[q];
                float* sl = base + (q == 9 ? 3 : g) * N;  // the multipliers, the same in all lanes of a shift
#pragma unroll
                for (int i2 = 0; i2 < N; i2++) {
                    const float inv = rcp_approx(piv), e = se[i2], l = e * inv;
                    x[i2] = y * inv;
                    sl[i2] = l;
                    if (i2 + 1 < N) {
                        piv = fmaf(-e, l, sd[i2 + 1] + s);
                        y = fmaf(-l, y, sR[(i2 + 1) * 12 + q]);
                    }
                }
                __syncwarp();
                acc[N - 1] = fmaf(w, x[N - 1], acc[N - 1]);
#pragma unroll
                for (int i2 = N - 2; i2 >= 0; i2--) {
                    x[i2] = fmaf(-sl[i2], x[i2 + 1], x[i2]);
                    acc[i2] = fmaf(w, x[i2], acc[i2]);
                }
                __syncwarp();
            }
            // the thirds together; every lane keeps the columns 3 u + g of its row
            const int l1 = lane < 30 ? (lane + 10) % 30 : 0, l2 = lane < 30 ? (lane + 20) % 30 : 0;
            constexpr int U = (N + 2) / 3;
            float z[U];
#pragma unroll
            for (int u = 0; u < U; u++) z[u] = 0.f;
#pragma unroll
            for (int i2 = 0; i2 < N; i2++) {
                const float f1 = __shfl_sync(0xffffffffu, acc[i2], l1), f2 = __shfl_sync(0xffffffffu, acc[i2], l2);
                const float t = (acc[i2] + f1) + f2;
                if (q == 9 && g == 0) sp[i2] = t;  // T^-1 g'
                if (i2 % 3 == g) z[i2 / 3] = t;
            }
            __syncwarp();
            {
                float s = 0.f;
#pragma unroll
                for (int u = 0; u < U; u++)
                    if (3 * u + g < N) s = fmaf(sR[(3 * u + g) * 12 + q], sp[3 * u + g], s);
                const float s1 = __shfl_sync(0xffffffffu, s, l1), s2 = __shfl_sync(0xffffffffu, s, l2);
                if (lane < kQ) sXs[12 + lane] = (s + s1) + s2;
            }
            __syncwarp();
            // ---- 3. back through the reflections: lane = (row, every third column)
#pragma unroll 1
            for (int k = n - 3; k >= 0; k--) {
                const float* v = sV + k * (2 * n - k - 1) / 2 - k - 1;  // entry i at v[i], i > k
                float vv[U];
                float a = 0.f;
#pragma unroll
                for (int u = 0; u < U; u++) {
                    const int i2 = 3 * u + g;
                    vv[u] = (i2 > k && i2 < n) ? v[i2] : 0.f;
                    a = fmaf(vv[u], z[u], a);
                }
                const float a1 = __shfl_sync(0xffffffffu, a, l1), a2 = __shfl_sync(0xffffffffu, a, l2);
                const float f = -st[k] * ((a + a1) + a2);
#pragma unroll
                for (int u = 0; u < U; u++) z[u] = fmaf(f, vv[u], z[u]);
            }
            if (lane < 30 && q < kQ)
#pragma unroll
                for (int u = 0; u < U; u++)
                    if (3 * u + g < N) sR[(3 * u + g) * 12 + q] = z[u];
            __syncwarp();
        }

        __syncthreads();
        // ---- the analysis members and their moments (update_xk + lbm2euler, letkf.cu:336-357); the rows of
        // Z are in sR [column][12]
#pragma unroll 1
        for (int m = lane; m < mx; m += LPP) {
            float xa[kQ];
            if constexpr (DUAL) {
                u64 acc[5];
                const int mm = min(m, M - 1);
                {
                    const ulonglong2 d0 = *reinterpret_cast<const ulonglong2*>(sX + 12 * mm);
                    const ulonglong2 d1 = *reinterpret_cast<const ulonglong2*>(sX + 12 * mm + 4);
                    acc[0] = d0.x; acc[1] = d0.y; acc[2] = d1.x; acc[3] = d1.y;
                    acc[4] = *reinterpret_cast<const u64*>(sX + 12 * mm + 8);
                }
#pragma unroll 2
                for (int o = 0; o < own_n; o++) {
                    const float y = sC[mm * N + o];
                    const u64 yy = pk(y, y);
                    const ulonglong2 z0 = *reinterpret_cast<const ulonglong2*>(sR + 12 * o);
                    const ulonglong2 z1 = *reinterpret_cast<const ulonglong2*>(sR + 12 * o + 4);
                    const u64 z2 = *reinterpret_cast<const u64*>(sR + 12 * o + 8);
                    acc[0] = fma2(yy, z0.x, acc[0]);
                    acc[1] = fma2(yy, z0.y, acc[1]);
                    acc[2] = fma2(yy, z1.x, acc[2]);
                    acc[3] = fma2(yy, z1.y, acc[3]);
                    acc[4] = fma2(yy, z2, acc[4]);
                }
#pragma unroll
                for (int q = 0; q < kQ; q++) {
                    const float zq = (q & 1) ? hi_of(acc[q / 2]) : lo_of(acc[q / 2]);
                    xa[q] = sXs[q] + fmaf(A.sqrt_beta, zq, sXs[12 + q]);
                }
            } else {
                const int mm = min(m, N - 1);
#pragma unroll
                for (int q = 0; q < kQ; q++) xa[q] = sXs[q] + fmaf(A.sqrt_beta, sR[mm * 12 + q], sXs[12 + q]);
            }
            if (active && m < M) {
#pragma unroll
                for (int q = 0; q < kQ; q++) {
                    bad |= !(xa[q] == xa[q]);
                    A.fout[(size_t(m) * kQ + q) * A.nxy + point] = xa[q];
                }
                float rsum = 0, mu = 0, mv = 0;
#pragma unroll
                for (int q = 0; q < kQ; q++) rsum += xa[q];
#pragma unroll
                for (int q = 0; q < kQ; q++) { mu += xa[q] * A.c * exq(q); mv += xa[q] * A.c * eyq(q); }
                float* mmac = A.mac + size_t(m) * 3 * A.nxy;
                mmac[point] = rsum;
                mmac[A.nxy + point] = mu / rsum;
                if (A.write_v) mmac[2 * A.nxy + point] = mv / rsum;
            }
        }
    }
    if (bad) atomicOr(A.stats + 2, 1);
    if (noconv) atomicAdd(A.stats + 1, noconv);
    if (tid == 0 && blockIdx.y == 0) {  // one direct solve per point, counted as one sweep
        const int w = max(0, min(tw, A.nx - bx0 * A.p)), h = max(0, min(A.nby * A.p, A.ny - by0 * A.p));
        atomicMax(A.stats + 0, 1);
        atomicAdd(A.stats + 3, w * h);
    }
}

// ---------------------------------------------------------------------------
// host side: the shifts
// ---------------------------------------------------------------------------
// Jacobi elliptic sn / cn of u for parameter m by the arithmetic-geometric mean
// (Abramowitz & Stegun 16.4, 17.6), and the complete integral K(m)
struct Agm {
    double a[24], c[24];
    int n = 0;
    explicit Agm(double m1) {  // m1 = 1 - m, the complementary parameter
        double b = std::sqrt(m1);
        a[0] = 1.0;
        c[0] = std::sqrt(1.0 - m1);
        while (n < 22 && std::fabs(c[n]) > 1e-16 * a[n]) {
            a[n + 1] = 0.5 * (a[n] + b);
            c[n + 1] = 0.5 * (a[n] - b);
            b = std::sqrt(a[n] * b);
            n++;
        }
    }
    double K() const { return M_PI / (2.0 * a[n]); }
    double tan_am(double u) const {  // sn / cn = tan(am u)
        double phi = std::ldexp(a[n] * u, n);
        for (int i = n; i > 0; i--) phi = 0.5 * (phi + std::asin(std::max(-1.0, std::min(1.0, c[i] / a[i] * std::sin(phi)))));
        return std::tan(phi);
    }
};

// t^-1/2 = D prod(t + c_2l) / prod(t + c_2l-1) on [1, kappa], c_l = (sn/cn)^2(l K / 2N) for
// m = 1 - 1/kappa (Zolotarev 1877), in partial fractions; D levels the relative error's two
// extremes, sampled at 16 points for each of its 2 N + 1 alternations.  Returns the error.
double zolotarev(double kappa, int N, double* s, double* w) {
    const Agm g(1.0 / kappa);
    const double K = g.K();
    double c[2 * kMaxPoles];  // (no allocation: the entry point is C's)
    for (int l = 1; l < 2 * N; l++) {
        const double t = g.tan_am(l * K / (2.0 * N));
        c[l] = t * t;
    }
    for (int i = 0; i < N; i++) {
        double v = 1.0;
        for (int l = 0; l < N - 1; l++) v *= (c[2 * l + 2] - c[2 * i + 1]) / (c[2 * (l < i ? l : l + 1) + 1] - c[2 * i + 1]);
        s[i] = c[2 * i + 1];
        w[i] = v;
    }
    double lo = 1e300, hi = -1e300;
    const int samples = 16 * (2 * N + 1);
    const double step = std::pow(kappa, 1.0 / samples);
    double t = 1.0;
    for (int e = 0; e <= samples; e++, t *= step) {
        double f = 0;
        for (int i = 0; i < N; i++) f += w[i] / (t + s[i]);
        f *= std::sqrt(t);
        lo = std::min(lo, f);
        hi = std::max(hi, f);
    }
    for (int i = 0; i < N; i++) w[i] *= 2.0 / (lo + hi);
    return (hi - lo) / (hi + lo);
}

const PoleTables& pole_tables() {
    static const PoleTables tables = [] {
        PoleTables T{};
        double kappa = 4.0;
        int n = 3;
        for (int b = 0; b < kTables; b++, kappa *= 4.0) {
            double s[kMaxPoles], w[kMaxPoles];
            while (zolotarev(kappa, n, s, w) > 2e-8 && n < kMaxPoles) n++;  // (a wider spectrum takes no fewer)
            T.n[b] = n;
            for (int i = 0; i < n; i++) {
                T.s[b][i] = float(s[i]);
                T.w[b][i] = float(w[i]);
            }
        }
        return T;
    }();
    return tables;
}

// the variants: order, lanes per point, dual
struct Variant {
    int n, lpp;
    bool dual;
    const void* fn;
};
const Variant kVariants[] = {
    {16, 16, false, (const void*)analysis_direct_kernel<16, 16, false>},
    {32, 32, false, (const void*)analysis_direct_kernel<32, 32, false>},
    {8, 16, true, (const void*)analysis_direct_kernel<8, 16, true>},
    {16, 16, true, (const void*)analysis_direct_kernel<16, 16, true>},
};

// The largest bound of a tile's traces of C^T C that the primal form solves; a tile with a larger one goes to the
// Jacobi kernel.  Rms error against FP64, of an increment, this kernel / the Jacobi kernel (64 x 32 points, an exact
// operator, by the largest trace):
//   primal  1e3: 16 members 1.3e-7 / 3.5e-7, 32 1.1e-7 / 5.6e-7; 1.4e4 (27 observations): 16 members 3.8e-7 / 3.2e-7,
//           32 1.4e-6 / 1.3e-6; 1.5e6: 6.0e-7 / 3.8e-7, 7.3e-5 / 2.9e-5; 1.5e7: 6.2e-7 / 3.7e-7, 1.2e-4 / 4.6e-5
//   dual    order 16, 32 members: 1e3 1.4e-8 / 2.9e-7, 1.6e5 1e-7 / 3.9e-4, 1e7 5e-6 / 5e-3, 1.6e8 2e-4 / 0.14, 6e8 5e-3 /
//           2e4 (not converged); order 8: 1.8e-8 up to 6e11: no limit
// The reduction keeps an eigenvalue to 2^-24 of the largest; in the member space, one of every window's is the
// smallest possible (the members' sum), in the observation space hardly any is.
float trace_limit(bool dual) { return dual ? INFINITY : 3e4f; }

template <int N, int LPP, bool DUAL>
int region_of(int mx) {
    using S = Shape<N, LPP, DUAL>;
    return region_floats(S::FIXED, N, DUAL, mx) * S::GPW;
}
int warp_floats(int v, int mx) {
    switch (v) {
        case 0: return region_of<16, 16, false>(mx);
        case 1: return region_of<32, 32, false>(mx);
        case 2: return region_of<8, 16, true>(mx);
        default: return region_of<16, 16, true>(mx);
    }
}

// the most observations of a point: window slots within the Gaspari-Cohn support (2 d_local); any number above
// 16 ends the search, since the observation space is then no choice.  (All p^2 patterns took the host 56 us a
// call at p = 32, 1 ms at 128; from p = 4 on the first one has more.)
int max_obs(int p, int nox, int nl_off, int nl, double dloc) {
    if (p == 1) return 3 * nox * nox;
    int best = 0;
    for (int pj = 0; pj < p; pj++)
        for (int pi = 0; pi < p; pi++) {
            int n = 0;
            for (int b = 0; b < nox; b++)
                for (int a = 0; a < nox; a++) {
                    const int di = pi - (a - nl_off) * p, dj = pj - (b - nl_off) * p;
                    if (std::abs(di) > nl * p || std::abs(dj) > nl * p) continue;
                    if (std::sqrt(double(di * di + dj * dj)) / (dloc + 1e-6) <= 2.0) n += 3;
                }
            best = std::max(best, n);
            if (best > 16) return best;
        }
    return best;
}

struct Plan {
    int variant = -1;
    int nbx = 1, nby = 1, ms = 0;
    size_t smem = 0;
};
Plan make_plan(int M, int p, int nox, int nl_off, int nl, double dloc, int nsx, int nsy) {
    Plan P;
    const int obs = max_obs(p, nox, nl_off, nl, dloc), nobs = 3 * nox * nox;
    // The smaller of the two spaces.  A call of the entry point, this way / all by the Jacobi kernel (us): pointwise (3
    // observations) at 128^2, 9 members 73 / 134, 16: 79 / 137, 17: 93 / 603, 32: 114 / 667; DA_XYPRUNE 2 (15) at 160 x 96,
    // 16: 95 / 173, 17: 103 / 689, 32: 159 / 776; DA_XYPRUNE 4, LETKF_RLOC_LEN 1 (42) at 256^2, 9: 289 / 420, 16: 353 / 467,
    // 17: 1071 / 2217, 32: 1658 / 2388.
    // Up to 8 members the gain was small (pointwise at 128^2, 4 members 70 / 51, 8: 72 / 80), and the entry point keeps
    // lbl_assimilate's analysis to the bit, within the 1e-7 that its velocities are held to there.
    if (M <= 8 || M > 32) return P;
    int v = 1;
    if (obs <= 16 && obs < M) v = obs <= 8 ? 2 : 3;
    else if (M <= 16) v = 0;
    const Variant& V = kVariants[v];
    // tiles of whole rounds: 12 x 4 points over twelve warps, 8 x 4 over eight (two points a warp)
    P.nbx = std::min(nsx, std::max(1, (V.lpp == 32 ? 12 : 8) / p));
    P.nby = std::min(nsy, std::max(1, 4 / p));
    const int mx = (M + 3) & ~3;
    P.ms = 4 * (((V.dual ? mx : V.n) / 4) | 1);
    for (;;) {
        const size_t slots = 3 * size_t(P.nbx + nox - 1) * (P.nby + nox - 1);
        P.smem = sizeof(float) * (slots * P.ms + ((slots + 3) & ~size_t(3)) + ((nobs + 3) & ~3) +
                                  size_t(warps_of(V.n)) * warp_floats(v, mx));
        if (P.smem <= kAnalysisSmemLimit) break;
        if (P.nbx > 1) P.nbx /= 2;
        else if (P.nby > 1) P.nby /= 2;
        else return P;  // the window alone is too large (none that the entry point accepts: 187 kB at most)
    }
    P.variant = v;
    return P;
}

void launch(const Plan& P, DirParams& A, cudaStream_t s) {
    A.nbx = P.nbx;
    A.nby = P.nby;
    A.ms = P.ms;
    const int tiles = ((A.nsx + P.nbx - 1) / P.nbx) * ((A.nsy + P.nby - 1) / P.nby);
    // A tile is at least one block of p x p points, whose rounds follow one another: from p = 9 or 10 on, CTAs of at
    // most six rounds share it (each stages the window).  With one CTA a tile, an analysis of 64^2 x 16 took 248 us
    // at p = 16 and 960 at p = 32, where the Jacobi kernel takes 159 and 149 (32 members: 826, 3200; 359, 310).
    const Variant& V = kVariants[P.variant];
    const int per_round = warps_of(V.n) * (32 / V.lpp);
    const int rounds = (P.nbx * A.p * P.nby * A.p + per_round - 1) / per_round;
    const int shares = (rounds + kMaxRounds - 1) / kMaxRounds;
    A.rounds = (rounds + shares - 1) / shares;
    PoleTables T = pole_tables();
    void* args[] = {&A, &T};
    cudaLaunchKernel(V.fn, dim3(tiles, shares), dim3(32 * warps_of(V.n)), args, P.smem, s);
}

}  // namespace

int direct_prepare() {
    int rc = 0;
    for (const Variant& v : kVariants)
        rc |= int(cudaFuncSetAttribute(v.fn, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kAnalysisSmemLimit)));
    (void)pole_tables();
    return rc;
}

Direct launch_analysis_direct_args(const AnalysisArgs& g, cudaStream_t s) {
    const int nsx = g.nx / g.p, nsy = g.ny / g.p;
    const Plan P = make_plan(g.M, g.p, g.nox, g.nl_off, g.nl, g.dloc, nsx, nsy);
    if (P.variant < 0) return Direct::kNone;
    DirParams A{};
    A.fin = g.f_in; A.fout = g.f_out; A.mac = g.mac_out; A.dY = g.dY; A.dyo = g.dyo;
    A.wtab = reinterpret_cast<const int4*>(g.wtab);
    A.wcnt = g.wtab + size_t(4) * g.p * g.p * g.nobs;
    A.stats = g.stats;
    A.nx = g.nx; A.ny = g.ny; A.nxy = g.nx * g.ny; A.M = g.M;
    A.p = g.p; A.nsx = nsx; A.nsy = nsy; A.nsites = nsx * nsy; A.nobs = g.nobs; A.nox = g.nox;
    A.nl_off = g.nl_off;
    A.inv_sqrt_a = float(1.0 / std::sqrt((g.M - 1) / g.covinf));
    A.sqrt_beta = float(std::sqrt(g.covinf));
    A.c = g.c;
    A.inv_m = 1.f / float(A.M);
    A.write_v = g.write_v;
    const Variant& V = kVariants[P.variant];
    A.limit = trace_limit(V.dual);
    launch(P, A, s);
    return std::isinf(A.limit) ? Direct::kAll : Direct::kLeavesSome;
}

}  // namespace lbl

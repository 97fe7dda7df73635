// The Cauchy step of a recursion level in exact double-precision integer arithmetic.
//
//   H[g, r, n] = hinf[gsrc[g], m, gj[g], n] + sum_{i < ncol[g]} 2 / (rowd[g, r] - cold[g, i]) res[col[g, i], n]
//
// with the terms of k_cauchy2 .. k_cauchy4: sign(x / d) floor(|x| 2^32 / |d|) for x aligned to the column's largest
// exponent, summed exactly and rounded once, then h_inf added (one rounding): bit-identical to them.
//
// The dividend X = x 2^32 is written in W-bit digits carrying x's sign, as doubles (k_cauchy_align_fp).  From
// the top digit down, c = r 2^W + digit (exact: |c| < 2^53), q = c / d rounded to the nearest integer by adding
// 1.5 2^52 (its low mantissa bits are then q), r = c - q d (exact).  q may miss the floor by one either way: the
// remainder is only required to stay near d / 2, and sum_j q_j 2^(W j) d + r = X holds all the same, so that one
// correction after the last digit (truncation towards zero from the sign of r) gives the exact quotient.  The bits
// of q + 1.5 2^52 are added into a 64-bit integer per digit position; the number of terms times the bits of
// 1.5 2^52 is subtracted at the end.
//
// Exactness: |inv - 1/d| <= 2^-53 / |d|, so |q - c / d| <= 1/2 + |c / d| 2^-53 and |r| <= |d| (1/2 + 1.52 2^(W - 53));
// with |d| <= dmax, |c| <= (dmax (1/2 + 1.52 2^(W-53)) + 1) 2^W, which cauchy_fp_bits keeps below 2^53; |q| <=
// 1.52 2^W + 1 < 2^51.
//
// What bounds it: latency (the digit steps of a chain depend on one another, 12 to 16 warps per SM by the 2 ND
// registers of the digit sums) and the rounding of each row; the double-precision pipe is a third busy (4 of its
// instructions per 46-bit digit).  The integer form spent a multiply-high at half the multiply rate, a shift, a mask,
// two multiplies, a compare, two selects and two shared-memory accesses on every 24-bit digit.
#pragma once
#include <atomic>

#include "kernels.cuh"

namespace b3d {

// digit width for divisors up to dmax (the exactness bound above)
B3D_CX int cauchy_fp_bits(i64 dmax) { return dmax <= 247 ? 46 : (dmax <= 480 ? 45 : (dmax <= 1900 ? 43 : 37)); }
B3D_CX int cauchy_fp_digits(int L, int W) { return (32 * (L + 1) + W - 1) / W; }
B3D_CX int cauchy_fp_table(int W) { return W == 46 ? 248 : (W == 45 ? 481 : (W == 43 ? 1901 : 1)); }
constexpr int kCauchyFpMaxThreads = 128;

// Column tiles of at most 32 columns, evenly sized (150 columns: five of 30).  The digits of a tile are contiguous,
// X[((g ntile + nt) Kc + i) ND TNp + j TNp + tn] with TNp = TN rounded up to even, so that the two terms of a
// stage are one run of 16-byte words.
struct CauchyFpTile {
    int ntile, TN, TNp;
};
B3D_CX CauchyFpTile cauchy_fp_tile(i64 N) {
    CauchyFpTile t{};
    t.ntile = (int)((N + 31) / 32);
    t.TN = t.ntile ? (int)((N + t.ntile - 1) / t.ntile) : 0;
    t.TNp = (t.TN + 1) / 2 * 2;
    return t;
}

// largest exponent of each column (g, n): 32 columns x 8 slices of the terms per block (a thread per column alone
// walked up to ncol dependent loads: 1.22 ms per 1024-bit task of 39 levels, 0.25 in slices; 1280 bits 5.1, 0.88)
constexpr int kColSlices = 8;

template <int L>
__global__ void __launch_bounds__(32 * kColSlices) k_cauchy_colmax(const int32_t* __restrict__ rm, const i64* __restrict__ re,
                                                                   i64 rplane, CauchyLevel lv, i64* __restrict__ oe) {
    __shared__ i64 part[kColSlices][32];
    const int lane = threadIdx.x & 31, sl = threadIdx.x >> 5;
    const i64 N = lv.N, total = lv.nb * N, t = blockIdx.x * (i64)32 + lane;
    i64 E = EZ;
    if (t < total) {
        i64 g, n;
        split2(t, N, total, n, g);
        const i64 ncol = lv.ncol[g];
        const i64* col = lv.col + g * lv.Kc;
#pragma unroll 4
        for (i64 i = sl; i < ncol; i += kColSlices) {
            const i64 ix = col[i] * N + n;
            const i64 ei = re[ix];
            if (rm[(L - 1) * rplane + ix] != 0 && ei > E) E = ei;
        }
    }
    part[sl][lane] = E;
    __syncthreads();
    if (sl == 0 && t < total) {
#pragma unroll
        for (int s = 1; s < kColSlices; s++) E = part[s][lane] > E ? part[s][lane] : E;
        oe[t] = E;
    }
}

// X[g][i][n] aligned to its column's exponent, as ND signed W-bit digits (digit 0: the top one, whose sign bit is
// x's sign even where the digit is zero), in the tiled order of CauchyFpTile
template <int L, int W>
__global__ void __launch_bounds__(128) k_cauchy_align_fp(const int32_t* __restrict__ rm, const i64* __restrict__ re, i64 rplane,
                                                         CauchyLevel lv, const i64* __restrict__ ce, CauchyFpTile tl,
                                                         double* __restrict__ om) {
    constexpr int ND = cauchy_fp_digits(L, W);
    const i64 t = blockIdx.x * (i64)blockDim.x + threadIdx.x;
    const i64 N = lv.N;
    if (t >= lv.nb * lv.Kc * N) return;
    i64 n, i, g;
    split3(t, N, lv.Kc, lv.nb * lv.Kc * N, n, i, g);
    if (i >= lv.ncol[g]) return;                             // never read
    const i64 E = ce[g * N + n];
    u32 a[L], s[L];
    bool neg = false;
    zero(s);
    if (E != EZ) {
        const i64 ix = lv.col[g * lv.Kc + i] * N + n;
        const i64 ei = re[ix];
        neg = load_mag<L>(rm, rplane, ix, a);
        if (is_zero(a) || ei == EZ || E - ei >= 32 * L) neg = false;
        else shr(a, (int)(E - ei), s);
    }
    const u32 sg = neg ? 0x80000000u : 0u;
    const int nt = (int)n / tl.TN;
    double* o = om + ((g * tl.ntile + nt) * lv.Kc + i) * (i64)(ND * tl.TNp) + ((int)n - nt * tl.TN);
#pragma unroll
    for (int j = 0; j < ND; j++) {
        const int lo = W * (ND - 1 - j), li = lo >> 5, bo = lo & 31;      // dividend limb k = s[k - 1], limb 0 is zero
        u32 w[3];
#pragma unroll
        for (int q = 0; q < 3; q++) w[q] = (li + q >= 1 && li + q <= L) ? s[li + q - 1] : 0u;
        const u32 l = fsr(w[0], w[1], bo), h = fsr(w[1], w[2], bo) & ((1u << (W - 32)) - 1u);
        const double v = __dadd_rn(__hiloint2double((int)(h | 0x43300000u), (int)l), -4503599627370496.0);
        o[j * tl.TNp] = __hiloint2double((int)((u32)__double2hiint(v) ^ sg), __double2loint(v));
    }
}

// digit sums acc (acc[j]: the sum of digit j, 0 = top) rounded and added to h_inf; stored at element t
template <int L, int W, int ND>
__device__ __forceinline__ void cauchy_fp_finish(const u64 (&acc)[ND], u64 bias, i64 E, const int32_t* hm, const i64* he,
                                                 i64 hplane, i64 hidx, int32_t* om, i64* oe, i64 oplane, i64 t) {
    u64 f[ND];                                               // W-bit fields, f[0] the lowest; the top one signed
    i64 carry = 0;
#pragma unroll
    for (int j = ND - 1; j > 0; j--) {
        const i64 v = (i64)(acc[j] - bias) + carry;
        f[ND - 1 - j] = (u64)v & ((1ull << W) - 1);
        carry = v >> W;
    }
    f[ND - 1] = (u64)((i64)(acc[0] - bias) + carry);
    u32 w[L + 3];                                            // two's complement limbs, value 2^(E - 31)
#pragma unroll
    for (int k = 0; k < L + 3; k++) {
        const int lo = 32 * k, x = lo / W < ND ? lo / W : ND - 1, b = lo - W * x;
        if (x == ND - 1) w[k] = (u32)((i64)f[x] >> (b < 63 ? b : 63));
        else w[k] = (u32)(f[x] >> b) | (W - b < 32 ? (u32)(f[x + 1] << (W - b)) : 0u);
    }
    const bool neg = (w[L + 2] >> 31) != 0;
    if (neg) negate(w);
    u32 s[L];
    i64 es;
    bool ns = false;
    if (E != EZ && round_mag<L>(w, E - 31, s, &es)) ns = neg;
    else { zero(s); es = EZ; }
    u32 h[L], out[L];
    const bool nh = load_mag<L>(hm, hplane, hidx, h);
    bool no;
    i64 eo;
    add_norm<L>(s, ns, es, h, nh, he[hidx], out, &no, &eo);
    store_signed<L>(om, oplane, t, out, no);
    oe[t] = eo;
}

// One block: TR rows x TN columns n of one group (thread = (row, n), columns innermost); four terms at a time, four
// independent chains.  The digits of the four are staged in shared memory by cp.async, the next four while these are
// divided: read from global memory where the digit steps need them, their latency was exposed at every digit (25.8 ms
// per 1024-bit task of six right-hand sides against 12.1; the integer form 23.0).  Other splits of the same chains, per
// 1024-bit / 1280-bit task: two rows x two terms 12.9 / 31.4, two rows x four terms 13.9 / 35.0, one row x two terms
// 12.5 / 33.7, one row x four terms 12.1 / 29.2 (five blocks per SM spill: 17.7; four at 31 digits: 41.7).
// grid: group-major, then column tiles, then row tiles.
constexpr int kCauchyFpTerms = 4;

template <int L, int W>
__global__ void __launch_bounds__(kCauchyFpMaxThreads, cauchy_fp_digits(L, W) <= 25 ? 4 : 3) k_cauchy5(
    const double* __restrict__ xm, const i64* __restrict__ xe, const int32_t* __restrict__ hm, const i64* __restrict__ he,
    i64 hplane, CauchyLevel lv, CauchyFpTile tl, int TR, int rtile, int32_t* __restrict__ om, i64* __restrict__ oe, i64 oplane) {
    constexpr int ND = cauchy_fp_digits(L, W), KT = kCauchyFpTerms;
    // (1 / d, d) by divisor -NT < d < NT (the plan's divisors are at most the bound of cauchy_fp_bits; W = 37
    // divides per term)
    constexpr int NT = cauchy_fp_table(W);
    constexpr double MG = 6755399441055744.0;                // 1.5 2^52
    extern __shared__ __align__(16) double c5_smem[];        // table | 2 stages x (KT terms, ND, TNp) digits
    double2* tab = reinterpret_cast<double2*>(c5_smem) + (NT - 1);
    const int TN = tl.TN, TNp = tl.TNp;
    double* xs = c5_smem + 2 * (2 * NT - 1);
    for (int v = (int)threadIdx.x - (NT - 1); v < NT; v += blockDim.x)
        tab[v] = make_double2(v ? __drcp_rn((double)v) : 0.0, (double)v);
    const int rt = blockIdx.x % (u32)rtile, gn = blockIdx.x / (u32)rtile, nt = gn % tl.ntile;
    const i64 g = gn / tl.ntile, N = lv.N;
    const int tr = threadIdx.x / TN, tn = threadIdx.x - tr * TN;
    const i64 n = (i64)nt * TN + tn, row = (i64)rt * TR + tr;
    const int nrow = (int)lv.nrow[g], ncol = (i64)rt * TR < nrow ? (int)lv.ncol[g] : 0;
    const bool active = tr < TR && n < N && row < lv.Mr, live = active && row < nrow;
    const i64* cold = lv.cold + g * lv.Kc;
    const int D = active ? (int)lv.rowd[g * lv.Mr + row] : 0;
    const i64 E = active ? xe[g * N + n] : EZ;
    const int term = ND * TNp;                               // doubles per term (even: 16-byte words)
    const double* x = xm + (g * tl.ntile + nt) * lv.Kc * (i64)term;
    auto fetch = [&](int i, int st) {                        // terms i .. i + KT - 1 of the tile
        const int words = (ncol - i < KT ? ncol - i : KT) * term / 2;
        const double* src = x + (i64)i * term;
        const u32 dst = (u32)__cvta_generic_to_shared(xs + st * KT * term);
        for (int q = threadIdx.x; q < words; q += blockDim.x)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + 16 * q), "l"(src + 2 * q) : "memory");
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    u64 acc[ND];
#pragma unroll
    for (int j = 0; j < ND; j++) acc[j] = 0;
    int st = 0;
    if (ncol > 0) fetch(0, 0);
    int cd[KT];
#pragma unroll
    for (int b = 0; b < KT; b++) cd[b] = b < ncol ? (int)cold[b] : 0;
#pragma unroll 1
    for (int i = 0; i < ncol; i += KT, st ^= 1) {
        if (i + KT < ncol) {
            fetch(i + KT, st ^ 1);
            asm volatile("cp.async.wait_group 1;" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
        }
        int cn[KT];
#pragma unroll
        for (int b = 0; b < KT; b++) cn[b] = i + KT + b < ncol ? (int)cold[i + KT + b] : 0;
        __syncthreads();
        if (live && E != EZ) {
            // a dead chain (vanishing difference, term beyond the last) keeps q = 0 and never feeds its remainder back
            const double* p[KT];
            int d[KT];
            double inv[KT], dd[KT], sw[KT], r[KT];
#pragma unroll
            for (int b = 0; b < KT; b++) {
                p[b] = xs + (st * KT + (i + b < ncol ? b : 0)) * term + tn;
                d[b] = i + b < ncol ? D - cd[b] : 0;
                if (NT > 1) {
                    const double2 e = tab[min(max(d[b], 1 - NT), NT - 1)];
                    inv[b] = e.x;
                    dd[b] = e.y;
                } else {
                    dd[b] = (double)d[b];
                    inv[b] = d[b] ? __drcp_rn(dd[b]) : 0.0;
                }
                sw[b] = d[b] ? (double)(1ull << W) : 0.0;
                r[b] = 0.0;
            }
            u32 xneg[KT];
#pragma unroll
            for (int j = 0; j < ND; j++) {
                double v[KT], cc[KT];
                u64 qb[KT];
#pragma unroll
                for (int b = 0; b < KT; b++) {
                    v[b] = p[b][j * TNp];
                    if (j == 0) xneg[b] = (u32)__double2hiint(v[b]) >> 31;
                }
#pragma unroll
                for (int b = 0; b < KT; b++) cc[b] = __fma_rn(r[b], sw[b], v[b]);
#pragma unroll
                for (int b = 0; b < KT; b++) {
                    const double qp = __fma_rn(cc[b], inv[b], MG);
                    qb[b] = (u64)__double_as_longlong(qp);
                    r[b] = __dadd_rn(qp, -MG);
                }
#pragma unroll
                for (int b = 0; b < KT; b++) r[b] = __fma_rn(-r[b], dd[b], cc[b]);
#pragma unroll
                for (int b = 0; b < KT; b += 2) acc[j] = acc[j] + qb[b] + qb[b + 1];
            }
#pragma unroll
            for (int b = 0; b < KT; b++) {                   // truncation towards zero
                const bool xn = xneg[b] != 0;
                if (d[b] != 0 && r[b] != 0.0 && (r[b] < 0.0) != xn) acc[ND - 1] -= xn != (d[b] < 0) ? ~0ull : 1ull;
            }
        }
#pragma unroll
        for (int b = 0; b < KT; b++) cd[b] = cn[b];
        __syncthreads();                                     // this stage is refilled next
    }
    if (!active) return;
    const u64 bias = (u64)((ncol + KT - 1) / KT * KT) * 0x4338000000000000ull;
    const i64 hidx = ((lv.gsrc[g] * lv.hlevels + lv.m) * lv.Jh + lv.gj[g]) * N + n;
    const i64 t = (g * lv.Mr + row) * N + n;
    if (live) {
        cauchy_fp_finish<L, W, ND>(acc, bias, E, hm, he, hplane, hidx, om, oe, oplane, t);
    } else {
        u32 z[L];
        zero(z);
        store_signed<L>(om, oplane, t, z, false);
        oe[t] = EZ;
    }
}

template <int L>
struct CauchyFpLaunch {
    static int align(const int32_t* rm, const i64* re, i64 rplane, const CauchyLevel& lv, i64 dmax, double* om, i64* oe,
                     cudaStream_t st);
    static int level(const double* xm, const i64* xe, const int32_t* hm, const i64* he, i64 hplane,
                     const CauchyLevel& lv, i64 dmax, int32_t* om, i64* oe, i64 oplane, cudaStream_t st);
};

#ifdef B3D_DEFINE_LAUNCH
template <int L>
int CauchyFpLaunch<L>::align(const int32_t* rm, const i64* re, i64 rplane, const CauchyLevel& lv, i64 dmax, double* om,
                             i64* oe, cudaStream_t st) {
    const i64 n = lv.nb * lv.N, ne = n * lv.Kc;
    if (n == 0) return 0;
    k_cauchy_colmax<L><<<(unsigned)((n + 31) / 32), 32 * kColSlices, 0, st>>>(rm, re, rplane, lv, oe);
    if (ne > 0) {
        const unsigned grid = (unsigned)((ne + 127) / 128);
        const CauchyFpTile tl = cauchy_fp_tile(lv.N);
        switch (cauchy_fp_bits(dmax)) {
            case 46: k_cauchy_align_fp<L, 46><<<grid, 128, 0, st>>>(rm, re, rplane, lv, oe, tl, om); break;
            case 45: k_cauchy_align_fp<L, 45><<<grid, 128, 0, st>>>(rm, re, rplane, lv, oe, tl, om); break;
            case 43: k_cauchy_align_fp<L, 43><<<grid, 128, 0, st>>>(rm, re, rplane, lv, oe, tl, om); break;
            default: k_cauchy_align_fp<L, 37><<<grid, 128, 0, st>>>(rm, re, rplane, lv, oe, tl, om); break;
        }
    }
    return (int)cudaGetLastError();
}

template <int L>
int CauchyFpLaunch<L>::level(const double* xm, const i64* xe, const int32_t* hm, const i64* he, i64 hplane,
                             const CauchyLevel& lv, i64 dmax, int32_t* om, i64* oe, i64 oplane, cudaStream_t st) {
    if (lv.nb == 0 || lv.Mr == 0 || lv.N == 0) return 0;
    const CauchyFpTile tl = cauchy_fp_tile(lv.N);
    int TR = kCauchyFpMaxThreads / tl.TN;                    // as many rows as fit the block
    if (TR > lv.Mr) TR = (int)lv.Mr;
    const i64 rtile = (lv.Mr + TR - 1) / TR, blocks = lv.nb * tl.ntile * rtile;
    if (blocks > 0x7FFFFFFF) return (int)cudaErrorInvalidConfiguration;
    const int th = (tl.TN * TR + 31) / 32 * 32;
    const unsigned long long dbit = device_bit();
    switch (cauchy_fp_bits(dmax)) {
#define B3D_C5(WB) {                                                                                                  \
        constexpr int per = 2 * kCauchyFpTerms * cauchy_fp_digits(L, WB), tab = 2 * (2 * cauchy_fp_table(WB) - 1);    \
        static std::atomic<unsigned long long> opted{0};     /* devices whose limit is raised */                      \
        if (!(opted.load(std::memory_order_relaxed) & dbit) || !dbit) {                                               \
            const int rc = (int)cudaFuncSetAttribute(k_cauchy5<L, WB>, cudaFuncAttributeMaxDynamicSharedMemorySize,   \
                                                     (tab + per * 32) * 8);                                           \
            if (rc) return rc;                                                                                        \
            opted.fetch_or(dbit, std::memory_order_relaxed);                                                          \
        }                                                                                                             \
        k_cauchy5<L, WB><<<(unsigned)blocks, th, (tab + per * tl.TNp) * 8, st>>>(xm, xe, hm, he, hplane, lv, tl, TR,  \
                                                                                (int)rtile, om, oe, oplane);          \
        break;                                                                                                        \
    }
        case 46: B3D_C5(46)
        case 45: B3D_C5(45)
        case 43: B3D_C5(43)
        default: B3D_C5(37)
#undef B3D_C5
    }
    return (int)cudaGetLastError();
}
#endif

}  // namespace b3d

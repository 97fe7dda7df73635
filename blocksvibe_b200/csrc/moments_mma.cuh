// The staged moments' flush on the sm_100a INT8 tensor cores (tcgen05.mma.kind::i8, s8 x s8 -> s32 in TMEM).
//
//   mom[row, k, c] (+)= round( sum_{w < W} n_w^k Y[w, row, c] ),   n_w = m0 + w + row_shift[row]
//
// is a contraction over the levels w with integer coefficients.  Per (row, c) the terms Y are aligned to the largest of
// them, cut PDV digits below it and written in balanced base-256 digits (the bytes of v + 0x80...80, each minus 128), as
// are the n^k.  With digit b = F cc + beta of n^k,
//     n^k Y = sum_cc 256^(F cc) sum_p 256^p D[(k, cc), p],   D[(k, cc), p] = sum_{beta < F, w} nk_{F cc + beta}[w] y_w[p - beta],
// and D is one GEMM: rows (k, cc) on the TMEM lanes, positions p on its columns, K = (beta, w).  The operand of step beta is
// the same digit matrix read beta rows earlier: in the canonical no-swizzle layout (8 rows of 16 bytes contiguous, SBO =
// 128) a row is 16 bytes, so a descriptor may start at any of them.  F = 4 makes the rows of an order a whole limb apart
// and keeps R = 27 in one tile of 128 lanes (314 rows at F = 1).  A lane carries its row of D into limbs along the columns
// (no transposition, two warps half of the limbs each), and a warp per (k, c), two limbs per lane, adds the rows
// of its order and rounds (carries and leading limbs by ballots).
//
// Cut: Y loses less than 2^(E - 8 PDV), E the exponent above the largest |Y|.  8 PDV = 32 (LO + 2) + 32 KW bits covers
// n^k < 2^(32 KW), so the sum is exact above 2^-(32 LO + 64) of its largest term, the contract of k_moments_flush, as long
// as that term has n >= 1: rows with n = 0 in the window stay with k_moments_flush.
//
// What bounds it: latency and integer issue of the limb work around the MMAs (per four columns of R = 11, W = 40: digits
// 11 K clocks, TMEM to limbs 13 K, sums and rounding 14 K, stores 4 K, the tensor pipe 5 % busy, two CTAs per SM).  The
// cost of a column grows with R but hardly with W, that of k_moments_flush with W R1: which form takes a window is
// flush_mma_pays, below.
#pragma once
#include <atomic>
#include <cmath>

#include "kernels.cuh"
#include "pole_mma.cuh"

namespace b3d {

constexpr int kFlushMmaThreads = 256;
constexpr int kFlushParts = kFlushMmaThreads / 128;        // warps that reach a TMEM lane
constexpr int kFlushMmaMaxR1 = 32;
constexpr int kFlushF = 4;                                 // digits of n^k per row: rows are whole limbs apart

struct FlushGeom {
    int CB;                 // columns per work item (a power of two)
    int Kp;                 // levels padded to the MMA's K step
    int PDV, PR, NCOL;      // digits kept of a term, rows of a digit matrix (16 zero rows on either side), MMA columns
    int VW, TW, P, RS;      // limbs read of a row of D, limbs of a sum, zero limbs below them, row stride of the limb buffers
    int Mrows;              // rows (k, cc)
    size_t a_bytes, b_stride, smem;
};

struct FlushMmaArgs {
    const int32_t* ym; const i64* ye; i64 yplane;
    const i64* row_shift;
    i64 m0, rows, N;
    int W, R1, NN, KW;
    const u32* nk; const int32_t* nkb;
    int32_t* mm; i64* me; i64 mplane;
    int* err;
};

// digits of n^k in balanced base 256 for a value of `bits` bits
B3D_CX int flush_digits(int bits) { return bits / 8 + 1; }

// geometry for orders k < R1 of integers n < NN; false where the tensor-core form does not apply
inline bool flush_mma_geom(int LO, int W, int R1, int NN, int KW, FlushGeom* out) {
    if (W < 1 || W > 128 || R1 > kFlushMmaMaxR1 || NN < 2) return false;
    constexpr int F = kFlushF;
    FlushGeom g{};
    const double lg = std::log2((double)(NN > 2 ? NN - 1 : 2));
    int last = 0;                                       // rows of the highest order
    for (int k = 0; k < R1; k++) {
        const int nd = flush_digits((int)std::floor(k * lg + 1e-9) + 1);      // the bit length of (NN - 1)^k, or one more
        last = (nd + F - 1) / F;
        g.Mrows += last;
    }
    if (g.Mrows > 128) return false;
    g.Kp = (W + 31) / 32 * 32;
    g.PDV = 4 * (LO + 2) + 4 * KW;
    const int PD = (g.PDV + 1 + 15) / 16 * 16;
    g.PR = PD + 32;
    g.NCOL = PD + 16;
    if (g.NCOL > 256) return false;
    g.TW = g.PDV / 4 + KW + 1;                          // |sum| < 2^(8 PDV + 32 KW + 7)
    if (g.TW > 64) return false;                        // two limbs per lane of a warp
    g.VW = g.NCOL / 4 < (g.TW + 3) / 4 * 4 ? g.NCOL / 4 : (g.TW + 3) / 4 * 4;
    g.RS = g.Mrows | 1;
    g.a_bytes = (size_t)F * 128 * g.Kp;
    g.b_stride = (size_t)g.PR * g.Kp + 16;
    g.P = last;
    for (g.CB = 4; g.CB >= 1; g.CB /= 2) {
        g.smem = g.a_bytes + (((size_t)g.CB * g.b_stride + 15) & ~(size_t)15) + (size_t)g.CB * g.RS * (4 * (g.P + g.TW + 3) + 16) +
                 (size_t)(4 * LO + 8) * R1 * g.CB + 32;
        if (g.smem <= 220 * 1024) break;
    }
    if (g.CB < 1) return false;
    *out = g;
    return true;
}

#ifdef B3D_DEFINE_LAUNCH
// bit i of a 64-bit mask: the predicate of limb i, two limbs per lane (i = lane, lane + 32)
__device__ __forceinline__ u64 ballot2(bool lo, bool hi) {
    return (u64)__ballot_sync(0xFFFFFFFFu, lo) | ((u64)__ballot_sync(0xFFFFFFFFu, hi) << 32);
}

// m[o] += the number of limbs x[i * st] and exponent e (one rounding).  A call: its operands would take the registers of
// the whole kernel, and only windows after the first come here.
template <int LO>
__device__ __noinline__ void flush_add(int32_t* m, i64* e, i64 plane, i64 o, const u32* x, int st, i64 ex) {
    u32 a[LO], b[LO], r[LO];
    const bool na = load_mag<LO>(m, plane, o, a), nb = load_mag<LO>(reinterpret_cast<const int32_t*>(x), st, 0, b);
    bool nr;
    i64 er;
    add_norm<LO>(a, na, e[o], b, nb, ex, r, &nr, &er);
    store_signed<LO>(m, plane, o, r, nr);
    e[o] = er;
}

template <int L, int LO>
__global__ void __launch_bounds__(kFlushMmaThreads, 2) k_moments_flush_mma(FlushMmaArgs a, FlushGeom g, int accumulate) {
    constexpr int NB = nb_bits(L), NBO = nb_bits(LO);               // NBO = 32 (LO - 1) + 30
    extern __shared__ __align__(128) uint8_t smem[];
    __shared__ __align__(8) uint64_t bar;
    __shared__ uint32_t tmem_sh;
    __shared__ int fail_sh;
    __shared__ long long E0[4];                                      // per column: exponent above the largest term
    __shared__ int ro[kFlushMmaMaxR1 + 1];                          // first row of each order
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    constexpr int F = kFlushF;
    const int CB = g.CB, Kp = g.Kp, RS = g.RS, W = a.W, R1 = a.R1;
    uint8_t* sA = smem;
    uint8_t* sB = smem + g.a_bytes;
    const int vcol = (g.P + g.TW + 3) * RS;                          // limbs of a column's rows
    u32* V = reinterpret_cast<u32*>(sB + (((size_t)CB * g.b_stride + 15) & ~(size_t)15));   // [column][P zeros, limb][row]
    int* CV = reinterpret_cast<int*>(V + (size_t)CB * vcol);         // [column][part][row]: carries out
    u32* OUT = reinterpret_cast<u32*>(CV + CB * kFlushParts * RS);                 // [limb][order, column]: rounded sums
    i64* EX = reinterpret_cast<i64*>((reinterpret_cast<uintptr_t>(OUT + (size_t)LO * R1 * CB) + 7) & ~(uintptr_t)7);   // exponents
    if (tid == 0) {
        fail_sh = 0;
        mbar_init(&bar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        int r = 0;
        for (int k = 0; k < R1; k++) {
            ro[k] = r;
            r += (flush_digits(a.nkb[k * a.NN + a.NN - 1]) + F - 1) / F;
        }
        ro[R1] = r;
        if (r > g.Mrows) fail_sh = 8;                               // the table does not hold n^k: nothing is written
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(smem_u32(&tmem_sh)), "r"(256) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    for (size_t q = tid; q < (g.a_bytes + (size_t)CB * g.b_stride) / 16; q += blockDim.x)
        reinterpret_cast<uint4*>(smem)[q] = make_uint4(0, 0, 0, 0);
    for (int q = tid; q < CB * vcol; q += blockDim.x) V[q] = 0;
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_sh;
    const int cs = CB == 4 ? 2 : CB - 1;                             // log2 CB
    const int KC = R1 << cs, kc = tid % KC, i_first = tid / KC, i_step = kFlushMmaThreads / KC;
    const uint32_t idesc = (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(g.NCOL >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
    const int lbo = g.PR * 16;
    const uint64_t da0 = umma_desc(smem_u32(sA), 2048, 128), db0 = umma_desc(smem_u32(sB), lbo, 128);
    // limbs [x h, (x + 1) h) of a row by warp x of those that reach its lanes, each from a zero carry
    constexpr int NX = kFlushParts;
    const int h = (g.VW / NX + 3) / 4 * 4;
    uint32_t phase = 0;
    bool pending = false, run = fail_sh == 0;                        // thread 0: a commit not yet waited for
    i64 shift_in_A = -1;
    const i64 groups = (a.N + CB - 1) / CB, items = a.rows * groups;
    // contiguous work: a CTA's items share the coefficients of a row
    const i64 per = (items + gridDim.x - 1) / gridDim.x, it0 = per * blockIdx.x, it1 = it0 + per < items ? it0 + per : items;
    for (i64 it = it0; it < it1 && run; it++) {
        const i64 row = it / groups, c0 = (it % groups) * CB;
        const int nc = (int)(a.N - c0 < CB ? a.N - c0 : CB);
        const i64 n0 = a.m0 + a.row_shift[row];                     // n of level w: n0 + w
        if (n0 <= 0) continue;                                       // k_moments_flush's rows
        if (n0 != shift_in_A) {                                      // digits of n^k (zero where n is beyond the table)
            shift_in_A = n0;
            for (int q = tid; q < R1 * W; q += blockDim.x) {
                const int k = q / W, w = q - k * W, nr = (ro[k + 1] - ro[k]) * F;
                const i64 n = n0 + w;
                const u32* src = a.nk + ((i64)k * a.NN + n) * a.KW;
                uint8_t* dst = sA + (w >> 4) * 2048 + (w & 15);
                u32 c = 0;
                for (int j = 0; 4 * j < nr; j++) {
                    const u64 s = (u64)(n < a.NN && j < a.KW ? src[j] : 0u) + 0x80808080u + c;
                    c = (u32)(s >> 32);
                    const u32 d = (u32)s ^ 0x80808080u;
                    for (int b = 4 * j; b < 4 * j + 4 && b < nr; b++) {
                        const int r = ro[k] + b / F;
                        dst[(size_t)(b % F) * 128 * Kp + (r >> 3) * 128 + (r & 7) * 16] = (uint8_t)(d >> (8 * (b & 3)));
                    }
                }
            }
        }
        if (tid < CB) E0[tid] = EZ;
        __syncthreads();
        for (int q = tid; q < W << cs; q += blockDim.x) {
            const int w = q >> cs, c = q & (CB - 1);
            if (c >= nc) continue;
            const i64 e = a.ye[(w * a.rows + row) * a.N + c0 + c];
            if (e != EZ && n0 + w < a.NN) atomicMax(&E0[c], (long long)(e + NB));
        }
        __syncthreads();
        bool any = false;
        for (int c = 0; c < nc; c++) any |= E0[c] != EZ;
        if (!any) {                                                  // rows of no pole, structures that do not occur
            for (int q = tid; q < R1 * nc && !accumulate; q += blockDim.x) {
                const i64 o = (row * R1 + q / nc) * a.N + c0 + q % nc;
#pragma unroll 1
                for (int i = 0; i < LO; i++) a.mm[i * a.mplane + o] = 0;
                a.me[o] = EZ;
            }
            __syncthreads();                                         // E0 is rewritten
            continue;
        }
        // digits of the terms: word i of floor(|y| 2^sh), complemented with a carry in for negative ones, plus 0x80...80
        for (int q = tid; q < W << cs; q += blockDim.x) {
            const int w = q >> cs, c = q & (CB - 1);
            if (c >= nc) continue;
            const i64 ix = (w * a.rows + row) * a.N + c0 + c, e = a.ye[ix], E = E0[c];
            const bool some = e != EZ && n0 + w < a.NN;
            const i64 sh = some ? 8 * (i64)g.PDV - (E - e) : 0;     // y's bit 0 on the grid (E - e >= NB)
            const int qq = sh < -32 * (L + 1) ? -(L + 1) : (int)(sh >= 0 ? sh >> 5 : -((-sh + 31) >> 5)), f = (int)(sh - 32 * (i64)qq) & 31;
            const u32 mask = some && a.ym[(L - 1) * a.yplane + ix] < 0 ? 0xFFFFFFFFu : 0u;
            uint8_t* dst = sB + (size_t)c * g.b_stride + (size_t)(w >> 4) * lbo + 256 + (w & 15);
            const int words = (g.PDV + 4) / 4;
            auto put = [&](int i, u32 d) {
                uint8_t* o = dst + 64 * i;                           // four rows of 16 bytes
                o[0] = (uint8_t)d;
                o[16] = (uint8_t)(d >> 8);
                o[32] = (uint8_t)(d >> 16);
                o[48] = (uint8_t)(d >> 24);
            };
            // grid word qq + k = limb k shifted by f bits; words outside [qq, qq + L + 1] are zero digits
            if (some) {
                u32 y[L];
#pragma unroll
                for (int k = 0; k < L; k++) y[k] = (u32)a.ym[k * a.yplane + ix] ^ mask;
                u32 prev = 0, cm = mask & 1u, ct = mask & 1u;        // carries: |y| from y, digits from the signed grid value
#pragma unroll
                for (int k = 0; k < L + 2; k++) {
                    u32 cur = 0;
                    if (k < L) {
                        const u64 s = (u64)y[k] + cm;
                        cm = (u32)(s >> 32);
                        cur = (u32)s;
                    }
                    const u32 word = fsl(prev, cur, f);
                    prev = cur;
                    if ((unsigned)(qq + k) < (unsigned)words) {
                        const u64 s = (u64)(word ^ mask) + 0x80808080u + ct;
                        ct = (u32)(s >> 32);
                        put(qq + k, (u32)s ^ 0x80808080u);
                    }
                }
            }
            const int lo = some ? qq : words, hi = some ? qq + L + 2 : words;
            for (int i = 0; i < lo; i++) put(i, 0);
            for (int i = hi > 0 ? hi : 0; i < words; i++) put(i, 0);
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // generic writes -> tensor-core reads
        for (int c = 0; c < nc; c++) {
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncthreads();                                         // operands written; the accumulators are read out
            if (tid == 0) {
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint64_t db = db0 + (uint64_t)(((size_t)c * g.b_stride) >> 4);
                for (int beta = 0; beta < F; beta++)
                    for (int ks = 0; ks < Kp / 32; ks++) {
                        const uint32_t acc = (beta > 0 || ks > 0) ? 1u : 0u;
                        asm volatile(
                            "{\n\t.reg .pred p;\n\t"
                            "setp.ne.b32 p, %4, 0;\n\t"
                            "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}"
                            ::"r"(tmem), "l"(da0 + (uint64_t)((beta * 128 * Kp + ks * 4096) >> 4)),
                              "l"(db + (uint64_t)(16 - beta + ((ks * 2 * lbo) >> 4))), "r"(idesc), "r"(acc) : "memory");
                    }
                asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
                             ::"r"(smem_u32(&bar)) : "memory");
                pending = true;
            }
            if (!mbar_wait(&bar, phase, kWaitLimit)) atomicExch(&fail_sh, 1);
            else pending = false;
            phase ^= 1;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const int r = (warp & 3) * 32 + lane, qt = warp >> 2;
            if ((warp & 3) * 32 < g.Mrows) {
                u32* v = V + c * vcol + g.P * RS + r;
                i64 cy = 0;
                const uint32_t ta = tmem + ((uint32_t)((warp & 3) * 32) << 16);
                const int i1 = qt == NX - 1 || (qt + 1) * h > g.VW ? g.VW : (qt + 1) * h;
                for (int i = qt * h; i < i1; i += 4) {
                    uint32_t d[16];
                    tmem_ld16(d, ta + (uint32_t)(4 * i));
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                    for (int u = 0; u < 4; u++) {
                        const i64 x = (i64)(int)d[4 * u] + (i64)(int)d[4 * u + 1] * 256 +
                                      ((i64)(int)d[4 * u + 2] + (i64)(int)d[4 * u + 3] * 256) * 65536;
                        const i64 s = x + cy;
                        if (r < g.Mrows) v[(i + u) * RS] = (u32)s;
                        cy = s >> 32;
                    }
                }
                if (r < g.Mrows) {
                    CV[(c * NX + qt) * RS + r] = (int)cy;             // |carries| < 2^18
                    if (qt == NX - 1)
                        for (int i = g.VW; i < g.TW; i++) v[i * RS] = 0;
                }
            }
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncthreads();
        run = fail_sh == 0;
        // each part's carry into the limbs above it (the last one is the sign of the limbs above VW)
        for (int q = tid; q < g.Mrows * nc && run; q += blockDim.x) {
            const int c = q / g.Mrows, r = q - c * g.Mrows;
            u32* v = V + c * vcol + g.P * RS + r;
#pragma unroll 1
            for (int x = 0; x < NX; x++) {
                i64 cy = CV[(c * NX + x) * RS + r];
                const int i0 = x == NX - 1 || (x + 1) * h > g.VW ? g.VW : (x + 1) * h;
                for (int i = i0; cy != 0 && i < g.TW; i++) {
                    const i64 s = (i64)v[i * RS] + cy;
                    v[i * RS] = (u32)s;
                    cy = s >> 32;
                }
            }
        }
        __syncthreads();
        // a warp per (order, column), two limbs per lane: the rows cc of the order (two's complement, sign extended) added
        // at their limb offsets modulo 2^(32 TW), carries, magnitude, one rounding
        for (int q = warp; q < KC && run; q += kFlushMmaThreads / 32) {
            const int k = q >> cs, c = q & (CB - 1);
            if (c >= nc) continue;
            const int r0 = ro[k], nr = ro[k + 1] - r0, i0 = lane, i1 = lane + 32;
            const bool in0 = i0 < g.TW, in1 = i1 < g.TW;
            u32* v = V + c * vcol + g.P * RS + r0;
            u64 s0 = in0 ? v[i0 * RS] : 0u, s1 = in1 ? v[i1 * RS] : 0u;
            for (int cc = 1; cc < nr; cc++) {
                const u32* x = v + (i0 - cc) * RS + cc;
                if (in0) s0 += x[0];
                if (in1) s1 += x[32 * RS];
            }
            u32 h0 = __shfl_up_sync(0xFFFFFFFFu, (u32)(s0 >> 32), 1), h1 = __shfl_up_sync(0xFFFFFFFFu, (u32)(s1 >> 32), 1);
            const u32 h31 = __shfl_sync(0xFFFFFFFFu, (u32)(s0 >> 32), 31);
            if (lane == 0) { h0 = 0; h1 = h31; }
            u32 x0 = (u32)s0 + h0, x1 = (u32)s1 + h1;
            // a limb that overflowed carries one into the next, and on through limbs of all ones
            const u64 seed = ballot2(x0 < h0, x1 < h1) << 1, ones = ballot2(x0 == ~0u, x1 == ~0u);
            const u64 carry = ((ones + (seed & ones)) ^ ones) | seed;
            x0 = in0 ? x0 + (u32)((carry >> i0) & 1) : 0u;
            x1 = in1 ? x1 + (u32)((carry >> i1) & 1) : 0u;
            const bool neg = (ballot2(x0 >> 31, x1 >> 31) >> (g.TW - 1)) & 1;
            const u64 nz = ballot2(x0 != 0, x1 != 0);
            const i64 E = E0[c];
            u32 res0 = 0, res1 = 0;
            i64 er = EZ;
            if (nz && E != EZ) {
                const int z = __ffsll((long long)nz) - 1;
                if (neg) {                                           // -x = ~x + 1: the 1 reaches the lowest nonzero limb
                    x0 = in0 ? (i0 > z ? ~x0 : (i0 == z ? 0u - x0 : 0u)) : 0u;
                    x1 = in1 ? (i1 > z ? ~x1 : (i1 == z ? 0u - x1 : 0u)) : 0u;
                }
                if (in0) v[i0 * RS] = x0;
                if (in1) v[i1 * RS] = x1;
                __syncwarp();
                const int top = 63 - __clzll((long long)ballot2(x0 != 0, x1 != 0));
                const int s = 32 * top + 32 - __clz(v[top * RS]) - NBO, w0 = s >> 5, f = s & 31;
                auto limb = [&](int i) { return (unsigned)i < (unsigned)g.TW ? v[i * RS] : 0u; };
                const bool half = s > 0 && ((limb((s - 1) >> 5) >> ((s - 1) & 31)) & 1u);
                res0 = i0 < LO ? fsr(limb(w0 + i0), limb(w0 + i0 + 1), f) : 0u;
                res1 = i1 < LO ? fsr(limb(w0 + i1), limb(w0 + i1 + 1), f) : 0u;
                er = E - 8 * (i64)g.PDV + s;
                if (half) {                                          // the top limb holds 30 bits: never all ones
                    const int kc1 = __ffsll((long long)~ballot2(res0 == ~0u, res1 == ~0u)) - 1;
                    res0 = i0 < kc1 ? 0u : res0 + (i0 == kc1);
                    res1 = i1 < kc1 ? 0u : res1 + (i1 == kc1);
                    const bool over = LO - 1 < 32 ? (lane == LO - 1 && (res0 >> 30)) : (lane == LO - 33 && (res1 >> 30));
                    if (__any_sync(0xFFFFFFFFu, over)) {             // rounded up to 2^NB
                        if (LO - 1 < 32) { if (lane == LO - 1) res0 >>= 1; }
                        else if (lane == LO - 33) res1 >>= 1;
                        er += 1;
                    }
                }
                if (neg) {
                    const int z2 = __ffsll((long long)ballot2(res0 != 0, res1 != 0)) - 1;
                    res0 = i0 > z2 ? ~res0 : (i0 == z2 ? 0u - res0 : 0u);
                    res1 = i1 > z2 ? ~res1 : (i1 == z2 ? 0u - res1 : 0u);
                }
            }
            if (i0 < LO) OUT[i0 * KC + q] = res0;
            if (i1 < LO) OUT[i1 * KC + q] = res1;
            if (lane == 0) EX[q] = er;
        }
        __syncthreads();
        if (run && !accumulate) {
            if (i_first < i_step && (kc & (CB - 1)) < nc) {          // columns innermost: runs of CB numbers per limb plane
                const i64 o = (row * R1 + (kc >> cs)) * a.N + c0 + (kc & (CB - 1));
                for (int i = i_first; i < LO; i += i_step) a.mm[i * a.mplane + o] = (int32_t)OUT[i * KC + kc];
                if (i_first == 0) a.me[o] = EX[kc];
            }
        } else if (run && tid < KC && (tid & (CB - 1)) < nc && EX[tid] != EZ) {
            const i64 o = (row * R1 + (tid >> cs)) * a.N + c0 + (tid & (CB - 1));
            flush_add<LO>(a.mm, a.me, a.mplane, o, OUT + tid, KC, EX[tid]);
        }
        __syncthreads();                                             // operands, limbs and E0 are rewritten
    }
    if (tid == 0 && pending) {                                       // bounded drain of our own MMAs
        if (!mbar_wait(&bar, phase ^ 1, kWaitLimit)) fail_sh = 2;
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(256) : "memory");
    }
    if (tid == 0 && fail_sh) atomicExch(a.err, fail_sh);
}

#endif

// CTAs resident at a time: two per SM where their shared memory allows (TMEM: 256 of 512 columns each)
inline i64 flush_mma_slots(const FlushGeom& g, int sms) { return (i64)sms * (g.smem <= 110 * 1024 ? 2 : 1); }

// Which form, by times of both on a B200 (1,344 windows: 6 to 42 limbs, 10 to 100 levels, 2 to 28 orders, 80 to 200,000
// columns).  The tensor cores need enough levels and terms, and either many terms (a column costs the CUDA cores W R1, the
// tensor cores R1) or so few columns that the CUDA-core form's thread per column leaves the SMs short of threads.  In
// microseconds, to 6 and 9 % in the median:
//     tensor cores  16 + columns per CTA (0.9 + 0.13 R1 + 0.045 LO + 0.00095 W LO)
//     CUDA cores    20 + W R1 ((0.09 + 0.014 NA) waves + 0.00036 cols NA / 1000)    NA = flush_words, waves >= 1 of the blocks an
//                                                                                SM's shared memory holds
// and where the first is well above the second the CUDA cores take the window (milliseconds, tensor / CUDA cores, every term
// present): 256 bits, W = 20, R1 = 7: 12,500 columns 0.15 / 0.08, 500 0.04 / 0.08; 1280 bits, W = 40, R1 = 4, 16,000 columns
// 0.36 / 0.19; 1280 bits, R1 = 28: 170,000 columns, W = 72 11.8 / 18.0, 200,000 columns, W = 32 9.0 / 10.2; 1024 bits, 200,000
// columns, R1 = 16, W = 48: 7.0 / 6.4, R1 = 12, W = 40: 4.1 / 3.1.
// The margin of 1.25 keeps every window measured on the tensor cores there whose time the estimates do not settle.
inline bool flush_mma_pays(const FlushGeom& g, int LO, int W, int R1, int KW, i64 cols, int sms) {
    const i64 terms = (i64)W * R1;
    if (terms < 900 && !(W >= 10 && terms >= 128 && cols < (i64)sms * 112)) return false;
    const int NA = flush_words(LO, KW);
    const i64 items = (cols + g.CB - 1) / g.CB, slots = flush_mma_slots(g, sms);
    const double columns = (double)g.CB * ((items + slots - 1) / slots);
    const double waves = std::fmax(1.0, (double)cols / (kFlushThreads * (double)sms * (227 / (NA + 1))));
    const double mma = 16.0 + columns * (0.9 + 0.13 * R1 + 0.045 * LO + 0.00095 * W * LO);
    const double cuda = 20.0 + (double)terms * ((0.09 + 0.014 * NA) * waves + 0.36e-6 * (double)cols * NA);
    return mma < 1.25 * cuda;
}

template <int L>
struct FlushMmaLaunch {
    static int flush(const FlushMmaArgs& a, int accumulate, int LO, cudaStream_t st);
};

#ifdef B3D_DEFINE_LAUNCH
template <int L, int LO>
static int flush_mma_launch(const FlushMmaArgs& a, const FlushGeom& g, int sms, int accumulate, cudaStream_t st) {
    static std::atomic<unsigned long long> opted{0};                // devices whose limit is raised
    const unsigned long long dbit = device_bit();
    if (!(opted.load(std::memory_order_relaxed) & dbit) || !dbit) {
        const int rc = (int)cudaFuncSetAttribute(k_moments_flush_mma<L, LO>, cudaFuncAttributeMaxDynamicSharedMemorySize, 220 * 1024);
        if (rc) return rc;
        opted.fetch_or(dbit, std::memory_order_relaxed);
    }
    const i64 items = a.rows * ((a.N + g.CB - 1) / g.CB), slots = flush_mma_slots(g, sms);
    k_moments_flush_mma<L, LO><<<(unsigned)(items < slots ? items : slots), kFlushMmaThreads, g.smem, st>>>(a, g, accumulate);
    return (int)cudaGetLastError();
}

template <int L>
int FlushMmaLaunch<L>::flush(const FlushMmaArgs& a, int accumulate, int LO, cudaStream_t st) {
    if (a.rows == 0 || a.N == 0 || a.W == 0) return 0;
    FlushGeom g;
    int dev = 0, sms = 0;
    int rc = (int)cudaGetDevice(&dev);
    if (!rc) rc = (int)cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (rc) return rc;
    const bool mma = flush_mma_geom(LO, a.W, a.R1, a.NN, a.KW, &g) && flush_mma_pays(g, LO, a.W, a.R1, a.KW, a.rows * a.N, sms);
    if (mma) rc = LO == L ? flush_mma_launch<L, L>(a, g, sms, accumulate, st) : flush_mma_launch<L, L + 4>(a, g, sms, accumulate, st);
    // all rows, or those with n = 0 in the window (n = m0 + shift there: none once m0 > 0)
    if (!rc && (!mma || a.m0 == 0))
        rc = Launch<L>::moments_flush(a.ym, a.ye, a.yplane, a.row_shift, a.m0, a.W, a.rows, a.N, a.R1, a.nk, a.nkb, a.NN, a.KW,
                                      accumulate, LO, a.mm, a.me, a.mplane, mma, st);
    return rc;
}
#endif

}  // namespace b3d

// Pole step on the sm_100a INT8 tensor cores (tcgen05.mma.kind::i8, s8 x s8 -> s32 accumulators in TMEM).
//
// One stage of the pole step is, per task t, Out[i, n] = sum_j C[i, j] X[j, n] over S x S multiprecision
// constants C (rows aligned, one exponent per row) and S x N numbers X (aligned per column n over j here),
// each output an exact sum rounded once: the same results as k_pole1 / k_pole2 bit for bit.
//
// The exact products are byte convolutions.  Both operands are written in balanced base-256 digits
// (d in [-128, 127]: the bytes of v + 0x8080...80, each minus 128), so that
//     sum_j C[i, j] X[j, n] = sum_p D[p, n] 256^p,   D[p, n] = sum_j sum_u c_ij[p - u] x_jn[u],
// and D is one int8 GEMM per row i: A[p, (j, u')] = c_ij[p - U + 1 + u'] (positions p on the 128 TMEM
// lanes, a Hankel matrix in (p, u')), B[n, (j, u')] = x_jn[U - 1 - u'] (the digits of each X entry reversed
// along K).  The Hankel operand is never materialised: its 16 x 16 blocks depend only on the sum of the
// block coordinates, so one 16-byte window of c_ij per byte offset o, stored at 16 o, is addressed by the
// canonical no-swizzle K-major descriptor with LBO = 256 (next K chunk = 16 offsets on) and SBO = 128
// (next 8 rows = 8 offsets on).  |D| <= S 4 L 2^14 < 2^31: no wrap.
//
// Positions below P0 (a multiple of 16) are not computed: their sum is below 2^(8 P0 + 17) in magnitude, at least 96
// bits under the rounding point of a sum as long as the operands allow.  The rounding is kept where no value that close
// rounds differently, and where it is not (deep cancellation, a sum at a rounding midpoint) the thread forms the exact sum
// from the operands in memory.
//
// One CTA (160 threads, three per SM) works through (task, column chunk of NC <= 32 columns) items.  Four front warps, per
// item: column exponents, the aligned X digits into the K-major B operand (16-byte stores); per row i: the padded digit
// strings of c_ij (the next row's constants load meanwhile), the Hankel windows (four per thread step, byte permutations
// of five words, stored in a rotated order that keeps the stores free of bank conflicts), one thread issues the MMAs (M =
// 128, N = NC, K = 32: two 16-digit chunks, the second of which may start the next entry, so that entries are not padded to
// 32 digits); then the accumulators go transposed (D[n][p]) into a shared-memory slot.  A back warp, a lane per column, takes
// the slot: the limbs of the sum by one carry chain in registers (the slot is free again), sign, one rounding, coalesced
// stores, while the front warps multiply the next row.  Slot and rows pass by mbarriers.
//
// What bounds it: latency, one row's windows, MMAs and transposition one after the other; at S = 5, L = 34 the MMAs (38
// clocks each, their 128-row A operand through shared memory) take 43 % of the time, the tensor pipe counts 20 % of the
// cycles, issue 30 %.  Per 1024-bit task (134,316 tasks of 30 columns, both stages): 18.4 ms, when first built 18.8;
// two CTAs of four front and four back warps 22.7 (26.9 and 24.8 with the next item's operands prefetched or preloaded:
// registers spill), TMEM read 32 columns at a time 26.5 (through local memory).  The form before handled a row in four warps
// by turns (windows, MMAs, carry segments, one header thread per column, limbs by run-time offsets) with all 256 positions:
// some 8,000 warp instructions and 10,000 clocks of a CTA per row, 27.8 ms.
// Every mbarrier wait is bounded; on expiry the CTA records an error code, waits (bounded) for its own MMAs,
// frees its TMEM and returns.
#pragma once
#include <cuda_runtime.h>

#include "kernels.cuh"
#include "rns.cuh"

namespace b3d {

template <int L>
struct PoleMmaGeom {
    static constexpr int NB = nb_bits(L);
    static constexpr int D = 4 * L;                                 // digits of a number
    static constexpr int U = 16 * ((D + 15) / 16);                  // digits per entry along K (chunks of 16)
    static constexpr int NCH = U / 16;
    static constexpr int p0_for(int mt) {
        return 8 * L - 1 - 128 * mt <= 0 ? 0 : 16 * ((8 * L - 1 - 128 * mt + 15) / 16);
    }
    // one tile of 128 positions where the dropped part stays 160 bits below the result's rounding point
    static constexpr int MT = (8 * p0_for(1) + 17 <= NB - 160) ? 1 : 2;
    // first position computed: as high as leaves 96 bits below the rounding point
    static constexpr int p0_high() { return NB - 96 - 17 < 128 ? 0 : 16 * ((NB - 96 - 17) / 128); }
    static constexpr int P0 = p0_high() > p0_for(MT) ? p0_high() : p0_for(MT);
    static constexpr int NP = 8 * L - P0;                           // positions computed (a multiple of 16)
    static constexpr int NWIN = NP + U - 16;                        // Hankel windows per entry (a multiple of 16)
    static constexpr int FAM = 16 * NWIN;                           // bytes of one entry's windows
    static constexpr int SPAN = 16 * (128 * MT + U + 16);            // bytes the MMAs may touch from an entry's windows on
    static constexpr int PADB = U - P0;                             // zero bytes before a digit string (negative: it starts P0 - U in)
    static constexpr int CW = (NP + U) / 4 + 2;                     // words of a padded digit string from byte P0 on
    static constexpr int NPW = NP / 4;                              // limbs of a sum from position P0 up
    static constexpr int DS = NP + 4;                               // words per transposed column (16-byte rows)
    static_assert(8 * P0 + 17 <= NB - 64 && NP > 0 && NP <= 128 * MT && NP % 16 == 0, "tiles must reach the rounding point");
    static_assert(PADB >= 0 && PADB % 4 == 0 && PADB / 4 + L <= CW, "digit string inside its padded buffer");
    static_assert(NWIN % 4 == 0, "window groups start one byte after a word");
};

struct PoleMmaArgs {
    const int32_t* xm; const i64* xe; i64 xplane;   // X: (rows, S, S, B) limb planes
    const int32_t* cm; const i64* ce; i64 cplane;   // constant tables (n, S, S), row exponents (n, S)
    const i64* t_x;                                 // (T) X row per task, or null (row t)
    const i64* t_c;                                 // (T) constant table per task
    const i64* t_o;                                 // (T) output row per task, or null (row t)
    int32_t* om; i64* oe; i64 oplane;               // output (rows, S, S, B)
    i64 T, B;
    int S;
    int stage;                                      // 1: X[a, j, k] summed over j; 2: X[j, b0, k] summed over j
    int NC, nchunks;                                // columns per CTA work item (multiple of 16), chunks per task
    int* err;                                       // device error flag (0 = ok)
};

constexpr int kPoleMmaThreads = 160;                            // four front warps, one back warp
constexpr int kPoleMmaMaxS = 8;
constexpr int kPoleMmaMaxNC = 32;

__host__ __device__ constexpr size_t pm_align(size_t x) { return (x + 127) & ~size_t(127); }

// dynamic shared memory: B operand (a zero chunk after an odd number of them) | Hankel windows | padded digit strings of two
// rows (this one and the next) | a slot of transposed accumulators | column exponents of the item and of the slot (and the
// slot's row exponent) | A descriptors of the K steps
template <int L>
struct PoleMmaSmem {
    using G = PoleMmaGeom<L>;
    static __host__ __device__ int steps(int S) { return (S * G::NCH + 1) / 2; }
    static __host__ __device__ size_t bop(int S, int NC) { return pm_align((size_t)steps(S) * 32 * NC); }
    static __host__ __device__ size_t hank(int S) { return pm_align((size_t)S * G::FAM); }
    static __host__ __device__ size_t cdig(int S) { return pm_align((size_t)2 * S * G::CW * 4); }   // two rows
    static __host__ __device__ size_t slot(int NC) { return pm_align((size_t)NC * G::DS * 4); }
    static __host__ __device__ size_t total(int S, int NC) {
        const size_t t = bop(S, NC) + hank(S) + cdig(S) + slot(NC) + 2 * (kPoleMmaMaxNC + 1) * 8 + (size_t)steps(S) * 8;
        const size_t read = bop(S, NC) + (size_t)(S - 1) * G::FAM + G::SPAN;
        return pm_align(t > read ? t : read);
    }
};

template <int L> B3D_CX bool P0_exact() { return PoleMmaGeom<L>::P0 == 0; }      // nothing is dropped

// v (two's complement, L words) -> balanced base-256 digits, four per word (little-endian bytes, as s8)
template <int L> __device__ __forceinline__ void to_balanced(u32 (&v)[L]) {
    u32 c = 0;
#pragma unroll
    for (int k = 0; k < L; k++) {
        const u64 s = (u64)v[k] + 0x80808080u + c;
        c = (u32)(s >> 32);
        v[k] = (u32)s ^ 0x80808080u;
    }
}

// Offsets inside a task's (S, S, B) block: X entry (j, column n) at coff(n) + j * jst, output (i, column n) at
// coff(n) + i * jst, with n = a B + k in stage 1 (X[a, j, k], Y[a, i, k]) and n = b0 B + k in stage 2
// (Y[j, b0, k], res[i, b0, k]).  32-bit arithmetic: a block holds S^2 B < 2^31 numbers.
__device__ __forceinline__ int pm_coff(const PoleMmaArgs& a, int n) {
    const int B = (int)a.B;
    return a.stage == 1 ? (n / B) * a.S * B + n % B : n;
}

__device__ __forceinline__ int pm_jst(const PoleMmaArgs& a) { return a.stage == 1 ? (int)a.B : a.S * (int)a.B; }

// one column of a row: its positions d4 from P0 -> limbs (two's complement, one more for the sign)
template <int L>
B3D_HD i64 pm_limbs(const int4* d4, u32 (&w)[PoleMmaGeom<L>::NPW + 1]) {
    constexpr int NPW = PoleMmaGeom<L>::NPW;
    i64 cy = 0;
#pragma unroll
    for (int q = 0; q < NPW; q++) {
        const int4 d = d4[q];
        const i64 x = (i64)d.x + (i64)d.y * 256 + ((i64)d.z + (i64)d.w * 256) * 65536;
        const i64 s = x + cy;
        w[q] = (u32)s;
        cy = s >> 32;
    }
    w[NPW] = (u32)cy;
    return cy;
}

// sign and one rounding of a column's limbs (value w 2^ein, left as its magnitude): magnitude r, exponent er (EZ: zero).
// false where a value within the dropped part (2^17 units of w either way) could round differently
template <int L>
B3D_HD bool pm_round(u32 (&w)[PoleMmaGeom<L>::NPW + 1], i64 ein, u32 (&r)[L], bool* negative, i64* er) {
    constexpr int NB = nb_bits(L), NPW = PoleMmaGeom<L>::NPW, NW = NPW + 1;
    const bool neg = (w[NPW] >> 31) != 0;
    if (neg) negate(w);
    *negative = neg;
    // bit length from the top limbs; the half bit of the rounding
    int bl = 0;
#pragma unroll
    for (int k = NW - 4; k < NW; k++)
        if (w[k]) bl = 32 * k + 32 - clz32(w[k]);
    const int hb = bl - NB - 1, q = hb >> 5, f = hb & 31;
    constexpr int Q0 = (32 * NPW - NB - 1) >> 5;                     // of a sum that fills its limbs; most lie in Q0 - 1, Q0
    if (Q0 >= 3 && bl != 0 && (q == Q0 || q == Q0 - 1)) {
        u32 x[L + 3];                                               // limbs q - 1 .. q + L + 1
#pragma unroll
        for (int k = 0; k < L + 3; k++) {
            const int hi = Q0 - 1 + k, lo = Q0 - 2 + k;
            x[k] = q == Q0 ? (hi < NW ? w[hi < NW ? hi : 0] : 0u) : (lo >= 0 && lo < NW ? w[lo >= 0 && lo < NW ? lo : 0] : 0u);
        }
        const u32 below = fsr(x[0], x[1], f);                       // the 32 bits under the half bit (all above the error)
        u32 t[L + 1];
#pragma unroll
        for (int k = 0; k <= L; k++) t[k] = fsr(x[k + 1], x[k + 2], f);
        const u32 half = t[0] & 1u;
        if (!P0_exact<L>() && below == (half ? 0u : ~0u)) return false;      // a midpoint within the dropped part
#pragma unroll
        for (int k = 0; k < L; k++) r[k] = fsr(t[k], t[k + 1], 1);
        add_bit(r, r, half);
        int s = hb + 1;
        if ((r[L - 1] >> (NB - 32 * (L - 1))) != 0) {                // rounded up to 2^NB
#pragma unroll
            for (int k = 0; k < L; k++) r[k] = fsr(r[k], k + 1 < L ? r[k + 1] : 0u, 1);
            s++;
        }
        *er = ein + s;
        return true;
    }
    if (!P0_exact<L>() && !round_safe<L, NW, 1>(w)) return false;    // other lengths: the general rounding
    if (!round_mag<L>(w, ein, r, er)) *er = EZ;
    return true;
}

// mbarrier wait, bounded, given up early once the CTA has failed
__device__ __forceinline__ bool pm_wait(uint64_t* bar, uint32_t parity, const int* fail) {
    const uint32_t addr = smem_u32(bar);
    for (uint32_t it = 0; it < kWaitLimit; it++) {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred P;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 P, [%1], %2;\n\t"
            "selp.b32 %0, 1, 0, P;\n\t}"
            : "=r"(done) : "r"(addr), "r"(parity) : "memory");
        if (done) return true;
        if ((it & 63) == 63 && *(const volatile int*)fail) return false;
    }
    return false;
}

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// sixteen TMEM columns of a warp's lanes (not waited for)
__device__ __forceinline__ void tmem_ld16(uint32_t* d, uint32_t addr) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3]), "=r"(d[4]), "=r"(d[5]), "=r"(d[6]), "=r"(d[7]), "=r"(d[8]),
          "=r"(d[9]), "=r"(d[10]), "=r"(d[11]), "=r"(d[12]), "=r"(d[13]), "=r"(d[14]), "=r"(d[15])
        : "r"(addr));
}

__device__ __forceinline__ void front_sync() { asm volatile("bar.sync 1, 128;" ::: "memory"); }

// barrier of the front warps; whether any of their threads passed true (the same answer for all)
__device__ __forceinline__ bool front_any(bool x) {
    int r;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.s32 p, %1, 0;\n\t"
        "barrier.cta.red.or.pred q, 1, 128, p;\n\t"
        "selp.s32 %0, 1, 0, q;\n\t}"
        : "=r"(r) : "r"((int)x) : "memory");
    return r != 0;
}

// warp 1, lane j < S: the digit string of c_ij (its magnitude and sign in c, ng) into a padded buffer
template <int L>
__device__ __forceinline__ void pm_put_digits(u32 (&c)[L], bool ng, u32* dst) {
    if (ng) negate(c);
    to_balanced(c);
#pragma unroll
    for (int k = 0; k < L; k++) dst[k] = c[k];
}

template <int L>
__global__ void __launch_bounds__(kPoleMmaThreads, 3) k_pole_mma(const __grid_constant__ PoleMmaArgs a) {
    using G = PoleMmaGeom<L>;
    using SM = PoleMmaSmem<L>;
    constexpr int U = G::U, NCH = G::NCH, MT = G::MT, CW = G::CW, FAM = G::FAM, NWIN = G::NWIN, DS = G::DS, NP = G::NP;
    extern __shared__ __align__(128) uint8_t smem[];
    __shared__ __align__(8) uint64_t bar, dfull, dempty;             // MMAs of a row; slot filled, slot read out
    __shared__ uint32_t tmem_sh;
    __shared__ int fail_sh;
    __shared__ i64 er_sh[kPoleMmaMaxS];                             // row exponents of the task's constant
    __shared__ int coff_sh[kPoleMmaMaxNC];                          // column offsets inside the task's block

    const int S = a.S, NC = a.NC, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const i64 N = (i64)S * a.B;
    uint8_t* bop = smem;
    uint8_t* hank = smem + SM::bop(S, NC);
    u32* cdig = reinterpret_cast<u32*>(hank + SM::hank(S));         // row r at cdig + (r % 2) S CW
    u32* dbuf = cdig + SM::cdig(S) / 4;                             // D[n][p]
    i64* ecol = reinterpret_cast<i64*>(reinterpret_cast<uint8_t*>(dbuf) + SM::slot(NC));   // the item's column exponents
    i64* inf = ecol + kPoleMmaMaxNC + 1;                            // the slot's, and its row's
    uint64_t* adesc = reinterpret_cast<uint64_t*>(inf + kPoleMmaMaxNC + 1);   // A descriptor of each K step
    const int nsteps = SM::steps(S);
    uint32_t ncols = 32;
    while (ncols < (uint32_t)(MT * NC)) ncols <<= 1;

    for (int q = tid; q < 2 * S * CW; q += blockDim.x) cdig[q] = 0;   // padding stays zero: digits go to [PADB, PADB + D)
    // K step s multiplies chunks 2 s and 2 s + 1 of the row of entries (entry g / NCH, 16 windows on per chunk)
    for (int q = tid; q < nsteps; q += blockDim.x) {
        auto at = [&](int g) { return (g / NCH) * FAM + (g % NCH) * 256; };
        const int g = 2 * q;
        adesc[q] = umma_desc(smem_u32(hank) + at(g), g + 1 < S * NCH ? at(g + 1) - at(g) : 256, 128);
    }
    for (int q = tid; q < NC; q += blockDim.x)                       // the chunk after the last entry: zero
        if ((S * NCH) & 1) *reinterpret_cast<uint4*>(bop + (size_t)S * NCH * 16 * NC + 16 * q) = make_uint4(0, 0, 0, 0);
    if (tid == 0) {
        fail_sh = 0;
        mbar_init(&bar, 1);
        mbar_init(&dfull, 128);
        mbar_init(&dempty, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(smem_u32(&tmem_sh)), "r"(ncols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_sh;
    const i64 items = a.T * a.nchunks;
    const int jst = pm_jst(a);
    bool pending = false;                                           // thread 0: a commit not yet waited for
    uint32_t phase = 0;

    if (warp == 4) {                                                // back warp
        u32 row = 0;
        bool stop = false;
        for (i64 w = blockIdx.x; w < items && !stop; w += gridDim.x) {
            const i64 t = w / a.nchunks, n0 = (w % a.nchunks) * (i64)NC;
            const int nn = (int)(N - n0 < NC ? N - n0 : NC);
            const i64 xrow = a.t_x ? a.t_x[t] : t, crow = a.t_c[t], orow = a.t_o ? a.t_o[t] : t;
            const i64 xbase = xrow * S * S * a.B, obase = orow * S * S * a.B;
            const int co = lane < nn ? pm_coff(a, (int)n0 + lane) : 0;
            for (int i = 0; i < S; i++, row++) {
                if (!__all_sync(0xFFFFFFFFu, pm_wait(&dfull, row & 1u, &fail_sh))) {
                    if (lane == 0) atomicCAS(&fail_sh, 0, 3);
                    stop = true;
                    break;
                }
                const i64 E = inf[lane & (NC - 1)], Er = inf[kPoleMmaMaxNC], oo = obase + co + (i64)i * jst;
                u32 wd[G::NPW + 1];
                pm_limbs<L>(reinterpret_cast<const int4*>(dbuf + (lane & (NC - 1)) * DS), wd);
                __syncwarp();
                if (lane == 0) mbar_arrive(&dempty);
                // the redo waits for the warp: its call never runs beside lanes that still hold a rounding of their own
                bool redo = false;
                if (lane < nn) {
                    if (E == EZ || Er == EZ) {
#pragma unroll
                        for (int k = 0; k < L; k++) a.om[k * a.oplane + oo] = 0;
                        a.oe[oo] = EZ;
                    } else {
                        u32 r[L];
                        bool neg;
                        i64 er;
                        redo = !pm_round<L>(wd, E + Er + 8 * G::P0, r, &neg, &er);
                        if (!redo) {
                            store_signed<L>(a.om, a.oplane, oo, r, neg && er != EZ);
                            a.oe[oo] = er;
                        }
                    }
                }
                __syncwarp();
                if (redo)
                    exact_dot<L>(a.cm, a.cplane, (crow * S + i) * S, a.xm, a.xe, a.xplane, xbase + co, jst, S, E, Er, a.om, a.oe,
                                 a.oplane, oo);
            }
        }
    } else {
        const int ncs = NC == 32 ? 5 : 4;                           // NC is 16 or 32
        const bool cthread = warp == 1 && lane < S;                 // the constants' digit strings
        // instruction descriptor: s32 accumulator, s8 x s8, both K-major, M = 128, N = NC
        const uint32_t idesc = (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(NC >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
        // B descriptor of the first K step; the others differ only in the 14-bit address field
        const uint64_t db0 = umma_desc(smem_u32(bop), 16 * NC, 128);
        u32 row = 0;
        bool stop = false;
        for (i64 w = blockIdx.x; w < items && !stop; w += gridDim.x) {
            const i64 t = w / a.nchunks, n0 = (w % a.nchunks) * (i64)NC;
            const int nn = (int)(N - n0 < NC ? N - n0 : NC);
            const i64 xrow = a.t_x ? a.t_x[t] : t, crow_now = a.t_c[t];

            // the constants of row 0 (digits now) and row 1 (loaded, converted during row 0), row exponents
            u32 cn[L];
            bool cneg = false;
            if (cthread) {
                cneg = load_mag<L>(a.cm, a.cplane, crow_now * S * S + lane, cn);
                er_sh[lane] = a.ce[crow_now * S + lane];
                pm_put_digits<L>(cn, cneg, cdig + lane * CW + G::PADB / 4);
                if (S > 1) cneg = load_mag<L>(a.cm, a.cplane, (crow_now * S + 1) * S + lane, cn);
            }
            const i64 xbase = xrow * S * S * a.B;
            // column exponents: the largest over j of the nonzero entries (all loads of a column issued at once)
            i64 Ec = EZ;
            if (tid < NC) {
                const int n = tid, co = n < nn ? pm_coff(a, (int)n0 + n) : 0;
                coff_sh[n] = co;
                if (n < nn) {
                    i64 ev[kPoleMmaMaxS];
                    int32_t tv[kPoleMmaMaxS];
#pragma unroll
                    for (int j = 0; j < kPoleMmaMaxS; j++) {
                        if (j < S) {
                            const i64 ix = xbase + co + j * jst;
                            ev[j] = a.xe[ix];
                            tv[j] = a.xm[(L - 1) * a.xplane + ix];
                        }
                    }
#pragma unroll
                    for (int j = 0; j < kPoleMmaMaxS; j++)
                        if (j < S && tv[j] != 0 && ev[j] > Ec) Ec = ev[j];
                }
                ecol[n] = Ec;
            }
            front_sync();
            // the aligned X digits into the B operand
            for (int it = tid; it < S * NC; it += 128) {
                const int j = it >> ncs, n = it & (NC - 1);
                u32 dg[L];
                zero(dg);
                const i64 E = ecol[n];
                if (n < nn) {
                    const i64 ix = xbase + coff_sh[n] + j * jst;
                    u32 x[L];
                    const bool neg = load_mag<L>(a.xm, a.xplane, ix, x);
                    const i64 ex = a.xe[ix];
                    if (E != EZ && !is_zero(x) && ex != EZ && E - ex < 32 * L) {
                        shr(x, (int)(E - ex), dg);
                        if (neg) negate(dg);
                    }
                }
                to_balanced(dg);
                uint8_t* col = bop + (n >> 3) * 128 + (n & 7) * 16;
#pragma unroll
                for (int c = 0; c < U / 16; c++) {
                    u32 q[4];
#pragma unroll
                    for (int r = 0; r < 4; r++) {
                        const int wd = U / 4 - 1 - (4 * c + r);        // reversed words, bytes reversed inside
                        q[r] = wd < L ? __byte_perm(dg[wd], 0, 0x0123) : 0u;
                    }
                    *reinterpret_cast<uint4*>(col + (size_t)(j * (U / 16) + c) * 16 * NC) = make_uint4(q[0], q[1], q[2], q[3]);
                }
            }
            for (int i = 0; i < S; i++, row++) {
                const i64 Er = er_sh[i];
                const u32* cd = cdig + (i & 1) * S * CW;
                if (Er != EZ) {
                    // windows o .. o + 3 (o a multiple of 4) start at bytes 1 + o .. of the padded string: words
                    // o / 4 .. o / 4 + 4 shifted by 1 to 4 bytes.  The thread stores them in the rotated order
                    // k' = (k + t / 2) % 4 so that the eight threads of each store phase cover all 32 banks.
                    for (int it = tid; it < S * (NWIN / 4); it += 128) {
                        const int j = it / (NWIN / 4), o = 4 * (it % (NWIN / 4));
                        const u32* cw = cd + j * CW + (o >> 2);
                        const u32 w0 = cw[0], w1 = cw[1], w2 = cw[2], w3 = cw[3], w4 = cw[4];
                        uint4* dst = reinterpret_cast<uint4*>(hank + (size_t)j * FAM + 16 * o);
#pragma unroll
                        for (int k = 0; k < 4; k++) {
                            const int kp = (k + (tid >> 1)) & 3;
                            const u32 sel = 0x4321u + 0x1111u * (u32)kp;
                            dst[kp] = make_uint4(__byte_perm(w0, w1, sel), __byte_perm(w1, w2, sel), __byte_perm(w2, w3, sel),
                                                 __byte_perm(w3, w4, sel));
                        }
                    }
                }
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // generic writes -> tensor-core reads
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                front_sync();
                if (tid == 0 && Er != EZ) {
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
                    for (int mt = 0; mt < MT; mt++) {
#pragma unroll 4
                        for (int ks = 0; ks < nsteps; ks++) {
                            const uint32_t accf = ks > 0 ? 1u : 0u;
                            asm volatile(
                                "{\n\t.reg .pred p;\n\t"
                                "setp.ne.b32 p, %4, 0;\n\t"
                                "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}"
                                ::"r"(tmem + (uint32_t)(mt * NC)), "l"(adesc[ks] + (uint64_t)(128 * mt)),
                                  "l"(db0 + (uint64_t)(2 * ks * NC)), "r"(idesc), "r"(accf) : "memory");
                        }
                    }
                    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
                                 ::"r"(smem_u32(&bar)) : "memory");
                    pending = true;
                }
                if (cthread && i + 1 < S) {                          // next row's digits while the MMAs run
                    pm_put_digits<L>(cn, cneg, cdig + ((i + 1) & 1) * S * CW + lane * CW + G::PADB / 4);
                    if (i + 2 < S) cneg = load_mag<L>(a.cm, a.cplane, (crow_now * S + i + 2) * S + lane, cn);
                }
                bool bad = false;
                if (Er != EZ) {
                    bad = !pm_wait(&bar, phase, &fail_sh);
                    if (bad) atomicCAS(&fail_sh, 0, 1);
                    else pending = false;
                    phase ^= 1;
                }
                if (!bad && row > 0 && !pm_wait(&dempty, (row - 1) & 1u, &fail_sh)) {
                    bad = true;
                    atomicCAS(&fail_sh, 0, 4);
                }
                if (front_any(bad)) { stop = true; break; }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                // accumulators -> D[n][p] of the slot (this lane's position p)
                if (Er != EZ) {
#pragma unroll 1
                    for (int mt = 0; mt < MT; mt++) {
                        if (mt * 128 + warp * 32 >= NP) break;
                        const int p = mt * 128 + warp * 32 + lane;
#pragma unroll 1
                        for (int c0 = 0; c0 < NC; c0 += 16) {
                            uint32_t d[16];
                            tmem_ld16(d, tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)(mt * NC + c0));
                            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                            if (p < NP) {
#pragma unroll
                                for (int q = 0; q < 16; q++) dbuf[(c0 + q) * DS + p] = d[q];
                            }
                        }
                    }
                }
                if (tid < NC) inf[tid] = Ec;
                if (tid == 0) inf[kPoleMmaMaxNC] = Er;
                mbar_arrive(&dfull);
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncwarp();
    __syncthreads();
    if (tid == 0 && pending) {                                       // bounded drain of our own MMAs
        if (!mbar_wait(&bar, phase ^ 1, kWaitLimit)) fail_sh = 2;
    }
    __syncthreads();
    if (warp == 0) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(ncols) : "memory");
    }
    if (tid == 0 && fail_sh) atomicExch(a.err, fail_sh);
}

#ifdef B3D_DEFINE_LAUNCH
// columns per work item: all of a task's S B columns up to kPoleMmaMaxNC, in multiples of 16 (the MMA's N step).  64 columns
// (the MMAs are bound by their A operand: a second 32 cost little) measured 0.84 to 1.0 of the time at S = 3 and 1.0 to 1.6
// at S = 4, 5, where fewer CTAs fit.
inline int pole_mma_nc(i64 N) { return (int)(N >= kPoleMmaMaxNC ? kPoleMmaMaxNC : ((N + 15) / 16) * 16); }

template <int L>
static int pole_mma_stage(PoleMmaArgs a, cudaStream_t st) {
    if (a.T == 0) return 0;
    const size_t smem = PoleMmaSmem<L>::total(a.S, a.NC);
    static unsigned long long configured = 0;                       // devices whose limits are raised
    const unsigned long long dbit = device_bit();
    if (!(configured & dbit) || !dbit) {
        int rc = (int)cudaFuncSetAttribute(k_pole_mma<L>, cudaFuncAttributeMaxDynamicSharedMemorySize, 220 * 1024);
        if (!rc) rc = (int)cudaFuncSetAttribute(k_pole_mma<L>, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
        if (rc) return rc;
        configured |= dbit;
    }
    int dev = 0, sms = 0;
    int rc = (int)cudaGetDevice(&dev);
    if (!rc) rc = (int)cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (rc) return rc;
    // resident CTAs per SM: three by the launch bounds (registers), fewer when the shared memory (228 KB per SM: static +
    // dynamic + 1 KB reserved per CTA) or the 512 TMEM columns do not hold three
    static size_t static_smem = 0;
    if (!static_smem) {
        cudaFuncAttributes fa;
        const int rc2 = (int)cudaFuncGetAttributes(&fa, k_pole_mma<L>);
        if (rc2) return rc2;
        static_smem = fa.sharedSizeBytes + 1;
    }
    int ncols = 32;
    while (ncols < PoleMmaGeom<L>::MT * a.NC) ncols <<= 1;
    int occ = (int)((228 * 1024) / (smem + static_smem + 1024));
    if (occ > 3) occ = 3;
    if (occ > 512 / ncols) occ = 512 / ncols;
    if (occ < 1) return (int)cudaErrorInvalidConfiguration;
    const i64 items = a.T * a.nchunks;
    const i64 grid = items < (i64)sms * occ ? items : (i64)sms * occ;
    k_pole_mma<L><<<(unsigned)grid, kPoleMmaThreads, smem, st>>>(a);
    return (int)cudaGetLastError();
}

template <int L>
int Launch<L>::pole_mma(const int32_t* hm, const i64* he, i64 hplane, const int32_t* Rm, const i64* Re, i64 Rplane,
                        const int32_t* Qm, const i64* Qe, i64 Qplane, const i64* t_hrow, const i64* t_R, const i64* t_qL,
                        const i64* t_slot, i64 T, i64 B, int S, int32_t* ym, i64* ye, i64 yplane,
                        int32_t* rm, i64* re, i64 rplane, int* err, cudaStream_t st) {
    if (T == 0) return 0;
    if (S > kPoleMmaMaxS || !err) return (int)cudaErrorInvalidValue;
    const int NC = pole_mma_nc((i64)S * B);
    const int nchunks = (int)(((i64)S * B + NC - 1) / NC);
    PoleMmaArgs s1{hm, he, hplane, Rm, Re, Rplane, t_hrow, t_R, nullptr, ym, ye, yplane, T, B, S, 1, NC, nchunks, err};
    int rc = pole_mma_stage<L>(s1, st);
    if (rc) return rc;
    PoleMmaArgs s2{ym, ye, yplane, Qm, Qe, Qplane, nullptr, t_qL, t_slot, rm, re, rplane, T, B, S, 2, NC, nchunks, err};
    return pole_mma_stage<L>(s2, st);
}
#endif

}  // namespace b3d

// Host check of the pole step's sums and roundings as the kernels compile them (csrc/pole_mma.cuh, csrc/mp.cuh), for
// tests/test_pole_host.py; host code only, no kernel is launched:
//   limbs  pm_limbs: positions of 256^p -> limbs, against a sum position by position
//   round  where pm_round keeps its rounding, every value within the dropped part rounds to it (midpoints planted)
//   redo   the same cases: how many it left to the exact sum, and how many of those had no midpoint within reach
//   win    mac_signed_win within 2^64 units of the exact sum's limbs from C0 up
//   high   mac_signed_high equal to mac_signed_mem
// Prints one "<check> <limbs> <cases> <failures>" line per check.
#include <cstdio>
#include <random>

#include "pole_mma.cuh"

using namespace b3d;
static std::mt19937_64 rng(20261205);

template <int N> void fill(u32 (&a)[N], int kind) {
    for (int k = 0; k < N; k++) a[k] = kind == 1 ? ~0u : (kind == 2 ? ((rng() & 1) ? ~0u : 0u) : (u32)rng());
}

// wide += sign v 256^p
template <int N> void add_at(u32 (&x)[N], i64 v, int byte) {
    const int k0 = byte / 4, sh = 8 * (byte % 4);
    const __int128 t = (__int128)v << sh;
    i64 c = 0;
    for (int k = k0; k < N; k++) {
        const int j = k - k0;
        const u32 word = j < 4 ? (u32)(t >> (32 * j)) : (v < 0 ? ~0u : 0u);
        const u64 s = (u64)x[k] + word + (u64)c;
        x[k] = (u32)s;
        c = (i64)(s >> 32);
    }
}

template <int L> void check_limbs(int iters) {
    using G = PoleMmaGeom<L>;
    constexpr int N = G::NPW + 1;
    long bad = 0;
    for (int it = 0; it < iters; it++) {
        int4 d[G::NPW];
        int* p = reinterpret_cast<int*>(d);
        const int mag = it % 3 == 0 ? (1 << 23) : 5 * 4 * L * 16384;      // S = 5 products of full digits
        for (int k = 0; k < G::NP; k++) p[k] = it % 5 == 0 ? (it & 1 ? mag : -mag) : (int)(rng() % (2 * (u64)mag + 1)) - mag;
        u32 w[N], x[N];
        zero(x);
        for (int k = 0; k < G::NP; k++) add_at(x, p[k], k);
        pm_limbs<L>(d, w);
        for (int k = 0; k < N; k++)
            if (w[k] != x[k]) { bad++; break; }
    }
    printf("limbs %d %d %ld\n", L, iters, bad);
}

template <int L> void check_round(int iters) {
    using G = PoleMmaGeom<L>;
    constexpr int NW = G::NPW + 1, NB = nb_bits(L), PW = G::P0 / 4, NX = NW + PW;
    long bad = 0, redo = 0, idle = 0;
    for (int it = 0; it < iters; it++) {
        u32 m[NW];                                                       // a magnitude of bl bits, often near a midpoint
        fill(m, 0);
        const int top = 32 * G::NPW - 1 - (int)(rng() % (it % 4 == 0 ? 32 * G::NPW - 1 : 90));
        const int bl = top < 1 ? 1 : top;
        for (int k = 0; k < NW; k++) {
            if (32 * k >= bl) m[k] = 0;
            else if (32 * k + 32 > bl) m[k] &= (1u << (bl - 32 * k)) - 1;
        }
        m[(bl - 1) >> 5] |= 1u << ((bl - 1) & 31);
        const int hb = bl - NB - 1, mode = (int)(rng() % 6);
        auto set = [&](int lo, int hi, bool one) {                       // bits [lo, hi)
            for (int b = lo < 0 ? 0 : lo; b < hi; b++) {
                if (one) m[b >> 5] |= 1u << (b & 31);
                else m[b >> 5] &= ~(1u << (b & 31));
            }
        };
        if (hb > 0 && mode < 4) {
            const int run = mode & 2 ? hb : (int)(rng() % (hb + 1));
            set(hb - run, hb, mode & 1);                                 // zeros or ones below the half bit
            if (rng() & 1) set(hb, hb + 1, !(mode & 1));                 // ... next to a midpoint
            if (rng() % 4 == 0) set(hb + 1, bl, true);                   // a carry to the top
        }
        u32 w[NW], r[L];
        for (int k = 0; k < NW; k++) w[k] = m[k];
        const bool minus = rng() & 1;
        if (minus) negate(w);
        bool neg;
        i64 er;
        const bool kept = pm_round<L>(w, 8 * G::P0, r, &neg, &er);
        bool near = false;                                               // some value within reach rounds differently
        for (int j = 0; j < 10; j++) {
            u32 v[NX];
            zero(v);
            for (int k = 0; k < NW; k++) v[PW + k] = m[k];
            if (G::P0 > 0) {                                             // |dropped part| < 2^(8 P0 + 17)
                const i64 part = j == 0 ? 131071 : (j == 1 ? -131071 : (j == 2 ? 0 : (i64)(rng() % 262143) - 131071));
                add_at(v, part, G::P0);
                add_at(v, (i64)(rng() >> 8) * (part < 0 ? -1 : 1), G::P0 - 8);
                if (v[NX - 1] >> 31) continue;                           // through zero: the sum changes its sign
            }
            u32 x[L];
            i64 ex;
            const bool nz = round_mag<L>(v, 0, x, &ex);
            bool same = nz ? (er == ex && neg == minus) : er == EZ;
            for (int k = 0; k < L && nz && kept; k++) same &= r[k] == x[k];
            if (kept && !same) { bad++; break; }
            if (!kept) {
                u32 y[L];
                i64 ey;
                u32 c[NX];
                zero(c);
                for (int k = 0; k < NW; k++) c[PW + k] = m[k];
                const bool nc = round_mag<L>(c, 0, y, &ey);
                bool eq = nc == nz && ey == ex;
                for (int k = 0; k < L; k++) eq &= x[k] == y[k];
                near |= !eq;
            }
        }
        if (!kept) { redo++; idle += !near && mode >= 4 && hb > 64; }    // an ordinary sum has no reason for the redo
    }
    printf("round %d %d %ld\n", L, iters, bad);
    printf("redo %d %ld %ld\n", L, redo, idle);
}

template <int L> void check_mac(int iters) {
    constexpr int NW = 2 * L + 2, C0 = trunc_cols<L>(), NF = NW - C0, X0 = L > kShort ? L - kShort : 0;
    long far = 0, differ = 0;
    for (int it = 0; it < iters; it++) {
        u32 ex[NW], hi[NW], win[NF];
        zero(ex);
        zero(win);
        const int n = 1 + (int)(rng() % 8);
        for (int t = 0; t < n; t++) {
            u32 a[L], b[L];
            fill(a, it % 3);
            fill(b, (it / 3) % 3);
            const bool neg = rng() & 1;
            mac_signed_mem<L, NW>(ex, 1, a, b, neg);
            mac_signed_win<L, NF, C0>(win, 1, a, b, neg);
            for (int k = 0; k < X0; k++) a[k] = 0;
            u32 full[NW];
            for (int k = 0; k < NW; k++) full[k] = hi[k] = ex[k];
            mac_signed_mem<L, NW>(full, 1, a, b, neg);
            mac_signed_high<L, NW, X0>(hi, 1, a, b, neg);
            for (int k = 0; k < NW; k++)
                if (full[k] != hi[k]) { differ++; break; }
        }
        u32 d[NF], e[NF];
        for (int k = 0; k < NF; k++) e[k] = ex[C0 + k];
        sub_borrow(d, e, win, 0u);
        if (d[NF - 1] >> 31) negate(d);
        for (int k = C0 > 0 ? 2 : 0; k < NF; k++)
            if (d[k]) { far++; break; }
    }
    printf("win %d %d %ld\n", L, iters, far);
    printf("high %d %d %ld\n", L, iters, differ);
}

template <int L> void all() {
    check_limbs<L>(300);
    check_round<L>(20000);
    check_mac<L>(60);
}

int main() {
    all<6>(); all<10>(); all<14>(); all<18>(); all<22>(); all<26>(); all<30>(); all<34>(); all<38>(); all<42>(); all<46>();
    return 0;
}

// The carry chains of mp.cuh on the device, for tests/test_gpu_carry_chains.py: one thread per case, operands and results as
// N words a case.
#include "mp.cuh"

using namespace b3d;

// results per case: add, add into a, add into b, sub, sub into a, sub into b, s + u, u n, u n (mul_small), u n into u, -a,
// the loop's u, (carry of add, borrow of sub)
constexpr int kResults = 13;

template <int N>
__global__ void k_check(const u32* in, u32* out, int cases, int turns) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= cases) return;
    u32 a[N], b[N], r[N], x[N];
    for (int k = 0; k < N; k++) { a[k] = in[(t * 2) * N + k]; b[k] = in[(t * 2 + 1) * N + k]; }
    const u32 c = t & 1, n = in[t * 2 * N] | 1u;
    u32* o = out + (size_t)t * kResults * N;
    int slot = 0;
    auto put = [&](const u32 (&v)[N]) { for (int k = 0; k < N; k++) o[slot * N + k] = v[k]; slot++; };
    auto copy = [&](const u32 (&v)[N]) { for (int k = 0; k < N; k++) x[k] = v[k]; };
    const u32 carry = add_carry(r, a, b, c);
    put(r);
    copy(a); add_carry(x, x, b, c); put(x);
    copy(b); add_carry(x, a, x, c); put(x);
    const u32 borrow = sub_borrow(r, a, b, c);
    put(r);
    copy(a); sub_borrow(x, x, b, c); put(x);
    copy(b); sub_borrow(x, a, x, c); put(x);
    copy(a); add_mul_small(x, r, b, n); put(x); put(r);
    mul_small(r, b, n); put(r);
    copy(b); mul_small(x, x, n); put(x);
    copy(a); negate(x); put(x);
    // limbs of a result carried into other limbs' variables from turn to turn
    u32 u[N], v[N];
    for (int k = 0; k < N; k++) { u[k] = a[k]; v[k] = b[k]; }
#pragma unroll 1
    for (int i = 0; i < turns; i++) {
        add_carry(r, u, v, c);
        sub_borrow(x, r, u, c);
#pragma unroll
        for (int k = 0; k < N; k++) { u[k] = r[(k + 1) % N]; v[k] = x[(k + N - 1) % N]; }
    }
    put(u);
    for (int k = 0; k < N; k++) r[k] = k == 0 ? carry | borrow << 1 : 0u;
    put(r);
}

extern "C" int mp_device_check(int n, const u32* in, u32* out, int cases, int turns) {
    const int blocks = (cases + 63) / 64;
    switch (n) {
#define CASE(N) case N: k_check<N><<<blocks, 64>>>(in, out, cases, turns); break;
        CASE(1) CASE(2) CASE(3) CASE(4) CASE(5) CASE(6) CASE(7) CASE(8) CASE(9) CASE(10)
        CASE(11) CASE(12) CASE(13) CASE(14) CASE(15) CASE(16) CASE(17) CASE(18) CASE(19) CASE(20)
#undef CASE
        default: return 1;
    }
    return (int)cudaGetLastError();
}

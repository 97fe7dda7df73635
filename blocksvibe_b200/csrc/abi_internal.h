// Shared by the C ABI translation units: error reporting and the dispatch on the limb count.
#pragma once
#include <string>

#include "kernels.cuh"
#include "rns.cuh"
#include "cauchy_rns.cuh"
#include "cauchy_fp.cuh"
#include "moments_mma.cuh"

namespace b3d {
#define B3D_DECL(L) extern template struct Launch<L>; extern template struct RnsLaunch<L>; extern template struct CauchyRnsLaunch<L>; \
    extern template struct CauchyFpLaunch<L>; extern template struct FlushMmaLaunch<L>;
B3D_FOR_EACH_L(B3D_DECL)
#undef B3D_DECL

// record `what` as the calling thread's last error (b3d_last_error) and return `code`
int fail(int code, const std::string& what);
// 0 for cudaSuccess, else the error code with its message recorded
int cuda_status(int code, const char* fn);
// tensor-core residue product and the Cauchy coefficient digits (rns_mma.cu)
int rns_mma_launch(const RnsMma& a, const RnsTables& tb, cudaStream_t st);
int cauchy_digits_launch(const CauchyLevel& lv, const uint32_t* table, int64_t dmax, int np, int64_t Rp, int64_t Kp,
                         int TR, int64_t mat_bytes, uint8_t* out, cudaStream_t st);
}  // namespace b3d

// return CALL with NAME the launcher template TYPE of the run-time limb count L
#define B3D_DISPATCH_AS(TYPE, NAME, L, CALL)                                                            \
    switch (L) {                                                                                        \
        case 6: { using NAME = b3d::TYPE<6>; return CALL; }                                             \
        case 10: { using NAME = b3d::TYPE<10>; return CALL; }                                           \
        case 14: { using NAME = b3d::TYPE<14>; return CALL; }                                           \
        case 18: { using NAME = b3d::TYPE<18>; return CALL; }                                           \
        case 22: { using NAME = b3d::TYPE<22>; return CALL; }                                           \
        case 26: { using NAME = b3d::TYPE<26>; return CALL; }                                           \
        case 30: { using NAME = b3d::TYPE<30>; return CALL; }                                           \
        case 34: { using NAME = b3d::TYPE<34>; return CALL; }                                           \
        case 38: { using NAME = b3d::TYPE<38>; return CALL; }                                           \
        case 42: { using NAME = b3d::TYPE<42>; return CALL; }                                           \
        case 46: { using NAME = b3d::TYPE<46>; return CALL; }                                           \
        default: return b3d::fail(B3D_E_LIMBS, "no kernels compiled for L = " + std::to_string(L));     \
    }
#define B3D_DISPATCH_RNS(L, CALL) B3D_DISPATCH_AS(RnsLaunch, RX, L, CALL)
#define B3D_DISPATCH_CAUCHY(L, CALL) B3D_DISPATCH_AS(CauchyRnsLaunch, CX, L, CALL)
#define B3D_DISPATCH_CFP(L, CALL) B3D_DISPATCH_AS(CauchyFpLaunch, FX, L, CALL)
#define B3D_DISPATCH_FLUSH(L, CALL) B3D_DISPATCH_AS(FlushMmaLaunch, MX, L, CALL)
#define B3D_DISPATCH(L, CALL) B3D_DISPATCH_AS(Launch, LX, L, CALL)

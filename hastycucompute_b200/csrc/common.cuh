// Shared helpers of libhasty_b200: status handling, complex arithmetic, launch sizing.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <string>

#include "hasty_b200.h"

namespace hb {

// Per-thread error message behind hb_last_error().
void set_error(const std::string& msg);
const char* get_error();

// Return-early helpers for functions returning an HB_* status.
#define HB_TRY(expr)                     \
    do {                                 \
        int hb_status_ = (expr);         \
        if (hb_status_ != HB_OK) return hb_status_; \
    } while (0)

#define HB_CUDA(call)                                                                   \
    do {                                                                                \
        cudaError_t hb_e_ = (call);                                                     \
        if (hb_e_ != cudaSuccess) {                                                     \
            hb::set_error(std::string(#call) + " failed: " + cudaGetErrorString(hb_e_)); \
            return HB_ERR_CUDA;                                                         \
        }                                                                               \
    } while (0)

#define HB_REQUIRE(cond, code, msg)  \
    do {                             \
        if (!(cond)) {               \
            hb::set_error(msg);      \
            return (code);           \
        }                            \
    } while (0)

// Checks the launch just issued on the current thread.
inline int check_launch(const char* what) {
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        set_error(std::string(what) + " launch failed: " + cudaGetErrorString(e));
        return HB_ERR_CUDA;
    }
    return HB_OK;
}

// ---- complex64 as float2 ------------------------------------------------------------------
__host__ __device__ __forceinline__ float2 cadd(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__host__ __device__ __forceinline__ float2 csub(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }
__host__ __device__ __forceinline__ float2 cmul(float2 a, float2 b) {
    return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
// a * conj(b)
__host__ __device__ __forceinline__ float2 cmulc(float2 a, float2 b) {
    return make_float2(a.x * b.x + a.y * b.y, a.y * b.x - a.x * b.y);
}
__host__ __device__ __forceinline__ float2 cscale(float2 a, float s) { return make_float2(a.x * s, a.y * s); }
__host__ __device__ __forceinline__ float2 conjf2(float2 a) { return make_float2(a.x, -a.y); }

// The reference's ToeplitzMultType applied to a (fft/kernels/toeplitz_load_3D.cu:2-15):
// 1 -> a*b, 2 -> a*conj(b), anything else -> a.
__device__ __forceinline__ float2 mult_typed(float2 a, float2 b, int type) {
    if (type == HB_MULT_MULT) return cmul(a, b);
    if (type == HB_MULT_MULT_CONJ) return cmulc(a, b);
    return a;
}

inline int64_t ceil_div(int64_t a, int64_t b) { return (a + b - 1) / b; }

constexpr int kNumSMs = 148;  // B200

// Lets a kernel whose dynamic shared memory differs from launch to launch have `smem` bytes. The limit belongs to
// the kernel, not to the launch, and is shared by all host threads: it is always set to the most a CTA can have, so no
// thread lowers it between another one's call and its launch. static_bytes: bound on the kernel's own __shared__ arrays.
constexpr size_t kMaxSmem = 227 * 1024;
template <class K>
int allow_smem(K* kern, size_t smem, const char* what, size_t static_bytes = 0) {
    const size_t most = kMaxSmem - static_bytes;
    if (smem > most) {
        set_error(std::string(what) + ": needs " + std::to_string(smem) + " bytes of shared memory, a CTA has " + std::to_string(most));
        return HB_ERR_CUDA;
    }
    HB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most));
    return HB_OK;
}

}  // namespace hb

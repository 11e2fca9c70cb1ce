// Pass operators between the caller's modes and the interleaved grids of a NUFFT plan.
#pragma once

#include "ops.cuh"

namespace hb {

#ifdef __CUDACC__

// ---- x-axis passes between the caller's [C][N..] modes and the interleaved buffers ----------
// Load modes f[e][a][l] (a = row over axes 0,1; l = axis 2) pre-scaled by 1/phihat.
struct OpModesIn {
    static constexpr bool kLoadLFast = true;
    static constexpr bool kStoreLFast = false;
    static constexpr bool kFusedK = false;
    static constexpr bool kChunkLoop = false;
    static constexpr bool kSenseReduce = false;
    const float2* f;
    float2* dst;  // [rows][nf2][C]
    const float* d0;
    const float* d1;
    const float* d2;
    int64_t N1, N2, nm;  // modes of axis 1, 2; modes per transform
    int64_t d_a, d_l;
    int64_t rows_f, fstride;  // frames: rows (N0 N1) and mode values (C nm) per frame; rows_f 0: one frame
    __device__ __forceinline__ float2 load(int64_t a, int l, int64_t e) const {
        // row a -> (frame, row of the frame) -> (mode 0, mode 1); 32-bit: F N0 N1 < 2^32 (setpts)
        uint32_t al = (uint32_t)a;
        int64_t fo = 0;
        if (rows_f) {
            const uint32_t fr = al / (uint32_t)rows_f;
            al -= fr * (uint32_t)rows_f;
            fo = (int64_t)fr * fstride;
        }
        const uint32_t i0 = al / (uint32_t)N1, i1 = al - i0 * (uint32_t)N1;
        const float sc = d0[i0] * d1[i1] * d2[l];
        return cscale(f[fo + e * nm + (int64_t)al * N2 + l], sc);
    }
    static constexpr int kPairShapes = 2;
    // pair access (fftp.cuh): a column is contiguous along the modes of axis 2
    struct CState {
        float sc;
    };
    __device__ __forceinline__ const float2* cin(int64_t a, int64_t e) const {
        uint32_t al = (uint32_t)a;
        int64_t fo = 0;
        if (rows_f) {
            const uint32_t fr = al / (uint32_t)rows_f;
            al -= fr * (uint32_t)rows_f;
            fo = (int64_t)fr * fstride;
        }
        return f + fo + e * nm + (int64_t)al * N2;
    }
    __device__ __forceinline__ CState cstate(int64_t a, int64_t, bool ok) const {
        if (!ok) return {0.f};
        uint32_t al = (uint32_t)a;
        if (rows_f) al %= (uint32_t)rows_f;
        const uint32_t i0 = al / (uint32_t)N1, i1 = al - i0 * (uint32_t)N1;
        return {d0[i0] * d1[i1]};
    }
    __device__ __forceinline__ float2 cvalue(const CState& st, int l, float2 v) const { return cscale(v, st.sc * d2[l]); }
    int rows_shared(int) const { return 0; }
    __device__ __forceinline__ const float2* row(int64_t, int64_t) const { return nullptr; }
    __device__ __forceinline__ void cstate_row(CState&, const float2*) const {}
    bool vout_even() const { return ((d_a | d_l) & 1) == 0; }
    const void* vout_base() const { return dst; }
    static constexpr bool kVecOut = true;
    using OState = float2*;
    __device__ __forceinline__ OState ostate(int64_t a, int64_t e, bool) const { return dst + a * d_a + e; }
    __device__ __forceinline__ void ostore(OState p, int o, float2 v) const { p[(int64_t)o * d_l] = v; }
    __device__ __forceinline__ int64_t vout_l() const { return d_l; }
    __device__ __forceinline__ c2 vout_value(c2 v) const { return v; }
    __device__ __forceinline__ int64_t kcol(int64_t) const { return 0; }
    __device__ __forceinline__ const float2* kptr(int64_t) const { return nullptr; }
    __device__ __forceinline__ const float2* srow(int64_t, int64_t) const { return nullptr; }
    __device__ __forceinline__ float2 product_s(float2 v, float2) const { return v; }
    __device__ __forceinline__ int64_t group(int64_t) const { return 0; }
    __device__ __forceinline__ int ngroups() const { return 1; }
    __device__ __forceinline__ float2 kval(int64_t, int, int64_t) const { return make_float2(0.f, 0.f); }
    __device__ __forceinline__ void store(int64_t a, int o, int64_t e, float2 v) const { dst[a * d_a + (int64_t)o * d_l + e] = v; }
    __device__ __forceinline__ float2 product(int64_t, int, int64_t, float2 v) const { return v; }
    __device__ __forceinline__ void write_row(int64_t, int, int, float2) const {}
    __device__ __forceinline__ void store_phase(const float2* res, const PassCfg& c, int64_t a0, int64_t e0, int, int,
                                                float2*) const {
        float2* d = dst;
        const int64_t da = d_a, dl = d_l;
        for_each_output<false>(res, c, a0, e0, [&](int64_t a, int o, int64_t e, float2 v) { d[a * da + (int64_t)o * dl + e] = v; });
    }
    __device__ __forceinline__ void finish(const PassCfg&, int64_t, float2*) const {}
};

// Store modes f[e][a][o] scaled by 1/phihat from the interleaved buffer.
struct OpModesOut {
    static constexpr bool kLoadLFast = false;
    static constexpr bool kStoreLFast = true;
    static constexpr bool kFusedK = false;
    static constexpr bool kChunkLoop = false;
    static constexpr bool kSenseReduce = false;
    const float2* src;  // [rows][nf2][C]
    float2* f;
    const float* d0;
    const float* d1;
    const float* d2;
    int64_t N1, N2, nm;
    int64_t s_a, s_l;
    int64_t rows_f, fstride;  // frames: rows (N0 N1) and mode values (C nm) per frame; rows_f 0: one frame
    __device__ __forceinline__ float2 load(int64_t a, int l, int64_t e) const { return src[a * s_a + (int64_t)l * s_l + e]; }
    static constexpr int kPairShapes = 1;
    struct OState {
        float2* p;
        float sc;
    };
    __device__ __forceinline__ OState ostate(int64_t a, int64_t e, bool ok) const {
        if (!ok) return {f, 0.f};
        uint32_t al = (uint32_t)a;
        int64_t fo = 0;
        if (rows_f) {
            const uint32_t fr = al / (uint32_t)rows_f;
            al -= fr * (uint32_t)rows_f;
            fo = (int64_t)fr * fstride;
        }
        const uint32_t i0 = al / (uint32_t)N1, i1 = al - i0 * (uint32_t)N1;
        return {f + fo + e * nm + (int64_t)al * N2, d0[i0] * d1[i1]};
    }
    __device__ __forceinline__ void ostore(const OState& s, int o, float2 v) const { s.p[o] = cscale(v, s.sc * d2[o]); }
    // pair access (fftp.cuh)
    bool vin_even() const { return ((s_a | s_l) & 1) == 0; }
    const void* vin_base() const { return src; }
    __device__ __forceinline__ const float2* vin(int64_t a, int64_t e) const { return src + a * s_a + e; }
    __device__ __forceinline__ int64_t vin_l() const { return s_l; }
    __device__ __forceinline__ int64_t kcol(int64_t) const { return 0; }
    __device__ __forceinline__ const float2* kptr(int64_t) const { return nullptr; }
    __device__ __forceinline__ const float2* srow(int64_t, int64_t) const { return nullptr; }
    __device__ __forceinline__ float2 product_s(float2 v, float2) const { return v; }
    __device__ __forceinline__ int64_t group(int64_t) const { return 0; }
    __device__ __forceinline__ int ngroups() const { return 1; }
    __device__ __forceinline__ float2 kval(int64_t, int, int64_t) const { return make_float2(0.f, 0.f); }
    __device__ __forceinline__ void store(int64_t a, int o, int64_t e, float2 v) const {
        uint32_t al = (uint32_t)a;
        int64_t fo = 0;
        if (rows_f) {
            const uint32_t fr = al / (uint32_t)rows_f;
            al -= fr * (uint32_t)rows_f;
            fo = (int64_t)fr * fstride;
        }
        const uint32_t i0 = al / (uint32_t)N1, i1 = al - i0 * (uint32_t)N1;
        const float sc = d0[i0] * d1[i1] * d2[o];
        f[fo + e * nm + (int64_t)al * N2 + o] = cscale(v, sc);
    }
    __device__ __forceinline__ float2 product(int64_t, int, int64_t, float2 v) const { return v; }
    __device__ __forceinline__ void write_row(int64_t, int, int, float2) const {}
    __device__ __forceinline__ void store_phase(const float2* res, const PassCfg& c, int64_t a0, int64_t e0, int, int,
                                                float2*) const {
        for_each_output<true>(res, c, a0, e0, [&](int64_t a, int o, int64_t e, float2 v) { store(a, o, e, v); });
    }
    __device__ __forceinline__ void finish(const PassCfg&, int64_t, float2*) const {}
};

HB_EXTERN_PASS(OpModesIn)
HB_EXTERN_PASS(OpModesOut)

#endif

}  // namespace hb

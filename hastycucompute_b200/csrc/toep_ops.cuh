// Pass operators of the Toeplitz convolution (see fft.cuh, fft2.cuh and fftp.cuh for the contract).
#pragma once

#include "ops.cuh"

namespace hb {

#ifdef __CUDACC__


struct OpToepIn {
    static constexpr int kHalfIO = 1;  // pass shape (pass2_kernel HM)
    static constexpr bool kLoadLFast = true;
    static constexpr bool kStoreLFast = false;
    static constexpr bool kFusedK = false;
    static constexpr bool kChunkLoop = false;
    static constexpr bool kSenseReduce = false;
    const float2* in;
    const float2* m1;
    const float2* m2;
    int in_m1, in_m2;
    float2* dst;
    int64_t N2, n, d_a, d_l;
    // frames: column e = f * cpf + c reads in[c] and m1[f] (cpf = 0: in[e], shared m1)
    int64_t cpf;
    __device__ __forceinline__ float2 load(int64_t a, int l, int64_t e) const {
        const int64_t idx = a * N2 + l;
        const int64_t ei = cpf ? e % cpf : e;
        const int64_t m1o = cpf ? (e / cpf) * n : 0;
        float2 v = in[ei * n + idx];
        if (m1) v = mult_typed(v, m1[m1o + idx], in_m1);
        if (m2) v = mult_typed(v, m2[idx], in_m2);
        return v;
    }
    struct CState {
        const float2 *f1, *f2;
    };
    // pair access (fftp.cuh)
    bool vout_even() const { return ((d_a | d_l) & 1) == 0; }
    const void* vout_base() const { return dst; }
    static constexpr bool kVecOut = true;
    using OState = float2*;
    __device__ __forceinline__ OState ostate(int64_t a, int64_t e, bool) const { return dst + a * d_a + e; }
    __device__ __forceinline__ void ostore(OState p, int o, float2 v) const { p[(int64_t)o * d_l] = v; }
    int rows_shared(int) const { return 0; }
    __device__ __forceinline__ const float2* row(int64_t, int64_t) const { return nullptr; }
    __device__ __forceinline__ void cstate_row(CState&, const float2*) const {}
    __device__ __forceinline__ int64_t vout_l() const { return d_l; }
    __device__ __forceinline__ c2 vout_value(c2 v) const { return v; }
    __device__ __forceinline__ const float2* cin(int64_t a, int64_t e) const { return in + (cpf ? e % cpf : e) * n + a * N2; }
    __device__ __forceinline__ CState cstate(int64_t a, int64_t e, bool ok) const {
        return {m1 ? m1 + (cpf && ok ? (e / cpf) * n : 0) + a * N2 : nullptr, m2 ? m2 + a * N2 : nullptr};
    }
    __device__ __forceinline__ float2 cvalue(const CState& f, int l, float2 v) const {
        if (f.f1) v = mult_typed(v, f.f1[l], in_m1);
        if (f.f2) v = mult_typed(v, f.f2[l], in_m2);
        return v;
    }
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

// P1 of the SENSE normal operator: column e = f * cpf + c reads S_c[idx] * x_f[idx] (cpf = 0: one
// frame, x shared by all coils), times the diagonal m2[idx] when kDiag. The product is fixed at
// compile time.
template <bool kDiag>
struct OpToepInSenseT : OpToepIn {
    __device__ __forceinline__ float2 load(int64_t a, int l, int64_t e) const {
        return cmul(load_col(a, l, e), row_at(a, l, e));
    }
    // pair access: x is one row for all columns of a CTA within one frame
    int rows_shared(int eb) const { return cpf == 0 || cpf % eb == 0; }
    __device__ __forceinline__ void cstate_row(CState& f, const float2* r) const { f.f1 = r; }
    __device__ __forceinline__ float2 cvalue(const CState& f, int l, float2 v) const {
        if constexpr (kDiag) v = cmul(v, f.f2[l]);
        return cmul(v, f.f1[l]);
    }
    // the image factor x is the same for every coil column of a row within one frame: when a
    // CTA's columns e0 .. e0+eb-1 lie in one frame the pass stages that row once per CTA
    static constexpr bool kStageRow = true;
    __device__ __forceinline__ bool row_shared(int64_t e0, int eb) const {
        return cpf == 0 || e0 / cpf == (e0 + eb - 1) / cpf;
    }
    __device__ __forceinline__ const float2* row(int64_t a, int64_t e0) const {
        return m1 + (cpf ? (e0 / cpf) * n : 0) + a * N2;
    }
    __device__ __forceinline__ float2 row_at(int64_t a, int l, int64_t e) const {
        return m1[(cpf ? (e / cpf) * n : 0) + a * N2 + l];
    }
    __device__ __forceinline__ float2 load_col(int64_t a, int l, int64_t e) const {
        const int64_t idx = a * N2 + l;
        float2 v = in[(cpf ? e % cpf : e) * n + idx];
        if constexpr (kDiag) v = cmul(v, m2[idx]);
        return v;
    }
};
using OpToepInSense = OpToepInSenseT<false>;

// The Toeplitz passes along the middle axis: zero-padding N -> 2N (forward) and cropping
// 2N -> N (inverse), both at offset 0.
// (kPrefetch is of the single-column kernel, which serves 512 and 640 points: there it measured slower for both, two
// or three CTAs per SM against four. The pair passes always copy the next job's samples ahead.)
struct OpStridedPad : OpStrided {
    static constexpr int kHalfIO = 1;
};
struct OpStridedCrop : OpStrided {
    static constexpr int kHalfIO = 2;
};

// In-place fused pass: FFT, * Kt[col][pos], IFFT, crop. buf[l][e] with row stride E.
struct OpToepMid {
    static constexpr int kHalfIO = 3;  // pass shape (pass2_kernel HM)
    static constexpr bool kPrefetch = true;  // persistent CTAs, next block's samples by cp.async
    static constexpr bool kLoadLFast = false;
    static constexpr bool kStoreLFast = false;
    static constexpr bool kFusedK = true;
    static constexpr bool kChunkLoop = false;
    static constexpr bool kSenseReduce = false;
    float2* buf;
    const float2* kt;
    int64_t E, B;
    int Lk;
    __device__ __forceinline__ float2 load(int64_t, int l, int64_t e) const { return buf[(int64_t)l * E + e]; }
    __device__ __forceinline__ const float2* sample_ptr(int64_t, int l, int64_t e) const { return buf + (int64_t)l * E + e; }
    // pair access (fftp.cuh); the fused pass works in place
    bool vin_even() const { return (E & 1) == 0; }
    const void* vin_base() const { return buf; }
    __device__ __forceinline__ const float2* vin(int64_t, int64_t e) const { return buf + e; }
    __device__ __forceinline__ int64_t vin_l() const { return E; }
    bool vout_even() const { return (E & 1) == 0; }
    const void* vout_base() const { return buf; }
    static constexpr bool kVecOut = true;
    using OState = float2*;
    __device__ __forceinline__ OState ostate(int64_t, int64_t e, bool) const { return buf + e; }
    __device__ __forceinline__ void ostore(OState p, int o, float2 v) const { p[(int64_t)o * E] = v; }
    __device__ __forceinline__ int64_t vout_l() const { return E; }
    __device__ __forceinline__ c2 vout_value(c2 v) const { return v; }
    int64_t cols_per_kernel() const { return B; }
    // kernel column of column e: a 32-bit division whenever the operands fit (every workspace
    // this library sizes), the 64-bit one otherwise
    __device__ __forceinline__ int64_t kcol(int64_t e) const {
        return ((uint64_t)e | (uint64_t)B) <= 0xffffffffull ? (int64_t)((uint32_t)e / (uint32_t)B) : e / B;
    }
    __device__ __forceinline__ const float2* kptr(int64_t kc) const { return kt + kc * Lk; }
    __device__ __forceinline__ const float2* srow(int64_t, int64_t) const { return nullptr; }
    __device__ __forceinline__ float2 product_s(float2 v, float2) const { return v; }
    __device__ __forceinline__ int64_t group(int64_t) const { return 0; }
    __device__ __forceinline__ int ngroups() const { return 1; }
    __device__ __forceinline__ float2 kval(int64_t, int pos, int64_t e) const { return kt[kcol(e) * Lk + pos]; }
    __device__ __forceinline__ void store(int64_t, int o, int64_t e, float2 v) const { buf[(int64_t)o * E + e] = v; }
    __device__ __forceinline__ float2 product(int64_t, int, int64_t, float2 v) const { return v; }
    __device__ __forceinline__ void write_row(int64_t, int, int, float2) const {}
    __device__ __forceinline__ void store_phase(const float2* res, const PassCfg& c, int64_t a0, int64_t e0, int, int,
                                                float2*) const {
        float2* d = buf;
        const int64_t EE = E;
        for_each_output<false>(res, c, a0, e0, [&](int64_t, int o, int64_t e, float2 v) { d[(int64_t)o * EE + e] = v; });
    }
    __device__ __forceinline__ void finish(const PassCfg&, int64_t, float2*) const {}
};

struct OpToepOutFlat {
    static constexpr int kHalfIO = 2;  // pass shape (pass2_kernel HM)
    static constexpr bool kLoadLFast = false;
    static constexpr bool kStoreLFast = true;
    static constexpr bool kFusedK = false;
    static constexpr bool kChunkLoop = false;
    static constexpr bool kSenseReduce = false;
    const float2* src;  // [rows][L2][B]
    int64_t s_a, s_l;
    const float2* in;
    const float2* m1;
    const float2* m2;
    int io_mult, out_m1, out_m2, accumulate;
    float2* out;
    int64_t N2, n;
    __device__ __forceinline__ float2 load(int64_t a, int l, int64_t e) const { return src[a * s_a + (int64_t)l * s_l + e]; }
    struct OState {
        int64_t idx, eo;  // image index of output 0, offset of the batch
    };
    __device__ __forceinline__ OState ostate(int64_t a, int64_t e, bool) const { return {a * N2, e * n}; }
    __device__ __forceinline__ void ostore(const OState& s, int o, float2 v) const {
        const int64_t idx = s.idx + o;
        if (m1) v = mult_typed(v, m1[idx], out_m1);
        if (m2) v = mult_typed(v, m2[idx], out_m2);
        if (io_mult) v = mult_typed(v, in[s.eo + idx], io_mult);
        float2* d = out + s.eo + idx;
        if (accumulate) v = cadd(v, *d);
        *d = v;
    }
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
        const int64_t idx = a * N2 + o;
        if (m1) v = mult_typed(v, m1[idx], out_m1);
        if (m2) v = mult_typed(v, m2[idx], out_m2);
        if (io_mult) v = mult_typed(v, in[e * n + idx], io_mult);
        float2* dst = out + e * n + idx;
        if (accumulate) v = cadd(v, *dst);
        *dst = v;
    }
    __device__ __forceinline__ float2 product(int64_t, int, int64_t, float2 v) const { return v; }
    __device__ __forceinline__ void write_row(int64_t, int, int, float2) const {}
    __device__ __forceinline__ void store_phase(const float2* res, const PassCfg& c, int64_t a0, int64_t e0, int, int,
                                                float2*) const {
        for_each_output<true>(res, c, a0, e0, [&](int64_t a, int o, int64_t e, float2 v) { store(a, o, e, v); });
    }
    __device__ __forceinline__ void finish(const PassCfg&, int64_t, float2*) const {}
};

// Last pass of the SENSE normal operator: out[f][a][o] = sum_c conj(S_c[a][o]) * v_{f,c}[a][o],
// columns e = f * cpf + c (one frame when cpf = B). The CTA walks every batch chunk of its rows and
// keeps one running sum per (row, frame) in shared memory (extra).
struct OpToepOutSense {
    static constexpr int kHalfIO = 2;  // pass shape (pass2_kernel HM)
    static constexpr bool kPrefetch = true;  // persistent rows, next chunk's samples by cp.async
    static constexpr bool kLoadLFast = false;
    static constexpr bool kStoreLFast = false;
    static constexpr bool kFusedK = false;
    static constexpr bool kChunkLoop = true;
    static constexpr bool kSenseReduce = true;
    const float2* src;
    int64_t s_a, s_l;
    const float2* smaps;
    float2* out;
    int64_t N2, n;
    int64_t cpf;  // coils per frame
    int nfr;      // frames
    const float2* odiag;  // optional: the coil sum is multiplied by conj(odiag[idx])
    int accumulate;       // add into out instead of overwriting it
    __device__ __forceinline__ void emit(int64_t oi, int64_t ii, float2 v) const {
        if (odiag) v = cmulc(v, odiag[ii]);
        if (accumulate) v = cadd(v, out[oi]);
        out[oi] = v;
    }
    __device__ __forceinline__ float2 load(int64_t a, int l, int64_t e) const { return src[a * s_a + (int64_t)l * s_l + e]; }
    __device__ __forceinline__ const float2* sample_ptr(int64_t a, int l, int64_t e) const { return src + a * s_a + (int64_t)l * s_l + e; }
    using OState = int;  // (no column outputs)
    // pair access (fftp.cuh)
    bool vin_even() const { return ((s_a | s_l) & 1) == 0; }
    const void* vin_base() const { return src; }
    __device__ __forceinline__ const float2* vin(int64_t a, int64_t e) const { return src + a * s_a + e; }
    __device__ __forceinline__ int64_t vin_l() const { return s_l; }
    __device__ __forceinline__ int64_t kcol(int64_t) const { return 0; }
    __device__ __forceinline__ const float2* kptr(int64_t) const { return nullptr; }
    __device__ __forceinline__ const float2* srow(int64_t a, int64_t e) const { return smaps + (e % cpf) * n + a * N2; }
    __device__ __forceinline__ float2 product_s(float2 v, float2 sv) const { return cmulc(v, sv); }
    __device__ __forceinline__ int64_t group(int64_t e) const { return e / cpf; }
    __device__ __forceinline__ int ngroups() const { return nfr; }
    __device__ __forceinline__ float2 kval(int64_t, int, int64_t) const { return make_float2(0.f, 0.f); }
    __device__ __forceinline__ void store(int64_t, int, int64_t, float2) const {}
    __device__ __forceinline__ float2 product(int64_t a, int o, int64_t e, float2 v) const {
        return cmulc(v, smaps[(e % cpf) * n + a * N2 + o]);
    }
    __device__ __forceinline__ void write_row(int64_t a, int o, int g, float2 v) const {
        emit(g * n + a * N2 + o, a * N2 + o, v);
    }
    // generic-kernel path: acc is [A_blk][nfr][Lout], zeroed on the first chunk
    __device__ __forceinline__ void store_phase(const float2* res, const PassCfg& c, int64_t a0, int64_t e0, int Ab, int Eb,
                                                float2* acc) const {
        const int ng = nfr;
        if (e0 == 0) {
            for (int i = threadIdx.x; i < Ab * ng * c.Lout; i += blockDim.x) acc[i] = make_float2(0.f, 0.f);
            __syncthreads();
        }
        const int tot = Ab * c.Lout;
        for (int idx = threadIdx.x; idx < tot; idx += blockDim.x) {
            const int o = idx % c.Lout, al = idx / c.Lout;
            const int64_t a = a0 + al;
            if (a >= c.A) continue;
            int pos = (o + c.out_shift) % c.L;
            if (pos < 0) pos += c.L;
            const int64_t idx_img = a * N2 + o;
            float2 run = make_float2(0.f, 0.f);
            int64_t gcur = group(e0);
            for (int el = 0; el < Eb; ++el) {
                const int64_t e = e0 + el;
                if (e >= c.E) break;
                const int64_t gg = group(e);
                if (gg != gcur) {
                    float2* dst = acc + ((int64_t)al * ng + gcur) * c.Lout + o;
                    *dst = cadd(*dst, run);
                    run = make_float2(0.f, 0.f);
                    gcur = gg;
                }
                const float2 v = res[pos * c.Wp + al * Eb + el];
                run = cadd(run, cmulc(v, smaps[(e % cpf) * n + idx_img]));
            }
            float2* dst = acc + ((int64_t)al * ng + gcur) * c.Lout + o;
            *dst = cadd(*dst, run);
        }
    }
    __device__ __forceinline__ void finish(const PassCfg& c, int64_t a0, float2* acc) const {
        const int ng = nfr;
        const int tot = c.A_blk * ng * c.Lout;
        for (int idx = threadIdx.x; idx < tot; idx += blockDim.x) {
            const int o = idx % c.Lout, rest = idx / c.Lout, gg = rest % ng, al = rest / ng;
            const int64_t a = a0 + al;
            if (a >= c.A) continue;
            emit(gg * n + a * N2 + o, a * N2 + o, acc[idx]);
        }
    }
};

HB_EXTERN_PASS(OpToepIn)
HB_EXTERN_PASS(OpToepInSenseT<false>)
HB_EXTERN_PASS(OpToepInSenseT<true>)
HB_EXTERN_PASS(OpStridedPad)
HB_EXTERN_PASS(OpStridedCrop)
HB_EXTERN_PASS(OpToepMid)
HB_EXTERN_PASS(OpToepOutFlat)
HB_EXTERN_PASS(OpToepOutSense)

#endif

}  // namespace hb

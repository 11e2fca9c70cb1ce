// Two-level register FFT pass (L = P * Q, radices up to 26) on pairs of columns, for every length
// the plans use that splits that way.
//
// For one column x[0..L), with n = t + Q j and k = k1 + P k2 (t, k2 < Q; j, k1 < P):
//     X[k1 + P k2] = sum_t W_Q^{t k2} [ W_L^{t k1} sum_j x[t + Q j] W_P^{j k1} ]
// Step 1: thread (t, pair) loads P samples, runs the P-point DFT and leaves it in shared memory;
// step 2: thread (k1, pair) reads Q values, runs the Q-point DFT and stores X[k1 + P k2]. One
// shared-memory round trip per transform. Fused kernel passes multiply, run the inverse Q-point
// DFT in place, and a third step runs the inverse P-point DFT.
//
// Every thread carries two columns: each value is a pair of packed f32x2 registers (re0, re1),
// (im0, im1). A packed instruction does two columns' arithmetic in one issue slot (the FMA pipe
// does the same work either way; these passes run out of issue slots before they run out of FMA
// or HBM), and adjacent columns load and store as one 16-byte access. A tile row of the transpose
// is kPairs x 16 bytes = 128 bytes, so a quarter-warp reads one row without bank conflicts.
//
// P and Q are run-time values: the steps are compiled once per radix and chosen by a uniform
// switch, so one kernel serves every length instead of one instance per length. Larger radices need
// more registers, so there are three such instances: radices up to 16, up to 20 and up to 26. The lengths 64, 128,
// 256 and 320 have instances with their radices as constants (launch_pair_dir).
//
// What bounds it at 320 points: not one unit but latency, with three CTAs of five warps an SM (128 registers). The
// fused Toeplitz pass (160^3, 8 coils: 0.87 ms) has DRAM at 32 %, the FMA pipe at 47 %, issue slots at 50 % and the
// shared-memory data path at 50 %; its warps wait for fixed latencies, barriers and shared memory. The plain
// passes stand at 66 % of DRAM, the first and the last one at 47 and 42 %.
//
// Against the shared-memory Stockham kernel that served these lengths before (B200): the SENSE normal
// operator at 88 x 104 x 110, 6 coils, 2.47 -> 0.53 ms; type 1 at 120 x 96 x 150, 12 transforms, 5.93 ->
// 2.93 ms (its FFT passes 3.95 -> 0.95 ms); type 2 at 90 x 110 x 75, 5 transforms, 1.21 -> 0.48 ms.
#pragma once

#include "fft2.cuh"

namespace hb {

#ifdef __CUDACC__

// ---- packed arithmetic ------------------------------------------------------------------------
typedef unsigned long long f2_t;  // two floats in a 64-bit register pair

__device__ __forceinline__ f2_t f2_pack(float a, float b) {
    f2_t d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(a), "f"(b));
    return d;
}
__device__ __forceinline__ void f2_unpack(f2_t v, float& a, float& b) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ f2_t f2_dup(float a) { return f2_pack(a, a); }
__device__ __forceinline__ f2_t f2_add(f2_t a, f2_t b) {
    f2_t d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ f2_t f2_sub(f2_t a, f2_t b) {
    f2_t d;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ f2_t f2_mul(f2_t a, f2_t b) {
    f2_t d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ f2_t f2_fma(f2_t a, f2_t b, f2_t c) {
    f2_t d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
// (as scalar negations of a factor: those fold into the multiply)
__device__ __forceinline__ f2_t f2_neg(f2_t v) {
    float a, b;
    f2_unpack(v, a, b);
    return f2_pack(-a, -b);
}

// one complex value of two columns
struct __align__(16) c2 {
    f2_t re, im;
};
__device__ __forceinline__ c2 c2_pack(float2 a, float2 b) { return {f2_pack(a.x, b.x), f2_pack(a.y, b.y)}; }
__device__ __forceinline__ void c2_unpack(c2 v, float2& a, float2& b) {
    f2_unpack(v.re, a.x, b.x);
    f2_unpack(v.im, a.y, b.y);
}
__device__ __forceinline__ c2 c2_add(c2 a, c2 b) { return {f2_add(a.re, b.re), f2_add(a.im, b.im)}; }
__device__ __forceinline__ c2 c2_sub(c2 a, c2 b) { return {f2_sub(a.re, b.re), f2_sub(a.im, b.im)}; }
// a + j b and a - j b with j = -i (forward) or +i (inverse)
template <bool INV>
__device__ __forceinline__ c2 c2_addj(c2 a, c2 b) {
    return INV ? c2{f2_sub(a.re, b.im), f2_add(a.im, b.re)} : c2{f2_add(a.re, b.im), f2_sub(a.im, b.re)};
}
// a * (wr + i wi), wr and wi the same or different for the two columns
__device__ __forceinline__ c2 c2_mul(c2 a, f2_t wr, f2_t wi) {
    return {f2_fma(f2_neg(a.im), wi, f2_mul(a.re, wr)), f2_fma(a.im, wr, f2_mul(a.re, wi))};
}
template <bool INV>
__device__ __forceinline__ c2 c2_mul_tw(c2 a, float2 w) {
    return c2_mul(a, f2_dup(w.x), f2_dup(INV ? -w.y : w.y));
}

// ---- DFTs in registers ------------------------------------------------------------------------
template <int R>
struct PrimeRadix {
    static constexpr bool value = R == 3 || R == 5 || R == 7 || R == 11 || R == 13;
};
// first factor of a composite radix: the largest power of two of an even one, else its smallest prime
template <int R>
constexpr int pair_factor() {
    if (R == 4 || R == 8 || R == 16) return R == 4 ? 2 : 4;
    if (R % 8 == 0) return 8;
    if (R % 4 == 0) return 4;
    if (R % 2 == 0) return 2;
    return R % 3 == 0 ? 3 : 5;
}
constexpr int ct_gcd(int a, int b) { return b == 0 ? a : ct_gcd(b, a % b); }
constexpr int ct_inv(int a, int m) {  // a^-1 mod m (coprime)
    for (int x = 1; x < m; ++x)
        if (a * x % m == 1) return x;
    return 1 % m;
}

// a * W_R^M (INV: the conjugate)
template <int R, int M, bool INV>
__device__ __forceinline__ c2 c2_tw(c2 a) {
    constexpr int m = ((M % R) + R) % R;
    if constexpr (m == 0) {
        return a;
    } else if constexpr (2 * m == R) {
        return {f2_neg(a.re), f2_neg(a.im)};
    } else if constexpr (4 * m == R || 4 * m == 3 * R) {
        constexpr bool plus = (4 * m == R) == INV;  // times +i, else -i
        return plus ? c2{f2_neg(a.im), a.re} : c2{a.im, f2_neg(a.re)};
    } else {
        constexpr float c = (float)ct_cos(ct_angle<R, m>());
        constexpr float s = (float)(INV ? ct_sin(ct_angle<R, m>()) : -ct_sin(ct_angle<R, m>()));
        return {f2_fma(a.im, f2_dup(-s), f2_mul(a.re, f2_dup(c))), f2_fma(a.im, f2_dup(c), f2_mul(a.re, f2_dup(s)))};
    }
}

template <bool INV>
__device__ __forceinline__ void c2_dft4(c2& x0, c2& x1, c2& x2, c2& x3) {
    const c2 t0 = c2_add(x0, x2), t1 = c2_sub(x0, x2), t2 = c2_add(x1, x3), t3 = c2_sub(x1, x3);
    x0 = c2_add(t0, t2);
    x2 = c2_sub(t0, t2);
    x1 = c2_addj<INV>(t1, t3);
    x3 = c2_addj<!INV>(t1, t3);
}

// odd primes by the symmetric pairs t_j = x_j + x_{R-j}, u_j = x_j - x_{R-j}:
//   y_k = x_0 + sum_j cos(2 pi jk/R) t_j -/+ i sum_j sin(2 pi jk/R) u_j
template <int R, bool INV>
__device__ __forceinline__ void c2_dft_odd(c2* v) {
    constexpr int H = (R - 1) / 2;
    c2 t[H], u[H];
#pragma unroll
    for (int j = 1; j <= H; ++j) {
        t[j - 1] = c2_add(v[j], v[R - j]);
        u[j - 1] = c2_sub(v[j], v[R - j]);
    }
    const c2 x0 = v[0];
    c2 sum = x0;
#pragma unroll
    for (int j = 0; j < H; ++j) sum = c2_add(sum, t[j]);
    static_for<H>([&](auto kk) {
        constexpr int k = decltype(kk)::value + 1;
        c2 a = x0, b{};
        static_for<H>([&](auto jj) {
            constexpr int j = decltype(jj)::value + 1;
            const f2_t c = f2_dup((float)ct_cos(ct_angle<R, j * k>()));
            const f2_t s = f2_dup((float)ct_sin(ct_angle<R, j * k>()));
            a.re = f2_fma(t[j - 1].re, c, a.re);
            a.im = f2_fma(t[j - 1].im, c, a.im);
            if constexpr (j == 1) {
                b.re = f2_mul(u[0].re, s);
                b.im = f2_mul(u[0].im, s);
            } else {
                b.re = f2_fma(u[j - 1].re, s, b.re);
                b.im = f2_fma(u[j - 1].im, s, b.im);
            }
        });
        v[k] = c2_addj<INV>(a, b);
        v[R - k] = c2_addj<!INV>(a, b);
    });
    v[0] = sum;
}

// R-point DFT in place. Composite radices split A x B: by the Chinese remainder theorem without
// twiddles where A and B are coprime (inputs n = B n1 + A n2, outputs k = k1 mod A = k2 mod B),
// by Cooley-Tukey with constant twiddles otherwise.
template <int R, bool INV>
__device__ __forceinline__ void c2_dft(c2* v) {
    if constexpr (R == 1) {
        return;
    } else if constexpr (R == 2) {
        const c2 a = v[0], b = v[1];
        v[0] = c2_add(a, b);
        v[1] = c2_sub(a, b);
    } else if constexpr (R == 4) {
        c2_dft4<INV>(v[0], v[1], v[2], v[3]);
    } else if constexpr (PrimeRadix<R>::value) {
        c2_dft_odd<R, INV>(v);
    } else {
        constexpr int A = pair_factor<R>(), B = R / A;
        c2 y[R];
        if constexpr (ct_gcd(A, B) == 1) {
            static_for<B>([&](auto nc) {
                constexpr int n2 = decltype(nc)::value;
                c2 a[A];
                static_for<A>([&](auto mc) {
                    constexpr int n1 = decltype(mc)::value;
                    a[n1] = v[(B * n1 + A * n2) % R];
                });
                c2_dft<A, INV>(a);
#pragma unroll
                for (int k1 = 0; k1 < A; ++k1) y[k1 * B + n2] = a[k1];
            });
            static_for<A>([&](auto kc) {
                constexpr int k1 = decltype(kc)::value;
                c2_dft<B, INV>(y + k1 * B);
                static_for<B>([&](auto lc) {
                    constexpr int k2 = decltype(lc)::value;
                    v[(k1 * B * ct_inv(B % A, A) + k2 * A * ct_inv(A % B, B)) % R] = y[k1 * B + k2];
                });
            });
        } else {
            static_for<B>([&](auto tc) {
                constexpr int t = decltype(tc)::value;
                c2 a[A];
#pragma unroll
                for (int j = 0; j < A; ++j) a[j] = v[t + B * j];
                c2_dft<A, INV>(a);
                static_for<A>([&](auto kc) {
                    constexpr int k1 = decltype(kc)::value;
                    y[k1 * B + t] = c2_tw<R, t * k1, INV>(a[k1]);
                });
            });
#pragma unroll
            for (int k1 = 0; k1 < A; ++k1) {
                c2_dft<B, INV>(y + k1 * B);
#pragma unroll
                for (int k2 = 0; k2 < B; ++k2) v[k1 + A * k2] = y[k1 * B + k2];
            }
        }
    }
}

// R-point DFT of v[0..R/2) followed by R/2 zeros (R even): X[2m] = DFT(v)[m],
// X[2m+1] = DFT(v_j W_R^j)[m]
template <int R, bool INV>
__device__ __forceinline__ void c2_dft_halfzero(c2* v) {
    constexpr int H = R / 2;
    c2 a[H], b[H];
    static_for<H>([&](auto jc) {
        constexpr int j = decltype(jc)::value;
        a[j] = v[j];
        b[j] = c2_tw<R, j, INV>(v[j]);
    });
    c2_dft<H, INV>(a);
    c2_dft<H, INV>(b);
#pragma unroll
    for (int m = 0; m < H; ++m) {
        v[2 * m] = a[m];
        v[2 * m + 1] = b[m];
    }
}

// ---- the pass -----------------------------------------------------------------------------------
constexpr int kPairs = 8;  // column pairs per CTA (kCW columns)
static_assert(2 * kPairs == kCW, "a CTA's columns");
constexpr int kRadixMax = 26;

// radices with a step function (one switch case each)
constexpr bool pair_radix(int r) {
    return (r >= 8 && r <= 16) || r == 18 || r == 20 || r == 21 || r == 22 || r == 24 || r == 25 || r == 26;
}
// the instance of a split (run-time radices), by its larger radix: the smallest radix it has a step for
constexpr int pair_rmin(int larger) { return larger <= 16 ? 8 : larger <= 20 ? 9 : 10; }

// (P, Q) of length L, the most even split into two radices of the set that one instance has; {0, 0} where there is
// none (189 = 9 x 21: the instance of 21 begins at 10). Of the two
// orders the one whose P (input_side) or Q is divisible by 4, else by 2: the side that a pass pads or crops.
constexpr void pair_split(int L, bool input_side, int* P, int* Q) {
    *P = *Q = 0;
    for (int hi = 8; hi <= kRadixMax; ++hi) {
        if (!pair_radix(hi) || L % hi != 0 || L / hi > hi || !pair_radix(L / hi) || L / hi < pair_rmin(hi)) continue;
        const int lo = L / hi;
        auto rank = [](int r) { return r % 4 == 0 ? 2 : r % 2 == 0 ? 1 : 0; };
        const bool lo_first = input_side ? rank(lo) >= rank(hi) : rank(hi) >= rank(lo);
        *P = lo_first ? lo : hi;
        *Q = L / *P;
        return;
    }
}
// every split is a product of two radices that its instance has
constexpr bool pair_splits_served() {
    for (int L = 1; L <= kRadixMax * kRadixMax; ++L) {
        for (int side = 0; side < 2; ++side) {
            int P = 0, Q = 0;
            pair_split(L, side != 0, &P, &Q);
            if (P == 0) continue;
            const int larger = P > Q ? P : Q, smaller = P > Q ? Q : P;
            if (P * Q != L || !pair_radix(P) || !pair_radix(Q) || smaller < pair_rmin(larger)) return false;
        }
    }
    return true;
}
static_assert(pair_splits_served(), "a radix without a step would leave its outputs unwritten");

struct PairCfg {
    int P, Q, L;
    int Lin, in_shift;    // sample l -> position (l + in_shift) mod L, in_shift in [0, L)
    int Lout, out_shift;
    int ph;               // centred input (1) / output (2): see pair_tw
    int vec_in, vec_out;  // pairs are 16-byte aligned neighbours
    int A_blk, E_blk;     // rows x inner columns per CTA (kSenseReduce: rows x inner pairs)
    int W;                 // columns of a job
    int in_stride, in_elems, s_stride, tw_n;
    int rows;              // kLoadLFast: the row factors are copied once per row
    int64_t n_jobs;
    int n_k;              // kFusedK: kernel columns staged in shared memory (0: read from global)
    unsigned n_eb;
    int64_t A, E;
    const float2* tw;
};


// Operators of the NUFFT axes: kPairShapes bit 0 = the input has full length (type 1 crops), bit 1 = the
// output has (type 2 pads). Where the other side is exactly half of it and centred, the pass runs the
// shapes of a fixed half side (HM 2 / 1); otherwise HM 4 / 8 with a position check per element. Operators with
// a fixed shape (kHalfIO) have that one.
template <class Op, class = void>
struct PairShapes {
    static constexpr int value = 0;
};
template <class Op>
struct PairShapes<Op, std::void_t<decltype(Op::kPairShapes)>> {
    static constexpr int value = Op::kPairShapes;
};

// How a pass gets its samples into shared memory (cp.async, issued while the previous job is
// transformed): an operator's columns lie side by side, sample (a, l, e) at vin(a, e) + l * vin_l(),
// and go to In[l][kPairs] as pairs (16-byte copies where pairs are aligned neighbours); or (kLoadLFast)
// each column is contiguous along l, at cin(a, e) + l, and goes to In[column][in_stride] (8-byte
// copies, odd stride: step 1 then reads different banks), where cvalue applies the operator's factors.
// kVecOut: a column's state is the address of output 0, outputs vout_l() apart, each through vout_value; a
// pair is one 16-byte store where vec_out.
template <class Op, class = void>
struct HasVecOut {
    static constexpr bool value = false;
};
template <class Op>
struct HasVecOut<Op, std::void_t<decltype(Op::kVecOut)>> {
    static constexpr bool value = true;
};

__device__ __forceinline__ void c2_st16(float2* p, c2 v) {
    float2 a, b;
    c2_unpack(v, a, b);
    *reinterpret_cast<float4*>(p) = make_float4(a.x, a.y, b.x, b.y);
}

// The two columns of a thread.
struct PairCols {
    int64_t a0, e0, a1, e1;
    bool ok0, ok1;
};

// Pair `cp` of the job at (a0, e0). Reducing operators keep a pair inside one row (E_blk pairs per
// row, the last one half empty when the row is odd); the others count columns through the rows.
template <class Op>
__device__ __forceinline__ PairCols pair_cols(const PairCfg& c, int64_t a0, int64_t e0, int cp) {
    PairCols k;
    if constexpr (Op::kSenseReduce) {
        const int al = c.A_blk == 1 ? 0 : cp / c.E_blk, pe = cp - al * c.E_blk;
        k.a0 = k.a1 = a0 + al;
        k.e0 = e0 + 2 * pe;
        k.e1 = k.e0 + 1;
        const bool in = al < c.A_blk && k.a0 < c.A;
        k.ok0 = in && k.e0 < c.E;
        k.ok1 = in && k.e1 < c.E;
    } else if (c.A_blk == 1) {
        k.a0 = k.a1 = a0;
        k.e0 = e0 + 2 * cp;
        k.e1 = k.e0 + 1;
        k.ok0 = 2 * cp < c.E_blk && k.e0 < c.E;
        k.ok1 = 2 * cp + 1 < c.E_blk && k.e1 < c.E;
    } else {
        const int q = 2 * cp, al0 = q / c.E_blk, al1 = (q + 1) / c.E_blk;
        k.a0 = a0 + al0;
        k.a1 = a0 + al1;
        k.e0 = q - al0 * c.E_blk;
        k.e1 = q + 1 - al1 * c.E_blk;
        k.ok0 = al0 < c.A_blk && k.a0 < c.A;
        k.ok1 = al1 < c.A_blk && k.a1 < c.A;
    }
    return k;
}

// slot of (row k1 * Q + t, pair cp) in the transpose: an operator whose lanes run along the outputs in step 2
// rotates the pairs of a row so that eight such lanes meet different banks
template <class Op>
__device__ __forceinline__ int pair_slot(int row, int k1, int cp) {
    return row * kPairs + (Op::kStoreLFast ? (cp ^ (k1 & (kPairs - 1))) : cp);
}

// Calls f(j, l) for the samples l of positions t + Q j, j < P, that the pass reads; z(j) for the others.
template <int P, int HM, class F, class Z>
__device__ __forceinline__ void pair_inputs(const PairCfg& c, int Q, int t, F&& f, Z&& z) {
    constexpr bool half = (HM & 1) != 0, full = (HM & 4) != 0 || (HM & 3) == 2;
#pragma unroll
    for (int j = 0; j < (half && P % 2 == 0 ? P / 2 : P); ++j) {
        const int pos = t + Q * j;
        if constexpr (full || (half && P % 2 == 0)) {
            f(j, pos);
        } else if constexpr (half) {
            if (2 * pos < c.L) f(j, pos); else z(j);
        } else {
            int l = pos - c.in_shift;
            if (l < 0) l += c.L;
            if (l < c.Lin) f(j, l); else z(j);
        }
    }
}

// Copies a job's samples into In (all threads).
template <int HM, class Op>
__device__ __forceinline__ void pair_fetch(const Op& op, const PairCfg& c, int64_t a0, int64_t e0, float4* In, float2* Rs) {
    if constexpr (Op::kLoadLFast) {
        // a warp per column
        for (int col = threadIdx.x >> 5; col < c.W; col += blockDim.x >> 5) {
            const int al = c.A_blk == 1 ? 0 : col / c.E_blk, el = col - al * c.E_blk;
            if (a0 + al >= c.A || e0 + el >= c.E) continue;
            const float2* p = op.cin(a0 + al, e0 + el);
            float2* d = reinterpret_cast<float2*>(In) + col * c.in_stride;
            for (int l = threadIdx.x & 31; l < c.Lin; l += 32) cp_async8(d + l, p + l);
        }
        if (c.rows) {
            for (int i = threadIdx.x; i < c.A_blk * c.Lin; i += blockDim.x) {
                const int al = c.A_blk == 1 ? 0 : i / c.Lin, l = i - al * c.Lin;
                if (a0 + al < c.A) cp_async8(Rs + i, op.row(a0 + al, e0) + l);
            }
        }
    } else {
        const int cp = threadIdx.x % kPairs;
        const PairCols k = pair_cols<Op>(c, a0, e0, cp);
        const int step = blockDim.x / kPairs;
        const int64_t sl = op.vin_l();
        if (c.vec_in) {
            if (!k.ok0) return;
            const float2* p = op.vin(k.a0, k.e0);
#pragma unroll 4
            for (int l = threadIdx.x / kPairs; l < c.Lin; l += step) cp_async16(In + l * kPairs + cp, p + l * sl);
        } else {
            const float2* p0 = k.ok0 ? op.vin(k.a0, k.e0) : nullptr;
            const float2* p1 = k.ok1 ? op.vin(k.a1, k.e1) : nullptr;
            for (int l = threadIdx.x / kPairs; l < c.Lin; l += step) {
                float2* d = reinterpret_cast<float2*>(In + l * kPairs + cp);
                if (p0) cp_async8(d, p0 + l * sl);
                if (p1) cp_async8(d + 1, p1 + l * sl);
            }
        }
    }
}

// Outer twiddle W_L^(t k1) of step 1. A centred half-length input (sample l at position l - L/4) is the
// transform of the unshifted input times i^k, and a centred output is the unshifted output of the input times
// i^n: with P (Q) divisible by 4 that is i^k1 (i^t), a quarter of the table added to the index
// (the table then holds two periods). The pass itself pads and crops at offset 0.
template <bool INV>
__device__ __forceinline__ c2 pair_tw(const PairCfg& c, int L, int t, int k1, const float2* tw, c2 v) {
    int at = t * k1;
    if (c.ph & 1) at += ((3 * k1) & 3) * (L / 4);
    if (c.ph & 2) at += ((3 * t) & 3) * (L / 4);
    return c2_mul_tw<INV>(v, tw[at]);
}

// Full-length samples of the plain operators share the transpose's memory: step 1 reads and writes the L slots of a
// pair's column set in place.
template <class Op, int HM>
constexpr bool kPairInPlace = !Op::kLoadLFast && !Op::kFusedK && ((HM & 4) != 0 || (HM & 3) == 2);

// Step 1 for radix P: the thread's samples, P-point DFT, outer twiddles, into the transpose.
template <int P, class Op, int HM, bool INV>
__device__ __forceinline__ void pair_step1(const Op& op, const PairCfg& c, int L, int Q, const PairCols& k, int t, int cp,
                                           const float2* tw, const float4* In, const float2* Rs, int64_t a0, c2* Y) {
    constexpr bool half = (HM & 1) != 0;
    constexpr bool prune = half && P % 2 == 0;
    constexpr bool PH = PairShapes<Op>::value != 0 && (HM & 3) != 0;  // operators with centred sides
    c2 v[P];
    const c2 zero{0ull, 0ull};
    if constexpr (Op::kLoadLFast) {
        auto f0 = op.cstate(k.a0, k.e0, k.ok0), f1 = op.cstate(k.a1, k.e1, k.ok1);
        if (c.rows) {  // the rows' factors were copied with the samples
            op.cstate_row(f0, Rs + (k.ok0 ? (k.a0 - a0) * c.Lin : 0));
            op.cstate_row(f1, Rs + (k.ok1 ? (k.a1 - a0) * c.Lin : 0));
        }
        pair_inputs<P, HM>(c, Q, t, [&](int j, int l) {
            const float2* x = reinterpret_cast<const float2*>(In) + 2 * cp * c.in_stride + l;
            v[j] = c2_pack(k.ok0 ? op.cvalue(f0, l, x[0]) : make_float2(0.f, 0.f),
                           k.ok1 ? op.cvalue(f1, l, x[c.in_stride]) : make_float2(0.f, 0.f));
        }, [&](int j) { v[j] = zero; });
    } else {
        pair_inputs<P, HM>(c, Q, t, [&](int j, int l) {
            const float4 x = In[l * kPairs + cp];
            v[j] = {f2_pack(x.x, x.z), f2_pack(x.y, x.w)};
        }, [&](int j) { v[j] = zero; });
    }
    if constexpr (prune)
        c2_dft_halfzero<P, INV>(v);
    else
        c2_dft<P, INV>(v);
    // rotated slots: a lane overwrites samples of the other lanes of its t (eight lanes of one warp, all of them here),
    // which must have read them first. Without rotation every lane writes the slots that it has read itself.
    if constexpr (kPairInPlace<Op, HM> && Op::kStoreLFast) __syncwarp(0xffu << (threadIdx.x & 24));
#pragma unroll
    for (int k1 = 0; k1 < P; ++k1) {
        if (k1 > 0 || (PH && (c.ph & 2))) v[k1] = PH ? pair_tw<INV>(c, L, t, k1, tw, v[k1]) : c2_mul_tw<INV>(v[k1], tw[t * k1]);
        Y[pair_slot<Op>(k1 * Q + t, k1, cp)] = v[k1];
    }
}

template <int Q, class Op, bool INV>
__device__ __forceinline__ void pair_read2(int k1, int cp, const c2* Y, c2* u) {
#pragma unroll
    for (int t = 0; t < Q; ++t) u[t] = Y[pair_slot<Op>(k1 * Q + t, k1, cp)];
    c2_dft<Q, INV>(u);
}

// Calls f(k2, o) for the outputs o of positions k1 + P k2 that the pass keeps.
template <int Q, int HM, class F>
__device__ __forceinline__ void pair_outputs(const PairCfg& c, int P, int k1, F&& f) {
    constexpr bool half = (HM & 2) != 0, full = (HM & 8) != 0 || (HM & 3) == 1;
#pragma unroll
    for (int k2 = 0; k2 < (half ? (Q + 1) / 2 : Q); ++k2) {
        const int pos = k1 + P * k2;
        if constexpr (full) {
            f(k2, pos);
        } else if constexpr (half) {
            if (Q % 2 == 0 || 2 * pos < c.L) f(k2, pos);
        } else {
            int o = pos - c.out_shift;
            if (o < 0) o += c.L;
            if (o < c.Lout) f(k2, o);
        }
    }
}

// Where an operator's outputs of one column go: operators without vout give a column state (OState ostate(a, e),
// computed once per column) and ostore(state, o, value).
template <class Op>
struct PairOut {
    const Op& op;
    const PairCfg& c;
    const PairCols& k;
    typename Op::OState s0, s1;
    __device__ __forceinline__ PairOut(const Op& op_, const PairCfg& c_, const PairCols& k_)
        : op(op_), c(c_), k(k_), s0(op_.ostate(k_.a0, k_.e0, k_.ok0)), s1(op_.ostate(k_.a1, k_.e1, k_.ok1)) {}
    __device__ __forceinline__ void operator()(int o, c2 v) const {
        if constexpr (HasVecOut<Op>::value) {
            if (c.vec_out) {
                if (k.ok0) c2_st16(s0 + o * op.vout_l(), op.vout_value(v));
                return;
            }
        }
        float2 x0, x1;
        c2_unpack(v, x0, x1);
        if (k.ok0) op.ostore(s0, o, x0);
        if (k.ok1) op.ostore(s1, o, x1);
    }
};

// Fused kernel pass: multiply the spectrum u (positions k1 + P k2) by the kernel, inverse Q-point DFT,
// inverse outer twiddles, back into the slots it came from.
template <int Q, class Op>
__device__ __forceinline__ void pair_kernel_mul(const Op& op, const PairCfg& c, int P, const PairCols& k, int k1, int cp,
                                                const float2* tw, c2* Y, const float2* Ks, int64_t kc0, c2* u) {
    const int64_t q0 = k.ok0 ? op.kcol(k.e0) : c.n_k ? kc0 : 0, q1 = k.ok1 ? op.kcol(k.e1) : q0;
    const float2* w0 = c.n_k ? Ks + (q0 - kc0) * c.L : op.kptr(q0);
    const float2* w1 = c.n_k ? Ks + (q1 - kc0) * c.L : op.kptr(q1);
    if (q0 == q1) {
#pragma unroll
        for (int k2 = 0; k2 < Q; ++k2) u[k2] = c2_mul_tw<false>(u[k2], w0[k1 + P * k2]);
    } else {
#pragma unroll
        for (int k2 = 0; k2 < Q; ++k2) {
            const c2 w = c2_pack(w0[k1 + P * k2], w1[k1 + P * k2]);
            u[k2] = c2_mul(u[k2], w.re, w.im);
        }
    }
    c2_dft<Q, true>(u);
#pragma unroll
    for (int n2 = 0; n2 < Q; ++n2) {
        if (n2 > 0) u[n2] = c2_mul_tw<true>(u[n2], tw[n2 * k1]);
        Y[(k1 * Q + n2) * kPairs + cp] = u[n2];
    }
}

// f(std::integral_constant<int, r>) for the radix r in [RMIN, RMAX]; RT != 0: r is RT
template <int RMIN, int RMAX, int RT, class F>
__device__ __forceinline__ void radix_switch(int r, F&& f) {
    if constexpr (RT != 0) {
        f(std::integral_constant<int, RT>{});
    } else {
#define HB_RADIX(n)                                                                        \
    case n:                                                                                \
        if constexpr (n >= RMIN && n <= RMAX) f(std::integral_constant<int, n>{});         \
        break;
        switch (r) {
            HB_RADIX(8) HB_RADIX(9) HB_RADIX(10) HB_RADIX(11) HB_RADIX(12)
            HB_RADIX(13) HB_RADIX(14) HB_RADIX(15) HB_RADIX(16) HB_RADIX(18) HB_RADIX(20) HB_RADIX(21) HB_RADIX(22)
            HB_RADIX(24) HB_RADIX(25) HB_RADIX(26)
        }
#undef HB_RADIX
    }
}

// Persistent CTAs walk the jobs (row block, column block) with a stride of the grid; a reducing operator
// takes all column blocks of a row block in turn. While a job is transformed the next one's samples are copied:
// into their own buffer In, free once step 1 has read it (INPL false), or -- full-length samples --
// into the transpose itself, free once step 2 has read it (INPL true: the eight lanes of a t read and write the
// same slots in step 1; half the shared memory, so more CTAs per SM).
template <class Op, int HM, bool INV, int RMIN, int RMAX, int PT, int QT, int MB, bool INPL>
__global__ void __launch_bounds__((RMAX * kPairs + 31) / 32 * 32, MB) pair_kernel(const Op op, const PairCfg c) {
    const int P = PT ? PT : c.P, Q = QT ? QT : c.Q, L = PT ? PT * QT : c.L;
    // in-place samples: the next job's copies go out between step 2's reads and stores, except where that spills
    constexpr bool kEarly = PT != 0 && (HM & 4) == 0;
    extern __shared__ float4 pair_smem[];
    c2* const Y = reinterpret_cast<c2*>(pair_smem);               // [L][kPairs]
    float4* const In = INPL ? pair_smem : pair_smem + L * kPairs;
    float2* const tw = reinterpret_cast<float2*>(pair_smem + L * kPairs) + (INPL ? 0 : c.in_elems);  // [tw_n]
    float2* const Rs = tw + c.tw_n;                               // rows: [A_blk][Lin] row factors
    float2* const Ks = tw + c.tw_n;                                  // kFusedK: [n_k][L]
    float2* const acc = tw + c.tw_n;                                 // kSenseReduce: [Lout][kPairs] running sums
    float2* const Ss = acc + c.Lout * kPairs;                     // kSenseReduce: [kCW][s_stride] factor rows
    const int tid = threadIdx.x;
    const int cp = tid % kPairs, t = tid / kPairs;                // step 1 (and 3): t < Q
    const int cp2 = Op::kStoreLFast ? tid / P : cp;               // step 2: k1 < P
    const int k1 = Op::kStoreLFast ? tid - cp2 * P : t;
    const bool in1 = t < Q, in2 = Op::kStoreLFast ? cp2 < kPairs : k1 < P;
    for (int i = tid; i < c.tw_n; i += blockDim.x) cp_async8(tw + i, c.tw + (i < L ? i : i - L));

    int64_t jq = blockIdx.x, ab = 0;
    unsigned eb = 0;
    auto split_job = [&]() -> bool {
        if (Op::kSenseReduce || c.n_eb == 1) {
            ab = jq;
            eb = 0;
        } else {  // fewer than 2^31 jobs (launcher)
            ab = (uint32_t)jq / c.n_eb;
            eb = (uint32_t)jq - (uint32_t)ab * c.n_eb;
        }
        return jq < c.n_jobs;
    };
    auto a0_of = [&](int64_t b) { return b * c.A_blk; };
    auto e_of = [&](unsigned b) { return (int64_t)b * (Op::kSenseReduce ? 2 * c.E_blk : c.E_blk); };
    // the kernel columns / factor rows of a job: with its samples for the first job, later ones under step 1
    int64_t kc0 = 0;
    auto fetch_side = [&](int64_t a0, int64_t e0) {
        if constexpr (Op::kFusedK) {
            if (c.n_k) {
                kc0 = op.kcol(e0);
                const int nk = (int)(op.kcol(min(e0 + c.E_blk, c.E) - 1) - kc0) + 1;
                const float2* src = op.kptr(kc0);  // the columns follow one another
                for (int i = tid; i < nk * L; i += blockDim.x) cp_async8(Ks + i, src + i);
            }
        }
        if constexpr (Op::kSenseReduce) {
            for (int col = tid >> 5; col < c.W; col += blockDim.x >> 5) {
                const int al = c.A_blk == 1 ? 0 : col / (2 * c.E_blk), el = col - al * 2 * c.E_blk;
                if (a0 + al >= c.A || e0 + el >= c.E) continue;
                const float2* src = op.srow(a0 + al, e0 + el);
                for (int o = tid & 31; o < c.Lout; o += 32) cp_async8(Ss + col * c.s_stride + o, src + o);
            }
        }
    };
    bool have = split_job(), first = true;
    if (have) {
        pair_fetch<HM>(op, c, a0_of(ab), e_of(eb), In, Rs);
        fetch_side(a0_of(ab), e_of(eb));
    }
    cp_async_commit();
    if constexpr (Op::kSenseReduce) {
        if (in2)
            for (int o = k1; o < c.Lout; o += P) acc[o * kPairs + cp] = make_float2(0.f, 0.f);
    }
    cp_async_wait_all();
    __syncthreads();
    while (have) {
        const int64_t a0 = a0_of(ab), e0 = e_of(eb);
        bool last_of_row = true;
        if (Op::kSenseReduce && eb + 1 < c.n_eb) {
            ++eb;
            last_of_row = false;
        } else {
            jq += gridDim.x;
            have = split_job();
        }
        if (!first) fetch_side(a0, e0);
        first = false;
        if (in1) {
            const PairCols k = pair_cols<Op>(c, a0, e0, cp);
            radix_switch<RMIN, RMAX, PT>(P, [&](auto rc) {
                pair_step1<decltype(rc)::value, Op, HM, INV>(op, c, L, Q, k, t, cp, tw, In, Rs, a0, Y);
            });
        }
        if (Op::kFusedK || Op::kSenseReduce) cp_async_wait_all();
        __syncthreads();
        if (!INPL && have) pair_fetch<HM>(op, c, a0_of(ab), e_of(eb), In, Rs);
        const PairCols k = pair_cols<Op>(c, a0, e0, cp2);
        radix_switch<RMIN, RMAX, QT>(Q, [&](auto rc) {
            constexpr int R = decltype(rc)::value;
            c2 u[R];
            if (in2) pair_read2<R, Op, INV>(k1, cp2, Y, u);
            if constexpr (INPL && kEarly) {
                __syncthreads();
                if (have) pair_fetch<HM>(op, c, a0_of(ab), e_of(eb), In, Rs);
            }
            if (in2) {
                if constexpr (Op::kFusedK) {
                    pair_kernel_mul<R>(op, c, P, k, k1, cp, tw, Y, Ks, kc0, u);
                } else if constexpr (Op::kSenseReduce) {
                    const float2* s0 = Ss + 2 * cp * c.s_stride;
                    pair_outputs<R, HM>(c, P, k1, [&](int k2, int o) {
                        float2 x0, x1;
                        c2_unpack(u[k2], x0, x1);
                        float2 r = acc[o * kPairs + cp];
                        if (k.ok0) r = cadd(r, op.product_s(x0, s0[o]));
                        if (k.ok1) r = cadd(r, op.product_s(x1, s0[c.s_stride + o]));
                        acc[o * kPairs + cp] = r;
                    });
                } else {
                    const PairOut<Op> put(op, c, k);
                    pair_outputs<R, HM>(c, P, k1, [&](int k2, int o) { put(o, u[k2]); });
                }
            }
        });
        if constexpr (Op::kSenseReduce) {
            if (last_of_row) {
                __syncthreads();
                // one thread per output of a row: the row's pairs in order, then cleared for the next row
                const int pe = c.E_blk;
                for (int idx = tid; idx < c.A_blk * c.Lout; idx += blockDim.x) {
                    const int al = idx / c.Lout, o = idx - al * c.Lout;
                    float2* r = acc + o * kPairs + al * pe;
                    float2 sum = r[0];
                    r[0] = make_float2(0.f, 0.f);
                    for (int i = 1; i < pe; ++i) {
                        sum = cadd(sum, r[i]);
                        r[i] = make_float2(0.f, 0.f);
                    }
                    if (a0 + al < c.A) op.write_row(a0 + al, o, 0, sum);
                }
            }
        }
        if constexpr (Op::kFusedK) {
            __syncthreads();
            if (in1) {
                const PairCols k3 = pair_cols<Op>(c, a0, e0, cp);
                radix_switch<RMIN, RMAX, PT>(P, [&](auto rc) {
                    constexpr int R = decltype(rc)::value;
                    static_assert(!Op::kFusedK || (HM & 3) == 3, "fused passes pad and crop to half");
                    c2 z[R];
#pragma unroll
                    for (int q = 0; q < R; ++q) z[q] = Y[(q * Q + t) * kPairs + cp];
                    c2_dft<R, true>(z);
                    const PairOut<Op> put(op, c, k3);
#pragma unroll
                    for (int n1 = 0; n1 < (R + 1) / 2; ++n1) {
                        const int pos = t + Q * n1;
                        if (R % 2 == 0 || 2 * pos < L) put(pos, z[n1]);
                    }
                });
            }
        }
        if constexpr (INPL && !kEarly) {
            __syncthreads();
            if (have) pair_fetch<HM>(op, c, a0_of(ab), e_of(eb), In, Rs);
        }
        // the next job's samples are in and nobody reads Y any more
        cp_async_wait_all();
        __syncthreads();
    }
}

template <class Op, int HM, bool INV, int RMIN, int RMAX, int PT, int QT, int MB>
int launch_pair_inst(const Op& op, PairCfg c, cudaStream_t s, const char* name) {
    constexpr bool INPL = kPairInPlace<Op, HM>;
    auto kern = pair_kernel<Op, HM, INV, RMIN, RMAX, PT, QT, MB, INPL>;
    c.W = kCW;
    c.in_stride = c.Lin | 1;
    c.s_stride = c.Lout | 1;
    c.in_elems = Op::kLoadLFast ? (kCW * c.in_stride + 1) / 2 * 2 : c.Lin * kCW;
    c.tw_n = c.ph ? 2 * c.L : c.L;
    size_t smem = (size_t)c.L * kPairs * sizeof(c2) + (size_t)c.tw_n * sizeof(float2);
    if (!INPL) smem += (size_t)c.in_elems * sizeof(float2);
    if constexpr (Op::kLoadLFast) {
        c.rows = op.rows_shared(c.E_blk);
        if (c.rows) smem += (size_t)c.A_blk * c.Lin * sizeof(float2);
    }
    if (Op::kFusedK) smem += (size_t)c.n_k * c.L * sizeof(float2);
    if (Op::kSenseReduce) smem += (size_t)(c.Lout * kPairs + kCW * c.s_stride) * sizeof(float2);
    const int threads = (std::max(c.P, c.Q) * kPairs + 31) / 32 * 32;
    HB_TRY(allow_smem(kern, smem, name));
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
    int per_sm = 0;
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, threads, smem);
    if (e != cudaSuccess) {
        set_error(std::string(name) + ": pass set-up failed: " + cudaGetErrorString(e));
        return HB_ERR_CUDA;
    }
    const int64_t grid = std::min<int64_t>(c.n_jobs, (int64_t)std::max(per_sm, 1) * kNumSMs);
    TimedSection ts(name, s);
    kern<<<(unsigned)grid, threads, smem, s>>>(op, c);
    return check_launch(name);
}

// CTAs per SM that the registers are held to: four of 128 threads, three of 160, two of 224.
template <class Op, int HM, bool INV>
int launch_pair_dir(const Op& op, const PairCfg& c, cudaStream_t s, const char* name) {
    const int r = std::max(c.P, c.Q);
    // the edges of the common matrix sizes have their radices as constants (the run-time switch costs 5 - 15 %)
    if (c.P == 8 && c.Q == 8) return launch_pair_inst<Op, HM, INV, 8, 8, 8, 8, 8>(op, c, s, name);
    if (c.P == 8 && c.Q == 16) return launch_pair_inst<Op, HM, INV, 8, 16, 8, 16, 4>(op, c, s, name);
    if (c.P == 16 && c.Q == 16) return launch_pair_inst<Op, HM, INV, 16, 16, 16, 16, 4>(op, c, s, name);
    if (c.P == 16 && c.Q == 20) return launch_pair_inst<Op, HM, INV, 16, 20, 16, 20, 3>(op, c, s, name);
    if (r <= 16) return launch_pair_inst<Op, HM, INV, pair_rmin(16), 16, 0, 0, 4>(op, c, s, name);
    if (r <= 20) return launch_pair_inst<Op, HM, INV, pair_rmin(20), 20, 0, 0, 3>(op, c, s, name);
    return launch_pair_inst<Op, HM, INV, pair_rmin(kRadixMax), kRadixMax, 0, 0, 2>(op, c, s, name);
}

inline bool aligned16(const void* p) { return ((uintptr_t)p & 15) == 0; }

// Runs the pass on column pairs. *done is false where the length or the pass's shape has no instance.
template <class Op>
int launch_pair_pass(const Op& op, const FftLen& f, int64_t A, int64_t E, int Lin, int in_shift, int Lout,
                     int out_shift, int inverse, cudaStream_t s, const char* name, bool* done) {
    constexpr int HMop = HalfIO<Op>::value;
    PairCfg c{};
    const int L = f.L;
    const bool crops = Lout < Lin;
    pair_split(L, !crops, &c.P, &c.Q);
    *done = c.P > 0;
    if (!*done) return HB_OK;
    c.L = L;
    c.Lin = Lin;
    c.in_shift = ((in_shift % L) + L) % L;
    c.Lout = Lout;
    c.out_shift = ((out_shift % L) + L) % L;
    c.A = A;
    c.E = E;
    c.tw = f.tw;
    const bool full_in = Lin == L && c.in_shift == 0, full_out = Lout == L && c.out_shift == 0;
    if (HMop != 0) {
        const bool ok_in = (HMop & 1) ? (2 * Lin == L && c.in_shift == 0) : full_in;
        const bool ok_out = (HMop & 2) ? (2 * Lout == L && c.out_shift == 0) : full_out;
        if (!ok_in || !ok_out || (inverse != 0) != ((HMop & 3) == 2)) {
            set_error(std::string(name) + ": pass shape does not match the operator's padding / crop");
            return HB_ERR_INVALID_ARG;
        }
    }
    if (Op::kSenseReduce) {
        c.E_blk = (int)std::min<int64_t>((E + 1) / 2, kPairs);  // pairs of a row
        c.A_blk = c.E_blk == kPairs ? 1 : (int)std::min<int64_t>(A, kPairs / c.E_blk);
        c.n_eb = (unsigned)ceil_div(E, 2 * c.E_blk);
    } else {
        c.E_blk = (int)std::min<int64_t>(E, kCW);
        c.A_blk = c.E_blk == kCW ? 1 : (int)std::min<int64_t>(A, kCW / c.E_blk);
        c.n_eb = (unsigned)ceil_div(E, c.E_blk);
    }
    // a pair is one 16-byte access where both columns always exist side by side: an even inner
    // extent, even strides and an aligned base
    if constexpr (!Op::kLoadLFast) c.vec_in = E % 2 == 0 && op.vin_even() && aligned16(op.vin_base());
    if constexpr (HasVecOut<Op>::value) c.vec_out = E % 2 == 0 && op.vout_even() && aligned16(op.vout_base());
    if constexpr (Op::kFusedK) {
        // distinct kernel columns under kCW columns: staged while at most kMaxKCols
        const int64_t per = op.cols_per_kernel();
        const int64_t nk = per >= kCW ? (per % kCW == 0 ? 1 : 2) : ceil_div(kCW, per) + 1;
        c.n_k = nk <= kMaxKCols ? (int)nk : 0;
    }
    const int64_t n_ab = ceil_div(A, c.A_blk);
    c.n_jobs = Op::kChunkLoop ? n_ab : n_ab * c.n_eb;
    if (c.n_jobs <= 0) return HB_OK;
    if (c.n_jobs > 0x7fffffffLL || ceil_div(E, c.E_blk) > 0x7fffffffLL) {
        set_error(std::string(name) + ": grid too large");
        return HB_ERR_INVALID_ARG;
    }
    if constexpr (HMop != 0) {
        return launch_pair_dir<Op, HMop, (HMop & 3) == 2>(op, c, s, name);
    } else {
        const int centred = L - L / 4;  // the shift -L/4
        if constexpr ((PairShapes<Op>::value & 1) != 0) {
            if (full_in && 2 * Lout == L && c.out_shift == centred && L % 4 == 0 && c.Q % 4 == 0) {
                c.out_shift = 0;
                c.ph = 2;
                return inverse ? launch_pair_dir<Op, 2, true>(op, c, s, name) : launch_pair_dir<Op, 2, false>(op, c, s, name);
            }
            if (full_in && !full_out)
                return inverse ? launch_pair_dir<Op, 4, true>(op, c, s, name) : launch_pair_dir<Op, 4, false>(op, c, s, name);
        }
        if constexpr ((PairShapes<Op>::value & 2) != 0) {
            if (full_out && 2 * Lin == L && c.in_shift == centred && L % 4 == 0 && c.P % 4 == 0) {
                c.in_shift = 0;
                c.ph = 1;
                return inverse ? launch_pair_dir<Op, 1, true>(op, c, s, name) : launch_pair_dir<Op, 1, false>(op, c, s, name);
            }
            if (full_out && !full_in)
                return inverse ? launch_pair_dir<Op, 8, true>(op, c, s, name) : launch_pair_dir<Op, 8, false>(op, c, s, name);
        }
        *done = false;
        return HB_OK;
    }
}

// Runs the pass kernel for the length: column pairs where L splits into two radices of 8 to 26 points and a side is
// padded or cropped, else launch_wide_pass.
// `extra_per_row` is the kSenseReduce accumulator size per outer row (bytes).
template <class Op>
int launch_fft_pass(const Op& op, const FftLen& f, int64_t A, int64_t E, int Lin, int in_shift, int Lout, int out_shift,
                    int inverse, size_t extra_per_row, cudaStream_t s, const char* name) {
    bool done = false;
    const int st = launch_pair_pass(op, f, A, E, Lin, in_shift, Lout, out_shift, inverse, s, name, &done);
    if (st != HB_OK || done) return st;
    return launch_wide_pass(op, f, A, E, Lin, in_shift, Lout, out_shift, inverse, extra_per_row, s, name);
}

// The passes of each operator are compiled in one file of their own (pass_*.cu).
#define HB_PASS_ARGS(Op) \
    const Op&, const FftLen&, int64_t, int64_t, int, int, int, int, int, size_t, cudaStream_t, const char*
#define HB_EXTERN_PASS(Op) extern template int launch_fft_pass<Op>(HB_PASS_ARGS(Op));
#define HB_INSTANTIATE_PASS(Op) template int launch_fft_pass<Op>(HB_PASS_ARGS(Op));

#endif  // __CUDACC__

}  // namespace hb

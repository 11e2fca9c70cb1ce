// Type-1 spreading in 3-D, widths 4 .. 7, with the transforms on the lanes, walking along z.
//
// One CTA owns a column of the fine grid, 8 (y) x 8 (x) cells by a segment of `seg` planes, for CC
// transforms. The 32 lanes of a warp are 32 / CC groups of CC transforms; every group owns 2 x 2 cells of the
// column, and a thread keeps them for its transform over the W planes that a footprint covers: 4 W
// complex accumulators. Candidates come in order of their first z cell (the points of a bin are
// sorted by it), so the W planes of a visit are the thread's W planes -- no z range to test, no weight of
// zero along z -- and when the walk moves on by one cell the lowest plane is finished and stored. Plane r
// stays in register slot r mod W: the z weights are staged rotated to their slots, so nothing moves
// between registers (shifting them cost 50 moves a visit). A point's footprint meets ((W + 1) / 2)^2 of the 2 x 2 blocks of
// its column and its neighbours (12 at W = 6, 73 % of whose cells it covers); the tile kernel this
// replaces visits 20 blocks of 2 x 2 x 8 cells.
//
// A visit is packed f32x2 arithmetic on (re, im): w_x v, w_y w_x v, then W multiply-adds per cell with
// weights that are staged twice over, so no register moves are needed: 24 + 6 packed operations of two cycles each
// at W = 6, of about 185 cycles that a visit takes per sub-core. No unit is full (96^3 x 32, 786 k radial points: issue
// slots 50 %, FMA pipe 42 %, shared-memory data path 39 %): 20 warps an SM do not cover the latency of the
// loads and of the multiply-adds. 160^3 x 32, 6.1 M points, w = 6: 12.6 ms, the tile kernel 20.1.
//
// Candidates are staged in chunks through a ring of three buffers by warps of their own, one thread per
// candidate: it finds the candidate, tests whether its footprint reaches the column, and writes its
// weights (tile-relative rows of 8 along y and x) and its CC values (cp.async). Spreading and staging warps
// meet only through each buffer's two mbarriers (staged / read by all warps): how many of a chunk's
// candidates touch a warp's block varies, and one barrier per chunk had the warps wait for the slowest a
// third of the time. A spreading warp first lists its candidates of a chunk, then visits the list.
//
// Segments with more than maxp candidates are spread in parts, one CTA each, into partial planes in
// scratch; k_walk_reduce adds a segment's parts in part order. No atomics, and the order of every sum is fixed for
// sorted points.
#pragma once

#include <algorithm>

#include "fftp.cuh"
#include "nufft.cuh"
#include "timing.cuh"

namespace hb {

// Geometry of the segments (walk_segments): sp planes each (the last of an axis may be shorter), ns per
// column, first cells r = 0 .. planes + W - 2 of a segment counted from z0 - (W - 1).
struct WalkArgs {
    int sp, ns;
    int64_t nseg;             // segments over all frames
    const int* fine;          // first sorted point of (bin, z cell): [bins * 8 + 1]
    const int4* parts;        // {segment, part, parts of the segment, first scratch plane of the segment}
    int n_parts;
    int2* range;              // first and last first-cell of each part
    float2* scratch;          // [plane][64 cells][C]
    int* err;                 // set when a wait ran out (never with a correct kernel)
    int tries;                // of a wait, up to 2 us each
};

constexpr int kWalkMaxCells = 32 + 6;  // first cells of a segment
// Visits after which a warp puts its sums away into their planes (and adds to them there): a sum of n equal terms
// rounds the same way at every step and drifts by up to n / 4 eps, and the points of a z cell at the centre of a
// trajectory are much alike. Error against FP64 gridding of a smooth image's samples, without putting away, with runs of
// 128 and of 64 visits (times of a type 1): 160^3 x 32, 6.1 M cones, w = 6: 3.5e-6, 3.9e-7, 1.6e-7 (17.2, 17.3,
// 17.5 ms; the tile kernel 7.3e-7); 64^3 x 8, 131 k radial, w = 4: 1.0e-6, 2.0e-7, 1.4e-7 (256, 263, 263 us; the
// tile kernel 1.4e-7); one transform 128^3, 2.1 M radial, w = 4: 2.2e-6, 4.6e-7, 1.9e-7 (0.92 ms each; the
// cell kernel 1.1e-6).
constexpr int kWalkRun = 64;

// CC >= 8: the lanes hold transforms (groups of CC, 2 x 2 cells each). CC = 1, 2, 4: the lanes hold cells (a warp
// 4 x 8 of the column's 8 x 8) and every thread all CC transforms of its cell.
template <int CC, int W>
struct WalkShape {
    static constexpr bool CELLS = CC <= 4;
    static constexpr int K = CELLS ? CC : 4;                        // accumulators per plane: transforms or cells
    static constexpr int G = 32 / CC;
    static constexpr int GY = G >= 2 ? 2 : 1, GX = G >= 4 ? 2 : 1;  // groups of a warp along y and x
    static constexpr int BY = CELLS ? 4 : 2 * GY, BX = CELLS ? 8 : 2 * GX;  // cells of a warp
    static constexpr int WARPS = (8 / BY) * (8 / BX);
    static constexpr int CH = CC == 32 ? 128 : CELLS ? 32 : 64;     // candidates per chunk
    static constexpr int NST = CH / 32;                             // staging warps
    static constexpr int NW = WARPS + NST, THREADS = NW * 32;
    static constexpr int RING = 3;                                  // buffers
    static constexpr int WZ = (W + 1) / 2 * 2;
    // floats per candidate: values [CC] | weights, each twice: z[WZ] | y[8] | x[8]
    static constexpr int OZ = CC == 1 ? 4 : 2 * CC, OY = OZ + 2 * WZ, OX = OY + 16, REC = OX + 16;
    static constexpr int kBufF = CH * REC + CH;                     // records | packed first cells
    static constexpr int kListN = CH + 2;
    static constexpr size_t smem_bytes() {
        return sizeof(float) * (size_t)(kCoefFloats + RING * kBufF + WARPS * kListN);
    }
    static_assert(CH * REC * 4 < (1 << 24), "record offsets take 24 bits");
    // CTAs per SM that the registers are held to
    static constexpr int MB = CC == 32 ? 1 : CC == 16 ? 2 : CC == 8 ? 3 : CC == 4 ? 5 : 8;
};

// tile index of (segment, plane r from the segment's first cell) and the bins of its column
__device__ __forceinline__ void walk_segment(const GridGeom& g, const WalkArgs& w, int64_t seg, int& fr, int& ts, int& ty, int& tx) {
    const int per = w.ns * g.nb[1] * g.nb[2];
    fr = g.nfr > 1 ? (int)(seg / per) : 0;
    const int s = (int)(seg - (int64_t)fr * per);
    tx = s % g.nb[2];
    ty = (s / g.nb[2]) % g.nb[1];
    ts = s / (g.nb[2] * g.nb[1]);
}
__device__ __forceinline__ int walk_planes(const GridGeom& g, const WalkArgs& w, int ts) { return min(w.sp, g.nf[0] - ts * w.sp); }
// index into `fine` of first cell r (from z0 - (W - 1)) of neighbour b (bit 0: the bin before along x, bit 1: along y)
__device__ __forceinline__ int64_t walk_bin(const GridGeom& g, int fr, int z, int ty, int tx, int b) {
    if (z < 0) z += g.nf[0];
    const int by = (b & 2) ? (ty > 0 ? ty - 1 : g.nb[1] - 1) : ty;
    const int bx = (b & 1) ? (tx > 0 ? tx - 1 : g.nb[2] - 1) : tx;
    return ((int64_t)fr * g.ntf + ((int64_t)(z >> 3) * g.nb[1] + by) * g.nb[2] + bx) * 8 + (z & 7);
}

// mbarrier helpers (shared-memory addresses)
__device__ __forceinline__ void mbar_init(uint64_t* b, unsigned count) {
    asm volatile("mbarrier.init.shared.b64 [%0], %1;" ::"r"((unsigned)__cvta_generic_to_shared(b)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* b) {
    asm volatile("mbarrier.arrive.shared.b64 _, [%0];" ::"r"((unsigned)__cvta_generic_to_shared(b)) : "memory");
}
// an arrival when the thread's cp.async copies so far have landed
__device__ __forceinline__ void mbar_arrive_copies(uint64_t* b) {
    asm volatile("cp.async.mbarrier.arrive.noinc.shared.b64 [%0];" ::"r"((unsigned)__cvta_generic_to_shared(b)) : "memory");
}
// Waits for the phase of the given parity; false when it did not come within `tries`. Lanes of a warp may differ, so
// they vote on it before any of them leaves.
__device__ __forceinline__ bool mbar_wait(uint64_t* b, unsigned parity, int tries) {
    const unsigned addr = (unsigned)__cvta_generic_to_shared(b);
    for (int i = 0; i < tries; ++i) {
        unsigned ok;
        asm volatile(
            "{\n.reg .pred p;\nmbarrier.try_wait.parity.shared.b64 p, [%1], %2, %3;\nselp.u32 %0, 1, 0, p;\n}"
            : "=r"(ok)
            : "r"(addr), "r"(parity), "r"(2000u)  // suspended up to 2 us a try
            : "memory");
        if (ok) return true;
    }
    return false;
}

// shared-memory loads by 32-bit address (volatile: they stay behind the waits above)
__device__ __forceinline__ unsigned lds32(unsigned a) {
    unsigned v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a));
    return v;
}
__device__ __forceinline__ f2_t lds64(unsigned a) {
    f2_t v;
    asm volatile("ld.shared.u64 %0, [%1];" : "=l"(v) : "r"(a));
    return v;
}
__device__ __forceinline__ ulonglong2 lds128(unsigned a) {
    ulonglong2 v;
    asm volatile("ld.shared.v2.u64 {%0, %1}, [%2];" : "=l"(v.x), "=l"(v.y) : "r"(a));
    return v;
}

// w taps of a point: kb_tap with the coefficients read four at a time. Coefficients above the degree are
// zero, so the longer chain gives the same value.
template <int W>
__device__ __forceinline__ void walk_taps(const float* coef, int deg, float s, float (&t)[W]) {
    if (deg < 12) {
#pragma unroll
        for (int d = 0; d < W; ++d) {
            const float4* c = reinterpret_cast<const float4*>(coef + d * (kMaxDeg + 1));
            const float4 c0 = c[0], c1 = c[1], c2 = c[2];
            float v = c2.w;
            v = fmaf(v, s, c2.z);
            v = fmaf(v, s, c2.y);
            v = fmaf(v, s, c2.x);
            v = fmaf(v, s, c1.w);
            v = fmaf(v, s, c1.z);
            v = fmaf(v, s, c1.y);
            v = fmaf(v, s, c1.x);
            v = fmaf(v, s, c0.w);
            v = fmaf(v, s, c0.z);
            v = fmaf(v, s, c0.y);
            t[d] = fmaf(v, s, c0.x);
        }
    } else {
#pragma unroll
        for (int d = 0; d < W; ++d) t[d] = kb_tap(coef, deg, d, s);
    }
}

template <int CC, int W>
__global__ void __launch_bounds__(WalkShape<CC, W>::THREADS, WalkShape<CC, W>::MB) k_spread_walk(const GridArgs a, const WalkArgs w) {
    using S = WalkShape<CC, W>;
    extern __shared__ float4 walk_f4[];
    float* const coef = reinterpret_cast<float*>(walk_f4);
    float* const ring = coef + kCoefFloats;
    __shared__ uint64_t m_full[S::RING], m_free[S::RING];
    __shared__ int s_st[kWalkMaxCells * 4];        // first sorted point of (cell, neighbour)
    __shared__ int s_pre[kWalkMaxCells * 4 + 1];   // candidates before (cell, neighbour)
    const GridGeom& g = a.g;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int grp = lane / CC, coil = S::CELLS ? 0 : lane % CC;
    const bool is_part = (int)blockIdx.x < w.n_parts;
    const int4 job = is_part ? w.parts[blockIdx.x] : make_int4((int)blockIdx.x - w.n_parts, 0, 1, 0);
    int fr, ts, ty, tx;
    walk_segment(g, w, job.x, fr, ts, ty, tx);
    const int z0 = ts * w.sp, planes = walk_planes(g, w, ts), ncell = planes + W - 1;
    const int org1 = ty * 8, org2 = tx * 8;
    const int nf1 = g.nf[1], nf2 = g.nf[2];
    float2* const gridf = a.grid + fr * g.fgrid;
    const float hw = a.kb.hw;
    const bool vec = (g.C % 2) == 0;
    const int cc0 = (int)blockIdx.y * CC;

    for (int i = tid; i < kCoefFloats; i += S::THREADS) coef[i] = (&a.kb.coef[0][0])[i];
    if (tid < S::RING) {
        mbar_init(m_full + tid, S::CH * 2);
        mbar_init(m_free + tid, S::WARPS);
    }
    // candidates of every (first cell, neighbour bin), one thread each, and their running sum
    static_assert(kWalkMaxCells * 4 <= 5 * 32, "five groups of 32 entries");
    __shared__ int s_sum[5];
    for (int v = warp; v < 5; v += S::NW) {
        const int e = v * 32 + lane;
        int st = 0, cnt = 0;
        if (e < ncell * 4) {
            const int64_t fb = walk_bin(g, fr, z0 - (W - 1) + (e >> 2), ty, tx, e & 3);
            st = w.fine[fb];
            cnt = w.fine[fb + 1] - st;
        }
        int incl = cnt;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += y;
        }
        if (e < ncell * 4) {
            s_st[e] = st;
            s_pre[e] = incl - cnt;
        }
        if (lane == 31) s_sum[v] = incl;
    }
    __syncthreads();
    for (int e = tid; e <= ncell * 4; e += S::THREADS) {  // the last entry is the total
        int before = 0;
        for (int v = 0; v < (min(e, ncell * 4 - 1) >> 5); ++v) before += s_sum[v];
        s_pre[e] = e < ncell * 4 ? s_pre[e] + before : before + s_sum[(ncell * 4 - 1) >> 5];
    }
    __syncthreads();
    const int total = s_pre[ncell * 4];
    if (!is_part) {
        if (total > a.maxp) return;  // spread in parts
        if (total == 0) {
            if (blockIdx.y != 0) return;
            // no point reaches the segment: rows of 8 cells x C values are contiguous and 16-byte aligned
            const int rowf4 = 4 * g.C;
            for (int i = tid; i < planes * 8 * rowf4; i += S::THREADS) {
                const int r = i / rowf4, c4 = i - r * rowf4;
                float4* dst = reinterpret_cast<float4*>(gridf + (((int64_t)(z0 + (r >> 3)) * nf1 + org1 + (r & 7)) * nf2 + org2) * g.C);
                dst[c4] = make_float4(0.f, 0.f, 0.f, 0.f);
            }
            return;
        }
    }
    // (m_full / m_free are initialised before the barrier above)
    const int k_begin = (int)((int64_t)job.y * total / job.z);
    const int k_end = (int)((int64_t)(job.y + 1) * total / job.z);

    // cell of candidate k, and its place among the cell's candidates, which are taken from the column's bins in turn (four
    // interleaved quarters of the cell's list), so that every chunk reaches all warps
    auto cell_of = [&](int k) -> int {
        int lo = 0, hi = ncell;
        while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if (s_pre[mid * 4] <= k) lo = mid; else hi = mid;
        }
        return lo;
    };
    auto sorted_index = [&](int k, int cell) -> int {
        const int p0 = s_pre[cell * 4], n = s_pre[cell * 4 + 4] - p0, j = k - p0, sg = j & 3;
        const int at = p0 + sg * (n >> 2) + min(sg, n & 3) + (j >> 2);
        int e = cell * 4;
        e += (at >= s_pre[e + 1]) + (at >= s_pre[e + 2]) + (at >= s_pre[e + 3]);
        return s_st[e] + (at - s_pre[e]);
    };

    const int nch = (k_end - k_begin + S::CH - 1) / S::CH;
    const int cell0 = is_part ? cell_of(k_begin) : 0;  // the walk's first cell
    // Stages chunk c, one thread per candidate; false (for a whole warp) when a wait ran out.
    auto stage = [&](int c, int q) -> bool {
        const int b = c % S::RING;
        float* buf = ring + b * S::kBufF;
        if (c >= S::RING && !__all_sync(0xffffffffu, mbar_wait(m_free + b, (c / S::RING - 1) & 1, w.tries))) return false;
        const int k = k_begin + c * S::CH + q;
        int pk = 0, cell = 0, pj = 0, ry = -16, rx = -16;  // past the end: reaches no block
        float fz = 0.f, fy = 0.f, fx = 0.f;
        if (k < k_end) {
            cell = cell_of(k);
            const int sidx = sorted_index(k, cell);
            fz = __fsub_rn(a.su[0][sidx], hw);
            fy = __fsub_rn(a.su[1][sidx], hw);
            fx = __fsub_rn(a.su[2][sidx], hw);
            pj = a.perm[sidx];
            auto rel_cell = [&](float f, int nf, int org) {
                int iw = (int)ceilf(f);
                if (iw < 0) iw += nf;
                if (iw >= nf) iw -= nf;
                int r = iw - org;
                if (r < 0) r += nf;
                if (r >= 8) r -= nf;  // a footprint reaching the column from below starts at -(W-1) .. -1
                return r;
            };
            ry = rel_cell(fy, nf1, org1);
            rx = rel_cell(fx, nf2, org2);
            pk = cell;
        }
        const bool reach = ry >= -(W - 1) && rx >= -(W - 1);
        // values: CC / 2 lanes per candidate, whole rows of CC x 8 bytes
        const unsigned reached = __ballot_sync(0xffffffffu, reach);
        if (CC >= 8 && vec && cc0 + CC <= g.C) {
            constexpr int LPC = CC >= 2 ? CC / 2 : 1, CPI = 32 / LPC;  // lanes per candidate, candidates per copy
            const int sub = lane / LPC, l2 = 2 * (lane % LPC);
#pragma unroll
            for (int i = 0; i < LPC; ++i) {
                const int qq = i * CPI + sub;
                const int pq = __shfl_sync(0xffffffffu, pj, qq);
                if ((reached >> qq) & 1u)
                    cp_async16(reinterpret_cast<float2*>(buf + ((q & ~31) + qq) * S::REC) + l2, a.inT + (int64_t)pq * g.C + cc0 + l2);
            }
        } else if (reach) {
            const float2* src = a.inT + (int64_t)pj * g.C + cc0;
            for (int c2 = 0; c2 < CC; ++c2) {
                float2* dst = reinterpret_cast<float2*>(buf + q * S::REC) + c2;
                if (cc0 + c2 < g.C) cp_async8(dst, src + c2); else *dst = make_float2(0.f, 0.f);
            }
        }
        if (reach) {
            pk |= ((ry + 16) << 8) | ((rx + 16) << 16);
            float* rec = buf + q * S::REC;
            auto frac = [](float f) { return fmaf(2.f, __fsub_rn(ceilf(f), f), -1.f); };
            float t[W];
            walk_taps<W>(coef, a.kb.deg, frac(fz), t);
            int sl = (cell - cell0) % W;  // slot of the first cell
#pragma unroll
            for (int d = 0; d < W; ++d) {
                *reinterpret_cast<float2*>(rec + S::OZ + 2 * sl) = make_float2(t[d], t[d]);
                sl = sl + 1 == W ? 0 : sl + 1;
            }
#pragma unroll 1
            for (int ax = 0; ax < 2; ++ax) {
                float2* row = reinterpret_cast<float2*>(rec + (ax == 0 ? S::OY : S::OX));
                const int r = ax == 0 ? ry : rx;
                walk_taps<W>(coef, a.kb.deg, frac(ax == 0 ? fy : fx), t);
#pragma unroll
                for (int cx = 0; cx < 8; cx += 2) *reinterpret_cast<float4*>(row + cx) = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
                for (int d = 0; d < W; ++d)
                    if ((unsigned)(r + d) < 8u) row[r + d] = make_float2(t[d], t[d]);
            }
        }
        reinterpret_cast<int*>(buf + S::CH * S::REC)[q] = pk;
        mbar_arrive_copies(m_full + b);
        mbar_arrive(m_full + b);
        return true;
    };

    if (warp >= S::WARPS) {  // staging warps
        bool ok = true;
        for (int c = 0; c < nch && ok; ++c) ok = stage(c, tid - S::WARPS * 32);
        cp_async_wait_all();
        if (!ok && lane == 0) atomicExch(w.err, 1);
        return;
    }

    // this warp's block, this group's 2 x 2 cells
    const int wy0 = (warp / (8 / S::BX)) * S::BY, wx0 = (warp % (8 / S::BX)) * S::BX;
    const int y0 = S::CELLS ? wy0 + lane / 8 : wy0 + 2 * (grp % S::GY), x0 = S::CELLS ? lane % 8 : wx0 + 2 * (grp / S::GY);
    f2_t acc[W][S::K];
#pragma unroll
    for (int d = 0; d < W; ++d)
#pragma unroll
        for (int k = 0; k < S::K; ++k) acc[d][k] = 0ull;

    int first = W - 1, stop = W - 1 + planes;  // planes r in [first, stop) are stored
    int cur = cell0;                           // first cell of the visits now; plane cur + d is in slot (cur - cell0 + d) mod W
    // this thread's cells of plane `cur`: in the grid, or in this part's scratch planes (strides below 2^31 values)
    float2* out;
    int plane_stride, row_stride;
    if (is_part) {
        const int zb = cell_of(k_end - 1);
        first = max(cell0, first);
        stop = min(zb + W, stop);
        if (tid == 0 && blockIdx.y == 0) w.range[blockIdx.x] = make_int2(cell0, zb);
        row_stride = 8 * g.C;
        plane_stride = 8 * row_stride;
        out = w.scratch + ((int64_t)job.w + (int64_t)job.y * W + cell0) * plane_stride;  // plane r at offset r
        out += y0 * row_stride + x0 * g.C + cc0 + coil;
    } else {
        row_stride = nf2 * g.C;
        plane_stride = nf1 * row_stride;
        out = gridf + (int64_t)(z0 - (W - 1)) * plane_stride + (int64_t)(org1 + y0) * row_stride + (org2 + x0) * g.C + cc0 + coil;
    }
    const bool coil_ok = cc0 + coil < g.C;
    // a visit's record is found by its shared address
    const unsigned at_v = (unsigned)coil * 8, at_y = (unsigned)(S::OY + 2 * y0) * 4, at_x = (unsigned)(S::OX + 2 * x0) * 4;
    auto visit = [&](unsigned rec) {
        // all loads first: one shared-memory latency per visit
        f2_t z[S::WZ], u[S::K];
        if constexpr (S::CELLS) {
            f2_t v[S::K];
            if constexpr (CC == 1) v[0] = lds64(rec);
#pragma unroll
            for (int k = 0; k + 1 < S::K; k += 2) {
                const ulonglong2 p = lds128(rec + 8 * k);
                v[k] = p.x;
                v[k + 1] = p.y;
            }
            const f2_t wx = lds64(rec + at_x), wy = lds64(rec + at_y);
#pragma unroll
            for (int d = 0; d < S::WZ; d += 2) {
                const ulonglong2 p = lds128(rec + S::OZ * 4 + 8 * d);
                z[d] = p.x;
                z[d + 1] = p.y;
            }
            const f2_t wyx = f2_mul(wy, wx);
#pragma unroll
            for (int k = 0; k < S::K; ++k) u[k] = f2_mul(wyx, v[k]);
        } else {
            const f2_t v = lds64(rec + at_v);
            const ulonglong2 wx = lds128(rec + at_x), wy = lds128(rec + at_y);
#pragma unroll
            for (int d = 0; d < S::WZ; d += 2) {
                const ulonglong2 p = lds128(rec + S::OZ * 4 + 8 * d);
                z[d] = p.x;
                z[d + 1] = p.y;
            }
            const f2_t v0 = f2_mul(v, wx.x), v1 = f2_mul(v, wx.y);
            u[0] = f2_mul(v0, wy.x);
            u[1] = f2_mul(v1, wy.x);
            u[2] = f2_mul(v0, wy.y);
            u[3] = f2_mul(v1, wy.y);
        }
#pragma unroll
        for (int d = 0; d < W; ++d)
#pragma unroll
            for (int k = 0; k < S::K; ++k) acc[d][k] = f2_fma(z[d], u[k], acc[d][k]);
    };

    const unsigned ring_at = (unsigned)__cvta_generic_to_shared(ring);
    const unsigned list_at = ring_at + (S::RING * S::kBufF + warp * S::kListN) * 4;
    constexpr unsigned kEnd = 0xff000000u, kDone = 0xfe000000u;  // end of a chunk's list, of the last chunk's
    bool ok = true;
    int c = -1;
    unsigned at = 0, e = kEnd;
    // visits since the last plane was stored or the sums were put away | slots with sums in `out` << 16
    unsigned run = 0;
    // this warp's candidates of the next chunk that has any: record address | first cell << 24
    auto next_list = [&]() {
        do {
            if (c >= 0) {
                __syncwarp();
                if (lane == 0) mbar_arrive(m_free + c % S::RING);
            }
            if (++c == nch) {
                e = kDone;
                return;
            }
            const int b = c % S::RING;
            ok = __all_sync(0xffffffffu, mbar_wait(m_full + b, (c / S::RING) & 1, w.tries));  // a warp stays together
            if (!ok) {
                e = kDone;
                return;
            }
            const unsigned buf_at = ring_at + b * S::kBufF * 4;
            int nh = 0;
#pragma unroll
            for (int q0 = 0; q0 < S::CH; q0 += 32) {
                const unsigned pk = lds32(buf_at + (S::CH * S::REC + q0 + lane) * 4);
                const int ry = (int)((pk >> 8) & 0xff) - 16, rx = (int)((pk >> 16) & 0xff) - 16;
                const bool hit = ry < wy0 + S::BY && ry + W > wy0 && rx < wx0 + S::BX && rx + W > wx0;
                const unsigned bits = __ballot_sync(0xffffffffu, hit);
                if (hit)
                    asm volatile("st.shared.u32 [%0], %1;" ::"r"(list_at + (nh + __popc(bits & ((1u << lane) - 1))) * 4),
                                 "r"((buf_at + (unsigned)(q0 + lane) * (S::REC * 4)) | (pk << 24))
                                 : "memory");
                nh += __popc(bits);
            }
            if (lane == 0) asm volatile("st.shared.u32 [%0], %1;" ::"r"(list_at + nh * 4), "r"(kEnd) : "memory");
            __syncwarp();
            at = list_at;
            e = lds32(at);
            run += nh;
        } while (e == kEnd);
    };
    // adds to the plane's sums in `out`, j planes above `cur`, those in slot `sl`
    auto put = [&](int j, int sl) {
        float2* const p = out + (int64_t)j * plane_stride;
        const bool add = (run >> (16 + sl)) & 1u;
        if constexpr (S::CELLS) {
#pragma unroll
            for (int k = 0; k < S::K; ++k)
                if (k < g.C) {
                    f2_t* q = reinterpret_cast<f2_t*>(p + k);
                    *q = add ? f2_add(acc[sl][k], *q) : acc[sl][k];
                }
        } else if (coil_ok) {
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                f2_t* q = reinterpret_cast<f2_t*>(p + (k >> 1) * row_stride + (k & 1) * g.C);
                *q = add ? f2_add(acc[sl][k], *q) : acc[sl][k];
            }
        }
#pragma unroll
        for (int k = 0; k < S::K; ++k) acc[sl][k] = 0ull;
    };
    // Visits the candidates of first cell `cur`, whose plane is in slot D, and stores the plane; false when the list
    // ends first.
    auto walk_cell = [&](auto dc) -> bool {
        constexpr int D = decltype(dc)::value;
        while ((int)(e >> 24) == cur) {
            const unsigned rec = e & 0xffffffu;
            at += 4;
            e = lds32(at);
            visit(rec);
        }
        if (e == kEnd) return false;
        if (cur >= first && cur < stop) put(0, D);
#pragma unroll
        for (int k = 0; k < S::K; ++k) acc[D][k] = 0ull;
        run &= ~(0xffffu | 0x10000u << D);
        ++cur;
        out += plane_stride;
        return true;
    };
    // the next list, with plane `cur` in slot d; before it the sums are put away after a long run
    auto refill = [&](int d) {
        if ((run & 0xffffu) >= (unsigned)kWalkRun) {
#pragma unroll
            for (int sl = 0; sl < W; ++sl) {
                const int j = sl < d ? sl - d + W : sl - d;
                if (cur + j >= first && cur + j < stop) {
                    put(j, sl);
                    run |= 0x10000u << sl;
                }
            }
            run &= ~0xffffu;
        }
        next_list();
    };
    // W cells a turn. With 32 transforms refill is compiled into every slot's loop; with fewer, where a list is shorter,
    // once, and a switch leads back to the slot (spreading, 160^3 x 32: 11.7 ms, by the switch 12.9; 120x96x150 x 12:
    // 1.22 ms, by the switch 1.13).
    if constexpr (CC == 32) {
        while (cur < stop) {
            static_for<W>([&](auto dc) {
                while (!walk_cell(dc)) refill(decltype(dc)::value);
            });
        }
    } else {
        int d = 0;
        while (cur < stop) {
            switch (d) {  // out of it with d < W where a list ended
#define HB_WALK_SLOT(n)                                                \
    case n:                                                            \
        if constexpr (n < W) {                                         \
            if (!walk_cell(std::integral_constant<int, n>{})) {        \
                d = n;                                                 \
                break;                                                 \
            }                                                          \
        }                                                              \
        [[fallthrough]];
                HB_WALK_SLOT(0) HB_WALK_SLOT(1) HB_WALK_SLOT(2) HB_WALK_SLOT(3) HB_WALK_SLOT(4) HB_WALK_SLOT(5) HB_WALK_SLOT(6)
#undef HB_WALK_SLOT
                default: d = W;
            }
            if (d == W)
                d = 0;
            else
                refill(d);
        }
    }
    if (!ok) {
        // a wait ran out, so the sums miss candidates: NaN in the last plane stored (the FFT passes take it to every
        // output; poisoning all planes kept `first` alive through the walk, 2 % of a type 1 of 12 transforms)
        float2* const p = out - (cur - stop + 1) * (int64_t)plane_stride;
        const float2 nan = make_float2(__int_as_float(0x7fffffff), __int_as_float(0x7fffffff));
        if constexpr (S::CELLS) {
            for (int k = 0; k < S::K; ++k)
                if (k < g.C) p[k] = nan;
        } else if (coil_ok) {
            p[0] = p[g.C] = p[row_stride] = p[row_stride + g.C] = nan;
        }
        if (lane == 0) atomicExch(w.err, 1);
    }
}

// Adds the parts of the dense segments: CTA blockIdx.x is part e.y of e.z of segment e.x and takes that share of
// the segment's planes x cells x transforms. A plane's parts follow one another (candidates are in z
// order); they are added in part order.
template <int W>
__global__ void __launch_bounds__(256) k_walk_reduce(const GridArgs a, const WalkArgs w) {
    const GridGeom& g = a.g;
    const int4 e = w.parts[blockIdx.x];
    int fr, ts, ty, tx;
    walk_segment(g, w, e.x, fr, ts, ty, tx);
    const int z0 = ts * w.sp, planes = walk_planes(g, w, ts);
    float2* const gridf = a.grid + fr * g.fgrid;
    const int2* range = w.range + ((int)blockIdx.x - e.y);
    const int64_t PE = (int64_t)64 * g.C, E = PE * planes;
    const int64_t i0 = e.y * E / e.z, i1 = (e.y + 1) * E / e.z;
    for (int p = (int)(i0 / PE); (int64_t)p * PE < i1; ++p) {
        const int r = p + W - 1;
        int s0 = 0, s1 = e.z;  // parts whose planes za .. zb + W - 1 hold r
        {
            int lo = 0, hi = e.z;  // first part with zb + W - 1 >= r
            while (lo < hi) {
                const int mid = (lo + hi) >> 1;
                if (range[mid].y + W - 1 >= r) hi = mid; else lo = mid + 1;
            }
            s0 = lo;
            hi = e.z;              // first part with za > r
            while (lo < hi) {
                const int mid = (lo + hi) >> 1;
                if (range[mid].x > r) hi = mid; else lo = mid + 1;
            }
            s1 = lo;
        }
        const int64_t b0 = max(i0, p * PE) - p * PE, b1 = min(i1, (p + 1) * PE) - p * PE;
        const float2* src = w.scratch + ((int64_t)e.w + r) * PE;
        for (int64_t i = b0 + threadIdx.x; i < b1; i += blockDim.x) {
            double re = 0., im = 0.;  // (parts alike, some hundred at the centre of a radial trajectory)
            for (int s = s0; s < s1; ++s) {
                const float2 v = src[(int64_t)s * W * PE + i];
                re += v.x;
                im += v.y;
            }
            const float2 sum = make_float2((float)re, (float)im);
            const int cell = (int)(i / g.C), c = (int)(i - (int64_t)cell * g.C);
            gridf[(((int64_t)(z0 + p) * g.nf[1] + ty * 8 + (cell >> 3)) * g.nf[2] + tx * 8 + (cell & 7)) * g.C + c] = sum;
        }
    }
}

template <int CC, int W>
inline int launch_spread_walk(const NufftPlan* p, const GridArgs& a, const WalkArgs& w, cudaStream_t s) {
    using S = WalkShape<CC, W>;
    auto kern = k_spread_walk<CC, W>;
    const size_t smem = S::smem_bytes();
    HB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    HB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared));
    {
        TimedSection ts("spread", s);
        kern<<<dim3((unsigned)(w.n_parts + w.nseg), (unsigned)ceil_div(a.g.C, CC)), S::THREADS, smem, s>>>(a, w);
        HB_TRY(check_launch("k_spread_walk"));
    }
    if (w.n_parts > 0) {
        TimedSection ts("spread_dense", s);
        k_walk_reduce<W><<<(unsigned)w.n_parts, 256, 0, s>>>(a, w);
        HB_TRY(check_launch("k_walk_reduce"));
    }
    return HB_OK;
}

template <int CC>
inline int launch_spread_walk_w(const NufftPlan* p, const GridArgs& a, const WalkArgs& w, cudaStream_t s) {
    switch (p->g.wa[2]) {
        case 4: return launch_spread_walk<CC, 4>(p, a, w, s);
        case 5: return launch_spread_walk<CC, 5>(p, a, w, s);
        case 6: return launch_spread_walk<CC, 6>(p, a, w, s);
        default: return launch_spread_walk<CC, 7>(p, a, w, s);
    }
}

}  // namespace hb

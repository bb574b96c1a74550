// K2W: the row stages of short rows (C = 16 .. 512 values), a warp at a time.
//
// A warp takes 512 / C consecutive rows of one prime (512 values of a and of b, 16 + 16 a
// lane), runs their forward stages, the products modulo X^4 - zeta and the inverse stages,
// and stores the product rows, without meeting any other warp: exchanges go through the
// warp's own shared memory behind __syncwarp.  Items are numbered (prime, rows)-major, all
// products of the same rows in a row, and each warp owns a contiguous range of them, so the
// rows' twiddles are staged once per range instead of once per product.
//
// The one-CTA-per-row-group kernel it replaces (k2_rows, now the fallback) read 4C bytes of
// twiddles per row and product, two thirds of what its data took, met CTA barriers at
// every exchange and kept 8 values a thread, so it exchanged twice or three times a direction.
// Here 16 values a lane leave one exchange (two at C = 512), with 16-byte shared accesses on
// the closing side.
//
// Measured in the same launches, k2_rows / this kernel (868-bit q unless said): 100 products at
// n = 8192 (C = 512) 247 / 235 us, 500 of 200 bits at n = 1024 (C = 64) 43.5 / 31.4, 60 of 517 bits at
// n = 4096 (C = 256) 47.1 / 47.0, and 130.2 / 124.7 for that whole call, as k2_rows is no dependent
// launch.  It runs the multiply pipe 66% of the time (a lazy butterfly, 8 pipe cycles, takes 9.2 in
// a loop of nothing else at 4 warps a sub-partition); 4 and 6 CTAs per SM instead of 5 measured
// within 2% of it either way.
//
// Layouts of a row of C values over T = C/16 lanes (t = lane % T):
//   first    value l*G + m of lane t is word t*G + m + D*l   (D = 16, or 32 at C = 512; G = D/T):
//            runs of G words, 64 to 128 contiguous bytes a row in global memory;
//   middle   (C = 512) lane 2k + h: word 32k + 4h + 8j + x in value 4j + x;
//   closing  lane t: words 16t .. 16t + 15.
#pragma once

#include <cstdint>

#include "pm_device.cuh"
#include "rows_persistent.cuh"

namespace pm {

constexpr int kWarpRowWords = 512;  // values of a (and of b) a warp takes at once
constexpr int kWarpRowWarps = 4;    // warps per CTA (independent of each other)

// rows of one item: 512 / C, at most the R rows of a plane
__host__ __device__ constexpr int warp_rows(int logc, int logr) {
    return (kWarpRowWords >> logc) < (1 << logr) ? (kWarpRowWords >> logc) : (1 << logr);
}

// `count` products of one plan: item = ((prime, rows), product)
struct PlanWarpRowWork {
    uint32_t* res;
    size_t ws_bstride;
    int n, logR, logC, P, count;
    __device__ int groups() const { return (1 << logR) / warp_rows(logC, logR); }  // row groups of a prime
    __device__ int total() const { return P * groups() * count; }
    __device__ RowItem item(int k) const {
        const int pair = k / count, z = k - pair * count;
        const int g = groups(), i = pair / g, r = (pair - i * g) * warp_rows(logC, logR);
        return RowItem{i, r, res + size_t(z) * ws_bstride + size_t(i) * n + (size_t(r) << logC), size_t(P) * n};
    }
};

// Exchange swizzle over the 512 words: 16-byte runs stay whole, and the lanes of every access
// phase above reach distinct banks (word bits 5 and 6 flip chunk bits {0,1} and {0,2}, bits 7
// and 8 chunk bit 2).  Linear over GF(2), so thread bits and element bits swizzle separately.
__host__ __device__ constexpr int swz_warp(int w) {
    return w ^ (((w >> 5) & 1) * 12) ^ (((w >> 6) & 1) * 20) ^ ((((w >> 7) ^ (w >> 8)) & 1) * 16);
}

template <int LOGC>
struct WarpRow {
    static_assert(LOGC >= 4 && LOGC <= 9, "rows of 16 .. 512 values");
    static constexpr int C = 1 << LOGC, T = C / 16, ROWS = kWarpRowWords / C;
    static constexpr bool MID = LOGC == 9;
    static constexpr int K1 = MID ? 4 : LOGC - 4;       // stages of the first pass
    static constexpr int D = MID ? 32 : 16;             // its stride
    static constexpr int G = 16 >> K1;                  // its groups per lane
    static constexpr int TWS = C / 4 + 1;               // twiddles of a row, padded (distinct banks across rows)
    static constexpr int SMEM_WORDS = 2 * kWarpRowWords + 2 * 2 * ROWS * TWS;  // a, b, forward and inverse twiddles
};

// G consecutive words at p (16-byte aligned when G >= 4), from or to registers v[0 .. G)
template <int G>
__device__ __forceinline__ void load_run(uint32_t* v, const uint32_t* p) {
    if constexpr (G == 1) {
        v[0] = *p;
    } else if constexpr (G == 2) {
        const uint2 x = *reinterpret_cast<const uint2*>(p);
        v[0] = x.x;
        v[1] = x.y;
    } else {
#pragma unroll
        for (int k = 0; k < G; k += 4) {
            const uint4 x = *reinterpret_cast<const uint4*>(p + k);
            v[k] = x.x;
            v[k + 1] = x.y;
            v[k + 2] = x.z;
            v[k + 3] = x.w;
        }
    }
}
template <int G>
__device__ __forceinline__ void store_run(uint32_t* p, const uint32_t* v) {
    if constexpr (G == 1) {
        *p = v[0];
    } else if constexpr (G == 2) {
        *reinterpret_cast<uint2*>(p) = make_uint2(v[0], v[1]);
    } else {
#pragma unroll
        for (int k = 0; k < G; k += 4) *reinterpret_cast<uint4*>(p + k) = make_uint4(v[k], v[k + 1], v[k + 2], v[k + 3]);
    }
}

// Shared accesses of the three layouts; `s` is the warp's 512 words, the swizzled lane parts
// are computed once per kernel (tb_*).
template <int LOGC, bool STORE>
__device__ __forceinline__ void first_exchange(uint32_t (&v)[16], uint32_t* s, int tb) {
    using W = WarpRow<LOGC>;
    constexpr int RUN = W::G < 4 ? W::G : 4;
#pragma unroll
    for (int l = 0; l < (1 << W::K1); ++l)
#pragma unroll
        for (int m = 0; m < W::G; m += RUN) {
            uint32_t* p = s + (tb ^ swz_warp(W::D * l + m));
            if (STORE)
                store_run<RUN>(p, v + l * W::G + m);
            else
                load_run<RUN>(v + l * W::G + m, p);
        }
}
template <bool STORE>
__device__ __forceinline__ void quad_exchange(uint32_t (&v)[16], uint32_t* s, int tb, int step) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        uint32_t* p = s + (tb ^ swz_warp(step * j));
        if (STORE)
            store_run<4>(p, v + 4 * j);
        else
            load_run<4>(v + 4 * j, p);
    }
}

// butterflies between v[e] and v[e + h] for the 16 values of a lane, twiddle by e / (2h)
template <bool FWD>
__device__ __forceinline__ void lane_stage(uint32_t (&v)[16], int h, const uint2* tw, uint32_t p, uint32_t two_p) {
#pragma unroll
    for (int e = 0; e < 16; ++e) {
        if (e & h) continue;
        if (FWD)
            ct_bfly(v[e], v[e + h], tw[e / (2 * h)], p, two_p);
        else
            gs_bfly(v[e], v[e + h], tw[e / (2 * h)], p, two_p);
    }
}

// the product of the rows a warp holds (first layout in, first layout out, over va)
template <int LOGC>
__device__ __forceinline__ void warp_row_product(uint32_t (&va)[16], uint32_t (&vb)[16], uint32_t* sa, uint32_t* sb,
                                                 const uint2* tf, const uint2* ti, int lane, const PrimeConst& pc) {
    using W = WarpRow<LOGC>;
    const int t = lane & (W::T - 1);
    const uint32_t p = pc.p, two_p = pc.two_p;
    const int tb1 = swz_warp((lane / W::T) * W::C + t * W::G);
    const int tb2 = swz_warp(32 * (lane >> 1) + 4 * (lane & 1)), tb3 = swz_warp(16 * lane);
    // --- forward: first pass (value l*G + m: stage u pairs l and l + 2^(K1-1-u)) ---
#pragma unroll
    for (int u = 0; u < W::K1; ++u) {
        lane_stage<true>(va, 8 >> u, tf + (1 << u), p, two_p);
        lane_stage<true>(vb, 8 >> u, tf + (1 << u), p, two_p);
    }
    if constexpr (W::MID) {
        first_exchange<LOGC, true>(va, sa, tb1);
        first_exchange<LOGC, true>(vb, sb, tb1);
        __syncwarp();
        quad_exchange<false>(va, sa, tb2, 8);
        quad_exchange<false>(vb, sb, tb2, 8);
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const uint2* w = tf + (16 << u) + ((t >> 1) << u);
            lane_stage<true>(va, 8 >> u, w, p, two_p);
            lane_stage<true>(vb, 8 >> u, w, p, two_p);
        }
        quad_exchange<true>(va, sa, tb2, 8);
        quad_exchange<true>(vb, sb, tb2, 8);
        __syncwarp();
        quad_exchange<false>(va, sa, tb3, 4);
        quad_exchange<false>(vb, sb, tb3, 4);
    } else if constexpr (W::K1 > 0) {
        first_exchange<LOGC, true>(va, sa, tb1);
        first_exchange<LOGC, true>(vb, sb, tb1);
        __syncwarp();
        quad_exchange<false>(va, sa, tb3, 4);
        quad_exchange<false>(vb, sb, tb3, 4);
    }
    // --- closing: the stages at distance 8 (in the middle layout already at C = 512) and 4 ---
    const uint2* w8 = tf + (W::C >> 4) + t;
    const uint2* w4 = tf + (W::C >> 3) + 2 * t;
    if constexpr (!W::MID) {
        lane_stage<true>(va, 8, w8, p, two_p);
        lane_stage<true>(vb, 8, w8, p, two_p);
    }
    lane_stage<true>(va, 4, w4, p, two_p);
    lane_stage<true>(vb, 4, w4, p, two_p);
    // quad 4t + k is modulo X^4 -+ w of the butterfly that split it from its sibling
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const uint2 w = w4[k >> 1];
        const uint2 zeta = (k & 1) ? shoup_negate(w, p) : w;
        quad_product(va[4 * k], va[4 * k + 1], va[4 * k + 2], va[4 * k + 3], vb[4 * k], vb[4 * k + 1], vb[4 * k + 2],
                     vb[4 * k + 3], zeta, p, two_p, pc.pinv);
    }
    // --- inverse ---
    lane_stage<false>(va, 4, ti + (W::C >> 3) + 2 * t, p, two_p);
    if constexpr (!W::MID) lane_stage<false>(va, 8, ti + (W::C >> 4) + t, p, two_p);
    if constexpr (W::MID) {
        quad_exchange<true>(va, sa, tb3, 4);
        __syncwarp();
        quad_exchange<false>(va, sa, tb2, 8);
#pragma unroll
        for (int u = 1; u >= 0; --u) lane_stage<false>(va, 8 >> u, ti + (16 << u) + ((t >> 1) << u), p, two_p);
        quad_exchange<true>(va, sa, tb2, 8);
        __syncwarp();
        first_exchange<LOGC, false>(va, sa, tb1);
    } else if constexpr (W::K1 > 0) {
        quad_exchange<true>(va, sa, tb3, 4);
        __syncwarp();
        first_exchange<LOGC, false>(va, sa, tb1);
    }
#pragma unroll
    for (int u = W::K1 - 1; u >= 0; --u) lane_stage<false>(va, 8 >> u, ti + (1 << u), p, two_p);
}

// One range of items per warp.  Dynamic shared memory: kWarpRowWarps * SMEM_WORDS words.
// Rows need 16-byte alignment (runs of 4 words): the host falls back to k2_rows otherwise.
// The rows are read straight into the first layout's registers; copying the next item's rows
// into shared memory ahead of time (cp.async) measured no faster (240 us against 236 for 100
// products at n = 8192): with 16 to 20 warps an SM the multiply pipe, not the loads, is the bound.
template <int LOGC, class Work>
__global__ void __launch_bounds__(32 * kWarpRowWarps, 5)
    k2w_rows(const __grid_constant__ Work w, const PrimeConst* __restrict__ pcs, const uint2* __restrict__ tw_fwd,
             const uint2* __restrict__ tw_inv, int logR) {
    using W = WarpRow<LOGC>;
    extern __shared__ __align__(16) uint32_t smem_rows[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t* sa = smem_rows + warp * kWarpRowWords * 2;
    uint32_t* sb = sa + kWarpRowWords;
    uint2* stf = reinterpret_cast<uint2*>(smem_rows + kWarpRowWarps * kWarpRowWords * 2) + warp * 2 * W::ROWS * W::TWS;
    uint2* sti = stf + W::ROWS * W::TWS;
    const int R = 1 << logR, rows = warp_rows(LOGC, logR);
    const int nw = int(gridDim.x) * kWarpRowWarps, wid = int(blockIdx.x) * kWarpRowWarps + warp;
    const int total = w.total();
    const int begin = int(int64_t(wid) * total / nw), end = int(int64_t(wid + 1) * total / nw);
    const int slot = lane / W::T, t = lane & (W::T - 1);
    const bool live = slot < rows;  // (planes of fewer than 512 values leave lanes idle)
    int cur_i = -1, cur_r = -1;
    PrimeConst pc{};
    // the rows' twiddles: row slot's entry j = 2^s + i' is Psi_rev[(R + r) 2^s + i'], s < log2 C - 2
    auto stage_twiddles = [&](const RowItem& it) {
        const uint2* gf = tw_fwd + size_t(it.i) * kNMax;
        const uint2* gi = tw_inv + size_t(it.i) * kNMax;
        for (int e = lane; e < rows * (W::C / 4); e += 32) {
            const int sl = e / (W::C / 4), j = e & (W::C / 4 - 1);
            if (j == 0) continue;
            const int s = 31 - __clz(j);
            const int g = ((R + it.r + sl) << s) + (j - (1 << s));
            stf[sl * W::TWS + j] = __ldg(gf + g);
            sti[sl * W::TWS + j] = __ldg(gi + g);
        }
        pc = pcs[it.i];
        cur_i = it.i;
        cur_r = it.r;
        __syncwarp();
    };
    grid_trigger();
    if (begin < end) stage_twiddles(w.item(begin));
    grid_wait();  // the conversion's planes
    for (int k = begin; k < end; ++k) {
        const RowItem it = w.item(k);
        uint32_t* ga = it.a + slot * W::C + t * W::G;
        const uint32_t* gb = ga + it.b_off;
        uint32_t va[16], vb[16];
        if (live) {
#pragma unroll
            for (int l = 0; l < (1 << W::K1); ++l) {
                load_run<W::G>(va + l * W::G, ga + W::D * l);
                load_run<W::G>(vb + l * W::G, gb + W::D * l);
            }
        } else {
#pragma unroll
            for (int e = 0; e < 16; ++e) va[e] = vb[e] = 0;
        }
        if (it.i != cur_i || it.r != cur_r) {
            __syncwarp();  // every lane is done with the previous rows' twiddles
            stage_twiddles(it);
        }
        const int ts = live ? slot : 0;
        warp_row_product<LOGC>(va, vb, sa, sb, stf + ts * W::TWS, sti + ts * W::TWS, lane, pc);
        if (live)
#pragma unroll
            for (int l = 0; l < (1 << W::K1); ++l) store_run<W::G>(ga + W::D * l, va + l * W::G);
    }
}

// grid and shared memory of a launch over `items` items
template <int LOGC>
constexpr size_t k2w_smem_bytes() {
    return size_t(kWarpRowWarps) * WarpRow<LOGC>::SMEM_WORDS * 4;
}
inline int k2w_grid(int64_t items, int sms) {
    const int64_t ctas = (items + kWarpRowWarps - 1) / kWarpRowWarps;
    return int(ctas < int64_t(sms) * 5 ? ctas : int64_t(sms) * 5);
}

}  // namespace pm

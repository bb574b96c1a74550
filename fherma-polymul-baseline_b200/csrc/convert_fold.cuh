// K1F: tensor-core conversion with the first column stages folded into the contraction.
//
// The residue of a coefficient and the first f forward column stages are both linear in the
// coefficients' bytes, so one contraction gives the stages' outputs directly.  With the rows of
// the 16 x C view in F = 2^f blocks of J = 16 / F rows, the value of prime i at row h J + j is
//   y_i(h, j) = sum_h' T_i[h][h'] sum_k x_k(h' J + j) 2^(8k)   (mod p_i),
// T_i the f butterfly stages over the blocks.  The weights are the stationary operand:
//   D_a[(h, i)][(j, c)] = sum_(h',k) byte_a(T_i[h][h'] 2^(8k) mod p_i) x_k(h' J + j, c)
// with M = 128 lanes = F blocks x 128/F primes, K = F x 256/F bytes, N = J rows x 8F columns = 128
// and one accumulator per byte a = 0 .. 3; every entry is at most 256 * 255^2 < 2^24.  A plan of at
// most 16 primes (q of up to 231 bits: 29 bytes of 32) folds three stages, of at most 32
// (59 bytes of 64) two, others one: the same K, M and N, so the tensor cores do the same work a
// tile while a tile holds 256, 512 or 1024 coefficients.
//
// What that changes against a coefficient per lane (convert_tile.cuh): a lane owns one prime
// and a block of rows, so its reduction constants stay in registers, the J rows of a column are
// values of one thread and the remaining 4 - f stages run on them straight from the
// accumulator -- no transpose through shared memory, no barrier between the reduction and the
// stages -- and the results leave in runs of 4F columns (32 to 128 contiguous bytes a row).
//
// One persistent CTA per SM: 128 KB of weights stay in shared memory, three 32 KB coefficient
// tiles are in flight by TMA, the accumulators fill the 512 TMEM columns.  N = 128 because an
// M = 128, K = 32 MMA takes 60 cycles at any N up to 64 and 64 at N = 128.  The accumulators of
// bytes 0 and 1 and of bytes 2 and 3 are two buffers: while the epilogue folds one pair into
// registers the MMAs fill the other, of this tile or the next.  A producer warp issues loads
// and MMAs (a warp of its own for the loads measured 5% slower); kFoldSets sets of four warps (the 128 TMEM lanes) take half tiles (half the columns)
// in turn, so one set's stages and stores overlap another's accumulator reads.
// Measured: 6.98 -> 5.60 us a product (868 bits, n = 32768, 128 products), 3.13 -> 2.72 us at
// n = 16384 (640 bits), 2.05 -> 1.53 us at n = 8192; 5.35 - 5.6 us at 32768 by box.  There it
// issues 24 instructions a residue (K1W 30) and moves 22.8 MB in 5.5 us (4.1 TB/s); left are
// the multiply pipe (busy 61% of its cycles), the 32-byte stores (each touches its own line: 29.5
// sectors an instruction; 16-byte ones cost 0.2 ms more) and the chain MMA - accumulator read -
// stages of few warps (three sets of 128 registers; two of 168 and four of 96 measured 1-2%
// and 23% slower).  The form without tensor maps converts 60 products of 517 bits (9 limbs,
// n = 4096) in 58 us against 47 for the same with 10 limbs by TMA (one loader warp 99, two 70);
// copying rows of even limbs 16 bytes at a time instead of by TMA measured 6% to 13% slower.
// Barriers: tma_full[3]; full[set][pair] (an accumulator pair is complete) and done[3] (the
// tile's buffer is free), from MMA commits; empty[pair] (one arrival a warp: the pair has been
// read); w_full.  Every wait is bounded; one that gives up stops the CTA, lets its
// copies land, frees the TMEM and sets the plan's error word.
#pragma once

#include "convert_tile.cuh"

namespace pm {

constexpr int kFoldSets = 3;
constexpr int kFoldLoaders = 3;                  // loader warps of the form without tensor maps
constexpr int kFoldTiles = 3;                    // coefficient tiles in flight
constexpr int kFoldTileBytes = 32768;            // 128 rows of 256 bytes
constexpr uint32_t kFoldWeightBytes = 4 * 32768;  // 4 bytes a, 128 rows, K = 256
constexpr size_t k1f_smem_bytes() { return 1024 + kFoldWeightBytes + kFoldTiles * kFoldTileBytes; }

// folded stages: the most whose 128 >> f lanes hold the primes, in rows long enough for a tile's
// 8 * 2^f columns; 0 when even one stage does not fit (rows of fewer than 16 values)
__host__ __device__ constexpr int fold_stages(int primes, int logc) {
    for (int f = 3; f >= 1; --f)
        if (primes <= (128 >> f) && logc >= f + 3) return f;
    return 0;
}

// `count` products of one plan: items (z, poly, column group) numbered product-major, or one
// polynomial's alone (poly_only = 0 or 1)
struct PlanFoldWork {
    CUtensorMap map_a, map_b;
    uint32_t* work;
    size_t ws_bstride;
    int n, logC, P, count;
    int log_groups;  // column groups per row = 2^log_groups
    PlainRows plain;            // (the form that loads rows without tensor maps)
    __device__ int total() const { return count << (log_groups + 1); }
    __device__ TileItem item(int k) const {
        const int g = log_groups, cg = k & ((1 << g) - 1);
        return TileItem{k >> (g + 1), (k >> g) & 1, cg};
    }
    __device__ ConvTarget target(int z, int poly) const {
        return ConvTarget{poly ? &map_b : &map_a, z, work + z * ws_bstride, n, logC, P};
    }
};

namespace tc {
// K-major operand rows of 32, 64 or 128 bytes in the swizzle of that span: 8-row groups are
// 8 * span bytes apart, 16-byte chunks are XORed with address bits 7 and up.
template <int SPAN>
__device__ __forceinline__ uint64_t swizzled_desc(uint32_t saddr) {
    static_assert(SPAN == 32 || SPAN == 64 || SPAN == 128, "swizzle spans");
    uint64_t d = uint64_t((saddr >> 4) & 0x3FFF);
    d |= uint64_t(1) << 16;
    d |= uint64_t((8 * SPAN) >> 4) << 32;
    d |= uint64_t(1) << 46;
    d |= uint64_t(SPAN == 128 ? 2 : (SPAN == 64 ? 4 : 6)) << 61;
    return d;
}

__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t (&v)[8]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
                 : "r"(taddr));
}
}  // namespace tc

// 8 consecutive words: one 32-byte store where the planes are 32-byte aligned
__device__ __forceinline__ void store8(uint32_t* p, const uint32_t (&v)[8], bool aligned32) {
    if (aligned32) {
        asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "r"(v[0]), "r"(v[1]),
                     "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
                     : "memory");
    } else {
        *reinterpret_cast<uint4*>(p) = make_uint4(v[0], v[1], v[2], v[3]);
        *reinterpret_cast<uint4*>(p + 4) = make_uint4(v[4], v[5], v[6], v[7]);
    }
}

constexpr int k1f_threads(bool plain) { return 32 * (4 * kFoldSets + 1 + (plain ? kFoldLoaders : 0)); }

// LOGF: folded stages f.  qbytes: bytes a coefficient can have (K steps past them are skipped).
// PLAIN: coefficient rows a tensor map cannot describe (w.plain); kFoldLoaders more warps copy
// them into the same swizzled layout, 8 bytes at a time, a tile ahead of the one they hand over.
template <int LOGF, class Work, bool PLAIN = false>
__global__ void __launch_bounds__(k1f_threads(PLAIN), 1)
    k1f_convert(const __grid_constant__ Work w, const PrimeConst* __restrict__ pcs, const uint8_t* __restrict__ weights,
                const uint2* __restrict__ tw_fwd, int qbytes, uint32_t* __restrict__ err) {
    constexpr int F = 1 << LOGF, J = 16 >> LOGF, PMAX = 128 >> LOGF;
    constexpr int COLS = 8 * F, HALF = 4 * F;    // a tile's columns, a warp's
    constexpr int SPAN = 256 >> LOGF;            // bytes of a coefficient in K
    constexpr int BOX = 128 * SPAN;              // one row block of a tile
    constexpr bool kDependent = std::is_same<Work, PlanFoldWork>::value;  // a plan's launch is a programmatic dependent
    constexpr int LOGJ = 4 - LOGF, NTW = J - 1;  // the remaining stages and their twiddles per lane
    // Tiles requested before the CTA's first barrier, where the other threads wait for the one that requests
    // a tile's 2^f copies: all three at f = 1, else one (500 products of 200 bits at n = 1024, whole, three /
    // one: 75.6 / 75.0 us).
    constexpr int FIRST = LOGF == 1 ? kFoldTiles : 1;
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t* sbase = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t* sW = sbase;                     // [4][2][128 rows x 128 B]
    uint8_t* sX = sbase + kFoldWeightBytes;  // [kFoldTiles][F][128 rows x SPAN B]
    __shared__ uint64_t tma_full[kFoldTiles], full[kFoldSets][2], done[kFoldTiles], empty[2], w_full;
    __shared__ uint32_t tmem_base;
    __shared__ volatile uint32_t s_abort;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int total = w.total();
    const int begin = int(int64_t(blockIdx.x) * total / gridDim.x);
    const int tiles = int(int64_t(blockIdx.x + 1) * total / gridDim.x) - begin;

    if constexpr (PLAIN)  // the bytes past the copied words stay zero
        for (int k = tid; k < kFoldTiles * kFoldTileBytes / 16; k += k1f_threads(PLAIN))
            reinterpret_cast<uint4*>(sX)[k] = make_uint4(0, 0, 0, 0);
    if (warp == 0) {
        tc::tmem_alloc(&tmem_base, 512);
        if (kDependent) grid_trigger();
    }
    auto issue = [&](int kk) {
        const TileItem it = w.item(begin + kk);
        const ConvTarget t = w.target(it.z, it.poly);
        const int b = kk % kFoldTiles;
        tc::mbar_expect_tx(&tma_full[b], uint32_t(kFoldTileBytes));
        for (int h = 0; h < F; ++h)
            tc::tma_load_4d(sX + b * kFoldTileBytes + h * BOX, t.map, 0, it.cg * COLS, h * J, t.mz, &tma_full[b]);
    };
    if (tid == 32 * 4 * kFoldSets) {
        for (int b = 0; b < kFoldTiles; ++b) {
            tc::mbar_init(&tma_full[b], PLAIN ? 32 * kFoldLoaders : 1);
            tc::mbar_init(&done[b], 1);
        }
        for (int b = 0; b < 2; ++b) {
            for (int g = 0; g < kFoldSets; ++g) tc::mbar_init(&full[g][b], 1);
            tc::mbar_init(&empty[b], 8);
        }
        tc::mbar_init(&w_full, 1);
        s_abort = 0;
        tc::fence_smem_async();
        if (tiles > 0) {
            tc::mbar_expect_tx(&w_full, kFoldWeightBytes);
            for (uint32_t o = 0; o < kFoldWeightBytes; o += 32768) tc::bulk_load(sW + o, weights + o, 32768u, &w_full);
        }
    }
    // Every warp waits for the previous kernel (the coefficients, and the planes' previous readers)
    // before its first bounded wait.  Here and not in the epilogue's branch: a wait (or, with tensor
    // maps, a barrier) between here and its loop took registers from the 128 of a thread, 700 -> 729 us for 128
    // products at n = 32768.  Rows without tensor maps: the warps that load wait below, all others meet
    // them at a barrier (60 products of 517 bits at n = 4096, whole: 125.6 us with no wait, 126.4 with a
    // wait in each branch, 124.7 so).
    if (!PLAIN && kDependent) {
        grid_wait();
        if (tid == 32 * 4 * kFoldSets)
            for (int kk = 0; kk < FIRST && kk < tiles; ++kk) issue(kk);
    }
    tc::fence_smem_async();
    tc::fence_before();
    __syncthreads();
    tc::fence_after();
    const uint32_t tbase = tmem_base;
    bool ok = true;

    if (warp == 4 * kFoldSets) {
        // --------------------- MMAs (and the tiles' TMA loads) ----------------
        auto wait = [&](uint64_t* bar, uint32_t parity) {
            const bool arrived = __all_sync(0xffffffffu, tc::mbar_wait(bar, parity));
            ok = ok && arrived;
            return arrived;
        };
        if (PLAIN) {
            grid_wait();
            __syncthreads();
        }
        int issued = 0, seen = 0, committed = 0;  // tiles requested, seen complete, given to the tensor cores
        bool w_pending = false;
        if (tiles > 0) {
            if (!PLAIN && kDependent) issued = min(FIRST, tiles);
            if (!PLAIN && (!kDependent || FIRST < kFoldTiles))
                for (; issued < kFoldTiles && issued < tiles; ++issued)
                    if (lane == 0) issue(issued);
            w_pending = !wait(&w_full, 0);
        }
        for (int kk = 0; kk < tiles && ok; ++kk) {
            if (__any_sync(0xffffffffu, s_abort != 0)) break;  // another warp gave up a wait
            const int b = kk % kFoldTiles;
            if (!wait(&tma_full[b], uint32_t(kk / kFoldTiles) & 1u)) break;
            ++seen;
            for (int pair = 0; pair < 2 && ok; ++pair) {  // bytes 0, 1, then 2, 3
                if (kk >= 1 && !wait(&empty[pair], uint32_t(kk - 1) & 1u)) break;
                tc::fence_after();
                if (lane == 0) {
                    constexpr uint32_t idesc = tc::idesc_u8(128, 128);
                    const uint32_t x0 = tc::smem_u32(sX + b * kFoldTileBytes), w0 = tc::smem_u32(sW) + 65536u * pair;
                    const uint32_t d0 = tbase + 256u * pair;
#pragma unroll
                    for (int a = 0; a < 2; ++a)
#pragma unroll
                        for (int s = 0; s < 8; ++s) {  // 32 bytes of K: byte ks of block h'
                            const int h = s / (SPAN / 32), ks = s % (SPAN / 32) * 32;
                            if (ks < qbytes)
                                tc::mma_u8(d0 + 128u * a, tc::sw128_desc(w0 + a * 32768 + (s >> 2) * 16384 + 32 * (s & 3)),
                                           tc::swizzled_desc<SPAN>(x0 + h * BOX + ks), idesc, s > 0);
                        }
                    tc::mma_commit(&full[(2 * kk) % kFoldSets][pair]);  // the sets of the tile's halves
                    tc::mma_commit(&full[(2 * kk + 1) % kFoldSets][pair]);
                    if (pair) tc::mma_commit(&done[b]);
                }
                __syncwarp();
            }
            if (!ok) break;
            ++committed;
            // the previous tile's MMAs have read its buffer: it takes the next tile to request
            if (!PLAIN && kk >= 1) {
                if (!wait(&done[(kk - 1) % kFoldTiles], uint32_t((kk - 1) / kFoldTiles) & 1u)) break;
                if (issued < tiles) {
                    if (lane == 0) issue(issued);
                    ++issued;
                }
            }
        }
        if (!ok) s_abort = 1;
        // copies requested but not consumed land before the CTA's shared memory goes away, and the
        // last MMAs complete before it frees the tensor memory
        for (; seen < issued; ++seen) tc::mbar_wait(&tma_full[seen % kFoldTiles], uint32_t(seen / kFoldTiles) & 1u);
        if (w_pending) tc::mbar_wait(&w_full, 0);
        if (committed)
            tc::mbar_wait(&done[(committed - 1) % kFoldTiles], uint32_t((committed - 1) / kFoldTiles) & 1u);
    } else if (PLAIN && warp > 4 * kFoldSets) {
        // ------------------------------ loaders -------------------------------
        if constexpr (PLAIN) {
            constexpr int T = 32 * kFoldLoaders;
            const int words = w.plain.copied;
            const int t0 = tid - k1f_threads(false);
            const int step_r = T / words, step_w = T - step_r * words;
            auto hand_over = [&](int kk) {  // this thread's copies of tile kk have landed
                tc::fence_smem_async();
                tc::mbar_arrive(&tma_full[kk % kFoldTiles]);
            };
            int loaded = 0;
            grid_wait();
            __syncthreads();
            for (int kk = 0; kk < tiles; ++kk, ++loaded) {
                const int b = kk % kFoldTiles;
                if (kk >= kFoldTiles)  // the MMAs have read the buffer's last tile
                    ok = tc::mbar_wait(&done[b], uint32_t(kk / kFoldTiles - 1) & 1u) && ok;
                if (__any_sync(0xffffffffu, !ok || s_abort)) break;
                const TileItem it = w.item(begin + kk);
                const ConvTarget t = w.target(it.z, it.poly);
                // row r of the tile: block r >> 7, then (row, column) n = r & 127; words in order
                int r = t0 / words, wd = t0 - r * words;
                while (r < 128 * F) {
                    const int n = r & 127, coef = (((r >> 7) * J + n / COLS) << t.logC) + it.cg * COLS + n % COLS;
                    const uint32_t off = uint32_t(n * SPAN + 8 * wd);
                    tc::cp_async8(sX + b * kFoldTileBytes + (r >> 7) * BOX + (off ^ (((off >> 7) & (SPAN / 16 - 1)) << 4)),
                                  w.plain.row(it.z, it.poly, t.n, coef) + wd);
                    r += step_r;
                    wd += step_w;
                    if (wd >= words) {
                        wd -= words;
                        ++r;
                    }
                }
                tc::cp_async_commit();
                if (kk >= 1) {
                    tc::cp_async_wait<1>();
                    hand_over(kk - 1);
                }
            }
            tc::cp_async_wait<0>();
            if (loaded) hand_over(loaded - 1);
            if (!ok) s_abort = 1;
        }
    } else {
        // ------------------------------ epilogue ------------------------------
        if (PLAIN) __syncthreads();
        const int set = warp >> 2;
        const int m = tid & 127;  // TMEM lane: block h of rows, prime i
        const int i = m % PMAX, h = m / PMAX;
        const PrimeConst pc = pcs[i];
        const uint32_t p = pc.p, two_p = pc.two_p, mu = pc.mu >> 13;  // floor(2^48 / p)
        // stage f + u splits block h into 2^u runs of rows: their twiddles
        uint2 tw[NTW > 0 ? NTW : 1];
#pragma unroll
        for (int u = 0; u < LOGJ; ++u)
#pragma unroll
            for (int b = 0; b < (1 << u); ++b)
                tw[(1 << u) - 1 + b] = __ldg(tw_fwd + size_t(i) * kNMax + (1 << (LOGF + u)) + (h << u) + b);
        // waits for an accumulator pair of this set's half tile; false stops the warp (and so the CTA)
        auto ready = [&](int pair, uint32_t parity) {
            ok = tc::mbar_wait(&full[set][pair], parity) && ok;
            const bool stop = __any_sync(0xffffffffu, !ok || s_abort);
            tc::fence_after();
            return !stop;
        };
        auto release = [&](int pair) {
            tc::fence_before();
            __syncwarp();
            if (lane == 0) tc::mbar_arrive(&empty[pair]);  // this warp's reads of the pair are complete
        };
        uint32_t parity = 0;
        for (int u = set; u < 2 * tiles; u += kFoldSets, parity ^= 1u) {
            const int half = u & 1;
            const uint32_t acc = tbase + (uint32_t(32 * (warp & 3)) << 16) + uint32_t(half * HALF);
            const TileItem it = w.item(begin + (u >> 1));
            const ConvTarget t = w.target(it.z, it.poly);
            // the thread's 64 values (row j, column c) are chunks of 8 columns: residue hi 2^16 + lo,
            // both sums below 257 * 256 * 255^2 < 2^32 - 2^16; in [0, 3p): butterfly inputs
            uint32_t v[64];
            if (!ready(0, parity)) break;
#pragma unroll
            for (int q = 0; q < 8; q += 2) {
                uint32_t d[4][8];
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    tc::tmem_ld8(acc + 128u * (e & 1) + uint32_t(8 * (q + (e >> 1)) / HALF * COLS + 8 * (q + (e >> 1)) % HALF),
                                 d[e]);
                tc::tmem_wait_ld();
#pragma unroll
                for (int e = 0; e < 16; ++e) v[8 * q + e] = d[2 * (e >> 3)][e & 7] + (d[2 * (e >> 3) + 1][e & 7] << 8);
            }
            release(0);
            if (!ready(1, parity)) break;
#pragma unroll
            for (int q = 0; q < 8; q += 2) {
                uint32_t d[4][8];
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    tc::tmem_ld8(acc + 256u + 128u * (e & 1) +
                                     uint32_t(8 * (q + (e >> 1)) / HALF * COLS + 8 * (q + (e >> 1)) % HALF),
                                 d[e]);
                tc::tmem_wait_ld();
#pragma unroll
                for (int e = 0; e < 16; ++e)
                    v[8 * q + e] = reduce48_lazy(v[8 * q + e], d[2 * (e >> 3)][e & 7] + (d[2 * (e >> 3) + 1][e & 7] << 8),
                                                 p, mu);
            }
            release(1);
            // the remaining stages; a row pair of the last one is stored while the next is computed
            // (the stores back to back stalled the warp: each touches 32 lines)
            uint32_t* dst = t.res + (size_t(it.poly) * t.P + i) * size_t(t.n) + (size_t(h * J) << t.logC) +
                            size_t(it.cg) * COLS + half * HALF;
            const bool aligned32 = (reinterpret_cast<uintptr_t>(t.res) & 31) == 0;
#pragma unroll
            for (int s = 0; s < LOGJ; ++s) {
                const int d = J >> (s + 1);
#pragma unroll
                for (int j = 0; j < J; ++j) {
                    if (j & d) continue;
#pragma unroll
                    for (int c = 0; c < HALF; ++c)
                        ct_bfly(v[j * HALF + c], v[(j + d) * HALF + c], tw[(1 << s) - 1 + (j >> (LOGJ - s))], p, two_p);
                    if (s == LOGJ - 1 && i < t.P)
#pragma unroll
                        for (int r = j; r <= j + 1; ++r)
#pragma unroll
                            for (int c = 0; c < HALF; c += 8) {
                                uint32_t o[8];
#pragma unroll
                                for (int e = 0; e < 8; ++e) o[e] = v[r * HALF + c + e];
                                store8(dst + (size_t(r) << t.logC) + c, o, aligned32);
                            }
                }
            }
        }
        if (!ok) s_abort = 1;
    }
    tc::fence_before();
    __syncthreads();
    if (warp == 0) {
        tc::fence_after();
        tc::tmem_dealloc(tbase, 512);
    }
    if (!ok) atomicOr(err, 1u);
}

}  // namespace pm

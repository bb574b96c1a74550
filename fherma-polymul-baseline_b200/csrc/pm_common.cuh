// Constants and modular arithmetic shared by the device kernels and the host
// code that prepares their tables.
#pragma once

#include <cstdint>

namespace pm {

constexpr int kLogNMax = 16;
constexpr int kNMax = 1 << kLogNMax;  // largest ring dimension; twiddle tables are this long
constexpr int kPMax = 64;             // largest prime basis
constexpr int kWMax = 28;             // largest q in 32-bit words (896 bits)
constexpr int kPowWords = 32;         // rows of 2^(32k) mod p kept per prime

struct PrimeConst {
    uint32_t p;
    uint32_t two_p;
    uint32_t mu;    // floor(2^61 / p), p in (2^29, 2^30)
    uint32_t pinv;  // p^-1 mod 2^32 (Montgomery reduction)
    uint64_t recip; // floor(2^64 / p)
};

// x * w mod p up to one extra p: result in [0, 2p) for any 32-bit x.
// w = (value, floor(value * 2^32 / p)).
__device__ __forceinline__ uint32_t shoup_mul(uint32_t x, uint2 w, uint32_t p) {
    return x * w.x - __umulhi(x, w.y) * p;
}

// [0, 2m) -> [0, m); the unsigned min picks x - m exactly when it did not wrap (written as one
// add-and-min: min(x, x - m) left to the compiler ran the row kernel 2.4% slower at n = 65536).
__device__ __forceinline__ uint32_t csub(uint32_t x, uint32_t m) { return __viaddmin_u32(x, 0u - m, x); }
// The same left to the compiler, for the plain method's CRT kernel (k3_cols_crt), which is one chain of
// such steps and shuffles a thread: with the fused form it took 65.7 us against 62.1 (32 products of
// n = 64, 896 bits) and 59.4 against 56.2 (one of n = 128, 831 bits).
__device__ __forceinline__ uint32_t csub_pair(uint32_t x, uint32_t m) { return min(x, x - m); }

// x mod p up to two extra p, for x < 2^60: Barrett with mu = floor(2^61/p), whose
// quotient estimate is at most 2 below floor(x/p), without the two corrections --
// the result lies in [0, 3p), enough for a forward butterfly input.
__device__ __forceinline__ uint32_t reduce60_lazy(uint64_t x, uint32_t p, uint32_t mu) {
    const uint32_t q = uint32_t((uint64_t(uint32_t(x >> 29)) * mu) >> 32);
    return uint32_t(x) - q * p;
}

// (hi 2^16 + lo) mod p up to two extra p, for hi < 2^32 - 2^16, any 32-bit lo
// and m = floor(2^48 / p), without forming the 48-bit value: u = hi + (lo >> 16)
// is its top part, u 2^16 <= v < u 2^16 + 2^16, and q = floor(u m / 2^32)
// satisfies v/p - 2 - 2^16/p < q <= v/p, so v - q p lies in [0, 3p) and is
// exact in 32-bit arithmetic.
__device__ __forceinline__ uint32_t reduce48_lazy(uint32_t lo, uint32_t hi, uint32_t p, uint32_t m) {
    const uint32_t q = __umulhi(hi + (lo >> 16), m);
    return lo + (hi << 16) - q * p;
}

// x * y * 2^-32 mod p up to one extra p, for x, y in [0, 2p): result in (0, 2p).
// Montgomery reduction with m = lo(xy) p^-1: xy - m p is a multiple of 2^32 and,
// as xy < 4p^2 < p 2^32, (xy - m p) / 2^32 lies in (-p, p).
__device__ __forceinline__ uint32_t mont_mul(uint32_t x, uint32_t y, uint32_t p, uint32_t pinv) {
    const uint64_t t = uint64_t(x) * y;
    const uint32_t m = uint32_t(t) * pinv;
    return uint32_t(t >> 32) - __umulhi(m, p) + p;
}

// The rows' transforms stop kDeferred stages early (fewer in rows of fewer than 4 values): a
// row ends as polynomials of 4 values modulo X^4 - zeta, multiplied as such (quad_product).
constexpr int kDeferred = 2;
__host__ __device__ constexpr int deferred_stages(int logc) { return logc < kDeferred ? logc : kDeferred; }

// (w, Shoup companion) of w mod p -> those of -w mod p: floor((p - w) 2^32 / p) is
// 2^32 - 1 - floor(w 2^32 / p), as p divides no w 2^32.
__device__ __forceinline__ uint2 shoup_negate(uint2 w, uint32_t p) { return make_uint2(p - w.x, ~w.y); }

// t 2^-32 mod p for t < 8p^2, in [0, 2p): (t - m p) / 2^32 with m = lo(t) p^-1 lies in (-p, 2p).
__device__ __forceinline__ uint32_t mont_reduce(uint64_t t, uint32_t p, uint32_t two_p, uint32_t pinv) {
    const uint32_t m = uint32_t(t) * pinv;
    return csub(uint32_t(t >> 32) - __umulhi(m, p) + p, two_p);
}

// a b 2^-32 mod (X^4 - zeta, p) over a: both factors in [0, 4p), the product in [0, 2p).
// a is taken to [0, p) and b (and zeta b) to [0, 2p), so each coefficient's four 64-bit
// products sum below 8p^2 and take one Montgomery reduction.  Against the two butterfly
// stages of a, b and the product and four pointwise products it replaces: 16 wide and 9 + 8
// other multiplies instead of 36 + 12 (112 multiplier-pipe cycles a warp against 136) and
// about half the instructions, and the last two stages' twiddles (three quarters of a row's
// table) are not needed at all.  Measured, row kernels: 11.36 -> 10.68 us a product at
// n = 32768 (868-bit q, 128 products), 3.12 -> 2.50 at n = 8192 (100 products).
__device__ __forceinline__ void quad_product(uint32_t& a0, uint32_t& a1, uint32_t& a2, uint32_t& a3, uint32_t b0,
                                             uint32_t b1, uint32_t b2, uint32_t b3, uint2 zeta, uint32_t p,
                                             uint32_t two_p, uint32_t pinv) {
    const uint32_t x0 = csub(csub(a0, two_p), p), x1 = csub(csub(a1, two_p), p);
    const uint32_t x2 = csub(csub(a2, two_p), p), x3 = csub(csub(a3, two_p), p);
    const uint32_t z1 = shoup_mul(b1, zeta, p), z2 = shoup_mul(b2, zeta, p), z3 = shoup_mul(b3, zeta, p);
    const uint32_t y0 = csub(b0, two_p), y1 = csub(b1, two_p), y2 = csub(b2, two_p), y3 = csub(b3, two_p);
    const auto wide = [](uint32_t x, uint32_t y) { return uint64_t(x) * y; };
    a0 = mont_reduce(wide(x0, y0) + wide(x1, z3) + wide(x2, z2) + wide(x3, z1), p, two_p, pinv);
    a1 = mont_reduce(wide(x0, y1) + wide(x1, y0) + wide(x2, z3) + wide(x3, z2), p, two_p, pinv);
    a2 = mont_reduce(wide(x0, y2) + wide(x1, y1) + wide(x2, y0) + wide(x3, z3), p, two_p, pinv);
    a3 = mont_reduce(wide(x0, y3) + wide(x1, y2) + wide(x2, y1) + wide(x3, y0), p, two_p, pinv);
}

// The same modulo X^2 - zeta (rows of 2 values): sums below 4p^2.
__device__ __forceinline__ void pair_product(uint32_t& a0, uint32_t& a1, uint32_t b0, uint32_t b1, uint2 zeta,
                                             uint32_t p, uint32_t two_p, uint32_t pinv) {
    const uint32_t x0 = csub(csub(a0, two_p), p), x1 = csub(csub(a1, two_p), p);
    const uint32_t z1 = shoup_mul(b1, zeta, p), y0 = csub(b0, two_p), y1 = csub(b1, two_p);
    a0 = mont_reduce(uint64_t(x0) * y0 + uint64_t(x1) * z1, p, two_p, pinv);
    a1 = mont_reduce(uint64_t(x0) * y1 + uint64_t(x1) * y0, p, two_p, pinv);
}

// Forward Cooley-Tukey butterfly, Harvey lazy: x, y in [0, 4p) -> [0, 4p).
__device__ __forceinline__ void ct_bfly(uint32_t& x, uint32_t& y, uint2 w, uint32_t p, uint32_t two_p) {
    uint32_t xr = csub(x, two_p);
    uint32_t t = shoup_mul(y, w, p);
    x = xr + t;
    y = xr - t + two_p;
}

// Inverse Gentleman-Sande butterfly, Harvey lazy: x, y in [0, 2p) -> [0, 2p).
__device__ __forceinline__ void gs_bfly(uint32_t& x, uint32_t& y, uint2 w, uint32_t p, uint32_t two_p) {
    uint32_t s = x + y;
    uint32_t d = x - y + two_p;
    x = csub(s, two_p);
    y = shoup_mul(d, w, p);
}

// Shared-memory swizzle: index bits 5, 6, 7 and 8 flip the bank bits {0, 2},
// {1, 3}, {0, 1, 4} and {0, 2, 3, 4}.  Only bits 0..4 change, as a function of
// bits that do not, so it maps every aligned power-of-two range onto itself and
// is linear over GF(2).  With it the 32 lanes of a warp reach 32 distinct banks
// in every pass layout of the row kernels at C = 1024..4096, with 8 or 16
// values a thread (passes at stride 2^logd, and the closing pass at stride 1,
// whose per-access element bits sit in the low bits and need lane bits XORed
// into them).
__device__ __forceinline__ int swz(int idx) {
    const int x = (idx >> 5) & 3;
    return idx ^ x ^ (x << 2) ^ (((idx >> 7) & 1) * 19) ^ (((idx >> 8) & 1) * 29);
}

}  // namespace pm

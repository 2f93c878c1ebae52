// The moduli of the int8 products (rns.cuh) and the arithmetic on one element: FP64 -> residues, a
// residue sum -> the CRT's digit, digits -> FP64.  Host and device.
#pragma once
#include <cstdint>

namespace mb {
namespace rns {

constexpr int kNum = 15;
// pairwise coprime, the largest such numbers <= 256: 2^8, 3 5 17, 11 23, 13 19, 7 31 and primes
constexpr int kMod[kNum] = {256, 255, 253, 251, 247, 241, 239, 233, 229, 227, 223, 217, 211, 199, 197};

using u128 = unsigned __int128;

constexpr u128 product() {
  u128 p = 1;
  for (int i = 0; i < kNum; ++i) p *= unsigned(kMod[i]);
  return p;
}
constexpr u128 kP = product();   // 2^117.78
static_assert(kP > (u128(1) << 117) && kP < (u128(1) << 118), "the scales below assume P between 2^117 and 2^118");
// A row of A is scaled to a 2-norm of at most 2^kTA, a column of B to 2^kTB: |sum| < 2^(kTA + kTB)
// (rounding to integers adds at most sqrt(K) / 2 < 2^8 to a norm), below P / 4 > 2^115
constexpr int kTA = 57, kTB = 58;
static_assert(kTA + kTB <= 115, "sums stay below P / 4");
constexpr uint64_t kOffset = uint64_t(1) << 59;   // makes the integers positive: |a'| <= 2^58

constexpr int inverse_mod(int a, int m) {
  for (int x = 1; x < m; ++x)
    if ((a * x) % m == 1) return x;
  return 1;
}

// Byte weights of one operand: an integer's residue is the weighted sum of its eight bytes.
struct Bytes {
  uint32_t lo[kNum];    // bytes k = 0..3: f 256^k mod m
  uint32_t hi[kNum];    // bytes k = 0..3: f 256^(k + 4) mod m
  uint32_t add[kNum];   // kFloat1 + (-f kOffset mod m)
};

constexpr int kGroups = kNum / 3;

struct Tables {
  uint32_t m[kNum];
  float minv[kNum];     // 1 / m
  Bytes a, b;           // A's residues (f = 1) and B's with the CRT's factor (f = (P / m)^-1 mod m)
  uint32_t inv[kNum];   // (P / m)^-1 mod m
  uint32_t mul[kNum];   // ceil(2^32 / m): exact quotients of numbers below 2^24
  uint32_t mulf[kNum];  // floor(2^32 / m): quotients of any 32-bit number, at most one too small
  uint32_t big[kNum];   // the multiple of m in [2^31, 2^31 + m)
  // Moduli three by three: y_a P/a + y_b P/b + y_c P/c = (y_a bc + y_b ac + y_c ab) P/(abc).  The bracket has
  // 26 bits, P/(abc) 94: four 24-bit parts, whose sums over the five groups are exact in FP64.
  uint32_t pair[kNum];               // product of the other two moduli of the group
  double w[4][kGroups];              // P/(abc) = sum of the parts w[0] (weight 2^72) .. w[3] (weight 1)
  double p[4];                       // P in the same parts (the first one 46 bits)
  double p_inv;
};
constexpr uint32_t kFloat1 = 0x4B000000u;   // bits of 2^23: kFloat1 + x reads as the float 2^23 + x, x < 2^23

constexpr double weight(u128 v, int shift) {   // v < 2^53
  double d = double(uint64_t(v));
  for (int i = 0; i < shift; ++i) d *= 2.0;
  return d;
}

constexpr Bytes make_bytes(bool with_inverse, const uint32_t (&inv)[kNum]) {
  Bytes t{};
  for (int i = 0; i < kNum; ++i) {
    const uint32_t m = uint32_t(kMod[i]), f = with_inverse ? inv[i] : 1u;
    uint32_t w = f % m;
    for (int k = 0; k < 8; ++k) {
      if (k < 4) t.lo[i] |= w << (8 * k);
      else t.hi[i] |= w << (8 * (k - 4));
      w = (w * 256u) % m;
    }
    t.add[i] = kFloat1 + (m - (uint32_t(kOffset % m) * f) % m) % m;
  }
  return t;
}

constexpr Tables make_tables() {
  Tables t{};
  const u128 mask = (u128(1) << 24) - 1;
  for (int i = 0; i < kNum; ++i) {
    const uint32_t m = uint32_t(kMod[i]);
    t.m[i] = m;
    t.minv[i] = 1.0f / float(kMod[i]);
    t.mul[i] = uint32_t(((uint64_t(1) << 32) + m - 1) / m);
    t.mulf[i] = uint32_t((uint64_t(1) << 32) / m);
    t.big[i] = uint32_t(((uint64_t(1) << 31) + m - 1) / m * m);
    t.inv[i] = uint32_t(inverse_mod(int(uint32_t((kP / m) % m)), int(m)));
  }
  t.a = make_bytes(false, t.inv);
  t.b = make_bytes(true, t.inv);
  for (int g = 0; g < kGroups; ++g) {
    const uint32_t x = t.m[3 * g], y = t.m[3 * g + 1], z = t.m[3 * g + 2];
    t.pair[3 * g] = y * z;
    t.pair[3 * g + 1] = x * z;
    t.pair[3 * g + 2] = x * y;
    const u128 q = kP / x / y / z;
    for (int h = 0; h < 4; ++h) t.w[h][g] = weight((q >> (72 - 24 * h)) & mask, 72 - 24 * h);
  }
  t.p[0] = weight(kP >> 72, 72);
  for (int h = 1; h < 4; ++h) t.p[h] = weight((kP >> (72 - 24 * h)) & mask, 72 - 24 * h);
  t.p_inv = 1.0 / (t.p[0] + t.p[1]);
  return t;
}

#ifdef __CUDA_ARCH__
__device__ __forceinline__ uint32_t dp4(uint32_t a, uint32_t b, uint32_t c) { return __dp4a(a, b, c); }
__device__ __forceinline__ uint32_t mulhi(uint32_t a, uint32_t b) { return __umulhi(a, b); }
__device__ __forceinline__ float bits_float(uint32_t u) { return __uint_as_float(u); }
__device__ __forceinline__ uint32_t float_bits(float f) { return __float_as_uint(f); }
__device__ __forceinline__ uint32_t least(uint32_t a, uint32_t b) { return min(a, b); }
#else
inline uint32_t dp4(uint32_t a, uint32_t b, uint32_t c) {
  for (int k = 0; k < 4; ++k) c += ((a >> (8 * k)) & 255u) * ((b >> (8 * k)) & 255u);
  return c;
}
inline uint32_t mulhi(uint32_t a, uint32_t b) { return uint32_t((uint64_t(a) * b) >> 32); }
inline float bits_float(uint32_t u) { float f; __builtin_memcpy(&f, &u, 4); return f; }
inline uint32_t float_bits(float f) { uint32_t u; __builtin_memcpy(&u, &f, 4); return u; }
inline uint32_t least(uint32_t a, uint32_t b) { return a < b ? a : b; }
#endif

// Low byte: a signed residue of f a' modulo m in [-m/2, m/2], for u = a' + kOffset (the upper bytes are not zero).
// The weighted byte sum x is below 8 * 255 * 255 + 256 < 2^20, an exact float; its quotient by m is rounded
// to nearest in the low bits of a float next to 1.5 2^23 (within 2^-12, so |r| <= 127 for m < 256, and 128 wraps
// to -128 for m = 256, which is the same residue).
__host__ __device__ __forceinline__ uint32_t residue(uint64_t u, const Bytes& w, const Tables& t, int i) {
  const uint32_t x = dp4(uint32_t(u >> 32), w.hi[i], dp4(uint32_t(u), w.lo[i], w.add[i]));
  const float q = fmaf(bits_float(x) - 8388608.0f, t.minv[i], 12582912.0f);
  return x - float_bits(q) * t.m[i];
}

// The CRT digit of a residue sum s, |s| <= 131071 * 2^14: s mod m, times (P / m)^-1 mod m where neither operand's
// residues carry that factor.
__host__ __device__ __forceinline__ uint32_t digit(int32_t s, const Tables& t, int i, bool with_inverse) {
  const uint32_t m = t.m[i];
  const uint32_t u = uint32_t(s) + t.big[i];                 // no wrap: |s| < 2^31 - 2^13
  const uint32_t r = u - mulhi(u, t.mulf[i]) * m;            // in [0, 2 m)
  if (!with_inverse) return least(r, r - m);
  const uint32_t x = r * t.inv[i];                           // below 2^17
  return x - mulhi(x, t.mul[i]) * m;
}

struct Crt {   // sum of y (P / m) over the moduli, in four exact parts
  double s[4] = {0.0, 0.0, 0.0, 0.0};
  __host__ __device__ __forceinline__ void add(uint32_t ya, uint32_t yb, uint32_t yc, const Tables& t, int g) {
    const double z = double(int(ya * t.pair[3 * g] + yb * t.pair[3 * g + 1] + yc * t.pair[3 * g + 2]));
#pragma unroll
    for (int h = 0; h < 4; ++h) s[h] = fma(z, t.w[h][g], s[h]);
  }
  // minus the multiple of P that leaves a number in (-P/4, P/4): every difference is exact, three roundings of
  // which only the last is not far below the result's
  __host__ __device__ __forceinline__ double value(const Tables& t) const {
    const double q = rint(s[0] * t.p_inv);
    return fma(-q, t.p[0], s[0]) + (fma(-q, t.p[1], s[1]) + (fma(-q, t.p[2], s[2]) + fma(-q, t.p[3], s[3])));
  }
};

}  // namespace rns
}  // namespace mb

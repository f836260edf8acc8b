// lela_b200/csrc/arith.cuh -- field arithmetic of the CUDA-core kernels
// (echelon panels, triangular inverses): exact inverses, residue arithmetic
// with 32-bit or 64-bit reductions, and the inverse of a 64 x 64 triangle.
#pragma once
#include <cstdint>

#include "common.cuh"

namespace lela {

// Exact inverse of a unit x modulo p (any p < 2^32): extended Euclid on
// unsigned remainders with 64-bit signed coefficients.  0 when gcd != 1.
__device__ __forceinline__ uint32_t inv_exact_u32(uint32_t p, uint32_t x) {
  uint32_t r0 = p, r1 = x;
  int64_t s0 = 0, s1 = 1;
  while (r1 != 0) {
    const uint32_t q = r0 / r1;
    const uint32_t r = r0 - q * r1;
    r0 = r1;
    r1 = r;
    const int64_t s = s0 - (int64_t)q * s1;
    s0 = s1;
    s1 = s;
  }
  if (r0 != 1) return 0;
  int64_t v = s0 % (int64_t)p;
  if (v < 0) v += p;
  return (uint32_t)v;
}

// The same for p < 2^31 in 32-bit coefficients (|s| <= p throughout).
__device__ __forceinline__ uint32_t inv_exact_i31(uint32_t p, uint32_t x) {
  uint32_t r0 = p, r1 = x;
  int s0 = 0, s1 = 1;
  while (r1 != 0) {
    const uint32_t q = r0 / r1;
    const uint32_t r = r0 - q * r1;
    r0 = r1;
    r1 = r;
    const int s = s0 - (int)q * s1;
    s0 = s1;
    s1 = s;
  }
  if (r0 != 1) return 0;
  s0 %= (int)p;
  return (uint32_t)(s0 < 0 ? s0 + (int)p : s0);
}

// sum of two products a*b + c*d modulo p (a, b, c, d < p < 2^32)
__device__ __forceinline__ uint32_t mod_dot2(uint32_t a, uint32_t b, uint32_t c, uint32_t d,
                                             const Modulus &mod, uint32_t two64) {
  const uint64_t x = (uint64_t)a * b, y = (uint64_t)c * d;
  uint64_t s = x + y;
  if (s < y) s += two64;
  return mod_reduce(s, mod);
}

// Field arithmetic for the panel kernels, in two forms chosen by the host:
// ArithSmall for p < 2^16 (every product fits in 32 bits; Barrett reduction
// with a 32-bit reciprocal, one correction) and ArithWide for any p < 2^32
// (64-bit products and Barrett reduction).  Both return canonical residues.
struct ArithSmall {
  uint32_t p, mu;  // mu = floor(2^32 / p)
  __host__ __device__ static ArithSmall make(uint32_t p) {
    ArithSmall a;
    a.p = p;
    a.mu = (uint32_t)((1ull << 32) / p);
    return a;
  }
  __device__ __forceinline__ uint32_t red(uint32_t x) const {
    const uint32_t r = x - __umulhi(x, mu) * p;
    return r >= p ? r - p : r;
  }
  __device__ __forceinline__ uint32_t mul(uint32_t a, uint32_t b) const { return red(a * b); }
  // a*b + c*d
  __device__ __forceinline__ uint32_t dot2(uint32_t a, uint32_t b, uint32_t c, uint32_t d) const {
    const uint32_t r = red(a * b) + red(c * d);
    return r >= p ? r - p : r;
  }
  // s += a*b for a sum of products reduced once at the end (sum): each
  // product is below 2^32, so up to 2^16 of them fit
  using Acc = uint64_t;
  __device__ __forceinline__ static Acc zero() { return 0; }
  __device__ __forceinline__ void acc(Acc &s, uint32_t a, uint32_t b) const {
    s += (uint64_t)a * b;
  }
  // s mod p for s < 2^48: (s mod 2^32 reduced) + (s / 2^32) (2^32 mod p)
  __device__ __forceinline__ uint32_t sum(Acc s) const {
    const uint32_t c32 = 0u - mu * p;
    return red(red((uint32_t)s) + (uint32_t)(s >> 32) * c32);
  }
};
struct ArithWide {
  Modulus mod;
  uint32_t p, two64;
  __host__ __device__ static ArithWide make(uint32_t p) {
    ArithWide a;
    a.mod = make_modulus(p);
    a.p = p;
    a.two64 = two64_mod(p);
    return a;
  }
  __device__ __forceinline__ uint32_t mul(uint32_t a, uint32_t b) const {
    return mod_mul(a, b, mod);
  }
  __device__ __forceinline__ uint32_t dot2(uint32_t a, uint32_t b, uint32_t c, uint32_t d) const {
    return mod_dot2(a, b, c, d, mod, two64);
  }
  // s += a*b in 96 bits, reduced once at the end (three instructions a term;
  // a 64-bit sum corrected by 2^64 mod p on each wrap takes about eight)
  struct Acc {
    uint32_t lo, hi, top;
  };
  __device__ __forceinline__ static Acc zero() { return {0u, 0u, 0u}; }
  __device__ __forceinline__ void acc(Acc &s, uint32_t a, uint32_t b) const {
    asm("mad.lo.cc.u32 %0, %3, %4, %0;\n\t"
        "madc.hi.cc.u32 %1, %3, %4, %1;\n\t"
        "addc.u32 %2, %2, 0;"
        : "+r"(s.lo), "+r"(s.hi), "+r"(s.top)
        : "r"(a), "r"(b));
  }
  __device__ __forceinline__ uint32_t sum(const Acc &s) const {
    const uint64_t r = (uint64_t)mod_reduce((uint64_t)s.hi << 32 | s.lo, mod) +
                       mod_mul(s.top, two64, mod);
    return (uint32_t)(r >= p ? r - p : r);
  }
};

// Inverse of a 64 x 64 triangular matrix X (upper or lower) in shared memory
// (row stride INV_LD), in place by doubling, by INV_THREADS threads (t = 0 ..):
// the inverse of [[A, B], [0, C]] is
// [[A^-1, -A^-1 B C^-1], [0, C^-1]] (lower: [[A^-1, 0], [-C^-1 B A^-1, C^-1]]),
// so the
// diagonal blocks of sizes 1, 2, 4, .., 32 are inverted level by level,
// each level two products of b x b blocks (through T, INV_T words) over
// all pairs at once.  On entry the diagonal holds the inverses of the
// diagonal entries and the rest of the triangle the matrix's entries, the
// other triangle zero (the products run over whole blocks, zeros included).
// The CTA may invert several matrices side by side, but every thread calls it
// (12 barriers).  The result is the one substitution gives with the same
// diagonal inverses: both apply the same linear map to the unit vectors.
// At the large levels a thread takes R rows of a product's column and reads the
// left factor four entries at a time (with one entry per thread they were
// bound by shared-memory reads, two per multiply-add), and the loops stay rolled:
// this code runs once per launch, at the rate its instructions are fetched
// (three cycles each measured; all levels unrolled took 15000 cycles).
constexpr int INV_THREADS = 256;
constexpr int INV_LD = 64 + 4;          // 16-byte rows
constexpr int INV_M = 64 * INV_LD;      // one matrix
constexpr int INV_T = 32 * (32 + 4);    // its scratch (rows of b + 4)
template <class A, int R>
__device__ __forceinline__ void tri64_level(uint32_t *X, uint32_t *T, bool upper, const A &ar,
                                            int t, int lb) {
  const uint32_t p = ar.p;
  const int B = 1 << lb, TLD = B + 4;
  // R rows from i0 of column jj of the product of pair q
  const int jj = t & (B - 1), i0 = ((t >> lb) * R) & (B - 1), q = t * R >> (2 * lb), r = 2 * B * q;
  const bool in = q < 32 >> lb;
  uint32_t *Tq = T + q * B * TLD;
#pragma unroll 1
  for (int half = 0; half < 2; ++half) {
    // T = B C^-1 (lower: B A^-1), then -A^-1 T (lower: -C^-1 T)
    const uint32_t *left = half ? X + (upper ? r * INV_LD + r : (r + B) * INV_LD + r + B)
                                : X + (upper ? r * INV_LD + r + B : (r + B) * INV_LD + r);
    const uint32_t *right = half ? Tq : X + (upper ? (r + B) * INV_LD + r + B : r * INV_LD + r);
    const int rld = half ? TLD : INV_LD;
    left += i0 * INV_LD;
    right += jj;
    if (in) {
      typename A::Acc acc[R];
#pragma unroll
      for (int u = 0; u < R; ++u) acc[u] = A::zero();
      if (R == 1 && B < 4) {
#pragma unroll 1
        for (int k = 0; k < B; ++k) ar.acc(acc[0], left[k], right[k * rld]);
      } else {
#pragma unroll 1
        for (int k = 0; k < B; k += 4) {
          uint32_t b[4];
#pragma unroll
          for (int w = 0; w < 4; ++w) b[w] = right[(k + w) * rld];
#pragma unroll
          for (int u = 0; u < R; ++u) {
            const uint4 a = *reinterpret_cast<const uint4 *>(left + u * INV_LD + k);
            ar.acc(acc[u], a.x, b[0]);
            ar.acc(acc[u], a.y, b[1]);
            ar.acc(acc[u], a.z, b[2]);
            ar.acc(acc[u], a.w, b[3]);
          }
        }
      }
#pragma unroll
      for (int u = 0; u < R; ++u) {
        const uint32_t v = ar.sum(acc[u]);
        if (half) {
          uint32_t *o = X + (upper ? (r + i0 + u) * INV_LD + r + B : (r + B + i0 + u) * INV_LD + r);
          o[jj] = v ? p - v : 0u;
        } else {
          Tq[(i0 + u) * TLD + jj] = v;
        }
      }
    }
    __syncthreads();
  }
}
// (n: the matrix is the identity from row n on; the same in every thread)
template <class A>
__device__ __forceinline__ void tri64_invert(uint32_t *X, uint32_t *T, bool upper, const A &ar, int t,
                                             int n = 64) {
#pragma unroll 1
  for (int lb = 0; lb < 4 && n > 1 << lb; ++lb) tri64_level<A, 1>(X, T, upper, ar, t, lb);
  if (n > 16) tri64_level<A, 2>(X, T, upper, ar, t, 4);
  if (n > 32) tri64_level<A, 4>(X, T, upper, ar, t, 5);
}

}  // namespace lela

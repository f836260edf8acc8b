// lela_b200/csrc/zp_gemm.cu -- dense gemm over Z/p (Modular<uint32>):
//   C <- alpha * A * B + beta * C  (mod p),  p in [2, 2^32).
//
// Replaces the per-entry delayed-reduction dot products of LELA's generic
// gemm (lela/blas/level3-generic.tcc:285-322 with _dot<Modular<uint32>,
// ZpModule> of lela/blas/level1-modular.tcc:135-158).  Two kernels:
//
// 1. zp_gemm_tc_kernel<L> -- limb-split INT8 tensor-core gemm.  Every entry
//    x in [0, p) is split into L unsigned 8-bit limbs, x = sum_i x_i 2^(8i),
//    with L = 1 (p <= 2^8), 2 (p <= 2^16) or 4 (p <= 2^32).  For each pair of
//    limbs (i, j) the tensor cores form P_ij = A_i * B_j with exact signed
//    32-bit accumulation (tcgen05.mma .kind::i8, accumulators in TMEM).
//    Overflow bound: a limb product is at most 255^2 = 65025, so a K-chunk
//    of at most 33025 terms cannot exceed 2^31 - 1; the host splits K into
//    chunks of KCHUNK = 32768 (the first chunk applies beta, the others add
//    with beta = 1).  The epilogue recombines
//        A*B = sum_s 2^(8s) D_s,   D_s = sum_{i+j=s} P_ij   (D_s < 4 * 2^31)
//    reduces mod p with Barrett reduction and applies alpha and beta; the
//    result is exact, i.e. bit-identical to LELA's.
//    Four limbs' products of some size go by residues instead of limbs (see
//    "residues of four limbs' work").
//
//    Data layout.  A is split into L planes of M x Kp bytes (K-major, i.e.
//    row-major A), B into L planes of N x Kp bytes (K-major, i.e. B^T); Kp =
//    K rounded up to 16 bytes (the TMA row-pitch rule).  One CTA owns a
//    128 x BN tile of C and stacks the limbs: the A operand of the i-th MMA
//    is A_i (128 rows), the B operand is [B_0; ..; B_{L-1}] (L*BN rows), so
//    one 128 x (L*BN) accumulator per A-limb holds P_i0 .. P_i(L-1) side by
//    side; L accumulators use all 512 TMEM columns for L = 2 and 4.
//
//    Pipeline (persistent, warp-specialised, 320 threads): warp 0 issues TMA
//    loads of 128-byte-swizzled K-blocks (128 bytes of K) into a ring of
//    shared-memory stages; warp 1 issues 4*L MMAs of K = 32 per stage and
//    releases stages with tcgen05.commit; warps 2-9 drain the accumulators
//    (one TMEM lane = one row of C per thread, two warps per lane quadrant
//    on the two halves of the tile's columns).  Every wait is bounded.
//
// 2. zp_gemm_plain_kernel -- the "plain GPU form": a CUDA-core tiled gemm
//    whose inner loop is exactly the reference's delayed-reduction dot
//    (64-bit sum of 32x32-bit products, + 2^64 mod p on wrap-around, one
//    final reduction).
// 3. zp_gemm_direct_kernel<L> -- the tensor-core tile product in one launch,
//    for the short-K updates of the triangular solve and the echelon panels,
//    where the first kernel's fixed cost (limb splits, tensor maps, pipeline
//    start) dominates: each CTA splits its own operands into shared memory.
// 4. zp_gemm_smallk_kernel -- CUDA-core gemm for small K: the smallest products.  For
//    p < 2^28 a 64-bit sum of 256 products cannot wrap, so the products are
//    summed without checks and the sums reduced every 256 terms.
#include <cuda.h>
#include <cudaTypedefs.h>

#include <algorithm>
#include <cstdio>
#include <mutex>

#include "common.cuh"
#include "../../include/lela_cuda.h"
#include "context.h"
#include "elem_rep.cuh"
#include "zp_gemm.h"

namespace lela {

// ------------------------------------------------------------ tile configs
//
// TcCfg<L, T>: tile variant T of the L-limb kernel.  BN = columns of C per
// tile, NMMA = L * BN (the N of one MMA: the L limbs of B stacked), STAGES
// = depth of the shared-memory ring, ACC = accumulator buffers in TMEM
// (each L * NMMA columns; at most 512 in all), EPI = epilogue warps.  With
// ACC = 2 the epilogue of one tile overlaps the MMAs of the next; with ACC =
// 1 the MMAs wait for the epilogue to drain TMEM, but each MMA is wider
// (more operations per byte of shared memory read).  The caller sees two
// shapes, wide (one limb: 256 columns; two limbs: 128 columns, one
// accumulator) and double-buffered (128 / 64 columns, two accumulators).
// Two limbs use 16 epilogue warps, one limb 16 or 8 chosen by K
// (zp_gemm_tile_pick): at short K the epilogue is most of a tile's time,
// and a tcgen05.ld wait covers all of a warp's outstanding TMEM loads, so
// only more warps hide their latency.  Four limbs have variant 0 only: with two accumulators a
// tile would be 16 columns wide, 8 per epilogue thread.
template <int L, int T>
struct TcCfg;
template <>
struct TcCfg<1, 0> {
  static constexpr int BN = 256, NMMA = 256, STAGES = 4, ACC = 2, EPI = 8;
};
template <>
struct TcCfg<1, 1> {
  static constexpr int BN = 128, NMMA = 128, STAGES = 6, ACC = 2, EPI = 16;
};
template <>
struct TcCfg<1, 2> {
  static constexpr int BN = 128, NMMA = 128, STAGES = 6, ACC = 2, EPI = 8;
};
// the GF(2) product at short K (one limb of 0/1 bytes, parity epilogue):
// wide tiles with 16 epilogue warps, 64 columns (one output word) each
template <>
struct TcCfg<1, 3> {
  static constexpr int BN = 256, NMMA = 256, STAGES = 4, ACC = 2, EPI = 16;
};
constexpr int GF2_TC_T = 3;
template <>
struct TcCfg<2, 0> {
  static constexpr int BN = 128, NMMA = 256, STAGES = 3, ACC = 1, EPI = 16;
};
template <>
struct TcCfg<2, 1> {
  static constexpr int BN = 64, NMMA = 128, STAGES = 4, ACC = 2, EPI = 16;
};
template <>
struct TcCfg<4, 0> {
  static constexpr int BN = 32, NMMA = 128, STAGES = 2, ACC = 1, EPI = 8;
};

constexpr int RNS_MAX = ZP_RESIDUE_MAX;
__host__ __device__ constexpr uint32_t rns_mod(int i) {
  return i == 0 ? 256 : i == 1 ? 255 : i == 2 ? 253 : i == 3 ? 251 : i == 4 ? 247 : i == 5 ? 241
       : i == 6 ? 239 : i == 7 ? 233 : i == 8 ? 229 : i == 9 ? 227 : 223;
}
// what the tensor-core kernel writes: residues modulo p, packed bits, or
// residue bytes modulo rns_mod(i) (rns_combine_kernel)
enum TcOut : int { OUT_ZP = 0, OUT_GF2 = 1, OUT_RNS = 2 };

constexpr int BM = 128;         // rows of C per tile (UMMA M)
constexpr int BK = 128;         // bytes (= limb elements) of K per stage
// Tile raster: groups of GROUP_M row-blocks, column-major inside a group,
// so the 148 tiles in flight share A's group panels and a few of B's.  B's
// limb planes are read once per group.  At 8192^3 (two limbs) a group's A
// planes are 32 MB and stay in L2 beside the streamed B panels; with 32
// row-blocks (64 MB) they did not: DRAM reads per launch went from 1.15 to
// 2.42 GB and the kernel took 4 % longer.
constexpr int GROUP_M = 16;
constexpr int TMEM_COLS = 512;
// warp 0: TMA, warp 1: MMA, warps 2 .. 2 + EPI - 1: epilogue (EPI / 4 per
// TMEM lane quadrant, each on BN / (EPI / 4) columns of a tile)
template <int L, int T>
constexpr int tc_threads() {
  return 64 + 32 * TcCfg<L, T>::EPI;
}

template <int L, int T>
struct TcLayout {
  using Cfg = TcCfg<L, T>;
  static_assert(Cfg::NMMA == L * Cfg::BN, "the B operand stacks the L limbs");
  static_assert(Cfg::ACC * L * Cfg::NMMA <= TMEM_COLS, "accumulators exceed TMEM");
  static_assert(Cfg::EPI % 4 == 0 && Cfg::BN % (Cfg::EPI / 4) == 0 &&
                    (Cfg::BN / (Cfg::EPI / 4)) % 16 == 0,
                "whole lane quadrants, 16-column chunks per epilogue warp");
  static constexpr int A_BYTES = L * BM * BK;
  static constexpr int B_BYTES = Cfg::NMMA * BK;
  static constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
  static constexpr int BAR_OFF = Cfg::STAGES * STAGE_BYTES;
  // full[S], empty[S], tfull[ACC], tempty[ACC], done, tmem base
  static constexpr int BAR_BYTES = 8 * (2 * Cfg::STAGES + 2 * Cfg::ACC + 1) + 8;
  static constexpr int SMEM = BAR_OFF + BAR_BYTES + 1024;
  static_assert(SMEM <= 227 * 1024, "shared memory per CTA exceeded");
};

__device__ __forceinline__ void tile_coords(int t, int tiles_m, int tiles_n, int &mb, int &nb) {
  int per_group = GROUP_M * tiles_n;
  int g = t / per_group;
  int first_m = g * GROUP_M;
  int gsize = min(GROUP_M, tiles_m - first_m);
  int w = t - g * per_group;
  mb = first_m + w % gsize;
  nb = w / gsize;
}

// Bounded wait that ignores the error word (used only to drain in-flight
// asynchronous operations before the block exits).
__device__ __forceinline__ void mbar_drain(uint64_t *bar, uint32_t parity, uint32_t *err) {
  uint64_t t0 = globaltimer_ns();
  while (!mbar_try_wait(bar, parity)) {
    if (globaltimer_ns() - t0 > WAIT_LIMIT_NS) {
      atomicOr(err, DEVERR_TIMEOUT);
      return;
    }
  }
}

// Reduction for one and two limbs (p <= 2^16): 32-bit Barrett with mu =
// floor(2^32 / p), whose quotient estimate for v < 2^32 is the quotient or
// one less, and c32 = 2^32 mod p for the high word of a two-limb product.
struct Mod32 {
  uint32_t p, mu, c32;
  __device__ __forceinline__ static Mod32 make(uint32_t p) {
    Mod32 m;
    m.p = p;
    m.mu = (uint32_t)((1ull << 32) / p);
    m.c32 = (uint32_t)((1ull << 32) % p);
    return m;
  }
  // v mod p, up to one multiple of p too large (r < 2p)
  __device__ __forceinline__ uint32_t lazy(uint32_t v) const { return v - __umulhi(v, mu) * p; }
  __device__ __forceinline__ uint32_t full(uint32_t v) const {
    const uint32_t r = lazy(v);
    return r >= p ? r - p : r;
  }
};

// How the product v (reduced) and C combine, chosen once per launch:
// C <- v + C (alpha = 1, beta = 1: the gemm C += A*B), C <- C - v
// (alpha = p - 1, beta = 1: the trsm and elimination updates), C <- alpha v
// (beta = 0), or the general alpha v + beta C.  The first three skip the two
// modular products of the general form (the epilogue is instruction-bound
// when K is small).
enum EpiMode : int { EPI_ADD = 0, EPI_SUB = 1, EPI_SET = 2, EPI_AXPBY = 3 };

// The mode is a template parameter: the epilogue's tile loop is
// instantiated once per mode and the launch runs one of them, so the hot
// code holds no per-element branches (the epilogue shares each
// sub-partition's instruction cache with the TMA and MMA warps).
// SMALL: p <= 2^16 (one and two limbs), where every product of two
// residues fits in 32 bits and the 32-bit reduction serves.
template <int MODE, bool SMALL>
__device__ __forceinline__ uint32_t epi_combine(uint32_t v, uint32_t c, const Modulus &mod,
                                                const Mod32 &m32, uint32_t alpha,
                                                uint32_t beta) {
  const uint32_t p = SMALL ? m32.p : (uint32_t)mod.p;
  auto mul = [&](uint32_t a, uint32_t b) -> uint32_t {
    if constexpr (SMALL) return m32.full(a * b);
    else return mod_mul(a, b, mod);
  };
  if constexpr (MODE == EPI_SET) return alpha == 1u ? v : mul(alpha, v);
  if constexpr (MODE == EPI_AXPBY) {
    if constexpr (SMALL) {
      const uint32_t r = mul(alpha, v) + mul(beta, c >= p ? m32.full(c) : c);
      return r >= p ? r - p : r;
    } else {
      return mod_axpby(alpha, v, beta, c, mod);
    }
  }
  if (c >= p) c = SMALL ? m32.full(c) : mod_reduce((uint64_t)c, mod);  // a caller's non-canonical C
  if constexpr (MODE == EPI_ADD) {
    const uint32_t t = p - v;  // v + c mod p without overflow
    return c >= t ? c - t : c + v;
  }
  return c >= v ? c - v : c + (p - v);
}

// The reduced products of 16 consecutive columns of one row, from the
// TMEM accumulators of a tile (tcol: the column of the first one in the
// accumulator of A-limb 0, B-limb 0).  Warp-collective: every lane of the
// warp runs it (tcgen05.ld is .sync.aligned).  The limb products P_ij are
// below 255^2 * 32768 < 2^31 (one K chunk).
template <int L, int BN, int NMMA>
__device__ __forceinline__ void chunk_products(uint32_t tcol, uint32_t (&v)[16],
                                               const Modulus &mod, const Mod32 &m32) {
  if constexpr (L == 1) {
    // one product P_00
    uint32_t r[16];
    tmem_ld16(tcol, r);
    tmem_ld_wait();
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = m32.full(r[i]);
  } else if constexpr (L == 2) {
    // x = 2^16 P_11 + 2^8 (P_01 + P_10) + P_00 < 2^48, as hi 2^32 + lo:
    // x = lo + hi c32 (mod p), and (lo mod p, < 2p) + hi c32 < 2^32 for
    // p <= 2^16 (p = 2^16 has c32 = 0)
    uint32_t p00[16], p01[16], p10[16], p11[16];
    tmem_ld16(tcol, p00);
    tmem_ld16(tcol + BN, p01);
    tmem_ld16(tcol + NMMA, p10);
    tmem_ld16(tcol + NMMA + BN, p11);
    tmem_ld_wait();
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const uint64_t x = ((uint64_t)p11[i] << 16) + ((uint64_t)(p01[i] + p10[i]) << 8) + p00[i];
      const uint32_t t = m32.lazy((uint32_t)x) + (uint32_t)(x >> 32) * m32.c32;
      v[i] = m32.full(t);
    }
  } else {
    // L = 4: x = sum_s 2^(8s) D_s with D_s = sum_{i+j=s} P_ij, gathered as
    // x = F_a + 2^24 F_b + 2^48 D_6 (F_a = D_0 + 2^8 D_1 + 2^16 D_2 < 2^49,
    // F_b likewise from D_3..D_5, D_6 = P_33 < 2^31), then three steps of
    // Horner in 2^24 with one reduction each ((r < 2^32) 2^24 + F < 2^57).
    // Eight columns at a time; the sixteen limb products in two waits.
#pragma unroll
    for (int h = 0; h < 16; h += 8) {
      uint64_t Fa[8], Fb[8];
      uint32_t D6[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        Fa[i] = 0;
        Fb[i] = 0;
      }
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        uint32_t r[2][4][8];
#pragma unroll
        for (int a = 0; a < 2; ++a)
#pragma unroll
          for (int lj = 0; lj < 4; ++lj)
            tmem_ld8(tcol + h + (2 * half + a) * NMMA + lj * BN, r[a][lj]);
        tmem_ld_wait();
#pragma unroll
        for (int a = 0; a < 2; ++a)
#pragma unroll
          for (int lj = 0; lj < 4; ++lj) {
            const int sd = 2 * half + a + lj;  // the digit of this limb product
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              if (sd == 6) D6[i] = r[a][lj][i];
              else if (sd < 3) Fa[i] += (uint64_t)r[a][lj][i] << (8 * sd);
              else Fb[i] += (uint64_t)r[a][lj][i] << (8 * (sd - 3));
            }
          }
      }
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        uint32_t acc = mod_reduce((uint64_t)D6[i], mod);
        acc = mod_reduce(((uint64_t)acc << 24) + Fb[i], mod);
        v[h + i] = mod_reduce(((uint64_t)acc << 24) + Fa[i], mod);
      }
    }
  }
}

// C row segments in registers.  load_c reads n consecutive entries of row
// `crow` from column gn (entries at columns >= N read as 0; crow == nullptr:
// a row past M); 16-byte loads where the row and column allow (vec: C and
// its row stride 16-byte aligned).  store_c writes them back.
template <int NV>
__device__ __forceinline__ void load_c(uint32_t (&c)[NV], const uint32_t *crow, int gn, int N,
                                       bool vec) {
  static_assert(NV % 4 == 0, "whole vectors");
#pragma unroll
  for (int j = 0; j < NV / 4; ++j) {
    const int g = gn + 4 * j;
    if (crow != nullptr && vec && g + 3 < N) {
      const uint4 u = *reinterpret_cast<const uint4 *>(crow + g);
      c[4 * j] = u.x;
      c[4 * j + 1] = u.y;
      c[4 * j + 2] = u.z;
      c[4 * j + 3] = u.w;
    } else {
#pragma unroll
      for (int i = 0; i < 4; ++i)
        c[4 * j + i] = (crow != nullptr && g + i < N) ? crow[g + i] : 0u;
    }
  }
}
template <int NV>
__device__ __forceinline__ void store_c(const uint32_t (&c)[NV], uint32_t *crow, int gn, int N,
                                        bool vec) {
  if (crow == nullptr) return;
#pragma unroll
  for (int j = 0; j < NV / 4; ++j) {
    const int g = gn + 4 * j;
    if (vec && g + 3 < N) {
      *reinterpret_cast<uint4 *>(crow + g) = make_uint4(c[4 * j], c[4 * j + 1], c[4 * j + 2], c[4 * j + 3]);
    } else {
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (g + i < N) crow[g + i] = c[4 * j + i];
    }
  }
}

// GF(2) output (OUT = 1, one limb of 0/1 bytes): the accumulator holds the
// integer count of the row/column bit products; its parity is the GF(2)
// product.  The 256 columns of a tile are packed into four 64-bit
// LittleEndian words (bit j of word w = column 64w + j) and combined as
// C <- (beta ? C : 0) XOR (alpha ? A*B : 0); bits of the last word at
// columns >= N keep their old values.
__device__ __forceinline__ void epilogue_gf2(uint32_t tcol, int gm, int gn0, int M, int N,
                                             uint64_t *C, size_t ldc_words, uint32_t alpha,
                                             uint32_t beta, int cbeg, int cend) {
  uint64_t word = 0;
#pragma unroll 1
  for (int c0 = cbeg; c0 < cend; c0 += 16) {
    uint32_t r[16];
    tmem_ld16(tcol + c0, r);
    tmem_ld_wait();
    uint64_t bits = 0;
#pragma unroll
    for (int i = 0; i < 16; ++i) bits |= (uint64_t)(r[i] & 1u) << i;
    word |= bits << (c0 & 63);
    if ((c0 & 63) == 48) {
      const int wcol = gn0 + (c0 & ~63);
      if (gm < M && wcol < N) {
        const int valid = min(64, N - wcol);
        const uint64_t mask = valid == 64 ? ~0ull : ((1ull << valid) - 1ull);
        uint64_t *dst = C + (size_t)gm * ldc_words + (wcol >> 6);
        const bool part = valid < 64;
        const uint64_t old = (beta || part) ? *dst : 0ull;
        const uint64_t v = (beta ? old : 0ull) ^ (alpha ? word : 0ull);
        *dst = (v & mask) | (old & ~mask);
      }
      word = 0;
    }
  }
}

// Epilogue of residue product z for one thread: its row's columns [cbeg, cend)
// of the tile modulo rns_mod(z), as bytes at plane z of C (M rows of `pitch`
// bytes each, pitch the columns rounded up to 16; the columns past N are zero), 32 at a time
// (one sector).
__device__ __forceinline__ void epilogue_rns(uint32_t tcol, int gm, int gn0, int M, uint8_t *C,
                                             size_t pitch, int z, int cbeg, int cend) {
  const uint32_t m = rns_mod(z), mu = 0xFFFFFFFFu / m;  // (the quotient, or one less)
  uint8_t *dst = C + ((size_t)z * M + gm) * pitch + gn0;
#pragma unroll 1
  for (int c0 = cbeg; c0 < cend; c0 += 32) {
    uint32_t r[2][16];
    tmem_ld16(tcol + c0, r[0]);
    tmem_ld16(tcol + c0 + 16, r[1]);
    tmem_ld_wait();
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      uint32_t w[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        w[j] = 0;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          uint32_t v = r[h][4 * j + i];
          v -= __umulhi(v, mu) * m;
          v = min(v, v - m);
          w[j] |= v << (8 * i);
        }
      }
      const int c = c0 + 16 * h;
      if (gm < M && (size_t)(gn0 + c) < pitch)
        *reinterpret_cast<uint4 *>(dst + c) = make_uint4(w[0], w[1], w[2], w[3]);
    }
  }
}

// K blocks [kb0, kb1) of the row tile starting at row m0: all of K, or,
// with per-row ranges kr (row r of A is zero outside columns [kr[r].x,
// kr[r].y) of the whole matrix; kbase = the whole matrix's column of this
// product's K = 0), the blocks covering the union of the tile's rows'
// ranges.  A tile whose rows are zero in all of K keeps one block: its
// product is zero either way.  Warp-collective (the warp's lanes share the
// rows), so every lane of the calling warp runs it.
__device__ __forceinline__ void tile_kblocks(const int2 *kr, int kbase, int m0, int M,
                                             int K, int &kb0, int &kb1) {
  const int nkb = (K + BK - 1) / BK;
  kb0 = 0;
  kb1 = nkb;
  if (kr == nullptr) return;
  int lo = 0x7fffffff, hi = -0x7fffffff;
  const int lane = threadIdx.x & 31;
  for (int r = m0 + lane; r < min(M, m0 + BM); r += 32) {
    const int2 v = kr[r];
    if (v.y > v.x) {
      lo = min(lo, v.x);
      hi = max(hi, v.y);
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    lo = min(lo, __shfl_xor_sync(0xffffffffu, lo, o));
    hi = max(hi, __shfl_xor_sync(0xffffffffu, hi, o));
  }
  if (hi <= lo) {  // no row of the tile has a nonzero anywhere
    kb1 = 1;
    return;
  }
  lo = max(lo - kbase, 0);
  hi = min(hi - kbase, K);
  if (hi <= lo) {  // none inside this product's K range
    kb1 = 1;
    return;
  }
  kb0 = lo / BK;
  kb1 = (hi + BK - 1) / BK;
}

// Epilogue of the Z/p product for one thread (TMEM lane `row` of quadrant
// q, columns cbeg.. of each tile) over this CTA's tiles.  This thread's row
// segment of a tile: W = BN / (EPI / 4) columns from gn0, in blocks of EPB
// columns.
// C's block 0 is loaded before the accumulator is ready (its latency hides
// behind the tile's MMAs), block b + 1 while block b is combined; TMEM is
// released after its last read, before the last block's stores.
template <int L, int T, int MODE>
__device__ __noinline__ void epilogue_tiles(uint32_t tmem, uint64_t *tfull, uint64_t *tempty,
                                               uint32_t *err, uint32_t *C, size_t ldc, int M,
                                               int N, int tiles_m, int tiles_n, int num_tiles,
                                               const Modulus &mod, uint32_t alpha, uint32_t beta,
                                               int row, int q, int cbeg) {
  using Cfg = TcCfg<L, T>;
  constexpr int ACC = Cfg::ACC, BN = Cfg::BN, NMMA = Cfg::NMMA;
  constexpr int W = BN / (Cfg::EPI / 4);
  constexpr int EPB = W < 32 ? W : 32;
  constexpr int NB = W / EPB;
  constexpr bool READC = MODE != EPI_SET;
  const Mod32 m32 = Mod32::make(L < 4 ? (uint32_t)mod.p : 3u);
  const bool vec = ((reinterpret_cast<uintptr_t>(C) & 15u) == 0) && ((ldc & 3u) == 0);
  int it = 0;
  for (int t = blockIdx.x; t < num_tiles; t += gridDim.x, ++it) {
    int mb, nb;
    tile_coords(t, tiles_m, tiles_n, mb, nb);
    const int a = it % ACC;
    const uint32_t aph = (uint32_t)(it / ACC) & 1u;
    const int gm = mb * BM + row;
    const uint32_t tbase = tmem + (uint32_t)(a * L * NMMA) + ((uint32_t)(q * 32) << 16);
    const int gn0 = nb * BN + cbeg;
    uint32_t *crow = gm < M ? C + (size_t)gm * ldc : nullptr;
    uint32_t cb[2][EPB];
    if (READC) load_c<EPB>(cb[0], crow, gn0, N, vec);
    if (!mbar_wait(&tfull[a], aph, err)) return;
    tc_fence_after();
#pragma unroll
    for (int b = 0; b < NB; ++b) {
      uint32_t(&cur)[EPB] = cb[b & 1];
      if (b + 1 < NB && READC) load_c<EPB>(cb[(b + 1) & 1], crow, gn0 + (b + 1) * EPB, N, vec);
#pragma unroll
      for (int h = 0; h < EPB / 16; ++h) {
        uint32_t v[16];
        chunk_products<L, BN, NMMA>(tbase + (uint32_t)(cbeg + b * EPB + 16 * h), v, mod, m32);
#pragma unroll
        for (int i = 0; i < 16; ++i)
          cur[16 * h + i] =
              epi_combine<MODE, (L < 4)>(v[i], READC ? cur[16 * h + i] : 0u, mod, m32, alpha, beta);
      }
      if (b == NB - 1) {
        tc_fence_before();
        mbar_arrive(&tempty[a]);
      }
      store_c<EPB>(cur, crow, gn0 + b * EPB, N, vec);
    }
  }
}

template <int L, int OUT, int T = 0>
__global__ void __launch_bounds__(tc_threads<L, T>(), 1)
    zp_gemm_tc_kernel(const __grid_constant__ CUtensorMap tmA,
                      const __grid_constant__ CUtensorMap tmB, void *Cv,
                      size_t ldc, int M, int N, int K, Modulus mod, uint32_t alpha, uint32_t beta,
                      uint32_t *err, const int2 *kr = nullptr, int kbase = 0) {
  static_assert(OUT == OUT_ZP || L == 1, "the byte outputs take one limb");
  uint32_t *C = static_cast<uint32_t *>(Cv);
  using Cfg = TcCfg<L, T>;
  using Lay = TcLayout<L, T>;
  constexpr int S = Cfg::STAGES, ACC = Cfg::ACC, BN = Cfg::BN, NMMA = Cfg::NMMA;
  constexpr uint32_t IDESC = idesc_u8_s32(BM, NMMA);

  extern __shared__ uint8_t smem_raw[];
  uint32_t base_off = smem_u32(smem_raw);
  uint8_t *smem = smem_raw + ((1024 - (base_off & 1023)) & 1023);
  uint64_t *full = reinterpret_cast<uint64_t *>(smem + Lay::BAR_OFF);
  uint64_t *empty = full + S;
  uint64_t *tfull = empty + S;
  uint64_t *tempty = tfull + ACC;
  uint64_t *done = tempty + ACC;
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(done + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tiles_m = (M + BM - 1) / BM, tiles_n = (N + BN - 1) / BN;
  // OUT_RNS: alpha products, plane z of A times plane z of B
  const int plane_tiles = tiles_m * tiles_n;
  const int num_tiles = OUT == OUT_RNS ? (int)alpha * plane_tiles : plane_tiles;

  if (threadIdx.x == 0) {
    for (int s = 0; s < S; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int a = 0; a < ACC; ++a) {
      mbar_init(&tfull[a], 1);
      mbar_init(&tempty[a], 32 * Cfg::EPI);
    }
    mbar_init(done, 1);
    fence_barrier_init();
    prefetch_tmap(&tmA);
    prefetch_tmap(&tmB);
  }
  if (warp == 1) tmem_alloc(tmem_slot, TMEM_COLS);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  pdl_enter();  // (after the TMEM allocation, see there)

  if (warp == 0) {
    // ------------------------------------------------------------ producer
    // The whole warp walks the tiles (their K ranges are warp-collective);
    // lane 0 issues the loads, and its status is shared each tile so that
    // the lanes leave together.
    uint32_t s = 0, ph = 0;
    uint32_t issued = 0, last_ph[S];
    for (int i = 0; i < S; ++i) last_ph[i] = 0;
    bool ok = true;
    for (int t = blockIdx.x; t < num_tiles; t += gridDim.x) {
      int mb, nb, kb0, kb1;
      const int z = OUT == OUT_RNS ? t / plane_tiles : 0;
      tile_coords(t - z * plane_tiles, tiles_m, tiles_n, mb, nb);
      tile_kblocks(kr, kbase, mb * BM, M, K, kb0, kb1);
      if (lane == 0) {
        for (int kb = kb0; kb < kb1; ++kb) {
          if (!mbar_wait(&empty[s], ph ^ 1, err)) { ok = false; break; }
          uint8_t *sa = smem + s * Lay::STAGE_BYTES;
          uint8_t *sb = sa + Lay::A_BYTES;
          mbar_arrive_expect_tx(&full[s], Lay::STAGE_BYTES);
          tma_load_3d(sa, &tmA, &full[s], kb * BK, mb * BM, z);
          tma_load_3d(sb, &tmB, &full[s], kb * BK, nb * BN, z);
          issued |= 1u << s;
          last_ph[s] = ph;
          if (++s == S) { s = 0; ph ^= 1; }
        }
      }
      if (!__shfl_sync(0xffffffffu, ok ? 1 : 0, 0)) break;
    }
    if (lane == 0 && !ok) {
      // Wait for the loads already in flight before the block may exit.
      for (int i = 0; i < S; ++i)
        if (issued & (1u << i)) mbar_drain(&full[i], last_ph[i], err);
    }
  } else if (warp == 1) {
    // ----------------------------------------------------------- MMA issue
    // As the producer: the warp walks the tiles, lane 0 issues the MMAs.
    uint32_t s = 0, ph = 0;
    int it = 0;
    bool ok = true;
    for (int t = blockIdx.x; t < num_tiles; t += gridDim.x, ++it) {
      int mb, nb, kb0, kb1;
      tile_coords(OUT == OUT_RNS ? t % plane_tiles : t, tiles_m, tiles_n, mb, nb);
      tile_kblocks(kr, kbase, mb * BM, M, K, kb0, kb1);
      if (lane == 0) {
        const int a = it % ACC;
        const uint32_t aph = (uint32_t)(it / ACC) & 1u;
        if (!mbar_wait(&tempty[a], aph ^ 1, err)) ok = false;
        tc_fence_after();
        const uint32_t dbase = tmem + (uint32_t)(a * L * NMMA);
        for (int kb = kb0; kb < kb1 && ok; ++kb) {
          if (!mbar_wait(&full[s], ph, err)) { ok = false; break; }
          tc_fence_after();
          uint8_t *sa = smem + s * Lay::STAGE_BYTES;
          uint8_t *sb = sa + Lay::A_BYTES;
          const uint64_t bd = smem_desc_sw128(sb);
#pragma unroll
          for (int l = 0; l < L; ++l) {
            const uint64_t ad = smem_desc_sw128(sa + l * BM * BK);
#pragma unroll
            for (int kk = 0; kk < BK / 32; ++kk) {
              // +32 bytes of K inside the 128-byte swizzled row = +2 in the
              // descriptor's (address >> 4) field.
              mma_u8(dbase + (uint32_t)(l * NMMA), ad + 2 * kk, bd + 2 * kk, IDESC,
                     (kb != kb0 || kk != 0) ? 1u : 0u);
            }
          }
          mma_commit(&empty[s]);
          if (++s == S) { s = 0; ph ^= 1; }
        }
        if (ok) mma_commit(&tfull[a]);
      }
      if (!__shfl_sync(0xffffffffu, ok ? 1 : 0, 0)) break;
    }
    if (lane == 0) {
      // All MMAs of this thread must finish before TMEM is released.
      mma_commit(done);
      mbar_drain(done, 0, err);
    }
  } else {
    // ------------------------------------------------------------ epilogue
    // EPI / 4 warps per TMEM lane quadrant, each on a BN / (EPI / 4) column
    // part of every tile
    const int q = warp & 3;  // TMEM lane quadrant this warp may access
    const int row = q * 32 + lane;
    const int part = (warp - 2) >> 2;
    const int cbeg = part * (BN / (Cfg::EPI / 4));
    if constexpr (OUT == OUT_ZP) {
      const int emode = beta == 0u ? EPI_SET
                        : (beta == 1u && alpha == 1u) ? EPI_ADD
                        : (beta == 1u && alpha == (uint32_t)mod.p - 1u) ? EPI_SUB
                                                                       : EPI_AXPBY;
#define LELA_EPI(MODE)                                                                          \
  epilogue_tiles<L, T, MODE>(tmem, tfull, tempty, err, C, ldc, M, N, tiles_m, tiles_n, num_tiles, \
                             mod, alpha, beta, row, q, cbeg)
      switch (emode) {
        case EPI_ADD: LELA_EPI(EPI_ADD); break;
        case EPI_SUB: LELA_EPI(EPI_SUB); break;
        case EPI_SET: LELA_EPI(EPI_SET); break;
        default: LELA_EPI(EPI_AXPBY); break;
      }
#undef LELA_EPI
    } else {
      int it = 0;
      for (int t = blockIdx.x; t < num_tiles; t += gridDim.x, ++it) {
        int mb, nb;
        const int z = OUT == OUT_RNS ? t / plane_tiles : 0;
        tile_coords(t - z * plane_tiles, tiles_m, tiles_n, mb, nb);
        const int a = it % ACC;
        const uint32_t aph = (uint32_t)(it / ACC) & 1u;
        const int gm = mb * BM + row;
        const uint32_t tbase = tmem + (uint32_t)(a * L * NMMA) + ((uint32_t)(q * 32) << 16);
        if (!mbar_wait(&tfull[a], aph, err)) break;
        tc_fence_after();
        if constexpr (OUT == OUT_RNS)
          epilogue_rns(tbase, gm, nb * BN, M, static_cast<uint8_t *>(Cv), ldc, z, cbeg,
                       cbeg + BN / (Cfg::EPI / 4));
        else
          epilogue_gf2(tbase, gm, nb * BN, M, N, static_cast<uint64_t *>(Cv), ldc, alpha, beta,
                       cbeg, cbeg + BN / (Cfg::EPI / 4));
        tc_fence_before();
        mbar_arrive(&tempty[a]);
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, TMEM_COLS);
  }
}

// ------------------------------------------------- one-launch tile kernel
// The same tile product without limb planes in memory, for short K and small
// problems, where the split launch and the tensor maps cost more than
// the product: a CTA loads its 128 x K rows of A and K x BN columns of B
// (u32), splits them into limbs on the way to shared memory (K-major, in the
// 128-byte swizzle the tensor cores read), multiplies, and writes its tile.  K
// goes in chunks of 128 through two stages, so a chunk's loads overlap the
// MMAs of the one before.  Every CTA splits its own operands, so it pays only
// where a tile's K is short or the tiles fill about one wave (zp_gemm_pick).
template <int L>
struct DirCfg {
  static constexpr int BN = L == 4 ? 32 : 64, NMMA = L * BN;
  static constexpr int TMEM = L * NMMA;  // 64, 256 or 512 columns
  static constexpr int A_BYTES = L * BM * BK, B_BYTES = NMMA * BK;
  static constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
  static constexpr int smem(int stages) { return stages * STAGE_BYTES + 64 + 1024; }
};
constexpr int DIR_THREADS = 256;

// Byte offset of (row r, K byte k) in a K-major operand with 128-byte rows:
// 16-byte pieces exchanged by the row's number in its group of eight.
__device__ __forceinline__ int sw128(int r, int k) {
  return r * 128 + ((((k >> 4) ^ r) & 7) << 4) + (k & 15);
}
// Limb l of four residues as four bytes.
__device__ __forceinline__ uint32_t limb4(const uint32_t (&v)[4], int l) {
  const uint32_t a = __byte_perm(v[0], v[1], (l | (4 + l) << 4) & 0xff);
  const uint32_t b = __byte_perm(v[2], v[3], (l | (4 + l) << 4) & 0xff);
  return (a & 0xffffu) | (b << 16);
}

template <int L, int MODE>
__device__ __noinline__ void dir_epilogue(uint32_t tmem, uint64_t *done, uint32_t *err, uint32_t *C,
                                          size_t ldc, int M, int N, const Modulus &mod,
                                          uint32_t alpha, uint32_t beta) {
  using Cfg = DirCfg<L>;
  constexpr int W = Cfg::BN / 2;  // two warps per lane quadrant
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, q = warp & 3;
  const int gm = blockIdx.y * BM + q * 32 + lane, cbeg = (warp >> 2) * W;
  const int gn = blockIdx.x * Cfg::BN + cbeg;
  const Mod32 m32 = Mod32::make(L < 4 ? (uint32_t)mod.p : 3u);
  const bool vec = ((reinterpret_cast<uintptr_t>(C) & 15u) == 0) && ((ldc & 3u) == 0);
  uint32_t *crow = gm < M ? C + (size_t)gm * ldc : nullptr;
  uint32_t c[W];
  if (MODE != EPI_SET) load_c<W>(c, crow, gn, N, vec);
  if (!mbar_wait(done, 0, err)) return;
  tc_fence_after();
  const uint32_t tbase = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)cbeg;
#pragma unroll
  for (int h = 0; h < W / 16; ++h) {
    uint32_t v[16];
    chunk_products<L, Cfg::BN, Cfg::NMMA>(tbase + 16 * h, v, mod, m32);
#pragma unroll
    for (int i = 0; i < 16; ++i)
      c[16 * h + i] = epi_combine<MODE, (L < 4)>(v[i], MODE != EPI_SET ? c[16 * h + i] : 0u, mod,
                                                 m32, alpha, beta);
  }
  store_c<W>(c, crow, gn, N, vec);
}

template <int L>
__global__ void __launch_bounds__(DIR_THREADS, L == 4 ? 1 : 2)
    zp_gemm_direct_kernel(const uint32_t *A, size_t lda,
                          const uint32_t *B, size_t ldb, uint32_t *C, size_t ldc,
                          int M, int N, int K, int stages, Modulus mod, uint32_t alpha,
                          uint32_t beta, uint32_t *err) {
  using Cfg = DirCfg<L>;
  constexpr int BN = Cfg::BN;
  constexpr uint32_t IDESC = idesc_u8_s32(BM, Cfg::NMMA);
  extern __shared__ uint8_t smem_raw[];
  uint8_t *smem = smem_raw + ((1024 - (smem_u32(smem_raw) & 1023)) & 1023);
  uint64_t *bars = reinterpret_cast<uint64_t *>(smem + stages * Cfg::STAGE_BYTES);
  uint64_t *freeb = bars, *done = bars + 2;  // stage read by the MMAs; all MMAs done
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(bars + 3);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  if (tid == 0) {
    mbar_init(&freeb[0], 1);
    mbar_init(&freeb[1], 1);
    mbar_init(done, 1);
    fence_barrier_init();
  }
  if (warp == 1) tmem_alloc(tmem_slot, Cfg::TMEM);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  pdl_enter();  // (after the TMEM allocation, see there)
  const bool vecA = ((reinterpret_cast<uintptr_t>(A) & 15u) == 0) && ((lda & 3u) == 0);
  bool ok = true;
  int c = 0;
  for (int k0 = 0; k0 < K; k0 += BK, ++c) {
    const int kc = min(BK, K - k0), kr = (kc + 31) & ~31;  // multiplied: whole MMAs of 32
    const int s = c & 1;
    uint8_t *sa = smem + s * Cfg::STAGE_BYTES, *sb = sa + Cfg::A_BYTES;
    // (two chunks before, this stage's)
    if (c >= 2 && !mbar_wait(&freeb[s], (uint32_t)((c >> 1) - 1) & 1u, err)) ok = false;
    if (__syncthreads_or(!ok)) {
      ok = false;
      break;
    }
    // A: a warp per row, four columns per lane
    constexpr int AU = 8;  // rows in flight per warp
#pragma unroll 1
    for (int r0 = warp * AU; r0 < BM; r0 += 8 * AU) {
      uint32_t v[AU][4];
      const int k = 4 * lane;
#pragma unroll
      for (int u = 0; u < AU; ++u) {
        const int gm = m0 + r0 + u;
        const uint32_t *src = A + (size_t)gm * lda + k0 + k;
        if (gm < M && vecA && k + 3 < kc) {
          const uint4 x = *reinterpret_cast<const uint4 *>(src);
          v[u][0] = x.x;
          v[u][1] = x.y;
          v[u][2] = x.z;
          v[u][3] = x.w;
        } else {
#pragma unroll
          for (int i = 0; i < 4; ++i) v[u][i] = (gm < M && k + i < kc) ? src[i] : 0u;
        }
      }
      if (k < kr)
#pragma unroll
        for (int u = 0; u < AU; ++u)
#pragma unroll
          for (int l = 0; l < L; ++l)
            *reinterpret_cast<uint32_t *>(sa + l * BM * BK + sw128(r0 + u, k)) = limb4(v[u], l);
    }
    // B: lanes on columns, four rows per thread and step
    constexpr int BG = BN / 32, BU = 4;  // column groups; steps in flight
#pragma unroll 1
    for (int e0 = warp * BU; e0 < BG * (kr / 4); e0 += 8 * BU) {
      uint32_t v[BU][4];
#pragma unroll
      for (int u = 0; u < BU; ++u) {
        const int e = e0 + u, k = 4 * (e / BG), n = n0 + (e % BG) * 32 + lane;
#pragma unroll
        for (int i = 0; i < 4; ++i)
          v[u][i] = (n < N && k + i < kc) ? *(B + (size_t)(k0 + k + i) * ldb + n) : 0u;
      }
#pragma unroll
      for (int u = 0; u < BU; ++u) {
        const int e = e0 + u, k = 4 * (e / BG), nr = (e % BG) * 32 + lane;
        if (k < kr)
#pragma unroll
          for (int l = 0; l < L; ++l)
            *reinterpret_cast<uint32_t *>(sb + sw128(l * BN + nr, k)) = limb4(v[u], l);
      }
    }
    fence_proxy_async();
    __syncthreads();
    if (tid == 0) {
      tc_fence_after();
      const uint64_t bd = smem_desc_sw128(sb);
      for (int l = 0; l < L; ++l) {
        const uint64_t ad = smem_desc_sw128(sa + l * BM * BK);
        for (int kk = 0; kk < kr / 32; ++kk)
          mma_u8(tmem + (uint32_t)(l * Cfg::NMMA), ad + 2 * kk, bd + 2 * kk, IDESC,
                 (c != 0 || kk != 0) ? 1u : 0u);
      }
      mma_commit(&freeb[s]);
    }
  }
  if (tid == 0) mma_commit(done);  // (also when a wait ran out: all MMAs end before TMEM goes)
  if (ok) {
    const int emode = beta == 0u ? EPI_SET
                      : (beta == 1u && alpha == 1u) ? EPI_ADD
                      : (beta == 1u && alpha == (uint32_t)mod.p - 1u) ? EPI_SUB
                                                                     : EPI_AXPBY;
    switch (emode) {
      case EPI_ADD: dir_epilogue<L, EPI_ADD>(tmem, done, err, C, ldc, M, N, mod, alpha, beta); break;
      case EPI_SUB: dir_epilogue<L, EPI_SUB>(tmem, done, err, C, ldc, M, N, mod, alpha, beta); break;
      case EPI_SET: dir_epilogue<L, EPI_SET>(tmem, done, err, C, ldc, M, N, mod, alpha, beta); break;
      default: dir_epilogue<L, EPI_AXPBY>(tmem, done, err, C, ldc, M, N, mod, alpha, beta); break;
    }
  }
  if (tid == 0) mbar_drain(done, 0, err);
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, Cfg::TMEM);
  }
}

// ------------------------------------------------ residues of four limbs' work
//
// Four limbs take sixteen byte products per entry product.  Where the planes' extra
// passes cost less, the product x = sum a b of the integers a, b < p, x < (p - 1)^2
// K, is instead formed modulo n pairwise coprime moduli m_i <= 256 with P = prod
// m_i > 2 x (n = 6 at p = 2^17, 10 at p = 2^31 and K = 4096): n one-limb products
// of residue bytes, which the tensor-core kernel's epilogue reduces modulo m_i to
// bytes again.  4096^3 at p = 2^31 - 1: 1015 -> 793 us a call on new operands (splits
// 140, products 455 at 3.0 Pop/s, rns_combine_kernel 80), 941 -> 680 for a few in a row
// on the same ones.  Row blocks whose planes stay in L2 are no
// faster (2048 rows 700 us, 1024 748, all 690).  A's residues carry the factor (P /
// m_i)^-1 mod m_i, so the bytes are y_i with
//     x = sum_i y_i (P / m_i) - t P,   t = floor(sum_i y_i / m_i),
// and rns_combine_kernel takes that sum modulo p.  Exact: x / P < 1/2, so t is
// floor(1/4 + sum y_i F_i / 2^15) with F_i = round(2^15 / m_i), whose error is
// at most 11 * 255 / 2 / 2^15 < 0.05.
// The bytes a split writes to plane l for four consecutive entries: limb l ...
template <int L>
struct LimbBytes {
  static constexpr int MAX = L;
  __device__ __forceinline__ constexpr int count() const { return L; }
  __device__ __forceinline__ uint32_t in(uint32_t x, uint32_t) const { return x; }
  __device__ __forceinline__ uint32_t word(const uint32_t (&v)[4], int l) const {
    uint32_t w = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) w |= ((v[i] >> (8 * l)) & 0xFFu) << (8 * i);
    return w;
  }
};
// ... or f_l x mod m_l: the bytes of x times those of coef (2^8b f_l mod m_l, at
// byte b) sum to r < 2^18.  m = 256: its low byte.  Odd m: in floats, four
// instructions at the full rate where the integer multiply-high and multiply go at
// less (the splits are issue-bound: 4096^2 entries, ten moduli, A's 66 us
// against 70, the limbs' 25).  2^23 + r is a float read from the bits; (r - (m - 1) / 2) / m
// rounds to floor(r / m), being at least 1 / 2m > 2^-9 from a half-integer with an error
// below 2^-13; 2^23 + r - q m is exact.
struct ResidueBytes {
  static constexpr int MAX = RNS_MAX;
  int n;
  uint32_t coef[RNS_MAX];
  __device__ __forceinline__ int count() const { return n; }
  __device__ __forceinline__ uint32_t in(uint32_t x, uint32_t p) const { return x < p ? x : x % p; }
  __device__ __forceinline__ uint32_t word(const uint32_t (&v)[4], int l) const {
    const int m = (int)rns_mod(l);
    uint32_t r[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      r[i] = __dp4a(v[i], coef[l], 0x4B000000u);
      if (m != 256) {
        const float f = __uint_as_float(r[i]);  // 2^23 + r
        const float q = fmaf(f - (8388608.0f + (m - 1) / 2), 1.0f / m, 12582912.0f) - 12582912.0f;
        r[i] = __float_as_uint(fmaf(q, (float)-m, f));
      }
    }
    const uint32_t w = __byte_perm(__byte_perm(r[0], r[1], 0x0040), __byte_perm(r[2], r[3], 0x0040), 0x5410);
    return w;
  }
};

// ------------------------------------------------------------ limb splits
// A (M x kc, row stride lda, elements T) -> L planes of bytes, row pitch Kp,
// `plane` bytes apart.  Bound by
// HBM (8192^2 of u32: 69 us, 402 MB); lanes on consecutive groups of four
// columns, a row per warp, so no index division; rows of at most 64 columns share a
// warp, as many as fill it (us a product, a row per warp / shared: p = 65521 262144 x 16 x
// 32 79 / 58, 200000 x 64 x 64 72 / 62; kernels of their own, since both in one
// slowed wider rows by up to 2 %).  part: 0 all columns; 1 (2) only those left
// (right) of the row's diagonal block of nb rows.
constexpr int SPLIT_ROWS = 8;  // warps per CTA
// The NARROW instances below, for rows enough to fill the SMs with fewer CTAs (8192 x 8192 x
// 64 at four limbs 605 us, narrow 610).
static bool split_narrow(int M, int kc) { return kc <= 64 && M >= 16384; }
// log2 of the lanes that a row of kc columns takes
__host__ __device__ __forceinline__ int split_lanes(int kc) {
  int l = 1;
  while (l < 5 && (4 << l) < kc) ++l;
  return l;
}
template <class W, class T, bool NARROW>
__device__ __forceinline__ void split_rows(const T *A, size_t lda, int M, int kc, uint32_t p,
                                           uint8_t *out, size_t Kp, size_t plane, int part, int nb,
                                           const W &planes, int bx, int by, int gx, int gy) {
  const int lb = NARROW ? split_lanes(kc) : 5, rows = SPLIT_ROWS * (32 >> lb);  // rows per CTA
  const int tx = threadIdx.x & ((1 << lb) - 1), ty = threadIdx.x >> lb;
  for (int r = by * rows + ty; r < M; r += gy * rows) {
    const T *src = A + (size_t)r * lda;
    uint8_t *dst = out + (size_t)r * Kp;
    const int kb = part == 2 ? min(kc, (r / nb + 1) * nb) : 0;
    const int ke = part == 1 ? min(kc, r / nb * nb) : kc;
    constexpr int U = 2;  // groups in flight
    const int step = gx << lb;
    for (int q = (kb >> 2) + (bx << lb) + tx; 4 * q < ke; q += U * step) {
      uint32_t v[U][4];
#pragma unroll
      for (int u = 0; u < U; ++u)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int k = 4 * (q + u * step) + i;
          v[u][i] = 4 * (q + u * step) < ke && k < kc ? planes.in(Rep<T>::in(src[k], p), p) : 0u;
        }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int k = 4 * (q + u * step);
        if (k >= ke) break;
#pragma unroll
        for (int l = 0; l < W::MAX; ++l)
          if (l < planes.count())
            *reinterpret_cast<uint32_t *>(dst + l * plane + k) = planes.word(v[u], l);
      }
    }
  }
}
template <class W, class T, bool NARROW>
__global__ void __launch_bounds__(32 * SPLIT_ROWS)
    split_rows_kernel(const T *A, size_t lda, int M, int kc, uint32_t p,
                      uint8_t *out, size_t Kp, size_t plane, int part, int nb, const W planes) {
  pdl_enter();
  split_rows<W, T, NARROW>(A, lda, M, kc, p, out, Kp, plane, part, nb, planes, blockIdx.x,
                           blockIdx.y, gridDim.x, gridDim.y);
}
static dim3 split_rows_grid(int num_sms, int M, int kc) {
  // one pass a warp up to 16 CTAs an SM, then more
  const int rows = SPLIT_ROWS * (split_narrow(M, kc) ? 32 >> split_lanes(kc) : 1);
  const int gy = std::min((M + rows - 1) / rows, num_sms * 16);
  return dim3(std::max(1, std::min(((kc + 3) / 4 + 31) / 32, num_sms * 16 / gy)), gy);
}

// B (kc x N, row stride ldb, elements T) -> L planes of N rows of kout <= Kp
// bytes (row pitch Kp, `plane` bytes apart; transposed), through a shared-memory tile of 64 k
// x NT columns (128 bytes of a row of the narrow types, 32 elements of the others).
template <class T>
constexpr int split_cols_nt() {
  return sizeof(T) < 4 ? 128 / (int)sizeof(T) : 32;
}
template <class W, class T>
__device__ __forceinline__ void split_cols(const T *B, size_t ldb, int kc, int N, uint32_t p,
                                           uint8_t *out, size_t Kp, size_t plane, int kout,
                                           const W &planes, int bx, int by) {
  using R = typename Rep<T>::Packed;
  constexpr int NT = split_cols_nt<T>();
  __shared__ R tile[64][NT + 4 / sizeof(R)];
  const int n0 = bx * NT, k0 = by * 64;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int k = k0 + ty + 8 * i;
#pragma unroll
    for (int u = 0; u < NT / 32; ++u) {
      const int n = n0 + tx + 32 * u;
      tile[ty + 8 * i][tx + 32 * u] =
          (k < kc && n < N) ? (R)Rep<T>::in(*(B + (size_t)k * ldb + n), p) : (R)0;
    }
  }
  __syncthreads();
#pragma unroll
  for (int j = 0; j < NT / 16; ++j) {
    const int w = threadIdx.x + 256 * j;
    const int n = w >> 4, kw = (w & 15) * 4;
    const int gn = n0 + n, gk = k0 + kw;
    if (gn < N && gk < kout) {
      uint32_t v[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) v[i] = planes.in(tile[kw + i][n], p);
#pragma unroll
      for (int l = 0; l < W::MAX; ++l)
        if (l < planes.count())
          *reinterpret_cast<uint32_t *>(out + l * plane + (size_t)gn * Kp + gk) = planes.word(v, l);
    }
  }
}
template <class W, class T>
__global__ void __launch_bounds__(256)
    split_cols_kernel(const T *B, size_t ldb, int kc, int N, uint32_t p,
                      uint8_t *out, size_t Kp, size_t plane, int kout, const W planes) {
  pdl_enter();
  split_cols<W, T>(B, ldb, kc, N, p, out, Kp, plane, kout, planes, blockIdx.x, blockIdx.y);
}
template <class T>
static dim3 split_cols_grid(int N, int Kp) {
  return dim3((N + split_cols_nt<T>() - 1) / split_cols_nt<T>(), (Kp + 63) / 64);
}

// Both operands' planes in one launch, A's (M x kc, planes from out_a, rows Kp
// apart) in the first gax * gay CTAs: a product of few tiles waits for each launch (512^3
// 17.6 us a call, 20.4 with two launches).
template <class W, class T, bool NARROW>
__global__ void __launch_bounds__(256)
    split_both_kernel(const T *A, size_t lda, const T *B, size_t ldb, int M, int N, int kc,
                      uint32_t p, uint8_t *out_a, uint8_t *out_b, int Kp, int gax, int gay, int gbx,
                      const W wa, const W wb) {
  static_assert(32 * SPLIT_ROWS == 256, "one block size");
  pdl_enter();
  const int b = blockIdx.x, na = gax * gay;
  if (b < na)
    split_rows<W, T, NARROW>(A, lda, M, kc, p, out_a, (size_t)Kp, (size_t)M * Kp, 0, 1, wa, b % gax,
                             b / gax, gax, gay);
  else
    split_cols<W, T>(B, ldb, kc, N, p, out_b, (size_t)Kp, (size_t)N * Kp, Kp, wb, (b - na) % gbx,
                     (b - na) / gbx);
}
template <class W, class T>
static void launch_split(bool early, int num_sms, cudaStream_t s, const T *A, size_t lda, const T *B,
                         size_t ldb, int M, int N, int kc, uint32_t p, uint8_t *out_a, uint8_t *out_b,
                         int Kp, const W &wa, const W &wb) {
  const dim3 ga = split_rows_grid(num_sms, M, kc), gb = split_cols_grid<T>(N, Kp);
  auto kern = split_narrow(M, kc) ? split_both_kernel<W, T, true> : split_both_kernel<W, T, false>;
  pdl_launch_if(early, kern, ga.x * ga.y + gb.x * gb.y, 256, 0, s, A, lda, B, ldb, M, N, kc, p, out_a,
                out_b, Kp, (int)ga.x, (int)ga.y, (int)gb.x, wa, wb);
}

// ------------------------------------------------- residues back to Z/p
// Weights of rns_combine_kernel: byte b of W[g][b] at position i is byte b of (P /
// m_(4g+i)) mod p, F[g] the F_i, neg = -P mod p.
struct RnsWeights {
  int n;
  uint32_t W[3][4], F[3], neg;
};
// C <- alpha x + beta C from the n residue planes Y (M rows of `pitch` bytes).
// 4096^2 entries and n = 10 take 80 us: 300 MB, issue at 68 %.
// Four columns a thread: the planes' words are transposed to words of one column and
// multiplied bytewise (5 dp4a per four residues), S = sum of y_i ((P / m_i) mod p)
// < 11 * 255 * 2^32 and t neg < 2^36 together, and one reduction.
template <int MODE>
__global__ void __launch_bounds__(256)
    rns_combine_kernel(const uint8_t *Y, size_t pitch, uint32_t *C, size_t ldc, int M, int N,
                       const RnsWeights rw, Modulus mod, uint32_t alpha, uint32_t beta) {
  pdl_enter();
  const int n = 4 * (blockIdx.x * 32 + threadIdx.x);
  if (n >= N) return;
  const bool vec = ((reinterpret_cast<uintptr_t>(C) & 15u) == 0) && ((ldc & 3u) == 0);
  const size_t plane = (size_t)M * pitch;
  for (int r = blockIdx.y * 8 + threadIdx.y; r < M; r += gridDim.y * 8) {
    const uint8_t *src = Y + (size_t)r * pitch + n;
    uint32_t y[12];
#pragma unroll
    for (int i = 0; i < 12; ++i)
      y[i] = i < RNS_MAX && i < rw.n ? *reinterpret_cast<const uint32_t *>(src + i * plane) : 0u;
    uint32_t *crow = C + (size_t)r * ldc;
    uint32_t c[4];
    if (MODE != EPI_SET) load_c<4>(c, crow, n, N, vec);
    uint32_t s[4][4], t[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      t[j] = 1u << 13;
#pragma unroll
      for (int b = 0; b < 4; ++b) s[j][b] = 0;
    }
#pragma unroll
    for (int g = 0; g < 3; ++g) {
      const uint32_t lo01 = __byte_perm(y[4 * g], y[4 * g + 1], 0x5140);
      const uint32_t lo23 = __byte_perm(y[4 * g + 2], y[4 * g + 3], 0x5140);
      const uint32_t hi01 = __byte_perm(y[4 * g], y[4 * g + 1], 0x7362);
      const uint32_t hi23 = __byte_perm(y[4 * g + 2], y[4 * g + 3], 0x7362);
      const uint32_t col[4] = {__byte_perm(lo01, lo23, 0x5410), __byte_perm(lo01, lo23, 0x7632),
                               __byte_perm(hi01, hi23, 0x5410), __byte_perm(hi01, hi23, 0x7632)};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        t[j] = __dp4a(col[j], rw.F[g], t[j]);
#pragma unroll
        for (int b = 0; b < 4; ++b) s[j][b] = __dp4a(col[j], rw.W[g][b], s[j][b]);
      }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const uint64_t S = s[j][0] + ((uint64_t)s[j][1] << 8) + ((uint64_t)s[j][2] << 16) +
                         ((uint64_t)s[j][3] << 24) + (uint64_t)(t[j] >> 15) * rw.neg;
      c[j] = epi_combine<MODE, false>(mod_reduce(S, mod), MODE != EPI_SET ? c[j] : 0u, mod, Mod32(),
                                      alpha, beta);
    }
    store_c<4>(c, crow, n, N, vec);
  }
}

// ------------------------------------------------------------ plain gemm
constexpr int PT = 64, PK = 32;

__global__ void __launch_bounds__(256)
    zp_gemm_plain_kernel(const uint32_t *__restrict__ A, size_t lda,
                         const uint32_t *__restrict__ B, size_t ldb, uint32_t *__restrict__ C,
                         size_t ldc, int M, int N, int K, Modulus mod, uint32_t two64,
                         uint32_t alpha, uint32_t beta) {
  __shared__ uint32_t As[PK][PT + 1];
  __shared__ uint32_t Bs[PK][PT + 1];
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  const int m0 = blockIdx.y * PT, n0 = blockIdx.x * PT;
  uint64_t acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0;

  for (int k0 = 0; k0 < K; k0 += PK) {
#pragma unroll
    for (int e = 0; e < (PT * PK) / 256; ++e) {
      int idx = threadIdx.x + 256 * e;
      int r = idx / PK, kk = idx % PK;  // A tile: 64 rows x 32 k
      int gm = m0 + r, gk = k0 + kk;
      As[kk][r] = (gm < M && gk < K) ? __ldg(A + (size_t)gm * lda + gk) : 0u;
      int kr = idx / PT, c = idx % PT;  // B tile: 32 k x 64 cols
      int gk2 = k0 + kr, gn = n0 + c;
      Bs[kr][c] = (gk2 < K && gn < N) ? __ldg(B + (size_t)gk2 * ldb + gn) : 0u;
    }
    __syncthreads();
#pragma unroll 4
    for (int kk = 0; kk < PK; ++kk) {
      uint32_t a[4], b[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) a[i] = As[kk][ty + 16 * i];
#pragma unroll
      for (int j = 0; j < 4; ++j) b[j] = Bs[kk][tx + 16 * j];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          uint64_t t = (uint64_t)a[i] * b[j];
          uint64_t s = acc[i][j] + t;
          acc[i][j] = (s < t) ? s + two64 : s;
        }
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    int gm = m0 + ty + 16 * i;
    if (gm >= M) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      int gn = n0 + tx + 16 * j;
      if (gn >= N) continue;
      uint32_t d = mod_reduce(acc[i][j], mod);
      uint32_t c = beta ? C[(size_t)gm * ldc + gn] : 0u;
      C[(size_t)gm * ldc + gn] = mod_axpby(alpha, d, beta, c, mod);
    }
  }
}

// Same tiling as the plain kernel.  NOWRAP (p < 2^28): unchecked sums,
// reduced modulo p after every 256 terms (256 (p-1)^2 < 2^64).
template <bool NOWRAP>
__global__ void __launch_bounds__(256)
    zp_gemm_smallk_kernel(const uint32_t *A, size_t lda, const uint32_t *B, size_t ldb, uint32_t *C,
                          size_t ldc, int M, int N, int K, Modulus mod, uint32_t two64,
                          uint32_t alpha, uint32_t beta) {
  pdl_enter();
  __shared__ uint32_t As[PK][PT + 1];
  __shared__ uint32_t Bs[PK][PT + 1];
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  const int m0 = blockIdx.y * PT, n0 = blockIdx.x * PT;
  uint64_t acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0;

  for (int k0 = 0; k0 < K; k0 += PK) {
#pragma unroll
    for (int e = 0; e < (PT * PK) / 256; ++e) {
      int idx = threadIdx.x + 256 * e;
      int r = idx / PK, kk = idx % PK;
      int gm = m0 + r, gk = k0 + kk;
      As[kk][r] = (gm < M && gk < K) ? A[(size_t)gm * lda + gk] : 0u;
      int kr = idx / PT, c = idx % PT;
      int gk2 = k0 + kr, gn = n0 + c;
      Bs[kr][c] = (gk2 < K && gn < N) ? B[(size_t)gk2 * ldb + gn] : 0u;
    }
    __syncthreads();
#pragma unroll 8
    for (int kk = 0; kk < PK; ++kk) {
      uint32_t a[4], b[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) a[i] = As[kk][ty + 16 * i];
#pragma unroll
      for (int j = 0; j < 4; ++j) b[j] = Bs[kk][tx + 16 * j];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const uint64_t t = (uint64_t)a[i] * b[j];
          if (NOWRAP) {
            acc[i][j] += t;
          } else {
            const uint64_t s = acc[i][j] + t;
            acc[i][j] = (s < t) ? s + two64 : s;
          }
        }
    }
    if (NOWRAP && ((k0 / PK) & 7) == 7)
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = mod_reduce(acc[i][j], mod);
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    int gm = m0 + ty + 16 * i;
    if (gm >= M) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      int gn = n0 + tx + 16 * j;
      if (gn >= N) continue;
      uint32_t d = mod_reduce(acc[i][j], mod);
      uint32_t c = beta ? C[(size_t)gm * ldc + gn] : 0u;
      C[(size_t)gm * ldc + gn] = mod_axpby(alpha, d, beta, c, mod);
    }
  }
}

// Scale C <- beta * C (mod p), used when K = 0 or alpha = 0.
__global__ void zp_scale_kernel(uint32_t *C, size_t ldc, int M, int N, Modulus mod,
                                uint32_t beta) {
  const size_t total = (size_t)M * N;
  for (size_t idx = blockIdx.x * (size_t)blockDim.x + threadIdx.x; idx < total;
       idx += (size_t)gridDim.x * blockDim.x) {
    size_t r = idx / N, c = idx % N;
    uint32_t *x = C + r * ldc + c;
    *x = beta ? mod_mul(*x, beta, mod) : 0u;
  }
}

// ------------------------------------------------------------------ host
static uint32_t host_two64(uint32_t p) {
  uint64_t t = 2;
  for (int i = 0; i < 6; ++i) t = (t * t) % p;
  return (uint32_t)t;
}

int zp_limbs_for(uint32_t p) { return p <= 256u ? 1 : (p <= 65536u ? 2 : 4); }

static int encode_3d(Ctx *c, CUtensorMap *tm, void *base, uint64_t d0, uint64_t d1, uint64_t d2,
                     uint64_t stride1, uint64_t stride2, uint32_t b0, uint32_t b1, uint32_t b2) {
  auto fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(c->encode_tiled);
  if (!fn) return ctx_fail(c, ST_CUDA, "cuTensorMapEncodeTiled unavailable");
  cuuint64_t dims[3] = {d0, d1, d2};
  cuuint64_t strides[2] = {stride1, stride2};
  cuuint32_t box[3] = {b0, b1, b2};
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = fn(tm, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, base, dims, strides, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    char msg[160];
    snprintf(msg, sizeof msg, "cuTensorMapEncodeTiled failed (%d) dims %llu %llu %llu", (int)r,
             (unsigned long long)d0, (unsigned long long)d1, (unsigned long long)d2);
    return ctx_fail(c, ST_CUDA, msg);
  }
  return ST_OK;
}

template <int L, int T = 0>
static int tc_attr(Ctx *c) {
  return ctx_smem_attr(c, (const void *)zp_gemm_tc_kernel<L, OUT_ZP, T>, TcLayout<L, T>::SMEM,
                       "cudaFuncSetAttribute(zp_gemm_tc)");
}

template <int L, int T, class E = uint32_t>
static int launch_tc(Ctx *c, int M, int N, int K, const Modulus &mod, uint32_t alpha,
                     const E *A, size_t lda, const E *B, size_t ldb, uint32_t beta,
                     uint32_t *C, size_t ldc, uint8_t *ws, const int2 *kr, int kbase) {
  using Cfg = TcCfg<L, T>;
  using Lay = TcLayout<L, T>;
  if (int st = tc_attr<L, T>(c)) return st;
  const int tiles = ((M + BM - 1) / BM) * ((N + Cfg::BN - 1) / Cfg::BN);
  // An early launch saves a few us, which long products do not need; 8192^3
  // under the power cap took 1845 us launched early and 1783 not.
  const bool early = (double)M * N * K < 1e11;
  uint32_t b = beta;
  for (int k0 = 0; k0 < K; k0 += ZP_KCHUNK) {
    const int kc = std::min(ZP_KCHUNK, K - k0);
    const int Kp = (kc + 15) & ~15;
    uint8_t *Al = ws;
    uint8_t *Bl = ws + (size_t)L * M * Kp;
    {
      const uint32_t p = (uint32_t)mod.p;
      int pi = prof_begin(c, "zp_split");
      launch_split(early, c->num_sms, c->stream, A + k0, lda, B + (size_t)k0 * ldb, ldb, M, N, kc, p,
                   Al, Bl, Kp, LimbBytes<L>{}, LimbBytes<L>{});
      prof_end(c, pi);
      ctx_launched(c);
    }
    CUtensorMap tmA, tmB;
    int st = encode_3d(c, &tmA, Al, (uint64_t)kc, (uint64_t)M, L, (uint64_t)Kp,
                       (uint64_t)M * Kp, BK, BM, L);
    if (st) return st;
    st = encode_3d(c, &tmB, Bl, (uint64_t)kc, (uint64_t)N, L, (uint64_t)Kp, (uint64_t)N * Kp, BK,
                   Cfg::BN, L);
    if (st) return st;
    const int grid = std::min(tiles, c->num_sms);
    int pi = prof_begin(c, "zp_gemm_tc");
    pdl_launch_if(early, zp_gemm_tc_kernel<L, OUT_ZP, T>, grid, tc_threads<L, T>(), Lay::SMEM, c->stream,
               tmA, tmB, C, ldc, M, N, kc, mod, alpha, b, c->dstatus, kr, kbase + k0);
    prof_end(c, pi);
    ctx_launched(c);
    b = 1;
  }
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return ctx_cuda(c, e, "zp_gemm_tc launch");
  return ST_OK;
}

// The residue split of a product of K terms modulo p: the moduli n (0: not
// enough of them), A's and B's coefficients and the weights.
static int rns_setup(uint32_t p, int K, ResidueBytes &ra, ResidueBytes &rb, RnsWeights &rw) {
  const unsigned __int128 need = 2 * (unsigned __int128)((uint64_t)(p - 1) * (p - 1)) * (unsigned)K;
  unsigned __int128 P = 1;
  int n = 0;
  while (n < RNS_MAX && P <= need) P *= rns_mod(n++);
  if (P <= need) return 0;
  ra = {};
  rb = {};
  rw = {};
  ra.n = rb.n = rw.n = n;
  for (int i = 0; i < n; ++i) {
    const uint32_t m = rns_mod(i);
    const unsigned __int128 q = P / m;
    uint32_t f = 1;  // (P / m)^-1 mod m
    while ((uint32_t)(q % m) * f % m != 1) ++f;
    const uint32_t w = (uint32_t)(q % p);
    for (int b = 0; b < 4; ++b) {
      const uint32_t e = (uint32_t)((1ull << (8 * b)) % m);
      rb.coef[i] |= e << (8 * b);
      ra.coef[i] |= e * f % m << (8 * b);
      rw.W[i / 4][b] |= (w >> (8 * b) & 0xFFu) << (8 * (i % 4));
    }
    rw.F[i / 4] |= (((1u << 15) + m / 2) / m) << (8 * (i % 4));
  }
  rw.neg = p - (uint32_t)(P % p);
  return n;
}

// The product by residues in blocks of `rows` rows of A and C (B's planes are
// made once).
template <class E>
static int launch_rns(Ctx *c, int M, int N, int K, int rows, const Modulus &mod, uint32_t alpha,
                      const E *A, size_t lda, const E *B, size_t ldb, uint32_t beta, uint32_t *C,
                      size_t ldc, uint8_t *ws, const ResidueBytes &ra, const ResidueBytes &rb,
                      const RnsWeights &rw) {
  using Lay = TcLayout<1, 0>;
  constexpr int BN = TcCfg<1, 0>::BN;
  if (int st = ctx_smem_attr(c, (const void *)zp_gemm_tc_kernel<1, OUT_RNS>, Lay::SMEM,
                             "cudaFuncSetAttribute(zp_gemm_tc)"))
    return st;
  const int n = rw.n;
  const size_t Kp = ((size_t)K + 15) & ~(size_t)15, Np = ((size_t)N + 15) & ~(size_t)15;
  const uint32_t p = (uint32_t)mod.p;
  uint8_t *Bl = ws, *Al = Bl + (size_t)n * N * Kp, *Y = Al + (size_t)n * rows * Kp;
  const bool early = (double)M * N * K < 1e11;  // (as launch_tc)
  int pi = prof_begin(c, "zp_split");
  pdl_launch_if(early, split_cols_kernel<ResidueBytes, E>, split_cols_grid<E>(N, (int)Kp), 256, 0,
                c->stream, B, ldb, K, N, p, Bl, Kp, (size_t)N * Kp, (int)Kp, rb);
  prof_end(c, pi);
  ctx_launched(c);
  CUtensorMap tmA, tmB;
  if (int st = encode_3d(c, &tmB, Bl, (uint64_t)K, (uint64_t)N, n, Kp, (uint64_t)N * Kp, BK, BN, 1))
    return st;
  for (int r0 = 0; r0 < M; r0 += rows) {
    const int m = std::min(rows, M - r0);
    uint32_t *Cr = C + (size_t)r0 * ldc;
    pi = prof_begin(c, "zp_split");
    pdl_launch_if(early, split_rows_kernel<ResidueBytes, E, false>, split_rows_grid(c->num_sms, m, K),
                  32 * SPLIT_ROWS, 0, c->stream, A + (size_t)r0 * lda, lda, m, K, p, Al, Kp,
                  (size_t)m * Kp, 0, 1, ra);
    prof_end(c, pi);
    if (int st = encode_3d(c, &tmA, Al, (uint64_t)K, (uint64_t)m, n, Kp, (uint64_t)m * Kp, BK, BM, 1))
      return st;
    const long long tiles = (long long)n * ((m + BM - 1) / BM) * ((N + BN - 1) / BN);
    pi = prof_begin(c, "zp_gemm_tc");
    pdl_launch_if(early, zp_gemm_tc_kernel<1, OUT_RNS>, (int)std::min<long long>(tiles, c->num_sms),
                  tc_threads<1, 0>(), Lay::SMEM, c->stream, tmA, tmB, Y, Np, m, N, K, mod,
                  (uint32_t)n, 0u, c->dstatus, nullptr, 0);
    prof_end(c, pi);
    pi = prof_begin(c, "zp_combine");
    const dim3 grid((N + 127) / 128, std::min((m + 7) / 8, 65535));
#define LELA_RC(MODE)                                                                           \
  pdl_launch_if(early, rns_combine_kernel<MODE>, grid, dim3(32, 8), 0, c->stream, Y, Np, Cr, ldc, \
                m, N, rw, mod, alpha, beta)
    if (beta == 0u) LELA_RC(EPI_SET);
    else if (beta == 1u && alpha == 1u) LELA_RC(EPI_ADD);
    else if (beta == 1u && alpha == p - 1u) LELA_RC(EPI_SUB);
    else LELA_RC(EPI_AXPBY);
#undef LELA_RC
    prof_end(c, pi);
    ctx_launched(c, 3);
  }
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? ST_OK : ctx_cuda(c, e, "zp_gemm_tc launch");
}

// Whether a four-limb product goes by n residues.  They save 16 - n of 16 byte
// products and cost planes n / 4 times as large and a pass over n bytes per entry of C.
// Measured on the B200 (us per call, a few in a row on the same operands, limbs / residues; p = 2^16 + 1 has n =
// 6, 2^24 - 3 8, 2^31 - 1 and 2^32 - 5 10): 4096^3 940 / 461, 576 and 693; 8192^3
// 7062 / 2763, 7071 / 3559, 7398 / 4560; 2048^3 160 / 115, 129 and 150; 4096^2 x 512
// 238 / 176, 201 and 226.  At n <= 8 down to 1024^2 x 2048 70 / 63 and 68, 512 x 8192 x
// 512 89 / 84 and 87, while 1024^3 56 / 58 and 768^3 44 / 47; at n = 10 1536^3 95 / 91, 2048^2 x
// 512 91 / 90, while 1024^2 x 8192 180 / 188, 512 x 8192 x 512 89 / 96, 1024^3 56 / 64.
static bool rns_pays(int M, int N, int K, int n) {
  return std::min(M, N) >= (n <= 8 ? 512 : 1536) && K >= 512 &&
         (double)M * N * K >= 2147483648.0;
}
constexpr size_t RNS_MAX_BYTES = ZP_RESIDUE_MAX_BYTES;
constexpr int RNS_MIN_ROWS = 2048;

// Whether the matrices X (rx rows of cx entries) and C share an entry.  Views of
// one matrix (equal strides) are compared as rectangles of it, others by their
// whole address ranges.
template <class E>
static bool share_entries(const E *X, size_t ldx, int rx, int cx, const uint32_t *C, size_t ldc,
                          int rc, int cc) {
  const uintptr_t x0 = reinterpret_cast<uintptr_t>(X), c0 = reinterpret_cast<uintptr_t>(C);
  const uintptr_t x1 = x0 + ((size_t)(rx - 1) * ldx + cx) * sizeof(E);
  const uintptr_t c1 = c0 + ((size_t)(rc - 1) * ldc + cc) * sizeof(uint32_t);
  if (x1 <= c0 || c1 <= x0) return false;
  if (sizeof(E) != sizeof(uint32_t) || ldx != ldc || (c0 - x0) % sizeof(uint32_t)) return true;
  // C starts q rows and s columns after X
  const long long ld = (long long)ldx, off = (long long)(c0 - x0) / (long long)sizeof(uint32_t);
  const long long q = off >= 0 ? off / ld : -((ld - 1 - off) / ld), s = off - q * ld;
  if (s < cx && q < rx && q + rc > 0) return true;
  return s + cc > ld && q + 1 < rx && q + 1 + rc > 0;  // its columns past the row's end
}

// The product by residues where shape and modulus favour it and its planes can be
// had: within RNS_MAX_BYTES in blocks of at least RNS_MIN_ROWS rows, and in a workspace
// that may grow to hold them (ctx_planes_fit: not inside a stream capture, not
// where little memory is left).  done says whether it was launched (else the limb
// planes, which take less room, serve).
template <class E>
static int rns_try(Ctx *c, int M, int N, int K, uint32_t p, uint32_t alpha, const E *A, size_t lda,
                   const E *B, size_t ldb, uint32_t beta, uint32_t *C, size_t ldc, bool &done) {
  done = false;
  // (shapes that no modulus sends here go before the moduli are set up, which takes
  // the host 2 to 5 us)
  if (zp_limbs_for(p) != 4 || K > ZP_KCHUNK || !rns_pays(M, N, K, 0)) return ST_OK;
  ResidueBytes ra, rb;
  RnsWeights rw;
  const int n = rns_setup(p, K, ra, rb, rw);
  if (n == 0 || !rns_pays(M, N, K, n)) return ST_OK;
  const size_t Kp = ((size_t)K + 15) & ~(size_t)15, Np = ((size_t)N + 15) & ~(size_t)15;
  const size_t fixed = (size_t)n * N * Kp, per_row = (size_t)n * (Kp + Np);
  if (fixed >= RNS_MAX_BYTES) return ST_OK;
  const size_t most = (RNS_MAX_BYTES - fixed) / per_row;
  int rows = M;
  if ((size_t)M > most) {
    if (most < RNS_MIN_ROWS) return ST_OK;
    if (share_entries(A, lda, M, K, C, ldc, M, N)) return ST_OK;  // a block's C may be a later one's A
    const int blocks = (int)((M + most - BM) / (most - BM + 1));
    rows = ((M + blocks - 1) / blocks + BM - 1) / BM * BM;
  }
  const size_t bytes = fixed + (size_t)rows * per_row;
  void *w = nullptr;
  if (!ctx_planes_fit(c, bytes) || ctx_workspace(c, bytes, &w)) return ST_OK;  // no room
  done = true;
  return launch_rns<E>(c, M, N, K, rows, make_modulus(p), alpha, A, lda, B, ldb, beta, C, ldc,
                       static_cast<uint8_t *>(w), ra, rb, rw);
}

template <int L>
static int launch_direct(Ctx *c, int M, int N, int K, const Modulus &mod, uint32_t alpha,
                         const uint32_t *A, size_t lda, const uint32_t *B, size_t ldb,
                         uint32_t beta, uint32_t *C, size_t ldc) {
  using Cfg = DirCfg<L>;
  if (int st = ctx_smem_attr(c, (const void *)zp_gemm_direct_kernel<L>, Cfg::smem(2),
                             "cudaFuncSetAttribute(zp_gemm_direct)"))
    return st;
  const int stages = K > BK ? 2 : 1;
  const dim3 grid((N + Cfg::BN - 1) / Cfg::BN, (M + BM - 1) / BM);
  int pi = prof_begin(c, "zp_gemm_direct");
  pdl_launch(zp_gemm_direct_kernel<L>, grid, DIR_THREADS, Cfg::smem(stages), c->stream, A,
             lda, B, ldb, C, ldc, M, N, K, stages, mod, alpha, beta, c->dstatus);
  prof_end(c, pi);
  ctx_launched(c);
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? ST_OK : ctx_cuda(c, e, "zp_gemm_direct launch");
}

size_t zp_gemm_workspace_bytes(uint32_t p, int M, int N, int K) {
  const int L = zp_limbs_for(p);
  const int kc = std::min(ZP_KCHUNK, K);
  const size_t Kp = (size_t)((kc + 15) & ~15);
  return (size_t)L * ((size_t)M + N) * Kp + 256;
}

int zp_gemm_tile_pick(const Ctx *c, int M, int N, int K, uint32_t p) {
  const int L = zp_limbs_for(p);
  if (L == 4) return 0;  // one variant for four limbs
  bool wide = c->gemm_tile == GEMM_TILE_WIDE;
  if (c->gemm_tile == GEMM_TILE_AUTO) {
    // Measured on the B200 (kernel us, wide / double-buffered).  Two limbs, wide
    // tiles of 128 columns: faster at long K (8192^3 1332 / 1922, 2000^3 54 /
    // 64, 512 x 4096 x 4096 40 / 48), at K = 256 slower (4096^2 49 / 41); with
    // at most half as many tiles as SMs the narrower tiles use twice the SMs
    // (1024^3 19 / 15, 512^3 16 / 13).  One limb, wide tiles of 256 columns: a
    // 128-column tile reads as many bytes of shared memory per cycle as there
    // are (8192^2 x 8192 407 / 582, x 2048 168 / 273; 3072 x 2816 x 4096 43 /
    // 57, 2000^3 25 / 27), but they need tiles for most SMs (512 x 4096 x
    // 4096 25 / 21) and K enough to hide their epilogue (4096^2 x 256 37 / 32).
    const long long tm = (M + BM - 1) / BM;
    if (L == 2)
      wide = K >= 512 && 2 * tm * ((N + 127) / 128) > c->num_sms;
    else
      wide = K >= 1024 && 5 * tm * ((N + 255) / 256) >= 4 * (long long)c->num_sms;
  }
  if (L == 2) return wide ? 0 : 1;
  return wide ? 0 : (K <= 2048 ? 1 : 2);
}

int zp_gemm_pick(const Ctx *c, int M, int N, int K, uint32_t p) {
  if (c->gemm_kernel != GEMM_AUTO) return c->gemm_kernel;
  // The one-launch tile kernel for short K while its tiles are few: it saves
  // the split launch, but every tile splits its own operands
  // and the CTAs do not overlap a tile's epilogue with the next tile's product.
  // Measured on the B200 (us per call, one-launch / split, then with a launch per
  // operand, 2.7 us more, and tensor cores, p = 65521): 64 x 960 x 64 9.6 / 16.2, 1000 x
  // 448 x 64 11.5 / 18.1, 2000 x 2000 x 64 (512 tiles) 24.6 / 28.9, 8000 x 960 x 64 (945)
  // 41 / 39, 1024^2 x 256 (128) 14.4 / 16.6, 512 x 4096 x 512 (256) 29.5 / 24.5, 512^3
  // (32) 20.5 / 17.6; four limbs: 64 x 9000 x 64 (282) 20.5 / 24.6, 4000 x 448 x 64 (448)
  // 37 / 35.  The CUDA-core kernel for small K is slower at all of them (14.4 us and more).
  const int L = zp_limbs_for(p), bn = L == 4 ? DirCfg<4>::BN : DirCfg<1>::BN;
  // The smallest products, with few entries of C a thread there, go to the CUDA-core
  // kernel for small K, which needs no barriers, TMEM or MMA (us per call alone, one-launch /
  // CUDA cores: p = 65521 1^3 19.2 / 17.4, 16 x 16 x 32 19.1 / 17.7, 32^3 19.5 / 18.7, 16 x
  // 64 x 32 19.6 / 18.5, 1000 x 16 x 32 19.9 / 19.2, while 64^3 20.0 / 25.3; p = 251 16^3
  // 18.4 / 17.4, 32^3 18.5 / 18.7; four limbs alike up to 16^3; a call among others 7.0
  // either way).
  if (L < 4 && K <= PK && std::min(M, PT) * std::min(N, PT) <= (L == 1 ? 256 : 1024) &&
      (long long)M * N <= 16384)
    return GEMM_SMALLK;
  const long long tiles = (long long)((M + BM - 1) / BM) * ((N + bn - 1) / bn);
  const long long most = K <= 128 ? (L == 4 ? 2 : 4) * c->num_sms : K <= 256 ? c->num_sms : 0;
  if (tiles <= most) return GEMM_DIRECT;
  // Beyond it, wide products of few rows and terms: the limb planes of B are most of the
  // split kernels' work, and four limbs' tiles are 32 columns wide (us per call, CUDA
  // cores / limb planes: p = 2^31 - 1 1 x 65536 x 5 55 / 99, 64 x 65536 x 5 72 / 131, x 32 72 / 85,
  // x 48 120 / 98, 80 x 65536 x 5 121 / 129; p = 65521 1 x 65536 x 32 27 / 33, 32 x 65536 x 16 35 /
  // 46, 64 x 65536 x 16 46 / 55, x 32 46 / 43).
  if (M <= PT && K <= PK && (L == 4 || (L == 2 && (K <= PK / 2 || M <= 16)))) return GEMM_SMALLK;
  return GEMM_TC;
}

// The tensor-core gemm for operands of type E (limb count and tile variant
// by modulus and shape).
template <class E>
static int tc_dispatch(Ctx *c, int M, int N, int K, uint32_t p, uint32_t alpha, const E *A,
                       size_t lda, const E *B, size_t ldb, uint32_t beta, uint32_t *C, size_t ldc,
                       uint8_t *ws, const int2 *kr, int kbase) {
  const Modulus mod = make_modulus(p);
  const int tv = zp_gemm_tile_pick(c, M, N, K, p);
#define LELA_TC(L, T) \
  launch_tc<L, T, E>(c, M, N, K, mod, alpha, A, lda, B, ldb, beta, C, ldc, ws, kr, kbase)
  switch (zp_limbs_for(p)) {
    case 1: return tv == 0 ? LELA_TC(1, 0) : tv == 1 ? LELA_TC(1, 1) : LELA_TC(1, 2);
    case 2: return tv == 0 ? LELA_TC(2, 0) : LELA_TC(2, 1);
    default: return LELA_TC(4, 0);
  }
#undef LELA_TC
}

int zp_gemm_dev(Ctx *c, int kernel, int M, int N, int K, uint32_t p, uint32_t alpha,
                const uint32_t *A, size_t lda, const uint32_t *B, size_t ldb, uint32_t beta,
                uint32_t *C, size_t ldc, uint8_t *ws_override, const int2 *kr, int kbase) {
  if (p < 2) return ctx_fail(c, ST_ARG, "modulus must be at least 2");
  if (M < 0 || N < 0 || K < 0) return ctx_fail(c, ST_ARG, "negative dimension");
  if (M == 0 || N == 0) return ST_OK;
  if (ldc < (size_t)N || (K > 0 && (lda < (size_t)K || ldb < (size_t)N)))
    return ctx_fail(c, ST_ARG, "leading dimension smaller than the row length");
  const Modulus mod = make_modulus(p);
  alpha %= p;
  beta %= p;
  if (K == 0 || alpha == 0) {
    if (beta == 1) return ST_OK;
    const size_t total = (size_t)M * N;
    int grid = (int)std::min<size_t>((total + 255) / 256, (size_t)c->num_sms * 8);
    zp_scale_kernel<<<grid, 256, 0, c->stream>>>(C, ldc, M, N, mod, beta);
    ctx_launched(c);
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? ST_OK : ctx_cuda(c, e, "zp_scale launch");
  }
  if (kernel == GEMM_AUTO) {
    kernel = zp_gemm_pick(c, M, N, K, p);
    // C may lie over A or B where the operands are split before C is written; the
    // one-launch kernels' CTAs read them while others already write
    const bool one = kernel == GEMM_DIRECT || kernel == GEMM_SMALLK;
    if (one && c->gemm_kernel == GEMM_AUTO &&
        (share_entries(A, lda, M, K, C, ldc, M, N) || share_entries(B, ldb, K, N, C, ldc, M, N)))
      kernel = GEMM_TC;
  }
  if (kernel == GEMM_SMALLK) {
    dim3 grid((N + PT - 1) / PT, (M + PT - 1) / PT);
    // (early only with few CTAs: more, waiting in turn beside those that still run, made a
    // row of 1000 x 448 x 64 products, 112 CTAs each, 28.5 us a call instead of 14.4)
    const bool early = (size_t)grid.x * grid.y <= 16;
    int pi = prof_begin(c, "zp_gemm_smallk");
    if (p < (1u << 28))
      pdl_launch_if(early, zp_gemm_smallk_kernel<true>, grid, 256, 0, c->stream, A, lda, B, ldb, C, ldc, M,
                    N, K, mod, host_two64(p), alpha, beta);
    else
      pdl_launch_if(early, zp_gemm_smallk_kernel<false>, grid, 256, 0, c->stream, A, lda, B, ldb, C, ldc, M,
                    N, K, mod, host_two64(p), alpha, beta);
    prof_end(c, pi);
    ctx_launched(c);
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? ST_OK : ctx_cuda(c, e, "zp_gemm_smallk launch");
  }
  if (kernel == GEMM_DIRECT) {
    switch (zp_limbs_for(p)) {
      case 1: return launch_direct<1>(c, M, N, K, mod, alpha, A, lda, B, ldb, beta, C, ldc);
      case 2: return launch_direct<2>(c, M, N, K, mod, alpha, A, lda, B, ldb, beta, C, ldc);
      default: return launch_direct<4>(c, M, N, K, mod, alpha, A, lda, B, ldb, beta, C, ldc);
    }
  }
  if (kernel == GEMM_PLAIN) {
    dim3 grid((N + PT - 1) / PT, (M + PT - 1) / PT);
    int pi = prof_begin(c, "zp_gemm_plain");
    zp_gemm_plain_kernel<<<grid, 256, 0, c->stream>>>(A, lda, B, ldb, C, ldc, M, N, K, mod,
                                                      host_two64(p), alpha, beta);
    prof_end(c, pi);
    ctx_launched(c);
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? ST_OK : ctx_cuda(c, e, "zp_gemm_plain launch");
  }
  uint8_t *ws = ws_override;
  if (!ws) {
    if (!kr) {
      bool done;
      const int st = rns_try<uint32_t>(c, M, N, K, p, alpha, A, lda, B, ldb, beta, C, ldc, done);
      if (st || done) return st;
    }
    void *w = nullptr;
    int st = ctx_workspace(c, zp_gemm_workspace_bytes(p, M, N, K), &w);
    if (st) return st;
    ws = static_cast<uint8_t *>(w);
  }
  return tc_dispatch<uint32_t>(c, M, N, K, p, alpha, A, lda, B, ldb, beta, C, ldc, ws, kr, kbase);
}

int zp_gemm_tc_elem_dev(Ctx *c, int elem, int M, int N, int K, uint32_t p, uint32_t alpha,
                        const void *A, size_t lda, const void *B, size_t ldb, uint32_t *V,
                        size_t ldv) {
  alpha %= p;
  if (elem == LELA_CUDA_ELEM_F64) {  // the only type with moduli of four limbs
    bool done;
    const int st = rns_try<double>(c, M, N, K, p, alpha, static_cast<const double *>(A), lda,
                                   static_cast<const double *>(B), ldb, 0u, V, ldv, done);
    if (st || done) return st;
  }
  void *w = nullptr;
  if (int st = ctx_workspace(c, zp_gemm_workspace_bytes(p, M, N, K), &w)) return st;
  uint8_t *ws = static_cast<uint8_t *>(w);
#define LELA_ELEM(E)                                                                           \
  tc_dispatch<E>(c, M, N, K, p, alpha, static_cast<const E *>(A), lda, static_cast<const E *>(B), \
                 ldb, 0u, V, ldv, ws, nullptr, 0)
  switch (elem) {
    case LELA_CUDA_ELEM_U8: return LELA_ELEM(uint8_t);
    case LELA_CUDA_ELEM_U16: return LELA_ELEM(uint16_t);
    case LELA_CUDA_ELEM_F32: return LELA_ELEM(float);
    case LELA_CUDA_ELEM_F64: return LELA_ELEM(double);
    default: return ctx_fail(c, ST_ARG, "unknown element type");
  }
#undef LELA_ELEM
}

// ------------------------------------------------- limb planes kept by callers
template <int L, int T>
static int launch_planes(Ctx *c, int M, int N, int K, const Modulus &mod, uint32_t alpha,
                         const ZpPlanes &A, const ZpPlanes &B, uint32_t beta, uint32_t *C,
                         size_t ldc, const int2 *kr, int kbase) {
  using Cfg = TcCfg<L, T>;
  if (int st = tc_attr<L, T>(c)) return st;
  const int tiles = ((M + BM - 1) / BM) * ((N + Cfg::BN - 1) / Cfg::BN);
  uint32_t b = beta;
  for (int k0 = 0; k0 < K; k0 += ZP_KCHUNK) {
    const int kc = std::min(ZP_KCHUNK, K - k0);
    CUtensorMap tmA, tmB;
    int st = encode_3d(c, &tmA, A.base + k0, (uint64_t)kc, (uint64_t)M, L, A.pitch, A.plane, BK, BM, L);
    if (!st) st = encode_3d(c, &tmB, B.base + k0, (uint64_t)kc, (uint64_t)N, L, B.pitch, B.plane, BK,
                            Cfg::BN, L);
    if (st) return st;
    int pi = prof_begin(c, "zp_gemm_tc");
    pdl_launch(zp_gemm_tc_kernel<L, OUT_ZP, T>, std::min(tiles, c->num_sms), tc_threads<L, T>(),
               TcLayout<L, T>::SMEM, c->stream,
               tmA, tmB, C, ldc, M, N, kc, mod, alpha, b, c->dstatus, kr, kbase + k0);
    prof_end(c, pi);
    ctx_launched(c);
    b = 1;
  }
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? ST_OK : ctx_cuda(c, e, "zp_gemm_tc launch");
}

int zp_gemm_planes_dev(Ctx *c, int M, int N, int K, uint32_t p, uint32_t alpha, const ZpPlanes &A,
                       const ZpPlanes &B, uint32_t beta, uint32_t *C, size_t ldc, const int2 *kr,
                       int kbase) {
  const Modulus mod = make_modulus(p);
  const int tv = zp_gemm_tile_pick(c, M, N, K, p);
#define LELA_PL(L, T) launch_planes<L, T>(c, M, N, K, mod, alpha, A, B, beta, C, ldc, kr, kbase)
  switch (zp_limbs_for(p)) {
    case 1: return tv == 0 ? LELA_PL(1, 0) : tv == 1 ? LELA_PL(1, 1) : LELA_PL(1, 2);
    case 2: return tv == 0 ? LELA_PL(2, 0) : LELA_PL(2, 1);
    default: return LELA_PL(4, 0);
  }
#undef LELA_PL
}

int zp_split_rows_dev(Ctx *c, uint32_t p, const uint32_t *A, size_t lda, int M, int K,
                      const ZpPlanes &out, int part, int nb) {
  const dim3 grid = split_rows_grid(c->num_sms, M, K), block(32 * SPLIT_ROWS);
#define LELA_SR(L) \
  pdl_launch(split_narrow(M, K) ? split_rows_kernel<LimbBytes<L>, uint32_t, true>         \
                                : split_rows_kernel<LimbBytes<L>, uint32_t, false>,       \
             grid, block, 0, c->stream, A, lda, M, K, p,                                  \
             out.base, out.pitch, out.plane, part, nb, LimbBytes<L>{})
  switch (zp_limbs_for(p)) {
    case 1: LELA_SR(1); break;
    case 2: LELA_SR(2); break;
    default: LELA_SR(4); break;
  }
#undef LELA_SR
  ctx_launched(c);
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? ST_OK : ctx_cuda(c, e, "zp_split launch");
}

int zp_split_cols_dev(Ctx *c, uint32_t p, const uint32_t *B, size_t ldb, int K, int N,
                      const ZpPlanes &out) {
  const int kout = (K + 15) & ~15;
  const dim3 grid = split_cols_grid<uint32_t>(N, kout);
#define LELA_SC(L) \
  pdl_launch(split_cols_kernel<LimbBytes<L>, uint32_t>, grid, 256, 0, c->stream, B, ldb, K, N, p, out.base, \
             out.pitch, out.plane, kout, LimbBytes<L>{})
  switch (zp_limbs_for(p)) {
    case 1: LELA_SC(1); break;
    case 2: LELA_SC(2); break;
    default: LELA_SC(4); break;
  }
#undef LELA_SC
  ctx_launched(c);
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? ST_OK : ctx_cuda(c, e, "zp_split launch");
}

// ============================================ pipelined host-pointer gemm
//
// The host-pointer gemm moves (M K + K N + 2 M N) * 4 bytes over the host
// link for 2 M N K operations on the GPU: at 8192^3 the copies take about
// ten times as long as the product.  The rows of C are therefore done in
// blocks: B goes over first, then A's and C's rows block by block on the
// copy_in stream; each block's product runs on the handle stream as soon as
// its rows are in, and its rows of C go back on the copy_out stream while
// later blocks still arrive (the two directions of the link run at once).
// The result is the same product: every output element is computed by the
// same kernel from the same operands, only the launches cover fewer rows.

bool zp_gemm_pipelined(const Ctx *c, int M, int N, int K, uint32_t p, uint32_t alpha) {
  return K > 0 && K <= ZP_KCHUNK && alpha % p != 0 && M >= 2 * PIPE_MIN_ROWS &&
         zp_gemm_pick(c, M, N, K, p) == GEMM_TC;
}

template <int L>
static int host_rows(Ctx *c, int M, int N, int K, const Modulus &mod, uint32_t alpha,
                     const uint32_t *hA, size_t lda, const uint32_t *hB, size_t ldb,
                     uint32_t beta, uint32_t *hC, size_t ldc, uint32_t *dA, uint32_t *dB,
                     uint32_t *dC, uint8_t *ws) {
  using Cfg = TcCfg<L, 0>;
  using Lay = TcLayout<L, 0>;
  if (int st = tc_attr<L>(c)) return st;
  const int Kp = (K + 15) & ~15;
  // row blocks: a multiple of the tile height, at most PIPE_MAX_BLOCKS
  const int per = (M + PIPE_MAX_BLOCKS - 1) / PIPE_MAX_BLOCKS;
  const int rb = std::max(PIPE_MIN_ROWS, (per + BM - 1) / BM * BM);
  const int nblk = (M + rb - 1) / rb;
  cudaEvent_t *ready = c->pipe_ev, *done = c->pipe_ev + PIPE_MAX_BLOCKS;
  cudaEvent_t ev_start = c->pipe_ev[2 * PIPE_MAX_BLOCKS], ev_b = c->pipe_ev[2 * PIPE_MAX_BLOCKS + 1],
              ev_out = c->pipe_ev[2 * PIPE_MAX_BLOCKS + 2];
  const size_t rowA = (size_t)K * 4, rowC = (size_t)N * 4;
  // the copies start after the work already queued on the handle stream
  cudaError_t e = cudaEventRecord(ev_start, c->stream);
  if (e == cudaSuccess) e = cudaStreamWaitEvent(c->copy_in, ev_start, 0);
  if (e == cudaSuccess) e = cudaStreamWaitEvent(c->copy_out, ev_start, 0);
  if (e == cudaSuccess)
    e = cudaMemcpy2DAsync(dB, rowC, hB, ldb * 4, rowC, (size_t)K, cudaMemcpyHostToDevice,
                          c->copy_in);
  if (e == cudaSuccess) e = cudaEventRecord(ev_b, c->copy_in);
  for (int j = 0; e == cudaSuccess && j < nblk; ++j) {
    const int r0 = j * rb, rows = std::min(rb, M - r0);
    e = cudaMemcpy2DAsync(dA + (size_t)r0 * K, rowA, hA + (size_t)r0 * lda, lda * 4, rowA,
                          (size_t)rows, cudaMemcpyHostToDevice, c->copy_in);
    if (e == cudaSuccess && beta)
      e = cudaMemcpy2DAsync(dC + (size_t)r0 * N, rowC, hC + (size_t)r0 * ldc, ldc * 4, rowC,
                            (size_t)rows, cudaMemcpyHostToDevice, c->copy_in);
    if (e == cudaSuccess) e = cudaEventRecord(ready[j], c->copy_in);
  }
  // B's limb planes once; block j's A planes in their own part of the
  // workspace, so that a block's split never overwrites planes an earlier
  // block's kernel still reads
  int st = ST_OK;
  uint8_t *Bl = ws + (size_t)L * M * Kp;
  CUtensorMap tmB;
  if (e == cudaSuccess) e = cudaStreamWaitEvent(c->stream, ev_b, 0);
  if (e == cudaSuccess) {
    int pi = prof_begin(c, "zp_split");
    pdl_launch(split_cols_kernel<LimbBytes<L>, uint32_t>, split_cols_grid<uint32_t>(N, Kp), 256, 0,
               c->stream, dB, (size_t)N, K, N, (uint32_t)mod.p, Bl, (size_t)Kp, (size_t)N * Kp, Kp,
               LimbBytes<L>{});
    prof_end(c, pi);
    ctx_launched(c);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess)
    st = encode_3d(c, &tmB, Bl, (uint64_t)K, (uint64_t)N, L, (uint64_t)Kp, (uint64_t)N * Kp, BK,
                   Cfg::BN, L);
  for (int j = 0; e == cudaSuccess && !st && j < nblk; ++j) {
    const int r0 = j * rb, rows = std::min(rb, M - r0);
    uint8_t *Al = ws + (size_t)L * r0 * Kp;
    e = cudaStreamWaitEvent(c->stream, ready[j], 0);
    if (e != cudaSuccess) break;
    int pi = prof_begin(c, "zp_split");
    pdl_launch(split_narrow(rows, K) ? split_rows_kernel<LimbBytes<L>, uint32_t, true>
                                     : split_rows_kernel<LimbBytes<L>, uint32_t, false>,
               split_rows_grid(c->num_sms, rows, K),
               32 * SPLIT_ROWS, 0, c->stream, dA + (size_t)r0 * K, (size_t)K, rows, K,
               (uint32_t)mod.p, Al, (size_t)Kp, (size_t)rows * Kp, 0, 1, LimbBytes<L>{});
    prof_end(c, pi);
    CUtensorMap tmA;
    st = encode_3d(c, &tmA, Al, (uint64_t)K, (uint64_t)rows, L, (uint64_t)Kp,
                   (uint64_t)rows * Kp, BK, BM, L);
    if (st) break;
    const int tiles = ((rows + BM - 1) / BM) * ((N + Cfg::BN - 1) / Cfg::BN);
    pi = prof_begin(c, "zp_gemm_tc");
    pdl_launch(zp_gemm_tc_kernel<L, OUT_ZP>, std::min(tiles, c->num_sms), tc_threads<L, 0>(),
               Lay::SMEM, c->stream, tmA, tmB, dC + (size_t)r0 * N, (size_t)N, rows, N, K, mod, alpha,
               beta, c->dstatus, nullptr, 0);
    prof_end(c, pi);
    ctx_launched(c, 2);
    e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaEventRecord(done[j], c->stream);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(c->copy_out, done[j], 0);
    if (e == cudaSuccess)
      e = cudaMemcpy2DAsync(hC + (size_t)r0 * ldc, ldc * 4, dC + (size_t)r0 * N, rowC, rowC,
                            (size_t)rows, cudaMemcpyDeviceToHost, c->copy_out);
  }
  // the handle stream ends after the last copy out
  if (e == cudaSuccess && !st) e = cudaEventRecord(ev_out, c->copy_out);
  if (e == cudaSuccess && !st) e = cudaStreamWaitEvent(c->stream, ev_out, 0);
  if (e != cudaSuccess || st) {
    // copies already queued may still use the caller's buffers
    cudaStreamSynchronize(c->copy_in);
    cudaStreamSynchronize(c->copy_out);
    return st ? st : ctx_cuda(c, e, "pipelined gemm");
  }
  return ST_OK;
}

int zp_gemm_host_rows(Ctx *c, int M, int N, int K, uint32_t p, uint32_t alpha,
                      const uint32_t *hA, size_t lda, const uint32_t *hB, size_t ldb,
                      uint32_t beta, uint32_t *hC, size_t ldc, uint32_t *dA, uint32_t *dB,
                      uint32_t *dC) {
  if (!zp_gemm_pipelined(c, M, N, K, p, alpha)) return ctx_fail(c, ST_ARG, "not a pipelined gemm");
  if (int st = ctx_pipe(c)) return st;
  void *w = nullptr;
  if (int st = ctx_workspace(c, zp_gemm_workspace_bytes(p, M, N, K), &w)) return st;
  uint8_t *ws = static_cast<uint8_t *>(w);
  const Modulus mod = make_modulus(p);
  alpha %= p;
  beta %= p;
  switch (zp_limbs_for(p)) {
    case 1:
      return host_rows<1>(c, M, N, K, mod, alpha, hA, lda, hB, ldb, beta, hC, ldc, dA, dB, dC, ws);
    case 2:
      return host_rows<2>(c, M, N, K, mod, alpha, hA, lda, hB, ldb, beta, hC, ldc, dA, dB, dC, ws);
    default:
      return host_rows<4>(c, M, N, K, mod, alpha, hA, lda, hB, ldb, beta, hC, ldc, dA, dB, dC, ws);
  }
}

}  // namespace lela

// ====================================================== no-allocation gemm
//
// lela_cuda_gemm_zp_u32_noalloc: the tensor-core Z/p gemm for callers that
// cannot allocate device memory -- code running under a memory manager that
// owns every device allocation (a host framework's caching allocator or a
// fixed per-process memory budget), or latency-critical paths where
// cudaMalloc/cudaFree, which may synchronise the device, are not allowed.
// Such a caller passes device pointers for A, B and C; the limb planes the
// kernel needs as scratch live in the fixed array below instead of a
// handle's workspace, so this entry point calls no cudaMalloc, cudaFree or
// other allocating routine and needs no handle.
//
// Limits and sharing:
//  - the scratch is NOALLOC_PLANE_BYTES = 64 MiB of limb planes, enough for
//    L * (m + n) * round16(min(k, 32768)) bytes, L = 1, 2 or 4 limbs for
//    p <= 2^8, 2^16, 2^32 (e.g. m = n = k = 4096 at p = 65521); larger
//    problems are rejected with LELA_CUDA_ERR_ARG before any GPU work;
//  - the array is a file-scope __device__ variable: every GPU that loads
//    this library holds it (plus 256 bytes of status) until the process
//    exits;
//  - all calls on a device share it and it keeps the last call's contents.
//    Each call writes every scratch byte its kernel reads (the K tail of a
//    row is never read: the TMA descriptors stop at k) and clears its
//    status word first, so nothing else must start at zero.  Calls whose
//    GPU work overlaps (different streams or host threads without
//    ordering) race on the scratch and give wrong results.
//  - The first call on a device does its set-up there, with that device
//    current: it looks up the array's device address with
//    cudaGetSymbolAddress and sets the kernels' shared-memory attribute.
//    Make that first call before any stream capture.  The set-up is kept
//    for the life of the process, so the entry point must not be called
//    after cudaDeviceReset (which unloads the module the address and the
//    attributes belong to).
namespace lela {

constexpr size_t NOALLOC_STATUS_BYTES = 256;
constexpr size_t NOALLOC_PLANE_BYTES = (size_t)64 << 20;
static __device__ __align__(256) uint8_t g_noalloc_scratch[NOALLOC_STATUS_BYTES + NOALLOC_PLANE_BYTES];

namespace {

constexpr int NOALLOC_MAX_DEVICES = 64;
struct NoallocDevice {
  bool ready;
  uint8_t *base;  // device address of g_noalloc_scratch on this device
  int num_sms;
};
NoallocDevice g_noalloc_dev[NOALLOC_MAX_DEVICES];
std::mutex g_noalloc_mu;
PFN_cuTensorMapEncodeTiled_v12000 g_noalloc_encode = nullptr;

// Once per device, with that device current.
int noalloc_setup(int dev, NoallocDevice *out) {
  std::lock_guard<std::mutex> lock(g_noalloc_mu);
  if (dev < 0 || dev >= NOALLOC_MAX_DEVICES) return ST_ARG;
  NoallocDevice &d = g_noalloc_dev[dev];
  if (!d.ready) {
    void *ptr = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&ptr, g_noalloc_scratch);
    if (e != cudaSuccess || ptr == nullptr) return ST_CUDA;
    int sms = 0;
    e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return ST_CUDA;
    e = cudaFuncSetAttribute(zp_gemm_tc_kernel<1, 0>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             TcLayout<1, 0>::SMEM);
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(zp_gemm_tc_kernel<2, 0>,
                               cudaFuncAttributeMaxDynamicSharedMemorySize, TcLayout<2, 0>::SMEM);
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(zp_gemm_tc_kernel<4, 0>,
                               cudaFuncAttributeMaxDynamicSharedMemorySize, TcLayout<4, 0>::SMEM);
    if (e != cudaSuccess) return ST_CUDA;
    if (!g_noalloc_encode) {
      void *fn = nullptr;
      cudaDriverEntryPointQueryResult q;
      e = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q);
      if (e != cudaSuccess || q != cudaDriverEntryPointSuccess || !fn) return ST_CUDA;
      g_noalloc_encode = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(fn);
    }
    d.base = static_cast<uint8_t *>(ptr);
    d.num_sms = sms;
    d.ready = true;
  }
  *out = d;
  return ST_OK;
}

bool noalloc_map(CUtensorMap *tm, void *base, uint64_t d0, uint64_t d1, uint64_t d2,
                 uint64_t stride1, uint64_t stride2, uint32_t b0, uint32_t b1, uint32_t b2) {
  cuuint64_t dims[3] = {d0, d1, d2};
  cuuint64_t strides[2] = {stride1, stride2};
  cuuint32_t box[3] = {b0, b1, b2};
  cuuint32_t estr[3] = {1, 1, 1};
  return g_noalloc_encode(tm, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, base, dims, strides, box, estr,
                          CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                          CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int L>
int noalloc_launch(cudaStream_t s, const NoallocDevice &d, int M, int N, int K,
                   const Modulus &mod, uint32_t alpha, const uint32_t *A, size_t lda,
                   const uint32_t *B, size_t ldb, uint32_t beta, uint32_t *C, size_t ldc) {
  using Cfg = TcCfg<L, 0>;
  using Lay = TcLayout<L, 0>;
  uint32_t *err = reinterpret_cast<uint32_t *>(d.base);
  uint8_t *planes = d.base + NOALLOC_STATUS_BYTES;
  const int tiles = ((M + BM - 1) / BM) * ((N + Cfg::BN - 1) / Cfg::BN);
  uint32_t b = beta;
  for (int k0 = 0; k0 < K; k0 += ZP_KCHUNK) {
    const int kc = std::min(ZP_KCHUNK, K - k0);
    const int Kp = (kc + 15) & ~15;
    uint8_t *Al = planes;
    uint8_t *Bl = planes + (size_t)L * M * Kp;
    const uint32_t p = (uint32_t)mod.p;
    launch_split(true, d.num_sms, s, A + k0, lda, B + (size_t)k0 * ldb, ldb, M, N, kc, p, Al, Bl, Kp,
                 LimbBytes<L>{}, LimbBytes<L>{});
    CUtensorMap tmA, tmB;
    if (!noalloc_map(&tmA, Al, (uint64_t)kc, (uint64_t)M, L, (uint64_t)Kp, (uint64_t)M * Kp,
                     BK, BM, L) ||
        !noalloc_map(&tmB, Bl, (uint64_t)kc, (uint64_t)N, L, (uint64_t)Kp, (uint64_t)N * Kp,
                     BK, Cfg::BN, L))
      return ST_CUDA;
    pdl_launch(zp_gemm_tc_kernel<L, OUT_ZP>, std::min(tiles, d.num_sms), tc_threads<L, 0>(), Lay::SMEM, s,
               tmA, tmB, C, ldc, M, N, kc, mod, alpha, b, err, nullptr, 0);
    b = 1;
  }
  return cudaGetLastError() == cudaSuccess ? ST_OK : ST_CUDA;
}

}  // namespace

}  // namespace lela

extern "C" int lela_cuda_gemm_zp_u32_noalloc(size_t m, size_t n, size_t k, uint32_t p,
                                             uint32_t a, const uint32_t *A, size_t lda,
                                             const uint32_t *B, size_t ldb, uint32_t b,
                                             uint32_t *C, size_t ldc, void *stream) {
  using namespace lela;
  if (p < 2) return ST_ARG;
  if (m > (size_t)INT32_MAX || n > (size_t)INT32_MAX || k > (size_t)INT32_MAX) return ST_ARG;
  if (m == 0 || n == 0) return ST_OK;
  if (!C || (k && (!A || !B))) return ST_ARG;
  if (ldc < n || (k && (lda < k || ldb < n))) return ST_ARG;
  const int L = zp_limbs_for(p);
  const size_t kc = std::min<size_t>(k, (size_t)ZP_KCHUNK);
  const size_t need = (size_t)L * (m + n) * ((kc + 15) & ~(size_t)15);
  if (need > NOALLOC_PLANE_BYTES) return ST_ARG;  // beyond the fixed scratch

  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return ST_CUDA;
  NoallocDevice d;
  int st = noalloc_setup(dev, &d);
  if (st) return st;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const Modulus mod = make_modulus(p);
  a %= p;
  b %= p;
  if (cudaMemsetAsync(d.base, 0, sizeof(uint32_t), s) != cudaSuccess) return ST_CUDA;
  if (k == 0 || a == 0) {
    if (b != 1) {
      const size_t total = m * n;
      int grid = (int)std::min<size_t>((total + 255) / 256, (size_t)d.num_sms * 8);
      zp_scale_kernel<<<grid, 256, 0, s>>>(C, ldc, (int)m, (int)n, mod, b);
      if (cudaGetLastError() != cudaSuccess) return ST_CUDA;
    }
  } else {
    switch (L) {
      case 1: st = noalloc_launch<1>(s, d, (int)m, (int)n, (int)k, mod, a, A, lda, B, ldb, b, C, ldc); break;
      case 2: st = noalloc_launch<2>(s, d, (int)m, (int)n, (int)k, mod, a, A, lda, B, ldb, b, C, ldc); break;
      default: st = noalloc_launch<4>(s, d, (int)m, (int)n, (int)k, mod, a, A, lda, B, ldb, b, C, ldc); break;
    }
    if (st) return st;
  }
  uint32_t word = 0;
  if (cudaMemcpyAsync(&word, d.base, sizeof word, cudaMemcpyDeviceToHost, s) != cudaSuccess)
    return ST_CUDA;
  if (cudaStreamSynchronize(s) != cudaSuccess) return ST_CUDA;
  return (word & DEVERR_TIMEOUT) ? ST_TIMEOUT : ST_OK;
}

// ======================================================= GF(2) on tensor cores
namespace lela {

// C (packed GF(2) words) <- (beta ? C : 0) XOR (alpha ? A*B : 0) from 0/1
// byte planes Ab (M x Kp, K-major) and Bb (N x Kp, K-major) of K columns:
// the one-limb tensor-core kernel with the bit-packing epilogue.
template <int T>
static int gf2_tc_launch(Ctx *c, int M, int N, int K, const uint8_t *Ab, const uint8_t *Bb,
                         int Kp, uint32_t alpha, uint32_t beta, uint64_t *C, size_t ldc_words) {
  using Cfg = TcCfg<1, T>;
  using Lay = TcLayout<1, T>;
  if (int st = ctx_smem_attr(c, (const void *)zp_gemm_tc_kernel<1, OUT_GF2, T>, Lay::SMEM,
                             "cudaFuncSetAttribute(gf2 tc)"))
    return st;
  CUtensorMap tmA, tmB;
  int st = encode_3d(c, &tmA, const_cast<uint8_t *>(Ab), (uint64_t)K, (uint64_t)M, 1,
                     (uint64_t)Kp, (uint64_t)M * Kp, BK, BM, 1);
  if (st) return st;
  st = encode_3d(c, &tmB, const_cast<uint8_t *>(Bb), (uint64_t)K, (uint64_t)N, 1, (uint64_t)Kp,
                 (uint64_t)N * Kp, BK, Cfg::BN, 1);
  if (st) return st;
  const int tiles = ((M + BM - 1) / BM) * ((N + Cfg::BN - 1) / Cfg::BN);
  int pi = prof_begin(c, "gf2_gemm_tc");
  pdl_launch_if(gf2_early(M, N, K), zp_gemm_tc_kernel<1, OUT_GF2, T>, std::min(tiles, c->num_sms),
                tc_threads<1, T>(), Lay::SMEM, c->stream, tmA, tmB, C, ldc_words, M, N, K,
                make_modulus(2), alpha, beta, c->dstatus, nullptr, 0);
  prof_end(c, pi);
  ctx_launched(c);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? ST_OK : ctx_cuda(c, e, "gf2 tc launch");
}

// 16 epilogue warps at short K (the echelon's block updates, K <= 512 bits:
// the 32768^2 echelon 62.0 -> 58.4 ms), 8 at long K (16384^3: 3.358 against
// 3.371 ms)
int gf2_gemm_tc_planes(Ctx *c, int M, int N, int K, const uint8_t *Ab, const uint8_t *Bb, int Kp,
                       uint32_t alpha, uint32_t beta, uint64_t *C, size_t ldc_words) {
  if (K <= 4096)
    return gf2_tc_launch<GF2_TC_T>(c, M, N, K, Ab, Bb, Kp, alpha, beta, C, ldc_words);
  return gf2_tc_launch<0>(c, M, N, K, Ab, Bb, Kp, alpha, beta, C, ldc_words);
}

}  // namespace lela

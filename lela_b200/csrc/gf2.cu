// lela_b200/csrc/gf2.cu -- dense GF(2) kernels on bit-packed matrices.
//
// Layout: LELA's DenseMatrix<bool> rows are BitVector<LittleEndian<uint64>>
// (lela/ring/gf2.h:311; bit j of word w = column 64w + j,
// lela/vector/bit-iterator.h:249-296), row stride in words.  Bits beyond the
// last column of a row are zero on input and kept zero on output.
//
// gemm  C <- a*A*B + b*C (a, b in {0, 1}).  Replaces the generic
// Row*Row*Row gemm over GF2 (lela/blas/level3-generic.tcc:243-263 ->
// _gemv<GF2> lela/blas/level2-gf2.tcc:132-155: row i of C is the XOR of the
// rows of B selected by row i of A) and M4RI's mzd_mul/mzd_addmul
// (lela/blas/level3-m4ri.tcc:78-80).  Two kernels:
//  * gf2_m4rm_kernel: bit-packed, "method of four Russians": per group of
//    8 rows of B a 256-entry table of all their XOR combinations is built in
//    shared memory, and each row of A then needs one table lookup per byte
//    instead of eight row XORs;
//  * the int8-expanded tensor-core variant (gf2_gemm_tc_planes in
//    zp_gemm.cu): bits become 0/1 bytes, tcgen05 .kind::i8 counts the
//    products exactly, and the parity of the count is the GF(2) entry.
//
// echelon  Non-reduced row-echelon form with LELA's pivot rule (first row
// at or below the current one with a 1 in the column, swapped in by a
// transposition; rows below with a 1 get the pivot row XOR-ed in), i.e.
// Elimination::echelonize on a Dense01 matrix (lela/algorithms/
// elimination.tcc:47-139, pivot-strategy.tcc:44-66), which the dense
// EchelonForm path (GaussJordan + move_L) reproduces.  Same exact panel
// scheme as the Z/p version (echelon.cu) with 64-column panels = one word
// per row; the words of a panel's block are updated by tables, those right of the block
// on the tensor cores (M4RM for few rows).
#include <algorithm>
#include <cstddef>
#include <mutex>
#include <vector>

#include "common.cuh"
#include "context.h"
#include "gf2.h"
#include "zp_gemm.h"

namespace lela {

// ------------------------------------------------------------------ M4RM
constexpr int M4_THREADS = 256;
constexpr int M4_KC = 32;     // rows of B per table round (4 tables of 8)

// C[r, w0 .. w0+M4_BW) for the CTA's rows (M4_ROWS per thread); tables
// T[g][w][s] in shared memory.
template <int M4_ROWS, int M4_BW>
__global__ void __launch_bounds__(M4_THREADS)
    gf2_m4rm_kernel(const uint64_t *A, size_t lda, const uint64_t *B,
                    size_t ldb, uint64_t *C, size_t ldc, int M, int Nw, int K,
                    uint64_t tail_mask, int alpha, int beta) {
  pdl_enter();
  extern __shared__ uint64_t m4_smem[];
  uint64_t(*T)[M4_BW][256] = reinterpret_cast<uint64_t(*)[M4_BW][256]>(m4_smem);
  uint64_t(*Bk)[M4_BW] = reinterpret_cast<uint64_t(*)[M4_BW]>(m4_smem + 4 * M4_BW * 256);
  const int w0 = blockIdx.x * M4_BW;
  const int r0 = blockIdx.y * (M4_THREADS * M4_ROWS);
  uint64_t acc[M4_ROWS][M4_BW];
#pragma unroll
  for (int i = 0; i < M4_ROWS; ++i)
#pragma unroll
    for (int w = 0; w < M4_BW; ++w) acc[i][w] = 0;

  for (int k0 = 0; k0 < K; k0 += M4_KC) {
    __syncthreads();
    for (int e = threadIdx.x; e < M4_KC * M4_BW; e += blockDim.x) {
      const int kk = e / M4_BW, w = e % M4_BW;
      Bk[kk][w] = (k0 + kk < K && w0 + w < Nw) ? B[(size_t)(k0 + kk) * ldb + w0 + w] : 0ull;
    }
    if (threadIdx.x < 4 * M4_BW) T[threadIdx.x / M4_BW][threadIdx.x % M4_BW][0] = 0ull;
    __syncthreads();
    // T[g][w][s + 2^j] = T[g][w][s] ^ B[8g + j][w] for s < 2^j
#pragma unroll 1
    for (int j = 0; j < 8; ++j) {
      const int half = 1 << j;
      for (int e = threadIdx.x; e < 4 * M4_BW * half; e += blockDim.x) {
        const int s = e % half, w = (e / half) % M4_BW, g = e / (half * M4_BW);
        T[g][w][s + half] = T[g][w][s] ^ Bk[8 * g + j][w];
      }
      __syncthreads();
    }
    const int wk = k0 >> 6, sh = k0 & 63;  // the 32 bits of A for k0 .. k0+31
#pragma unroll
    for (int i = 0; i < M4_ROWS; ++i) {
      const int r = r0 + i * M4_THREADS + threadIdx.x;
      uint32_t bits = 0;
      if (r < M) {
        bits = (uint32_t)(A[(size_t)r * lda + wk] >> sh);
        if (K - k0 < 32) bits &= (1u << (K - k0)) - 1u;
      }
      const uint32_t b0 = bits & 255u, b1 = (bits >> 8) & 255u, b2 = (bits >> 16) & 255u,
                     b3 = bits >> 24;
#pragma unroll
      for (int w = 0; w < M4_BW; ++w)
        acc[i][w] ^= T[0][w][b0] ^ T[1][w][b1] ^ T[2][w][b2] ^ T[3][w][b3];
    }
  }
#pragma unroll
  for (int i = 0; i < M4_ROWS; ++i) {
    const int r = r0 + i * M4_THREADS + threadIdx.x;
    if (r >= M) continue;
    uint64_t *crow = C + (size_t)r * ldc;
#pragma unroll
    for (int w = 0; w < M4_BW; ++w) {
      const int gw = w0 + w;
      if (gw >= Nw) break;
      // bits of the last word at columns >= N keep their old values (they
      // may belong to the next columns of a strided view)
      const bool part = gw == Nw - 1 && tail_mask != ~0ull;
      const uint64_t old = (beta || part) ? crow[gw] : 0ull;
      uint64_t v = (beta ? old : 0ull) ^ (alpha ? acc[i][w] : 0ull);
      if (part) v = (v & tail_mask) | (old & ~tail_mask);
      crow[gw] = v;
    }
  }
}

int gf2_m4rm_dev(Ctx *c, int M, int N, int K, int alpha, const uint64_t *A, size_t lda,
                 const uint64_t *B, size_t ldb, int beta, uint64_t *C, size_t ldc) {
  if (M <= 0 || N <= 0) return ST_OK;
  const int Nw = (N + 63) / 64;
  const uint64_t tail = (N & 63) ? ((1ull << (N & 63)) - 1ull) : ~0ull;
  // Eight words and four rows per thread per CTA; one row when that leaves
  // fewer than two CTAs per SM; two words as well when even that does (few
  // rows, e.g. a panel's 64 pivot rows against a wide B: the tables, which
  // dominate there, are then built by four times as many CTAs, each a
  // quarter of them).
  auto smem_for = [](int bw) { return (4 * bw * 256 + M4_KC * bw) * 8; };
  if (int st = ctx_smem_attr(c, (const void *)gf2_m4rm_kernel<4, 8>, smem_for(8),
                             "cudaFuncSetAttribute(gf2_m4rm)"))
    return st;
  if (int st = ctx_smem_attr(c, (const void *)gf2_m4rm_kernel<1, 8>, smem_for(8),
                             "cudaFuncSetAttribute(gf2_m4rm)"))
    return st;
  const size_t enough = 2u * c->num_sms;
  const int gx8 = (Nw + 7) / 8, gx2 = (Nw + 1) / 2;
  const int gy4 = (M + M4_THREADS * 4 - 1) / (M4_THREADS * 4), gy1 = (M + M4_THREADS - 1) / M4_THREADS;
  int pi = prof_begin(c, "gf2_m4rm");
  if ((size_t)gx8 * gy4 >= enough)
    pdl_launch(gf2_m4rm_kernel<4, 8>, dim3(gx8, gy4), M4_THREADS, smem_for(8), c->stream,
        A, lda, B, ldb, C, ldc, M, Nw, K, tail, alpha, beta);
  else if ((size_t)gx8 * gy1 >= enough)
    pdl_launch(gf2_m4rm_kernel<1, 8>, dim3(gx8, gy1), M4_THREADS, smem_for(8), c->stream,
        A, lda, B, ldb, C, ldc, M, Nw, K, tail, alpha, beta);
  else
    pdl_launch(gf2_m4rm_kernel<1, 2>, dim3(gx2, gy1), M4_THREADS, smem_for(2), c->stream,
        A, lda, B, ldb, C, ldc, M, Nw, K, tail, alpha, beta);
  prof_end(c, pi);
  ctx_launched(c);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? ST_OK : ctx_cuda(c, e, "gf2_m4rm launch");
}

// ------------------------------------------------- int8 expansion for TC
// Four bits to four 0/1 bytes: the multiplier's copies at bits 0, 7, 14, 21
// put bit i at bit 8i.
__device__ __forceinline__ uint32_t spread4(uint32_t nibble) {
  return ((nibble & 15u) * 0x00204081u) & 0x01010101u;
}
// Sixteen bits to sixteen 0/1 bytes.
__device__ __forceinline__ uint4 spread16(uint32_t h) {
  return make_uint4(spread4(h), spread4(h >> 4), spread4(h >> 8), spread4(h >> 12));
}

// Ab[r][k] = bit k0+k of row r of A (K-major bytes, row pitch Kp, a multiple
// of 64; bytes past kc are never read).  Sixteen bits to a 16-byte store per
// thread, lanes along the row.  Bound: the bytes written (16384^2: 268 MB;
// four bytes a thread and an index division took 209 us).
constexpr int UNPACK_ROWS = 8;  // rows (warps) per CTA
__global__ void __launch_bounds__(32 * UNPACK_ROWS)
    gf2_unpack_rows_kernel(const uint64_t *A, size_t lda, int M, int k0,
                           uint8_t *out, int Kp) {
  pdl_enter();
  const int per = Kp / 16;
  for (int r = blockIdx.y * UNPACK_ROWS + threadIdx.y; r < M; r += gridDim.y * UNPACK_ROWS) {
    const uint16_t *src = reinterpret_cast<const uint16_t *>(A + (size_t)r * lda + (k0 >> 6));
    uint4 *dst = reinterpret_cast<uint4 *>(out + (size_t)r * Kp);
    for (int q = blockIdx.x * 32 + threadIdx.x; q < per; q += gridDim.x * 32)
      dst[q] = spread16(src[q]);
  }
}

// Bb[n][k] = bit n of row k0+k of B.  A CTA takes UNPACK_W words of UNPACK_K
// rows: a warp holds 32 rows' words, a 32 x 32 bit transposition per half word
// (five exchanges of bit blocks between lanes) gives each column's 32 bits,
// kept in shared memory; then a warp writes a column's UNPACK_K bytes at
// once, 16 per lane.  Bound: the bytes written (16384^2, 268 MB: 580 us with
// one column per thread and a 64-bit shift per byte, 162 us with 16-byte
// stores a row pitch apart from the lanes of the transposition).
constexpr int UNPACK_K = 512, UNPACK_W = 4, UNPACK_WARPS = 8;
__device__ __forceinline__ uint32_t transpose32(uint32_t x, int lane) {
#pragma unroll
  for (int j = 16; j > 0; j >>= 1) {
    const uint32_t low = j == 16  ? 0x0000ffffu
                         : j == 8 ? 0x00ff00ffu
                         : j == 4 ? 0x0f0f0f0fu
                         : j == 2 ? 0x33333333u
                                  : 0x55555555u;
    const uint32_t y = __shfl_xor_sync(0xffffffffu, x, j);
    x = (lane & j) ? (x & ~low) | ((y & ~low) >> j) : (x & low) | ((y & low) << j);
  }
  return x;
}
__global__ void __launch_bounds__(32 * UNPACK_WARPS)
    gf2_unpack_cols_kernel(const uint64_t *B, size_t ldb, int k0, int kc, int N,
                           uint8_t *out, int Kp) {
  pdl_enter();
  __shared__ uint32_t bits[64 * UNPACK_W][UNPACK_K / 32 + 1];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int w0 = blockIdx.x * UNPACK_W, kb0 = blockIdx.y * UNPACK_K;
  const int words = min(UNPACK_W, (N + 63) / 64 - w0);
  for (int u = wid; u < UNPACK_K / 32; u += UNPACK_WARPS) {
    const int k = kb0 + 32 * u + lane;
    const uint64_t *src = B + (size_t)(k0 + k) * ldb + w0;
    uint64_t v[UNPACK_W];
#pragma unroll
    for (int j = 0; j < UNPACK_W; ++j) v[j] = k < kc && j < words ? src[j] : 0ull;
#pragma unroll
    for (int j = 0; j < UNPACK_W; ++j) {
      bits[64 * j + lane][u] = transpose32((uint32_t)v[j], lane);
      bits[64 * j + lane + 32][u] = transpose32((uint32_t)(v[j] >> 32), lane);
    }
  }
  __syncthreads();
  const int kk = 16 * lane;  // this lane's bytes of a column
  if (kb0 + kk >= Kp) return;
  const int cols = min(64 * UNPACK_W, N - 64 * w0);
  for (int n = wid; n < cols; n += UNPACK_WARPS) {
    const uint32_t h = bits[n][kk >> 5] >> (kk & 16);
    *reinterpret_cast<uint4 *>(out + (size_t)(64 * w0 + n) * Kp + kb0 + kk) = spread16(h);
  }
}
static_assert(UNPACK_K == 32 * 16, "a warp writes a column's bytes at once");

static void unpack_rows(Ctx *c, const uint64_t *A, size_t lda, int M, int k0, uint8_t *out, int Kp) {
  // one pass a warp up to 16 CTAs an SM, then more
  const int gy = std::min((M + UNPACK_ROWS - 1) / UNPACK_ROWS, c->num_sms * 16);
  const int gx = std::max(1, std::min((Kp / 16 + 31) / 32, c->num_sms * 16 / gy));
  pdl_launch(gf2_unpack_rows_kernel, dim3(gx, gy), dim3(32, UNPACK_ROWS), 0, c->stream, A, lda, M,
             k0, out, Kp);
  ctx_launched(c);
}
static void unpack_cols(Ctx *c, const uint64_t *B, size_t ldb, int k0, int kc, int N, uint8_t *out,
                        int Kp, bool early) {
  const int Nw = (N + 63) / 64;
  const dim3 grid((Nw + UNPACK_W - 1) / UNPACK_W, (Kp + UNPACK_K - 1) / UNPACK_K);
  pdl_launch_if(early, gf2_unpack_cols_kernel, grid, 32 * UNPACK_WARPS, 0, c->stream, B, ldb, k0, kc, N,
                out, Kp);
  ctx_launched(c);
}

int gf2_gemm_dev(Ctx *c, int kernel, int M, int N, int K, int alpha, const uint64_t *A,
                 size_t lda, const uint64_t *B, size_t ldb, int beta, uint64_t *C, size_t ldc) {
  if (M < 0 || N < 0 || K < 0) return ctx_fail(c, ST_ARG, "negative dimension");
  if (M == 0 || N == 0) return ST_OK;
  const int Nw = (N + 63) / 64, Kw = (K + 63) / 64;
  if (ldc < (size_t)Nw || (K > 0 && (lda < (size_t)Kw || ldb < (size_t)Nw)))
    return ctx_fail(c, ST_ARG, "leading dimension smaller than the row length");
  alpha &= 1;
  beta &= 1;
  if (kernel == GF2_AUTO) kernel = c->gf2_kernel == GF2_AUTO ? GF2_TC : c->gf2_kernel;
  if (K == 0 || alpha == 0 || kernel == GF2_M4RM)
    return gf2_m4rm_dev(c, M, N, (alpha && K > 0) ? K : 0, alpha, A, lda, B, ldb, beta, C, ldc);
  // tensor cores on 0/1 bytes, K in chunks of 32768 (the counts stay exact)
  const int kcmax = std::min(K, ZP_KCHUNK);
  const int Kpmax = (kcmax + 63) & ~63;
  void *w = nullptr;
  int st = ctx_workspace(c, (size_t)(M + N) * Kpmax + 256, &w);
  if (st) return st;
  uint8_t *Ab = static_cast<uint8_t *>(w);
  uint32_t b = (uint32_t)beta;
  for (int k0 = 0; k0 < K; k0 += ZP_KCHUNK) {
    const int kc = std::min(ZP_KCHUNK, K - k0);
    const int Kp = (kc + 63) & ~63;
    uint8_t *Bb = Ab + (size_t)M * Kp;
    int pi = prof_begin(c, "gf2_unpack");
    unpack_rows(c, A, lda, M, k0, Ab, Kp);
    unpack_cols(c, B, ldb, k0, kc, N, Bb, Kp, gf2_early(M, N, kc));
    prof_end(c, pi);
    if ((st = gf2_gemm_tc_planes(c, M, N, kc, Ab, Bb, Kp, 1u, b, C, ldc))) return st;
    b = 1;
  }
  return ST_OK;
}

// ---------------------------------------------- host-pointer row blocks
constexpr int GF2_PIPE_MIN_ROWS = 512;

bool gf2_gemm_pipelined(const Ctx *c, int M, int N, int K, int alpha) {
  const int kernel = c->gf2_kernel == GF2_AUTO ? GF2_TC : c->gf2_kernel;
  return kernel == GF2_TC && (alpha & 1) && K > 0 && K <= ZP_KCHUNK && N > 0 &&
         M >= 2 * GF2_PIPE_MIN_ROWS;
}

int gf2_gemm_host_rows(Ctx *c, int M, int N, int K, const uint64_t *hA, size_t lda,
                       const uint64_t *hB, size_t ldb, int beta, uint64_t *hC, size_t ldc,
                       uint64_t *dA, uint64_t *dB, uint64_t *dC) {
  if (!gf2_gemm_pipelined(c, M, N, K, 1)) return ctx_fail(c, ST_ARG, "not a pipelined gemm");
  if (int st = ctx_pipe(c)) return st;
  const int Kp = (K + 63) & ~63;
  const int Kw = (K + 63) / 64, Nw = (N + 63) / 64;
  void *w = nullptr;
  if (int st = ctx_workspace(c, (size_t)(M + N) * Kp + 256, &w)) return st;
  uint8_t *Ab = static_cast<uint8_t *>(w), *Bb = Ab + (size_t)M * Kp;
  // row blocks: a multiple of 128 rows (the tensor-core tile), at most
  // PIPE_MAX_BLOCKS of them
  const int per = (M + PIPE_MAX_BLOCKS - 1) / PIPE_MAX_BLOCKS;
  const int rb = std::max(GF2_PIPE_MIN_ROWS, (per + 127) / 128 * 128);
  const int nblk = (M + rb - 1) / rb;
  cudaEvent_t *ready = c->pipe_ev, *done = c->pipe_ev + PIPE_MAX_BLOCKS;
  cudaEvent_t ev_start = c->pipe_ev[2 * PIPE_MAX_BLOCKS], ev_b = c->pipe_ev[2 * PIPE_MAX_BLOCKS + 1],
              ev_out = c->pipe_ev[2 * PIPE_MAX_BLOCKS + 2];
  const size_t rowA = (size_t)Kw * 8, rowB = (size_t)Nw * 8;
  // C's rows come in when b = 1, and for the bits past column N of each
  // row's last word, which the product leaves as they were
  const bool cin = (beta & 1) || (N & 63);
  cudaError_t e = cudaEventRecord(ev_start, c->stream);
  if (e == cudaSuccess) e = cudaStreamWaitEvent(c->copy_in, ev_start, 0);
  if (e == cudaSuccess) e = cudaStreamWaitEvent(c->copy_out, ev_start, 0);
  if (e == cudaSuccess)
    e = cudaMemcpy2DAsync(dB, rowB, hB, ldb * 8, rowB, (size_t)K, cudaMemcpyHostToDevice,
                          c->copy_in);
  if (e == cudaSuccess) e = cudaEventRecord(ev_b, c->copy_in);
  for (int j = 0; e == cudaSuccess && j < nblk; ++j) {
    const int r0 = j * rb, rows = std::min(rb, M - r0);
    e = cudaMemcpy2DAsync(dA + (size_t)r0 * Kw, rowA, hA + (size_t)r0 * lda, lda * 8, rowA,
                          (size_t)rows, cudaMemcpyHostToDevice, c->copy_in);
    if (e == cudaSuccess && cin)
      e = cudaMemcpy2DAsync(dC + (size_t)r0 * Nw, rowB, hC + (size_t)r0 * ldc, ldc * 8, rowB,
                            (size_t)rows, cudaMemcpyHostToDevice, c->copy_in);
    if (e == cudaSuccess) e = cudaEventRecord(ready[j], c->copy_in);
  }
  // B's bytes once; each block's A bytes in its own part of the workspace
  int st = ST_OK;
  if (e == cudaSuccess) e = cudaStreamWaitEvent(c->stream, ev_b, 0);
  if (e == cudaSuccess) {
    int pi = prof_begin(c, "gf2_unpack");
    unpack_cols(c, dB, (size_t)Nw, 0, K, N, Bb, Kp, false);
    prof_end(c, pi);
    e = cudaGetLastError();
  }
  for (int j = 0; e == cudaSuccess && !st && j < nblk; ++j) {
    const int r0 = j * rb, rows = std::min(rb, M - r0);
    uint8_t *Aj = Ab + (size_t)r0 * Kp;
    e = cudaStreamWaitEvent(c->stream, ready[j], 0);
    if (e != cudaSuccess) break;
    int pi = prof_begin(c, "gf2_unpack");
    unpack_rows(c, dA + (size_t)r0 * Kw, (size_t)Kw, rows, 0, Aj, Kp);
    prof_end(c, pi);
    st = gf2_gemm_tc_planes(c, rows, N, K, Aj, Bb, Kp, 1u, (uint32_t)(beta & 1),
                            dC + (size_t)r0 * Nw, (size_t)Nw);
    if (st) break;
    e = cudaEventRecord(done[j], c->stream);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(c->copy_out, done[j], 0);
    if (e == cudaSuccess)
      e = cudaMemcpy2DAsync(hC + (size_t)r0 * ldc, ldc * 8, dC + (size_t)r0 * Nw, rowB, rowB,
                            (size_t)rows, cudaMemcpyDeviceToHost, c->copy_out);
  }
  // the handle stream ends after the last copy out
  if (e == cudaSuccess && !st) e = cudaEventRecord(ev_out, c->copy_out);
  if (e == cudaSuccess && !st) e = cudaStreamWaitEvent(c->stream, ev_out, 0);
  if (e != cudaSuccess || st) {
    // copies already queued may still use the caller's buffers
    cudaStreamSynchronize(c->copy_in);
    cudaStreamSynchronize(c->copy_out);
    return st ? st : ctx_cuda(c, e, "pipelined gf2 gemm");
  }
  return ST_OK;
}

// --------------------------------------------------------------- echelon
//
// Per 64-column panel (one word per row), the Z/p panel scheme of
// echelon.cu with GF(2) arithmetic:
//  * gf2_heads_kernel: first set bit of each row's panel word, the head
//    histogram and the last row with a nonzero word;
//  * gf2_search_kernel: the reference's pivot choice on a window in registers,
//    and lazily past it;
//  * the host replays the transpositions and moves the rows;
//  * gf2_solve_kernel: per row from the first pivot down to the last
//    possibly nonzero row, the reference's elimination steps on the word
//    (pivot k XOR-ed in when bit pcol_k is set) give the multipliers; pivot
//    rows become U_k, rows below become zero; one CTA solves the block's words of
//    U12 = L11^-1 A12 besides;
//  * gf2_block_words_kernel: C ^= L21 U12 on the block's words; right of the block, once per
//    block, gf2_block_solve_kernel and one tensor-core (few rows: M4RM) update.
constexpr int GW = 64;
constexpr uint8_t GF2_HEAD_NONE = 64;

__device__ __forceinline__ int gf2_row_at(int pos, const int *p2r, const int *stamp, int epoch) {
  return stamp[pos] == epoch ? p2r[pos] : pos;
}

constexpr int GF2_HEADS_THREADS = 256;
// hist counts only the rows from position hist0 on (those the search reads
// lazily, past its register window).
__global__ void __launch_bounds__(GF2_HEADS_THREADS)
    gf2_heads_kernel(const uint64_t *D, size_t ld, int i0, int m, int wc,
                     uint64_t pmask, uint8_t *head, uint8_t *act,
                     int *hist, int *last, int hist0) {
  pdl_enter();
  __shared__ int s_last;
  __shared__ int s_hist[GW + 1];
  if (threadIdx.x == 0) s_last = -1;
  if (threadIdx.x <= GW) s_hist[threadIdx.x] = 0;
  __syncthreads();
  int my_last = -1;
  for (int r = i0 + blockIdx.x * blockDim.x + threadIdx.x; r < m; r += gridDim.x * blockDim.x) {
    const uint64_t v = D[(size_t)r * ld + wc] & pmask;
    const int h = v ? __ffsll((long long)v) - 1 : GF2_HEAD_NONE;
    head[r] = (uint8_t)h;
    act[r] = v != 0ull;
    if (r >= hist0) atomicAdd(&s_hist[h], 1);
    if (v) my_last = r;
  }
  if (my_last >= 0) atomicMax(&s_last, my_last);
  __syncthreads();
  if (threadIdx.x == 0 && s_last >= 0) atomicMax(last, s_last);
  if (threadIdx.x <= GW && s_hist[threadIdx.x]) atomicAdd(&hist[threadIdx.x], s_hist[threadIdx.x]);
}

// One warp.  The words of positions i0 .. i0 + GF2_WR - 1 (the window) sit
// in registers by columns: lane l holds the window's bits of columns l and l +
// 32, position i0 + e at bit e, and they are eliminated
// eagerly: when the pivot of column c is chosen, every other window row at
// or below the current position with bit c set gets the pivot word XOR-ed
// in, so the pivot of a column is the first window position at or below
// the current one with the bit set, and a
// pivot row's word is its final U_k (reduced by the pivots before it, as the
// reference's elimination leaves it).  A column step hands the column's 128 bits
// to the warp (four exchanges); the pivot position, the bits to clear and the two
// bits to trade follow from them alike in every lane, and each lane
// applies them to its own columns where those hold a pivot bit.  (Rows on
// lanes, the pivot from four ballots and __ffs, took 900 cycles a column, 30 us
// a panel.)  Rows past the window are tested
// lazily: the pivot rows are also kept as a reduced basis g_k (bit pcol_j of
// g_k is delta_kj) with, per column c, the mask M[c] = (1 << c) | sum_k
// g_k[c] << pcol_k, so bit c of a row reduced by all pivots so far is
// parity(v & M[c]); head[] holds a lower bound of the first set bit of each
// such row's reduced word and cnt[h] counts them by that bound, so the scan
// past the window runs only when a row there may hold the pivot.  Outputs:
// Gf2PanelOut, U (the pivot rows' final words); the host's copy as words of a
// value and the sequence number (as the Z/p search's).  Resets *last_act and
// hist[] for the next panel.
constexpr int GF2_WR = 128;               // window positions
constexpr int GF2_WU = GF2_WR / 32;       // words of a column
enum : int {
  GF2_W_T = 0,     // pivots
  GF2_W_LAST = 1,  // last_pos
  GF2_W_PIV = 2,   // per pivot: transposition target
  GF2_WORDS = GF2_W_PIV + GW
};
static_assert(PANEL_WORDS_OFF + GF2_WORDS * 8 <= PANEL_FLAG_OFF, "words below the flag");
__global__ void __launch_bounds__(32)
    gf2_search_kernel(const uint64_t *D, size_t ld, int i0, int m, int wc, int w,
                      uint64_t pmask, uint8_t *head, const uint8_t *act,
                      int *hist, int *last_act, int *p2r,
                      int *stamp, int epoch, uint64_t *Uout, uint32_t *pcol_out,
                      volatile uint64_t *hout, uint32_t seq) {
  pdl_enter();
  constexpr unsigned FULL = 0xffffffffu;
  __shared__ uint64_t G[GW], M[GW];
  __shared__ int s_pcol[GW], s_tq[GW], s_wr[GF2_WR];
  __shared__ int s_cnt[GW + 1];
  const int lane = threadIdx.x;
  const int wend = min(i0 + GF2_WR, m);  // positions past the window start here
  // cnt: the rows from wend on (the heads kernel counted only those)
  for (int h = lane; h <= GW; h += 32) {
    s_cnt[h] = hist[h];
    hist[h] = 0;
  }
  uint32_t c0[GF2_WU], c1[GF2_WU];  // columns lane, lane + 32
  {
    uint64_t v[GF2_WU];
#pragma unroll
    for (int u = 0; u < GF2_WU; ++u) {
      const int pos = i0 + lane + 32 * u;
      s_wr[lane + 32 * u] = pos < m ? pos : -1;  // row at the position: none has moved yet
      v[u] = pos < m ? D[(size_t)pos * ld + wc] & pmask : 0ull;
    }
#pragma unroll
    for (int u = 0; u < GF2_WU; ++u) {
      c0[u] = transpose32((uint32_t)v[u], lane);
      c1[u] = transpose32((uint32_t)(v[u] >> 32), lane);
    }
  }
  M[lane] = 1ull << lane;
  M[lane + 32] = 1ull << (lane + 32);
  __syncwarp();
  // the word of the window row at position i0 + e, e < 64 (the same in every lane)
  auto row_word = [&](int e) -> uint64_t {
    const uint32_t a = e < 32 ? c0[0] : c0[1], b = e < 32 ? c1[0] : c1[1];
    const uint32_t lo = __ballot_sync(FULL, (a >> (e & 31)) & 1u);
    const uint32_t hi = __ballot_sync(FULL, (b >> (e & 31)) & 1u);
    return (uint64_t)hi << 32 | lo;
  };
  auto set_row = [&](int e, uint64_t word) {
    const uint32_t b0 = e < 32 ? 1u << e : 0u, b1 = e < 32 ? 0u : 1u << (e & 31);
    const bool lo = (word >> lane) & 1ull, hi = (word >> (lane + 32)) & 1ull;
    c0[0] = lo ? c0[0] | b0 : c0[0] & ~b0;
    c0[1] = lo ? c0[1] | b1 : c0[1] & ~b1;
    c1[0] = hi ? c1[0] | b0 : c1[0] & ~b0;
    c1[1] = hi ? c1[1] | b1 : c1[1] & ~b1;
  };
  // The basis g_k and masks M: pivot U at column c makes g_k ^= U where g_k
  // has bit c, and M[c'] ^= M[c] for the columns c' > c where U has a bit.
  // Only the scan past the window uses them, so they are built when it first
  // runs (replaying the pivots so far) and kept from then on.
  auto basis_add = [&](uint64_t U, int c, int k) {
    const uint64_t mcol = M[c], b = 1ull << c;
    __syncwarp();
    if (lane < k && (G[lane] & b)) G[lane] ^= U;
    if (lane + 32 < k && (G[lane + 32] & b)) G[lane + 32] ^= U;
    for (int cc = lane; cc < w; cc += 32)
      if (cc > c && ((U >> cc) & 1ull)) M[cc] ^= mcol;
    __syncwarp();
    if (lane == 0) G[k] = U;
    __syncwarp();
  };
  bool basis = false;
  int t = 0;  // pivots so far; the current position is i0 + t, bit t
#pragma unroll 1
  for (int col = 0; col < w && i0 + t < m; ++col) {
    // the column's bits, at or below the current position
    uint32_t v[GF2_WU];
#pragma unroll
    for (int u = 0; u < GF2_WU; ++u) v[u] = __shfl_sync(FULL, col < 32 ? c0[u] : c1[u], col & 31);
    static_assert(GF2_WU == 4 && GW <= 64, "four words, the current position in the first two");
    v[0] &= t < 32 ? ~0u << t : 0u;
    v[1] &= t < 32 ? ~0u : ~0u << (t & 31);
    const int wq = v[0] ? 0 : v[1] ? 1 : v[2] ? 2 : 3;  // the pivot's word, its bit
    const uint32_t x = v[0] ? v[0] : v[1] ? v[1] : v[2] ? v[2] : v[3];
    const uint32_t pb = x & (0u - x);
    int q = -1;  // the pivot's position - i0
    if (x) {
      q = 32 * wq + (31 - __clz((int)pb));
      // rows to clear (the pivot's own bit stays); rows t and q trade places,
      // row t having a 0 in this column when q > t
      const uint32_t tb = 1u << (t & 31);
      const bool swap = q != t;
      uint32_t e[GF2_WU], sw[GF2_WU];
#pragma unroll
      for (int u = 0; u < GF2_WU; ++u) {
        e[u] = v[u] ^ (u == wq ? pb : 0u);
        sw[u] = swap ? (u == wq ? pb : 0u) ^ (u == (t >> 5) ? tb : 0u) : 0u;
      }
      auto apply = [&](uint32_t(&cc)[GF2_WU]) {
        const uint32_t cq = wq == 0 ? cc[0] : wq == 1 ? cc[1] : wq == 2 ? cc[2] : cc[3];
        const uint32_t ct = t < 32 ? cc[0] : cc[1];
        const bool bq = (cq & pb) != 0u, bt = (ct & tb) != 0u;
#pragma unroll
        for (int u = 0; u < GF2_WU; ++u) cc[u] ^= (bq ? e[u] : 0u) ^ (bq != bt ? sw[u] : 0u);
      };
      apply(c0);
      apply(c1);
      if (swap && lane == 0) {
        const int r = s_wr[t];
        s_wr[t] = s_wr[q];
        s_wr[q] = r;
      }
    } else {
      // none in the window: rows past it whose bound allows a pivot here
      int cand = 0;
      for (int h = lane; h <= col; h += 32) cand += s_cnt[h];
      cand = __reduce_add_sync(FULL, cand);
      if (cand == 0) continue;  // no pivot in this column
      if (!basis) {
        for (int k = 0; k < t; ++k) basis_add(row_word(k), s_pcol[k], k);
        basis = true;
      }
      uint64_t pw = 0ull;
      for (int base = wend; base < m && cand > 0; base += 32) {
        const int pos = base + lane;
        int is_cand = 0, hit = 0;
        uint64_t pv = 0ull;
        if (pos < m) {
          const int r = gf2_row_at(pos, p2r, stamp, epoch);
          const int hr = head[r];
          if (hr <= col) {
            is_cand = 1;
            pv = D[(size_t)r * ld + wc] & pmask;
            int c = col;
            while (c < w && !(__popcll(pv & M[c]) & 1)) ++c;
            const int hn = c < w ? c : GF2_HEAD_NONE;
            if (hn != hr) {
              head[r] = (uint8_t)hn;
              atomicSub(&s_cnt[hr], 1);
              atomicAdd(&s_cnt[hn], 1);
            }
            hit = c == col;
          }
        }
        cand -= __popc(__ballot_sync(FULL, is_cand));
        const unsigned hb = __ballot_sync(FULL, hit);
        if (hb) {
          const int l = __ffs(hb) - 1;
          q = base + l - i0;
          pw = __shfl_sync(FULL, pv, l);
          break;
        }
      }
      __syncwarp();
      if (q < 0) continue;  // no pivot in this column
      // the pivot row reduced by the pivots so far: U = v ^ sum_{k: v bit pcol_k} g_k
      uint64_t xg = 0;
      if (lane < t && ((pw >> s_pcol[lane]) & 1ull)) xg ^= G[lane];
      if (lane + 32 < t && ((pw >> s_pcol[lane + 32]) & 1ull)) xg ^= G[lane + 32];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) xg ^= __shfl_xor_sync(FULL, xg, o);
      const uint64_t U = pw ^ xg;
      // transposition (i, q): the pivot row takes position i; the window row
      // there (bit col clear, reduced by every pivot) goes to position q, with
      // the bound of its reduced word
      const uint64_t vi = row_word(t);
      const int ap = gf2_row_at(i0 + q, p2r, stamp, epoch);  // before the maps change
      __syncwarp();
      if (lane == 0) {
        const int ri = s_wr[t];
        const int hv = vi ? __ffsll((long long)vi) - 1 : GF2_HEAD_NONE;
        atomicSub(&s_cnt[head[ap]], 1);  // the pivot row leaves the counts
        head[ri] = (uint8_t)hv;
        atomicAdd(&s_cnt[hv], 1);
        p2r[i0 + q] = ri;
        stamp[i0 + q] = epoch;
        s_wr[t] = ap;
      }
      __syncwarp();
      set_row(t, U);
    }
    if (basis) basis_add(row_word(t), col, t);
    if (lane == 0) {
      s_pcol[t] = col;
      s_tq[t] = i0 + q;
    }
    ++t;
    __syncwarp();
  }
  const int i = i0 + t;
  // last final position of a non-pivot row with a nonzero word
  int hi = i - 1;
  for (int k = lane; k < t; k += 32) hi = max(hi, s_tq[k]);
  hi = __reduce_max_sync(FULL, hi);
  int last = -1;
#pragma unroll
  for (int u = 0; u < GF2_WU; ++u) {
    const int pos = i0 + lane + 32 * u, r = s_wr[lane + 32 * u];
    if (pos >= i && pos <= hi && r >= 0 && act[r]) last = max(last, pos);
  }
  for (int pos = max(i, wend) + lane; pos <= hi && pos < m; pos += 32)
    if (act[gf2_row_at(pos, p2r, stamp, epoch)]) last = max(last, pos);
  last = __reduce_max_sync(FULL, last);
  const auto word = [seq](uint32_t v) { return (uint64_t)seq << 32 | v; };
  if (lane == 0) {
    const int la = *last_act;
    if (la > hi) last = la;
    *last_act = -1;
    hout[GF2_W_T] = word((uint32_t)t);
    hout[GF2_W_LAST] = word((uint32_t)max(last, 0));
  }
  // rows 0 .. t - 1 of the window are the pivot rows
  uint64_t U[2];
#pragma unroll
  for (int u = 0; u < 2; ++u)
    U[u] = (uint64_t)transpose32(c1[u], lane) << 32 | transpose32(c0[u], lane);
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    const int k = lane + 32 * u;
    if (k < t) {
      hout[GF2_W_PIV + k] = word((uint32_t)s_tq[k]);
      Uout[k] = U[u];
      pcol_out[k] = (uint32_t)s_pcol[k];
    }
  }
}

// Rows i0..r1 at their final positions: the reference's elimination steps
// on the panel word give the multipliers (L11 row of pivot row k over the
// pivots before it; L21 row of the rows below over all t) and the final
// word (U_k; zero below).  One thread per row.  With Lb the multipliers also go
// into the block's rows of bits (GB words a row, at bit offset off; the caller
// zeroed the block's rows) and, when the block has words right of the panel (w1
// .. wend, at most GB), the first CTA, which holds all pivot rows, solves U12 =
// L11^-1 A12 there in place: a warp per word as gf2_l11_solve_kernel.  (The
// three steps as kernels of their own took 7.3, 3.2 and 5.6 us.)
constexpr int GB = 8;  // panels (words) per block of delayed updates
constexpr int GF2_SOLVE_THREADS = 256;
__device__ __forceinline__ void gf2_u12_word(uint64_t *D, size_t ld, int i0, int t, int w,
                                             uint64_t l0, uint64_t l1, int lane) {
  uint64_t x0 = lane < t ? D[(size_t)(i0 + lane) * ld + w] : 0ull;
  uint64_t x1 = lane + 32 < t ? D[(size_t)(i0 + lane + 32) * ld + w] : 0ull;
  for (int k = 0; k < t - 1; ++k) {
    const uint64_t xk = __shfl_sync(0xffffffffu, k < 32 ? x0 : x1, k & 31);
    if (lane > k && ((l0 >> k) & 1ull)) x0 ^= xk;
    if ((l1 >> k) & 1ull) x1 ^= xk;  // L11 is strictly lower: bit k set means k < the row
  }
  if (lane < t) D[(size_t)(i0 + lane) * ld + w] = x0;
  if (lane + 32 < t) D[(size_t)(i0 + lane + 32) * ld + w] = x1;
}
__global__ void __launch_bounds__(GF2_SOLVE_THREADS)
    gf2_solve_kernel(uint64_t *D, size_t ld, int i0, int r1, int wc, uint64_t pmask, int t,
                     const uint32_t *pcol, const uint64_t *Uin, uint64_t *L11, uint64_t *L21,
                     uint64_t *Lb, int off, int w1, int wend) {
  pdl_enter();
  __shared__ uint64_t sU[GW], sL[GW];
  __shared__ int sP[GW];
  if (threadIdx.x < GW) {
    sU[threadIdx.x] = threadIdx.x < t ? Uin[threadIdx.x] : 0ull;
    sP[threadIdx.x] = threadIdx.x < t ? (int)pcol[threadIdx.x] : 0;
    sL[threadIdx.x] = 0ull;
  }
  __syncthreads();
  static_assert(GF2_SOLVE_THREADS >= GW, "the first CTA's first pass holds the pivot rows");
  const int r0 = i0 + t;
  for (int pos = i0 + blockIdx.x * blockDim.x + threadIdx.x; pos <= r1;
       pos += gridDim.x * blockDim.x) {
    uint64_t *x = D + (size_t)pos * ld + wc;
    const uint64_t old = *x;
    uint64_t v = old & pmask;
    const int kk = pos - i0, lim = kk < t ? kk : t;
    uint64_t l = 0;
#pragma unroll 4
    for (int k = 0; k < lim; ++k) {
      const bool b = (v >> sP[k]) & 1ull;
      v ^= b ? sU[k] : 0ull;
      l |= (uint64_t)b << k;
    }
    *x = (old & ~pmask) | v;
    if (kk < t) {
      L11[kk] = l;
      sL[kk] = l;
    } else {
      L21[pos - r0] = l;
    }
    if (Lb) {
      uint64_t *row = Lb + (size_t)pos * GB;
      const int wq = off >> 6, sh = off & 63;
      row[wq] |= l << sh;
      if (sh && sh + t > 64) row[wq + 1] |= l >> (64 - sh);
    }
  }
  if (Lb == nullptr || blockIdx.x != 0 || w1 >= wend) return;
  __syncthreads();
  const int lane = threadIdx.x & 31, w = w1 + (threadIdx.x >> 5);
  static_assert(GF2_SOLVE_THREADS / 32 >= GB, "a warp per word of the block");
  if (w < wend) gf2_u12_word(D, ld, i0, t, w, sL[lane], sL[lane + 32], lane);
}

// C ^= L21 U12 on the words w1 .. w1 + nw - 1 (nw <= GB) of the rows r0 .. r1 of
// D: the words of the panel's block right of it.  U12: rows i0 .. i0 + t - 1.
// Sixteen tables of the XORs of four rows of U12 in shared memory, a thread
// per row and word (a row's words on neighbouring threads), sixteen lookups.
// The general four-Russians kernel, which builds tables of 256 entries per word
// pair, took 14 us a panel here.
constexpr int GF2_BW_THREADS = 256;
__global__ void __launch_bounds__(GF2_BW_THREADS)
    gf2_block_words_kernel(uint64_t *D, size_t ld, int n, int i0, int t, int w1, int nw, int r0,
                           int r1, const uint64_t *L21) {
  pdl_enter();
  __shared__ uint64_t sU[GW][GB], T[GW / 4][16][GB];
  for (int e = threadIdx.x; e < GW * GB; e += GF2_BW_THREADS) {
    const int k = e / GB, w = e % GB;
    // (bits past column n of the last word stay as they are)
    const int cols = n - 64 * (w1 + w);
    const uint64_t mask = cols >= 64 ? ~0ull : cols > 0 ? (1ull << cols) - 1ull : 0ull;
    sU[k][w] = k < t && w < nw ? D[(size_t)(i0 + k) * ld + w1 + w] & mask : 0ull;
  }
  __syncthreads();
  {
    static_assert(GF2_BW_THREADS == GW / 4 * 16, "a table entry per thread");
    const int g = threadIdx.x >> 4, e = threadIdx.x & 15;
#pragma unroll
    for (int w = 0; w < GB; ++w) {
      uint64_t v = 0;
#pragma unroll
      for (int b = 0; b < 4; ++b) v ^= (e >> b) & 1 ? sU[4 * g + b][w] : 0ull;
      T[g][e][w] = v;
    }
  }
  __syncthreads();
  const int w = threadIdx.x % GB;
  for (int r = r0 + blockIdx.x * (GF2_BW_THREADS / GB) + threadIdx.x / GB; r <= r1;
       r += gridDim.x * (GF2_BW_THREADS / GB)) {
    const uint64_t l = L21[r - r0];
    uint64_t *x = D + (size_t)r * ld + w1 + w;
    uint64_t v = w < nw ? *x : 0ull;
#pragma unroll
    for (int g = 0; g < GW / 4; ++g) v ^= T[g][(l >> (4 * g)) & 15][w];
    if (w < nw) *x = v;
  }
}

// Row permutation in one launch: each CTA takes GF2_PERM_WORDS words of
// every moved row of D, the last ones of the block's multipliers Lb (nwb words a
// row; 0: none).  Its threads load all their words of the source rows at
// once (at most GF2_PERM_PER each, into registers), wait at the barrier,
// then store them to the destination rows; the CTAs own disjoint words, so
// no grid-wide ordering is needed.  cnt <= 2 * GW rows.
constexpr int GF2_PERM_THREADS = 256, GF2_PERM_WORDS = 16;
constexpr int GF2_PERM_PER = 2 * GW * GF2_PERM_WORDS / GF2_PERM_THREADS;
__global__ void __launch_bounds__(GF2_PERM_THREADS)
    gf2_permute_rows_kernel(uint64_t *D, size_t ld, int nw, uint64_t *Lb, int nwb,
                            const int *src, const int *dst, int cnt) {
  pdl_enter();
  const int own = (nw + GF2_PERM_WORDS - 1) / GF2_PERM_WORDS;
  const bool lb = (int)blockIdx.x >= own;
  uint64_t *X = lb ? Lb : D;
  const size_t ldx = lb ? (size_t)nwb : ld;
  const int nx = lb ? nwb : nw;
  const int w0 = ((int)blockIdx.x - (lb ? own : 0)) * GF2_PERM_WORDS, total = cnt * GF2_PERM_WORDS;
  uint64_t v[GF2_PERM_PER];
#pragma unroll
  for (int u = 0; u < GF2_PERM_PER; ++u) {
    const int e = threadIdx.x + u * GF2_PERM_THREADS, w = w0 + e % GF2_PERM_WORDS;
    v[u] = (e < total && w < nx) ? X[(size_t)src[e / GF2_PERM_WORDS] * ldx + w] : 0ull;
  }
  __syncthreads();
#pragma unroll
  for (int u = 0; u < GF2_PERM_PER; ++u) {
    const int e = threadIdx.x + u * GF2_PERM_THREADS, w = w0 + e % GF2_PERM_WORDS;
    if (e < total && w < nx) X[(size_t)dst[e / GF2_PERM_WORDS] * ldx + w] = v[u];
  }
}

// U12 = L11^-1 A12 over GF(2): pivot rows i0..i0+t-1, words w1 .. nw-1;
// row k gets the XOR of the earlier pivot rows j whose bit is set in
// L11[k].  One warp per word, lane l holding rows l and l + 32: step k hands
// the finished row k to the warp (one shuffle) and the later rows whose
// L11 row has bit k XOR it in (right-looking, 64 short steps per word
// instead of a thread's 2016 dependent XORs).
constexpr int GF2_L11_THREADS = 256;
__global__ void __launch_bounds__(GF2_L11_THREADS)
    gf2_l11_solve_kernel(uint64_t *D, size_t ld, int i0, int t, int w1, int nw,
                         const uint64_t *L11) {
  pdl_enter();
  const int lane = threadIdx.x & 31;
  const int w = w1 + (int)((blockIdx.x * (size_t)GF2_L11_THREADS + threadIdx.x) >> 5);
  if (w >= nw) return;  // whole warps
  const uint64_t l0 = lane < t ? L11[lane] : 0ull, l1 = lane + 32 < t ? L11[lane + 32] : 0ull;
  gf2_u12_word(D, ld, i0, t, w, l0, l1, lane);
}

// U12 = L11^-1 A12 of a whole block, on the words w1 .. nw - 1 of its T pivot rows
// (T <= GB GW, from row i0 of D): L11 is unit lower triangular, row q's bits before
// q in its GB words of Lb.  A CTA solves BS_WORDS words, in shared memory, 64 rows at a time: a
// warp per word substitutes (gf2_u12_word's steps), then the rows after get
// their sums of the 64 solved ones from sixteen tables of four rows, a thread per row
// and word.  Bound: the 64-step chains (eight of about 2500 cycles).  Panel by panel, each panel a
// four-Russians product for the rows before it and a substitution of its
// own, a block of the 32768^2 form took 200 us.
constexpr int BS_WORDS = 2, BS_THREADS = 256;
__global__ void __launch_bounds__(BS_THREADS)
    gf2_block_solve_kernel(uint64_t *D, size_t ld, int i0, int T, int w1, int nw,
                           const uint64_t *Lb) {
  pdl_enter();
  constexpr int ROWS = GB * GW;
  constexpr int LS = ROWS + 2;  // (the 16 words of two rows in different banks)
  __shared__ uint64_t sL[GB * LS], X[ROWS][BS_WORDS], tab[GW / 4][16][BS_WORDS];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int wb = w1 + blockIdx.x * BS_WORDS;
  for (int e = tid; e < ROWS * GB; e += BS_THREADS) {
    const int r = e / GB, q = e % GB;
    sL[q * LS + r] = r < T ? Lb[(size_t)(i0 + r) * GB + q] : 0ull;
  }
  for (int e = tid; e < ROWS * BS_WORDS; e += BS_THREADS) {
    const int r = e / BS_WORDS, j = e % BS_WORDS;
    X[r][j] = r < T && wb + j < nw ? D[(size_t)(i0 + r) * ld + wb + j] : 0ull;
  }
  __syncthreads();
  for (int c = 0; GW * c < T; ++c) {
    const uint64_t *L = sL + c * LS;
    if (warp < BS_WORDS) {
      const int r = GW * c + lane;
      const uint64_t l0 = L[r] & ((1ull << lane) - 1), l1 = L[r + 32] & ((1ull << (lane + 32)) - 1);
      uint64_t x0 = X[r][warp], x1 = X[r + 32][warp];
#pragma unroll 4
      for (int k = 0; k < 32; ++k) {
        const uint64_t xk = __shfl_sync(0xffffffffu, x0, k);
        x0 ^= (l0 >> k) & 1ull ? xk : 0ull;
        x1 ^= (l1 >> k) & 1ull ? xk : 0ull;
      }
#pragma unroll 4
      for (int k = 0; k < 31; ++k) {
        const uint64_t xk = __shfl_sync(0xffffffffu, x1, k);
        x1 ^= (l1 >> (k + 32)) & 1ull ? xk : 0ull;
      }
      X[r][warp] = x0;
      X[r + 32][warp] = x1;
    }
    if (GW * (c + 1) >= T) break;
    __syncthreads();
    for (int e = tid; e < GW / 4 * 16 * BS_WORDS; e += BS_THREADS) {
      const int j = e % BS_WORDS, v = (e / BS_WORDS) & 15, g = e / (16 * BS_WORDS);
      uint64_t x = 0;
#pragma unroll
      for (int b = 0; b < 4; ++b)
        if ((v >> b) & 1) x ^= X[GW * c + 4 * g + b][j];
      tab[g][v][j] = x;
    }
    __syncthreads();
    for (int e = GW * (c + 1) * BS_WORDS + tid; e < T * BS_WORDS; e += BS_THREADS) {
      const int r = e / BS_WORDS, j = e % BS_WORDS;
      const uint64_t l = L[r];
      uint64_t x = X[r][j];
#pragma unroll
      for (int g = 0; g < GW / 4; ++g) x ^= tab[g][(l >> (4 * g)) & 15][j];
      X[r][j] = x;
    }
    __syncthreads();
  }
  __syncthreads();
  for (int e = tid; e < T * BS_WORDS; e += BS_THREADS) {
    const int r = e / BS_WORDS, j = e % BS_WORDS;
    if (wb + j < nw) D[(size_t)(i0 + r) * ld + wb + j] = X[r][j];
  }
}

int gf2_echelon_dev(Ctx *c, int m, int n, uint64_t *D, size_t ld, size_t *rank_out) {
  if (m < 0 || n < 0) return ctx_fail(c, ST_ARG, "negative dimension");
  const int nw = (n + 63) / 64;
  if (m > 0 && n > 0 && ld < (size_t)nw) return ctx_fail(c, ST_ARG, "leading dimension too small");
  size_t rank = 0;
  if (m == 0 || n == 0) {
    *rank_out = 0;
    return ST_OK;
  }
  const size_t out_bytes = GW * sizeof(uint32_t);  // pivot columns
  // p2r, stamp (m each); permutation lists (4 GW); last row (1); histogram (GW + 1)
  const size_t i_bytes =
      (((size_t)2 * m + 4 * GW + 1 + GW + 1) * sizeof(int) + 255) & ~(size_t)255;
  const size_t h_bytes = ((size_t)2 * m + 255) & ~(size_t)255;
  void *base = nullptr;
  const size_t lb_bytes = (size_t)m * GB * 8;  // block bits
  int st = ctx_buffer(c, BUF_GF2_0,
                      out_bytes + i_bytes + h_bytes + (size_t)m * 8 + 2 * GW * 8 + lb_bytes + 1024,
                      &base);
  if (st) return st;
  uint8_t *b8 = static_cast<uint8_t *>(base);
  uint32_t *d_pcol = reinterpret_cast<uint32_t *>(b8);
  int *d_p2r = reinterpret_cast<int *>(b8 + out_bytes);
  int *d_stamp = d_p2r + m;
  int *d_perm = d_stamp + m;      // 4*GW ints
  int *d_last = d_perm + 4 * GW;  // largest row with a nonzero word
  int *d_hist = d_last + 1;       // GW + 1 head counts
  uint8_t *d_head = b8 + out_bytes + i_bytes;
  uint8_t *d_act = d_head + m;
  uint64_t *d_L21 = reinterpret_cast<uint64_t *>(b8 + out_bytes + i_bytes + h_bytes);
  uint64_t *d_L11 = d_L21 + m;
  uint64_t *d_U = d_L11 + GW;
  uint64_t *d_Lb = d_U + GW;  // m x GB words
  void *mh = nullptr, *md = nullptr;
  if ((st = ctx_panel_map(c, &mh, &md))) return st;
  int *hperm = reinterpret_cast<int *>(static_cast<char *>(mh) + PANEL_PERM_OFF);
  static_assert(2 * (2 * GW) <= (int)PANEL_PERM_INTS, "staging layout");
  auto words = [](void *map) {
    return reinterpret_cast<volatile uint64_t *>(static_cast<char *>(map) + PANEL_WORDS_OFF);
  };
  volatile uint64_t *hwords = words(mh), *hwords_dev = words(md);
  cudaError_t e = cudaMemsetAsync(d_stamp, 0xff, (size_t)m * sizeof(int), c->stream);
  if (e == cudaSuccess) e = cudaMemsetAsync(d_last, 0xff, sizeof(int), c->stream);
  if (e == cudaSuccess) e = cudaMemsetAsync(d_hist, 0, (GW + 1) * sizeof(int), c->stream);
  if (e != cudaSuccess) return ctx_cuda(c, e, "gf2 echelon: scratch");

  int tq[GW];
  std::vector<int> at, src, dst;
  int i = 0, epoch = 0;
  const int head_grid = std::max(1, std::min((m + GF2_HEADS_THREADS - 1) / GF2_HEADS_THREADS,
                                             c->num_sms * 2));
  // Blocks of GB words (delayed updates), as in the Z/p form: when the
  // block's first panel with pivots has at least DELAY_ROWS rows below it,
  // the block's panels update only the block's words; the words right of it
  // get, per block, U12 = L11^-1 A12 on the block's pivot rows and one C ^= L21
  // U12 with K = the block's pivots (up to 64 GB bits) on the rows
  // below.  d_Lb row q (GB words) holds the multipliers of the row at
  // position q, panel k of the block at bits Tb_k .. Tb_k + t_k - 1; later
  // panels' transpositions move d_Lb's rows with D's.
  constexpr int DELAY_ROWS = 512;
  int ib = 0, Tb = 0, R = -1, bw1 = 0, delayed = 0;
  auto flush = [&]() -> int {
    if (Tb == 0 || bw1 >= nw) return ST_OK;
    const int nrest = n - 64 * bw1;  // bits right of the block
    pdl_launch(gf2_block_solve_kernel, (nw - bw1 + BS_WORDS - 1) / BS_WORDS, BS_THREADS, 0, c->stream,
               D, ld, ib, Tb, bw1, nw, d_Lb);
    ctx_launched(c);
    const int rb = ib + Tb;
    if (R < rb) return ST_OK;
    int pi = prof_begin(c, "gf2_block_update");
    int s = gf2_gemm_dev(c, GF2_AUTO, R - rb + 1, nrest, Tb, 1, d_Lb + (size_t)rb * GB, GB,
                         D + (size_t)ib * ld + bw1, ld, 1, D + (size_t)rb * ld + bw1, ld);
    prof_end(c, pi);
    return s;
  };
  for (int wc = 0; wc < nw && i < m; ++wc) {
    const int w = std::min(64, n - 64 * wc);
    if (wc % GB == 0) {
      if ((st = flush())) return st;
      ib = i;
      Tb = 0;
      R = -1;
      bw1 = std::min(nw, wc + GB);
      delayed = -1;  // decided at the block's first panel with pivots
    }
    const uint64_t pmask = (w == 64) ? ~0ull : ((1ull << w) - 1ull);
    int pi = prof_begin(c, "gf2_heads");
    pdl_launch(gf2_heads_kernel, head_grid, GF2_HEADS_THREADS, 0, c->stream,
        D, ld, i, m, wc, pmask, d_head, d_act, d_hist, d_last, i + GF2_WR);
    prof_end(c, pi);
    const uint32_t seq = ++c->panel_seq;
    pi = prof_begin(c, "gf2_search");
    pdl_launch(gf2_search_kernel, 1, 32, 0, c->stream,
        D, ld, i, m, wc, w, pmask, d_head, d_act, d_hist, d_last, d_p2r, d_stamp, epoch++, d_U,
        d_pcol, hwords_dev, seq);
    prof_end(c, pi);
    ctx_launched(c, 2);
    auto word = [&](int k, int *v) -> int {
      const int s = ctx_wait_flag(c, reinterpret_cast<volatile uint32_t *>(hwords + k) + 1, seq,
                                  "gf2 echelon: panel");
      if (s == ST_OK) *v = (int)(uint32_t)hwords[k];
      return s;
    };
    int t = 0, last_pos = 0;
    if ((st = word(GF2_W_T, &t)) || (st = word(GF2_W_LAST, &last_pos))) return st;
    t = std::min(t, GW);
    if (t == 0) continue;
    int hi = i;
    for (int k = 0; k < t; ++k) {
      if ((st = word(GF2_W_PIV + k, &tq[k]))) return st;
      hi = std::max(hi, tq[k]);
    }
    at.resize(hi - i + 1);
    for (int q = i; q <= hi; ++q) at[q - i] = q;
    for (int k = 0; k < t; ++k) std::swap(at[k], at[tq[k] - i]);
    src.clear();
    dst.clear();
    for (int q = i; q <= hi; ++q)
      if (at[q - i] != q) {
        dst.push_back(q);
        src.push_back(at[q - i]);
      }
    const int cnt = (int)src.size();
    if (cnt > 2 * GW) return ctx_fail(c, ST_ARG, "gf2 echelon: permutation larger than expected");
    if (cnt > 0) {
      for (int k = 0; k < cnt; ++k) {
        hperm[k] = src[k];
        hperm[cnt + k] = dst[k];
      }
      e = cudaMemcpyAsync(d_perm, hperm, (size_t)2 * cnt * sizeof(int), cudaMemcpyHostToDevice,
                          c->stream);
      if (e != cudaSuccess) return ctx_cuda(c, e, "gf2 echelon: permutation");
      // (the block's earlier multipliers move with their rows)
      static_assert(GB <= GF2_PERM_WORDS, "one CTA for the block's multipliers");
      pdl_launch(gf2_permute_rows_kernel,
                 (nw + GF2_PERM_WORDS - 1) / GF2_PERM_WORDS + (Tb > 0 ? 1 : 0), GF2_PERM_THREADS, 0,
                 c->stream, D, ld, nw, d_Lb, GB, d_perm, d_perm + cnt, cnt);
      ctx_launched(c);
    }
    const int r0 = i + t;
    const int r1 = last_pos >= r0 ? last_pos : r0 - 1;
    const int below = r1 - r0 + 1;
    if (delayed < 0) {
      delayed = below >= DELAY_ROWS && bw1 < nw;
      if (delayed) {  // rows the panels' solves do not reach hold zero multipliers
        e = cudaMemsetAsync(d_Lb + (size_t)i * GB, 0, (size_t)(m - i) * GB * 8, c->stream);
        if (e != cudaSuccess) return ctx_cuda(c, e, "gf2 echelon: multipliers");
      }
    }
    // the rest of the block's words (delayed), or of all words
    const int w1 = wc + 1, wend = delayed ? bw1 : nw;
    {
      const int rows = r1 - i + 1;
      pi = prof_begin(c, "gf2_solve");
      pdl_launch(gf2_solve_kernel,
                 std::max(1, std::min((rows + GF2_SOLVE_THREADS - 1) / GF2_SOLVE_THREADS, c->num_sms * 4)),
                 GF2_SOLVE_THREADS, 0, c->stream, D, ld, i, r1, wc, pmask, t, d_pcol, d_U, d_L11, d_L21,
                 delayed ? d_Lb : nullptr, Tb, w1, wend);
      prof_end(c, pi);
      ctx_launched(c);
    }
    if (w1 < wend) {
      if (!delayed) {
        pdl_launch(gf2_l11_solve_kernel,
                   (wend - w1 + GF2_L11_THREADS / 32 - 1) / (GF2_L11_THREADS / 32), GF2_L11_THREADS, 0,
                   c->stream, D, ld, i, t, w1, wend, d_L11);
        ctx_launched(c);
      }
      if (below > 0) {
        // rows r0..r1, those words: C ^= L21 (one word of t bits per row) * U12
        pi = prof_begin(c, "gf2_update");
        if (wend - w1 <= GB) {
          pdl_launch(gf2_block_words_kernel, std::min((below + 31) / 32, c->num_sms * 4),
                     GF2_BW_THREADS, 0, c->stream, D, ld, n, i, t, w1, wend - w1, r0, r1, d_L21);
          ctx_launched(c);
        } else {
          st = gf2_m4rm_dev(c, below, std::min(n, 64 * wend) - 64 * w1, t, 1, d_L21, 1,
                            D + (size_t)i * ld + w1, ld, 1, D + (size_t)r0 * ld + w1, ld);
        }
        prof_end(c, pi);
        if (st) return st;
      }
    }
    if (delayed) {
      R = std::max(R, std::max(r1, hi));
      Tb += t;
    }
    rank += t;
    i += t;
  }
  if ((st = flush())) return st;
  *rank_out = rank;
  return ST_OK;
}

}  // namespace lela

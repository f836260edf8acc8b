// lela_b200/csrc/zp_gemm.h -- dense Z/p gemm entry points (device pointers).
#pragma once
#include <cstddef>
#include <cstdint>

#include <cuda_runtime.h>

#include "context.h"

namespace lela {

// Largest K handled by one tensor-core launch: 32768 * 255^2 < 2^31.
constexpr int ZP_KCHUNK = 32768;

int zp_limbs_for(uint32_t p);
size_t zp_gemm_workspace_bytes(uint32_t p, int M, int N, int K);

// A product modulo p > 2^16 by residues takes up to ZP_RESIDUE_MAX byte planes of A, B and C
// in the workspace, at most ZP_RESIDUE_MAX_BYTES.
constexpr int ZP_RESIDUE_MAX = 11;
constexpr size_t ZP_RESIDUE_MAX_BYTES = (size_t)4 << 30;

// C <- alpha*A*B + beta*C mod p on the handle's stream (asynchronous).
// kernel: a GemmKernel.  B may be C itself (same rows and columns, beta = 0)
// for GEMM_TC with K <= ZP_KCHUNK, and for GEMM_DIRECT with M <= 128 and K <=
// 256: every product that reads a tile's columns of B precedes its stores.
// ws_override, when non-null,
// is used instead of the handle workspace for the limb planes and must hold
// zp_gemm_workspace_bytes(p, M, N, K) bytes.  kr (device, optional): per
// row r of A, a column range [kr[r].x, kr[r].y) of the whole matrix outside
// which row r is zero (y <= x: the row is zero), and kbase the whole
// matrix's column of A's column 0; the tensor-core kernel then multiplies,
// per 128-row tile, only the K blocks its rows can touch (the other
// kernels ignore it: the result is the same).
int zp_gemm_dev(Ctx *c, int kernel, int M, int N, int K, uint32_t p, uint32_t alpha,
                const uint32_t *A, size_t lda, const uint32_t *B, size_t ldb, uint32_t beta,
                uint32_t *C, size_t ldc, uint8_t *ws_override, const int2 *kr = nullptr,
                int kbase = 0);

// V <- alpha*A*B mod p on the tensor cores, A and B of element type elem
// (LELA_CUDA_ELEM_*, not uint32; p one of its moduli), V residues.  K > 0.
int zp_gemm_tc_elem_dev(Ctx *c, int elem, int M, int N, int K, uint32_t p, uint32_t alpha,
                        const void *A, size_t lda, const void *B, size_t ldb, uint32_t *V,
                        size_t ldv);

// The kernel GEMM_AUTO resolves to for this shape (the handle's forced
// kernel, else the CUDA-core kernel for the smallest products, the one-launch
// tile kernel for short K and few tiles, and for the others the
// limb-plane one).
int zp_gemm_pick(const Ctx *c, int M, int N, int K, uint32_t p);
// The tensor-core tile variant (TcCfg<L, T>'s T: 0, 1, or 2 for one limb)
// for this shape and modulus: the handle's forced shape (wide or
// double-buffered), else by limbs, K and the number of tiles; for one limb the
// number of epilogue warps of the double-buffered tiles follows K.
int zp_gemm_tile_pick(const Ctx *c, int M, int N, int K, uint32_t p);

// Limb planes a caller keeps: L = zp_limbs_for(p) planes `plane` bytes apart,
// rows of bytes `pitch` apart (pitch and the addresses used multiples of 16),
// K along a row: a row of A, or a column of B.
struct ZpPlanes {
  uint8_t *base;
  size_t pitch, plane;
  ZpPlanes at(size_t row, size_t k) const { return {base + row * pitch + k, pitch, plane}; }
};
// The planes of the M x K matrix A (part 1 / 2: only the columns left / right of each
// row's diagonal block of nb rows), or of the K x N matrix B (its row K up to a
// multiple of 16, zero there).
int zp_split_rows_dev(Ctx *c, uint32_t p, const uint32_t *A, size_t lda, int M, int K,
                      const ZpPlanes &out, int part, int nb);
int zp_split_cols_dev(Ctx *c, uint32_t p, const uint32_t *B, size_t ldb, int K, int N,
                      const ZpPlanes &out);
// C <- alpha*A*B + beta*C on the tensor cores from planes (K > 0; kr, kbase
// as zp_gemm_dev).
int zp_gemm_planes_dev(Ctx *c, int M, int N, int K, uint32_t p, uint32_t alpha, const ZpPlanes &A,
                       const ZpPlanes &B, uint32_t beta, uint32_t *C, size_t ldc,
                       const int2 *kr = nullptr, int kbase = 0);

// Whether the host-pointer gemm of this shape is done in row blocks with
// its copies overlapped (tensor-core path, one K chunk, at least two blocks
// of PIPE_MIN_ROWS rows).
constexpr int PIPE_MIN_ROWS = 512;
bool zp_gemm_pipelined(const Ctx *c, int M, int N, int K, uint32_t p, uint32_t alpha);

// C <- alpha*A*B + beta*C mod p with A, B, C in host memory (row strides
// lda, ldb, ldc) through the device buffers dA (M x K), dB (K x N), dC
// (M x N, packed): the row-block pipeline above.  Asynchronous on the
// handle stream, which ends after the last copy back; the caller
// synchronises it.  Only for shapes zp_gemm_pipelined accepts.
int zp_gemm_host_rows(Ctx *c, int M, int N, int K, uint32_t p, uint32_t alpha,
                      const uint32_t *hA, size_t lda, const uint32_t *hB, size_t ldb,
                      uint32_t beta, uint32_t *hC, size_t ldc, uint32_t *dA, uint32_t *dB,
                      uint32_t *dC);

}  // namespace lela

namespace lela {
// Whether a GF(2) product's kernels after the first are launched early (us per product,
// early / in order: 1590 x 753 x 3420 21.8 / 27.3, 810 x 8264 x 523 19.9 / 23.4,
// 2048^3 24.4 / 24.9; 13564 x 3189 x 1074 75.9 / 61.3 after a kernel that is not of
// this chain, 4096^3 65.2 / 60.5, 16384^2 x 1024 212 / 197).
inline bool gf2_early(int M, int N, int K) { return (double)M * N * K < 1e10; }
// GF(2) product on the tensor cores from 0/1 byte planes (see zp_gemm.cu).
int gf2_gemm_tc_planes(Ctx *c, int M, int N, int K, const uint8_t *Ab, const uint8_t *Bb, int Kp,
                       uint32_t alpha, uint32_t beta, uint64_t *C, size_t ldc_words);
}  // namespace lela

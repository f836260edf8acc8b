// lela_b200/csrc/echelon.cu -- non-reduced row-echelon form over Z/p with
// LELA's pivot rule, in place on a dense device matrix.
//
// Reference semantics (bit-exact target): Elimination::echelonize
// (lela/algorithms/elimination.tcc:47-139) with DensePivotStrategy
// (lela/algorithms/pivot-strategy.tcc:19-42), which EchelonForm's dense path
// (GaussJordan::echelonize + move_L, lela/solutions/echelon-form.h:103-134)
// reproduces (tests/test-gauss-jordan.C:91-99).  At current row i and column
// c the pivot is the first nonzero of column c at or below row i (columns
// without one are skipped); it is swapped into row i by a transposition,
// multiplies det, and every row below with a nonzero a in column c gets
// row_i * (-a/x) added.  Pivots are not normalised.
//
// Blocked right-looking form, exact.  The columns are taken in panels of
// W = 64.  Facts the design rests on, for one panel:
//  * the value of a row after elimination by the panel's pivot rows
//    U_0..U_{t-1} is the unique vector of v + span(U) that is zero in the
//    pivot columns, whatever order the eliminations take, and so are the
//    multipliers l (v = l U + reduced);
//  * after the whole panel every row below the pivots is zero in all W
//    columns (a skipped column was zero in every row at or below the
//    current row, and every later pivot row is zero there as well);
//  * the pivot of column c is the first row at or below the current row
//    whose reduced entry in c is nonzero, and that entry only involves the
//    row's entries in the pivot columns found so far and in c.
// So per panel:
//  1. panel_heads_kernel: each row at or below the current row records the
//     first nonzero column of its panel part (64: none), with a histogram;
//  2. panel_search_kernel (one CTA) replays the reference's pivot choice on
//     a window of the first rows, four columns at a time: one warp chooses
//     their pivots with the columns in registers, then all warps update the
//     rest of the window in shared memory.  For p up to 65521 the pivots are
//     inverted from a table; above, the elimination goes without division (a row
//     W becomes y W - W[c] P for pivot row P with pivot value y) and the
//     inverses come at the end.  Rows below the window are reduced only
//     when the head histogram says one of them may hold a pivot the window
//     lacks.  After the host has been signalled it inverts, for p < 2^31, the pivot
//     block U_P (the pivot rows at the pivot columns) and L11;
//  3. the host replays the recorded transpositions and moves the affected
//     rows (at most two per pivot) with one gather;
//  4. panel_solve_inv_kernel (p < 2^31) / panel_solve_kernel (all SMs, one
//     warp per row): for every row from the first pivot to the last possibly
//     nonzero row, its multipliers (the L11 row of a pivot row, the L21 row
//     otherwise): a_P U_P^-1 from its entries a_P at the pivot columns, or
//     the reference's elimination steps on its panel part; the panel becomes
//     U_k in pivot row k and zero below;
//  5. U12 = L11^-1 A12 (a tensor-core product with the search's inverse, in place;
//     by substitution on CUDA cores for p >= 2^31 and on wide panels) and A22 -= L21 U12 on the
//     tensor cores over the rows down to the last possibly nonzero row,
//     for the columns of the panel's block of EB columns; the columns right
//     of the block get one such update per block, with the multipliers of
//     all its panels (K up to EB = 16 W instead of W: a sixteenth of the
//     passes over the trailing matrix).
// F4 Schur complements are staircase-shaped (rows sorted by head), so few
// rows are touched per panel; dense matrices make every row active and the
// scheme becomes ordinary blocked LU with LELA's pivot choice.
#include <algorithm>
#include <cstddef>
#include <mutex>
#include <type_traits>
#include <vector>

#include "arith.cuh"
#include "common.cuh"
#include "context.h"
#include "echelon.h"
#include "tri.h"
#include "zp_gemm.h"

namespace lela {

constexpr int EW = 64;                     // panel width
constexpr int EB = 16 * EW;                // block of panels sharing one trailing update
constexpr int PS_THREADS = 512;            // panel search CTA
constexpr int PS_FAST = PS_THREADS / 32;   // positions tested per column by whole warps
constexpr uint8_t HEAD_NONE = 64;

// The host's copy of a panel's result, in mapped host memory: words of the
// value (low half) and the search's sequence number (high half).  Each word
// is written whole, so the host takes a word when its sequence number has
// arrived and nothing orders the words among themselves.
enum : int {
  PANEL_W_T = 0,     // pivots (bits 0-7), U_P^-1 written (bit 8), an inverse failed (bit 9)
  PANEL_W_LAST = 1,  // last_pos
  PANEL_W_DET = 2,
  PANEL_W_PIV = 4,   // per pivot: column, transposition target
  PANEL_WORDS = PANEL_W_PIV + 2 * EW
};
static_assert(PANEL_WORDS_OFF + PANEL_WORDS * 8 <= PANEL_FLAG_OFF, "words below the flag");

// Row index currently at position pos: positions touched by this panel's
// transpositions carry the panel's epoch stamp.
__device__ __forceinline__ int row_at(int pos, const int *p2r, const int *stamp, int epoch) {
  return stamp[pos] == epoch ? p2r[pos] : pos;
}

// 1. First nonzero column of each row's panel part, rows i0..m-1 (one warp
// per row); the histogram of these heads (hist[0..64], which the caller
// has zeroed) and the largest row index with a nonzero panel (*last, which
// the caller has set to -1).  Entries of the panel that are not reduced (a
// caller's may not be) are, in place: the search looks inverses up by
// their value.  (A 4096^2 form takes 5 to 15 us of 4740 more for the check; in the
// search, at its loads, it took 15 to 45.)
constexpr int HEADS_THREADS = 256;
__global__ void __launch_bounds__(HEADS_THREADS)
    panel_heads_kernel(uint32_t *D, size_t ld, int i0, int m, int c0, int w, uint32_t p,
                       uint8_t *head, uint8_t *act, int *hist, int *last) {
  pdl_enter();
  __shared__ int s_last;
  __shared__ int s_hist[EW + 1];
  if (threadIdx.x == 0) s_last = -1;
  if (threadIdx.x <= EW) s_hist[threadIdx.x] = 0;
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const int warps = (gridDim.x * blockDim.x) >> 5;
  int my_last = -1;
  for (int r = i0 + ((blockIdx.x * blockDim.x + threadIdx.x) >> 5); r < m; r += warps) {
    uint32_t *row = D + (size_t)r * ld + c0;
    uint32_t a = lane < w ? row[lane] : 0u;
    uint32_t b = lane + 32 < w ? row[lane + 32] : 0u;
    if (max(a, b) >= p) {
      if (lane < w) row[lane] = a %= p;
      if (lane + 32 < w) row[lane + 32] = b %= p;
    }
    const unsigned ba = __ballot_sync(0xffffffffu, a != 0u);
    const unsigned bb = __ballot_sync(0xffffffffu, b != 0u);
    const int h = ba ? __ffs(ba) - 1 : (bb ? 32 + __ffs(bb) - 1 : HEAD_NONE);
    if (lane == 0) {
      head[r] = (uint8_t)h;
      act[r] = h < HEAD_NONE;
      atomicAdd(&s_hist[h], 1);
    }
    if (h < HEAD_NONE) my_last = r;
  }
  if (lane == 0 && my_last >= 0) atomicMax(&s_last, my_last);
  __syncthreads();
  if (threadIdx.x == 0 && s_last >= 0) atomicMax(last, s_last);
  if (threadIdx.x <= EW && s_hist[threadIdx.x]) atomicAdd(&hist[threadIdx.x], s_hist[threadIdx.x]);
}

// Field arithmetic of the panel search, in three forms chosen by the host.
//
// SearchSmall, 32 <= p <= 65521 (the largest prime below 2^16): signed
// residues |v| <= p/2 + 4 and pivots inverted from a table of the inverses
// of 0 .. p/2 + 5 (u16, 0: none), which the CTA holds in shared memory, so a row is reduced
// with its true multiplier l: w - l P (NORM below).  Reduction: q = (x mu +
// 2^(31+s)) >> (32 + s) with mu = round (2^(32+s) / p) in [2^30, 2^31) (s = 14
// for p > 2^15, one less per halving of p) is x / p rounded, up to an error of
// |x| / 2^(33+s) from mu, for |x| < 2^31; so |x - q p| <= p/2 + 1, and x = 0 mod p
// gives q = x / p exactly: a zero is stored as 0 (s >= 3 here).  The product
// and the rounding are one 64-bit multiply-add (four issue cycles a warp measured, as
// many as a 32-bit high product, after which the rounding is an instruction more).  Two products
// and one more term fit 32 bits (2 (p/2 + 4)^2 + p/2 + 4 < 2^31).  Four and one more are
// halved for the quotient, which then is off by 2 / p more: half of |w| + 4 |l P|, with
// |l| <= p/2 + 1 and |P|, |w| <= p/2 + 4, must be below 2^31, and is (4 x 32761 x 32764 +
// 32764 < 2^32 at p = 65521, with 0.03 % to spare).
//
// SearchMont and SearchPlain reduce without division (an inverse costs more
// than a whole column there): one elimination step is upd(y, w, na, P) = k (y
// w + na P) and a product mul(a, b) = k a b, with a unit k fixed per form;
// lin(s, w, a, P) = k (s w + a[0] P[0] + .. + a[3] P[3]); plain(a, b) = a b. A
// window row then holds S_t times its reduced row with S_{t+1} = k S_t y_t,
// whatever k is, so the reductions may carry a factor of their own.
// neg(a) = -a, one() the identity of mul, canon(v) the residue in [0, p).
struct SearchSmall {
  using V = int;
  using V4 = int4;
  static constexpr bool NORM = true;
  int p, mu, s;
  long long half;
  const uint16_t *table;  // inverses of 0 .. p / 2 + 5
  __host__ static bool takes(uint32_t p) { return p >= 32 && p <= 65521; }
  __host__ static SearchSmall make(uint32_t p, const uint16_t *table) {
    SearchSmall a;
    a.p = (int)p;
    a.s = 0;
    while (((1ull << (33 + a.s)) + p) / (2ull * p) < (1ull << 30)) ++a.s;
    a.mu = (int)(((1ull << (33 + a.s)) + p) / (2ull * p));
    a.half = 1ll << (31 + a.s);
    a.table = table;
    return a;
  }
  // round (x / p), sh = s; of x / 2, sh = s - 1
  __device__ __forceinline__ int quot(int x, int sh) const {
    long long d;
    asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(d) : "r"(x), "r"(mu), "l"(sh == s ? half : half >> 1));
    return (int)(d >> 32) >> sh;
  }
  __device__ __forceinline__ int red(int x) const { return x - quot(x, s) * p; }
  // (reduced entries only, see panel_heads_kernel)
  __device__ __forceinline__ int load(uint32_t v) const {
    return (int)v > (p >> 1) ? (int)v - p : (int)v;
  }
  // w - l P
  __device__ __forceinline__ int step(int w, int l, int P) const { return red(w - l * P); }
  __device__ __forceinline__ int step2(int w, int l, int P, int l2, int P2) const {
    return red(w - l * P - l2 * P2);
  }
  // w - l[0] P[0] - .. - l[3] P[3]
  __device__ __forceinline__ int lin(int w, const int4 &l, const int (&P)[4]) const {
    const long long x = (long long)w - (long long)l.x * P[0] - (long long)l.y * P[1] -
                        (long long)l.z * P[2] - (long long)l.w * P[3];
    return (int)x - quot((int)(x >> 1), s - 1) * p;
  }
  // a b, also for one factor in (-p, p)
  __device__ __forceinline__ int plain(int a, int b) const { return red(a * b); }
  // 1 / |v| in [0, p), 0 if there is none
  __device__ __forceinline__ int inverse_abs(const uint16_t *tab, int v) const { return tab[abs(v)]; }
  __device__ __forceinline__ uint32_t canon(int v) const { return (uint32_t)(v < 0 ? v + p : v); }
};

// The inverses of 0 .. p / 2 + 5 modulo p < 2^16, 0 for those that have none.
__global__ void inverse_table_kernel(uint32_t p, uint16_t *__restrict__ table) {
  const uint32_t x = blockIdx.x * blockDim.x + threadIdx.x;
  if (x <= p / 2 + 5) table[x] = (uint16_t)inv_exact_u32(p, x);
}

// SearchMont, other odd p < 2^31: canonical residues, Montgomery reduction
// (P. Montgomery, 1985) with k = 2^-32: T = y w + na P < 2 p^2 and m p <
// 2^32 p sum to less than 2^64, and (T + m p) / 2^32 < 2 p.
struct SearchMont {
  using V = uint32_t;
  using V4 = uint4;
  static constexpr bool NORM = false;
  uint32_t p, np, r1, r2;  // -1/p mod 2^32, 2^32 mod p, 2^64 mod p
  __host__ static bool takes(uint32_t p) { return (p & 1u) && p > 2 && p < 0x80000000u; }
  __host__ static SearchMont make(uint32_t p) {
    SearchMont a;
    a.p = p;
    uint32_t inv = p;  // Newton: 3 correct bits, doubled four times
    for (int k = 0; k < 4; ++k) inv *= 2u - p * inv;
    a.np = 0u - inv;
    a.r1 = (uint32_t)((1ull << 32) % p);
    a.r2 = (uint32_t)((uint64_t)a.r1 * a.r1 % p);
    return a;
  }
  __device__ __forceinline__ uint32_t redc(uint64_t T) const {
    const uint32_t m = (uint32_t)T * np;
    const uint32_t r = (uint32_t)((T + (uint64_t)m * p) >> 32);
    return r >= p ? r - p : r;
  }
  __device__ __forceinline__ uint32_t load(uint32_t v) const { return v; }
  __device__ __forceinline__ uint32_t upd(uint32_t y, uint32_t w, uint32_t na, uint32_t P) const {
    return redc((uint64_t)y * w + (uint64_t)na * P);
  }
  __device__ __forceinline__ uint32_t add(uint32_t a, uint32_t b) const {
    const uint32_t r = a + b;  // below 2 p < 2^32
    return r >= p ? r - p : r;
  }
  __device__ __forceinline__ uint32_t lin(uint32_t s0, uint32_t w, const uint4 &a,
                                          const uint32_t (&P)[4]) const {
    return add(add(upd(s0, w, a.x, P[0]), upd(a.y, P[1], a.z, P[2])), mul(a.w, P[3]));
  }
  __device__ __forceinline__ uint32_t mul(uint32_t a, uint32_t b) const {
    return redc((uint64_t)a * b);
  }
  __device__ __forceinline__ uint32_t plain(uint32_t a, uint32_t b) const {
    return mul(mul(a, b), r2);
  }
  __device__ __forceinline__ uint32_t neg(uint32_t a) const { return a ? p - a : 0u; }
  __device__ __forceinline__ uint32_t one() const { return r1; }
  __device__ __forceinline__ uint32_t canon(uint32_t v) const { return v; }
};
// SearchPlain, any p < 2^32 (even moduli, p below 3 and p >= 2^31): canonical
// residues, Barrett reduction, k = 1.  Below 2^16 with ArithSmall's 32-bit
// reductions, which count where rows past the window, a warp per row and all
// its pivots, are reduced for each column without a pivot: a 3000 x 500 matrix of
// rank 166 modulo 2 takes 2490 us, with ArithWide's 4550.
template <class A>
struct SearchPlain {
  using V = uint32_t;
  using V4 = uint4;
  static constexpr bool NORM = false;
  A w;
  uint32_t p;
  __host__ static SearchPlain make(uint32_t p) {
    SearchPlain a;
    a.w = A::make(p);
    a.p = p;
    return a;
  }
  __device__ __forceinline__ uint32_t load(uint32_t v) const { return v; }
  __device__ __forceinline__ uint32_t upd(uint32_t y, uint32_t x, uint32_t na, uint32_t P) const {
    return w.dot2(y, x, na, P);
  }
  __device__ __forceinline__ uint32_t lin(uint32_t s0, uint32_t x, const uint4 &a,
                                          const uint32_t (&P)[4]) const {
    uint64_t s = (uint64_t)upd(s0, x, a.x, P[0]) + upd(a.y, P[1], a.z, P[2]) + w.mul(a.w, P[3]);
    if (s >= p) s -= p;
    return (uint32_t)(s >= p ? s - p : s);
  }
  __device__ __forceinline__ uint32_t mul(uint32_t a, uint32_t b) const { return w.mul(a, b); }
  __device__ __forceinline__ uint32_t plain(uint32_t a, uint32_t b) const { return w.mul(a, b); }
  __device__ __forceinline__ uint32_t neg(uint32_t a) const { return a ? p - a : 0u; }
  __device__ __forceinline__ uint32_t one() const { return 1u % p; }
  __device__ __forceinline__ uint32_t canon(uint32_t v) const { return v; }
};

// 2. The reference's pivot choice on the panel (see the file comment).
// The window: the first wcap <= PW_R rows at or below i0, by position, with a
// nonzero in the panel, kept in shared memory.  With NORM arithmetic a window
// row holds its row reduced by the pivots so far; otherwise the elimination is
// division-free: when pivot row P (pivot value y) is chosen, every window row
// W becomes k (y W - W[col] P), so a window row holds S_t times its row
// reduced by the t pivots so far (S_0 = 1, S_{t+1} = k S_t y_t), and at the end
// S_t is inverted and the S_k^-1, the pivots x_k and their inverses follow
// from scans of products.  Pivot rows move to PV (U_k, or S_k U_k).  Rows
// between window
// rows are zero in the panel and can never hold a pivot.  The pivot of a
// column is the first window row, by position, with a nonzero there; rows
// past the last window position are reached only when no window row has one
// and the head histogram says one of them may: they are then reduced by the
// same recurrence, in position order.
// Outputs: the pivot columns (relative to c0); U (t x EW, row stride EW: the pivot
// rows' final panel values) and the pivot inverses; the host's copy of the result as words of
// a value and the call's sequence number (hout), so that no fence orders
// them.  Resets *last_act to -1 and hist[] to zero for the next panel.
//
// Blocks of PB = 4 columns.  Warp 0 alone chooses the pivots of a block: the
// live rows in position order, entry e in register group e / 32 of lane e %
// 32, the block's columns in registers; a column's pivot is the first live entry with
// a nonzero there (a warp-wide minimum), its row comes by shuffles, and the elimination runs
// on the block's columns and keeps each row's coefficients of the block's pivot rows
// (its multipliers l; or, division-free, the row's current value as sc times
// its value before the block plus cf[j] times that of the pivot row of the
// block's column j).  No barrier is on that chain.  The pivot row reduces to
// zero by itself and so leaves.  Then all warps form the remaining columns of
// the window rows and of the block's pivot rows from those coefficients (rows
// on warps, columns on lanes).
//
// With NORM arithmetic warp 0 goes on to the next block at once: it applies the
// block before to its four columns itself, while twelve warps on the other
// three schedulers form the columns further right.
//
// Bound: the instructions on warp 0's dependent chain, four to five cycles each.
// Measured on a 64 x 64 window (p = 65521, a panel of a dense 4096^2 matrix),
// cycles a block of four columns: 1200 to load and bring up its columns, 1650 for
// the pivots, 350 for lists and barrier; 56000 for the panel's sixteen.  With
// the updates of a block between its pivots and the next block's 60800, and with
// all fifteen other warps on them, sharing warp 0's scheduler, 58400.  Forms with one
// barrier per column and all 16 warps on it (window in shared memory, lanes
// on rows; or rows in registers, a warp per row) took 1640 cycles a column
// (80 us a panel, at 2^31 - 1 102 us).  Rolled loops, the panel's inverse
// included, were slower.  On this
// chip a ballot takes 26 cycles, __ffs 40, __reduce_min_sync 22, so the pivot's
// lane comes from the reduction.
//
// Bookkeeping (warp 0): s_ent[e] / s_epos[e] are the slot and the position
// of live entry e, rewritten per block.  A transposition (i, q) moves the row
// at position i to q: if it is a window row, it is the first entry and takes
// the pivot's entry; a row outside the window (zero in the panel) is recorded
// in p2r / stamp.  wrow[slot] is the row index in D.  Rows past the window
// carry in head[] a lower bound of the first nonzero column of their reduced
// panel part; cnt[h] counts them by that bound.
constexpr int PW_R = 80;               // window rows
constexpr int PW_RPW = PW_R / PS_FAST; // window rows per warp
constexpr int PW_G = (PW_R + 31) / 32; // most window rows per lane of warp 0
constexpr int PB = 4;                  // columns per block
static_assert(PW_R % PS_FAST == 0, "whole rows per warp");
// window rows padded to EW + 1 words: a column read across rows touches
// every bank once
constexpr int PW_LD = EW + 1;
// dynamic shared memory: the window rows, later the two inverses and their
// scratch; the multipliers of the window's rows (by slot) and of pivots from
// past it; then the table of inverses (NORM)
constexpr int INV_WORDS = 2 * (INV_M + INV_T);
static_assert(PS_THREADS == 2 * INV_THREADS, "half of the CTA per inverse");
constexpr int PW_AREA = PW_R * PW_LD > INV_WORDS ? PW_R * PW_LD : INV_WORDS;
constexpr int PW_LROWS = PW_R + EW;
constexpr size_t PW_SMEM = ((size_t)(PW_AREA + PW_LROWS * PW_LD) * 4 + 15) / 16 * 16;
constexpr size_t PW_TABLE = 65536 + 64;
// positions a thread looks at per pass of the window's compaction
constexpr int PW_U = 4;

template <class SA, class A>
__global__ void __launch_bounds__(PS_THREADS, 1)
    panel_search_kernel(const uint32_t *D, size_t ld, int i0, int m, int c0, int w,
                        SA sa, A ar, uint8_t *head, const uint8_t *act,
                        int *hist, int *last_act, int *p2r,
                        int *stamp, int epoch, uint32_t *Uout,
                        uint32_t *xinv_out, uint32_t *Uinv_out,
                        uint32_t *Linv_out, uint32_t *pcol_out, volatile uint64_t *hout, uint32_t seq,
                        int wcap) {
  using V = typename SA::V;
  using V4 = typename SA::V4;
  extern __shared__ __align__(16) uint32_t dyn_w[];
  V(*Wv)[PW_LD] = reinterpret_cast<V(*)[PW_LD]>(dyn_w);  // PW_R rows
  V(*Lm)[PW_LD] = reinterpret_cast<V(*)[PW_LD]>(dyn_w + PW_AREA);  // [slot][pivot] (division-free: raw)
  const uint16_t *s_inv = reinterpret_cast<const uint16_t *>(dyn_w + PW_SMEM / 4);
  __shared__ V PV[EW][EW];
  // per block, double-buffered (warp 0 is one block ahead): per slot the
  // coefficients of the block's pivot rows, by pivot; division-free by column, and
  // z of the block's pivot rows when chosen, their slots (-1: no pivot in the
  // column) and scales, and the other rows' scale
  __shared__ V4 s_coef[2][PW_R], s_pcoef[2][PB];
  __shared__ __align__(16) int s_pj[2][PB];
  __shared__ V s_psc[2][PB], s_sc[2];
  // the block's end, its stop, the pivots before and after it, live entries after it
  __shared__ int s_next[2], s_rare[2], s_t0[2], s_t[2], s_nl[2], s_col0;
  __shared__ V s_red[PS_FAST][EW];    // rows past the window, reduced (one per warp),
  __shared__ V s_rl[PS_FAST][EW];     // and their multipliers (raw)
  __shared__ int s_ent[2][PW_R], s_epos[2][PW_R], wrow[PW_R];
  __shared__ int2 s_piv[EW];          // pivot column, transposition target
  __shared__ int s_prow[EW];          // the pivot's row of Lm
  __shared__ V s_y[EW], s_sinv[EW];   // pivot values (in window rows' scale), 1 / S_k
  __shared__ V s_yinv[EW];            // 1 / s_y (division-free, p < 2^31)
  __shared__ int s_xi[EW];            // pivots' inverses (NORM: in (-p, p))
  __shared__ uint32_t s_det;
  __shared__ int s_cnt[EW + 1];
  __shared__ int s_first[PS_FAST], s_wcnt[PW_U * PS_FAST];
  __shared__ int s_list[PS_THREADS], s_lrow[PS_THREADS], s_lhead[PS_THREADS];
  __shared__ int s_err, s_last, s_hi, s_wlast, s_uinv;
  const uint32_t p = (uint32_t)sa.p;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  constexpr unsigned FULL = 0xffffffffu;

  if constexpr (SA::NORM) {
    // the table of inverses, on its way while the window is formed
    char *dst = reinterpret_cast<char *>(dyn_w) + PW_SMEM;
    for (int e = tid; e < (int)(p / 2 + 6 + 7) / 8; e += PS_THREADS)
      cp_async16(dst + 16 * e, reinterpret_cast<const char *>(sa.table) + 16 * e);
  }
  // (the table was complete before the memsets that precede the first panel)
  pdl_enter();
  // the window: ordered compaction of the rows with a nonzero panel
  int nl = 0;
  if (tid == 0) {
    s_wlast = m - 1;
    s_err = 0;
    s_last = -1;
  }
  if (tid <= EW) {
    s_cnt[tid] = hist[tid];
    hist[tid] = 0;
  }
  for (int base = i0; base < m && nl < wcap; base += PW_U * PS_THREADS) {
    int hd[PW_U];
#pragma unroll
    for (int u = 0; u < PW_U; ++u) {
      const int pos = base + u * PS_THREADS + tid;
      hd[u] = pos < m ? (int)head[pos] : (int)HEAD_NONE;
    }
    unsigned bal[PW_U];
#pragma unroll
    for (int u = 0; u < PW_U; ++u) {
      bal[u] = __ballot_sync(FULL, hd[u] < HEAD_NONE);
      if (lane == 0) s_wcnt[u * PS_FAST + wid] = __popc(bal[u]);
    }
    __syncthreads();
    static_assert(PW_U * PS_FAST == 64, "two counts per lane");
    int a = s_wcnt[lane], b = s_wcnt[lane + 32];  // inclusive scan of the 64 counts
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int x = __shfl_up_sync(FULL, a, o), y = __shfl_up_sync(FULL, b, o);
      if (lane >= o) {
        a += x;
        b += y;
      }
    }
    b += __shfl_sync(FULL, a, 31);
    const int cnt = __shfl_sync(FULL, b, 31);
    const int take = min(cnt, wcap - nl);
#pragma unroll
    for (int u = 0; u < PW_U; ++u) {
      const int gp = u * PS_FAST + wid - 1;  // the count before this warp's
      const int before = gp < 0 ? 0 : __shfl_sync(FULL, gp < 32 ? a : b, gp & 31);
      const int off = before + __popc(bal[u] & ((1u << lane) - 1u));
      if (hd[u] < HEAD_NONE && off < take) {
        const int slot = nl + off, pos = base + u * PS_THREADS + tid;
        s_ent[0][slot] = slot;
        s_epos[0][slot] = pos;
        wrow[slot] = pos;
        atomicSub(&s_cnt[hd[u]], 1);  // the window's rows leave the counts
        if (off == wcap - 1 - nl) s_wlast = pos;
      }
    }
    nl += take;
    __syncthreads();  // s_wcnt is rewritten by the next pass
  }
  // the window rows' panel values: rows on warps, columns on lanes
  {
    uint32_t a0[PW_RPW], a1[PW_RPW];
#pragma unroll
    for (int r = 0; r < PW_RPW; ++r) {
      const int slot = wid + r * PS_FAST;
      const uint32_t *row = D + (size_t)(slot < nl ? wrow[slot] : i0) * ld + c0;
      a0[r] = lane < w ? row[lane] : 0u;
      a1[r] = lane + 32 < w ? row[lane + 32] : 0u;
    }
#pragma unroll
    for (int r = 0; r < PW_RPW; ++r) {
      const int slot = wid + r * PS_FAST;
      Wv[slot][lane] = sa.load(a0[r]);
      Wv[slot][lane + 32] = sa.load(a1[r]);
    }
  }
  if constexpr (SA::NORM) cp_async_wait_all();
  __syncthreads();
  const int wlast = s_wlast;  // rows past it are outside the window
  // the final values of the nb pivot rows of a block (buffer b, from pivot tb) in
  // one column, in place: U_k = P_k - sum l_kj U_j
  [[maybe_unused]] auto finish = [&](V(&P)[PB], int b, int tb, int nb) {
    if constexpr (SA::NORM) {
      const V4 l1 = s_coef[b][s_prow[tb + (1 < nb ? 1 : 0)]], l2 = s_coef[b][s_prow[tb + (2 < nb ? 2 : 0)]];
      V4 l3 = s_coef[b][s_prow[tb + (3 < nb ? 3 : 0)]];
      l3.w = 0;
      P[1] = 1 < nb ? sa.step(P[1], l1.x, P[0]) : 0;
      P[2] = 2 < nb ? sa.step2(P[2], l2.x, P[0], l2.y, P[1]) : 0;
      const V u3 = sa.lin(P[3], l3, P);
      P[3] = 3 < nb ? u3 : 0;
    }
  };
  int t = 0, col0 = 0;  // pivots so far; the current row is i0 + t
  int buf = 0;          // the block's buffer; the live entries on entry are list `buf`

  // A. warp 0: the pivots of the block's columns, with NG groups of entries.
  // z holds, per entry, the block's columns from the current one on, and
  // behind them (division-free) the coefficients of the block's pivot rows
  // chosen so far: each column drops z[0] and appends its own.  `ahead`: the
  // block's columns still lack the block before, which the other warps are
  // applying to the columns right of it (B): warp 0 applies it here.
  auto choose = [&](auto ng_c, bool ahead) {
    constexpr int NG = decltype(ng_c)::value;
    constexpr uint32_t NONE = 255;
    V z[PB][NG];
    int ent[NG], pos[NG];
    uint32_t live[NG];  // the entry's number, NONE when it is not live
    auto sel = [&](const auto &r, int g) {  // r[g], g the same in every lane
      auto v = r[0];
#pragma unroll
      for (int u = 1; u < NG; ++u)
        if (g == u) v = r[u];
      return v;
    };
#pragma unroll
    for (int g = 0; g < NG; ++g) {
      const int e = lane + 32 * g;
      const bool in = e < nl;
      live[g] = in ? (uint32_t)e : NONE;
      ent[g] = in ? s_ent[buf][e] : 0;
      pos[g] = in ? s_epos[buf][e] : 0;
#pragma unroll
      for (int j = 0; j < PB; ++j) z[j][g] = (in && col0 + j < w) ? Wv[ent[g]][col0 + j] : 0;
    }
    if constexpr (SA::NORM)
      if (ahead) {
        const int pb = buf ^ 1, tb = s_t0[pb], nb = t - tb, c = col0 + (lane & (PB - 1));
        V P[PB];
#pragma unroll
        for (int k = 0; k < PB; ++k) P[k] = k < nb && c < w ? Wv[s_prow[tb + k]][c] : 0;
        finish(P, pb, tb, nb);
        V U[PB][PB];  // [column][pivot], from lanes 0 .. PB - 1
#pragma unroll
        for (int j = 0; j < PB; ++j)
#pragma unroll
          for (int k = 0; k < PB; ++k) U[j][k] = __shfl_sync(FULL, P[k], j);
#pragma unroll
        for (int g = 0; g < NG; ++g) {
          const V4 cf = s_coef[pb][ent[g]];
          if (live[g] != NONE) {
#pragma unroll
            for (int j = 0; j < PB; ++j) {
              z[j][g] = sa.lin(z[j][g], cf, U[j]);
              Wv[ent[g]][min(col0 + j, PW_LD - 1)] = z[j][g];
            }
          }
        }
      }
    if (!SA::NORM && lane < PB) s_pj[buf][lane] = -1;
    __syncwarp();
    const int t0 = t;
    [[maybe_unused]] V sc = 0;
    if constexpr (!SA::NORM) sc = sa.one();
    int next = min(col0 + PB, w), rare = -1;
    V *coef[NG];
#pragma unroll
    for (int g = 0; g < NG; ++g) coef[g] = reinterpret_cast<V *>(&s_coef[buf][ent[g]]);
#pragma unroll
    for (int j = 0; j < PB; ++j) {
      const int zn = SA::NORM ? PB - j : PB;  // entries of z in use
      const int col = col0 + j, nb = t - t0;
      // the pivot's entry (columns past w are zero)
      uint32_t key = NONE;
#pragma unroll
      for (int g = 0; g < NG; ++g) key = min(key, z[0][g] != 0 ? live[g] : NONE);
      [[maybe_unused]] int inv[NG];  // each row's inverse, looked up meanwhile
      if constexpr (SA::NORM) {
#pragma unroll
        for (int g = 0; g < NG; ++g) inv[g] = sa.inverse_abs(s_inv, z[0][g]);
      }
      key = __reduce_min_sync(FULL, rare < 0 ? key : NONE);
      V znew[NG];
#pragma unroll
      for (int g = 0; g < NG; ++g) znew[g] = 0;
      if (key == NONE) {
        // none in the window: rows past it whose bound allows a pivot here
        // end the block (all warps look for it)
        if (wlast < m - 1 && col < next && i0 + t < m) {
          const int v = (lane <= col ? s_cnt[lane] : 0) + (lane + 32 <= col ? s_cnt[lane + 32] : 0);
          if (__reduce_add_sync(FULL, v) > 0) {
            rare = col;
            next = col;
          }
        }
      } else {
        const int pg = (int)key >> 5, pl = (int)key & 31;
        V pv[PB];  // the pivot row's z
        [[maybe_unused]] int iv = 0;
#pragma unroll
        for (int k = 0; k < PB; ++k) pv[k] = k < zn ? __shfl_sync(FULL, sel(z[k], pg), pl) : 0;
        if constexpr (SA::NORM) {
          iv = __shfl_sync(FULL, sel(inv, pg), pl);
          iv = pv[0] < 0 ? -iv : iv;
        }
        const int q = __shfl_sync(FULL, sel(pos, pg), pl);
        if constexpr (SA::NORM) {
#pragma unroll
          for (int g = 0; g < NG; ++g) {
            const V l = sa.plain(z[0][g], iv);  // 1 for the pivot row
#pragma unroll
            for (int k = 1; k < PB; ++k)
              if (k < zn) z[k][g] = sa.step(z[k][g], l, pv[k]);
            if (live[g] != NONE) coef[g][nb] = l;  // by slot
          }
        } else {
#pragma unroll
          for (int g = 0; g < NG; ++g) {
            const V na = sa.neg(z[0][g]);
            if (live[g] != NONE) Lm[ent[g]][t] = z[0][g];
            znew[g] = sa.mul(na, sc);
#pragma unroll
            for (int k = 1; k < PB; ++k) z[k][g] = sa.upd(pv[0], z[k][g], na, pv[k]);
          }
        }
        if (lane == pl) {
          s_piv[t] = make_int2(col, q);
          s_prow[t] = sel(ent, pg);
          s_y[t] = pv[0];
          if constexpr (SA::NORM) {
            s_xi[t] = iv;
          } else {
            s_psc[buf][j] = sc;
            s_pj[buf][j] = sel(ent, pg);
            V4 c4;  // (only the coefficients of earlier columns are read)
            c4.x = pv[0];
            c4.y = pv[1];
            c4.z = pv[2];
            c4.w = pv[3];
            s_pcoef[buf][j] = c4;
          }
        }
        if constexpr (!SA::NORM) sc = sa.mul(pv[0], sc);
        uint32_t gone = key;  // the entry that goes
        if (q != i0 + t) {
          // position i: the first entry's row, or a row outside the window
          const int i = i0 + t;
          uint32_t fkey = NONE;
#pragma unroll
          for (int g = 0; g < NG; ++g) fkey = min(fkey, live[g]);
          fkey = __reduce_min_sync(FULL, fkey);
          const int fg = (int)fkey >> 5, fl = (int)fkey & 31;
          const int f = __shfl_sync(FULL, sel(pos, fg), fl);
          if (f != i) {
            if (lane == 0) {
              p2r[q] = row_at(i, p2r, stamp, epoch);
              stamp[q] = epoch;
            }
          } else {
            // the first entry's row moves to the pivot's entry (and position)
            gone = fkey;
            const int en = __shfl_sync(FULL, sel(ent, fg), fl);
            const V vn = __shfl_sync(FULL, sel(znew, fg), fl);
#pragma unroll
            for (int k = 1; k < PB; ++k) {
              const V vx = __shfl_sync(FULL, sel(z[k], fg), fl);
#pragma unroll
              for (int g = 0; g < NG; ++g)
                if (g == pg && lane == pl) z[k][g] = vx;
            }
#pragma unroll
            for (int g = 0; g < NG; ++g)
              if (g == pg && lane == pl) {
                ent[g] = en;
                znew[g] = vn;
                coef[g] = reinterpret_cast<V *>(&s_coef[buf][en]);
              }
          }
        }
#pragma unroll
        for (int g = 0; g < NG; ++g)
          if (live[g] == gone) live[g] = NONE;
        ++t;
      }
#pragma unroll
      for (int g = 0; g < NG; ++g) {
#pragma unroll
        for (int k = 0; k + 1 < PB; ++k) z[k][g] = z[k + 1][g];
        z[PB - 1][g] = znew[g];
      }
    }
    // the live entries closed up (division-free: and their coefficients of the
    // block's pivot rows, which stand in z by column)
    __syncwarp();
    int base = 0;
#pragma unroll
    for (int g = 0; g < NG; ++g) {
      const unsigned alive = __ballot_sync(FULL, live[g] != NONE);
      if (live[g] != NONE) {
        const int e = base + __popc(alive & ((1u << lane) - 1u));
        s_ent[buf ^ 1][e] = ent[g];
        s_epos[buf ^ 1][e] = pos[g];
        if constexpr (!SA::NORM) {
          V4 c4;
          c4.x = z[0][g];
          c4.y = z[1][g];
          c4.z = z[2][g];
          c4.w = z[3][g];
          s_coef[buf][ent[g]] = c4;
        }
      }
      base += __popc(alive);
    }
    if (lane == 0) {
      s_sc[buf] = sc;
      s_next[buf] = next;
      s_rare[buf] = rare;
      s_t0[buf] = t0;
      s_t[buf] = t;
      s_nl[buf] = base;
    }
    nl = base;
    if (lane == 0) s_col0 = col0;
    col0 = next;
    __syncwarp();
  };

  bool ahead = false;
  while (col0 < w && i0 + t < m) {
    if (wid == 0) {
      if (nl <= 32) choose(std::integral_constant<int, 1>{}, ahead);
      else if (nl <= 64) choose(std::integral_constant<int, 2>{}, ahead);
      else choose(std::integral_constant<int, PW_G>{}, ahead);
    }
    // the block's pivots are known, and the block before is applied to all
    // columns right of this one
    __syncthreads();
    const int rare = s_rare[buf], tb = s_t0[buf], blk0 = wid == 0 ? s_col0 : col0;
    col0 = s_next[buf];
    t = s_t[buf];
    nl = s_nl[buf];
    // B. the other warps: the columns right of the block, from the rows'
    // values before it; not those of the next block, which warp 0 takes
    // itself while it chooses there (unless this one was cut short)
    // (the twelve warps of the other three schedulers, so that warp 0 does not
    // share its issue slots; division-free, where warp 0's own share costs more
    // than it hides, all warps and all columns, and a barrier)
    if ((!SA::NORM || (wid & 3) != 0) && t > tb) {
      const int right = SA::NORM && rare < 0 ? col0 + PB : col0;
      // a warp takes one half of the columns while both have some left, and
      // every sixth (eighth) row, then every twelfth (sixteenth) of the upper half
      const bool both = blk0 < 32;
      const int v0 = SA::NORM ? (wid >> 2) * 3 + (wid & 3) - 1 : wid;
      const int warps = SA::NORM ? 12 : PS_FAST, wh = both ? v0 >> 1 : v0, nw = both ? warps / 2 : warps;
      const int c = lane + (both ? 32 * (v0 & 1) : 32), nb = t - tb;
      V P[PB];  // the block's pivot rows, before it (by pivot; division-free by column)
      const int4 pj = SA::NORM ? make_int4(0, 0, 0, 0) : *reinterpret_cast<const int4 *>(s_pj[buf]);
      const int slots[PB] = {pj.x, pj.y, pj.z, pj.w};
#pragma unroll
      for (int k = 0; k < PB; ++k) {
        const bool there = SA::NORM ? k < nb : slots[k] >= 0;
        P[k] = there && c >= blk0 ? Wv[SA::NORM ? s_prow[tb + k] : slots[k]][c] : 0;
      }
      if constexpr (SA::NORM) finish(P, buf, tb, nb);
      {
        // the pivot rows to PV, a warp each (and half)
        int k = wh - (nw - PB), tk = tb + k;
        bool mine = k >= 0 && k < nb;
        if constexpr (!SA::NORM) {
          mine = false;
          tk = tb;
#pragma unroll
          for (int x = 0; x < PB; ++x) {
            if (x < k) tk += slots[x] >= 0;
            if (x == k) mine = slots[x] >= 0;
          }
        }
        if (mine) {
          V u = P[0];
#pragma unroll
          for (int x = 1; x < PB; ++x)
            if (x == k) u = P[x];
          if constexpr (!SA::NORM) {
            // at its choice in column k the row's coefficients of columns 0 .. k - 1
            // stood behind the 4 - k columns left
            const V *zz = reinterpret_cast<const V *>(&s_pcoef[buf][k]);
            V4 cf;
            cf.x = k > 0 ? zz[PB - k] : 0;
            cf.y = k > 1 ? zz[PB - k + 1] : 0;
            cf.z = k > 2 ? zz[PB - k + 2] : 0;
            cf.w = 0;
            u = sa.lin(s_psc[buf][k], u, cf, P);
          } else if (c == lane + 32 && lane < k) {  // (one of the halves)
            Lm[s_prow[tb + k]][tb + lane] = reinterpret_cast<const V *>(&s_coef[buf][s_prow[tb + k]])[lane];
          }
          if (c >= blk0) PV[tk][c] = u;
        }
        [[maybe_unused]] const V sc = s_sc[buf];
#pragma unroll 2
        for (int e = wh; e < nl; e += nw) {
          const int slot = s_ent[buf ^ 1][e];
          const V4 cf = s_coef[buf][slot];
          V v = Wv[slot][c];
          if constexpr (SA::NORM) {
            v = sa.lin(v, cf, P);
            if (c == lane + 32 && lane < nb)
              Lm[slot][tb + lane] = lane == 0 ? cf.x : lane == 1 ? cf.y : lane == 2 ? cf.z : cf.w;
          } else {
            v = sa.lin(sc, v, cf, P);
          }
          if (c >= right) Wv[slot][c] = v;
        }
      }
    }
    ahead = SA::NORM && rare < 0 && t > tb;
    buf ^= 1;
    if constexpr (!SA::NORM) __syncthreads();
    if (rare < 0) continue;

    // C. column `rare`: no window row has a pivot, rows past the window may
    __syncthreads();  // the window and PV are complete
    const int col = rare, i = i0 + t;
    const bool z = nl > 0 && s_epos[buf][0] == i;  // the row at position i is the first entry's
    int cand;
    {
      const int v = (lane <= col ? s_cnt[lane] : 0) + (lane + 32 <= col ? s_cnt[lane + 32] : 0);
      cand = __reduce_add_sync(FULL, v);
    }
    col0 = col + 1;
    __syncthreads();  // every thread has its count before s_cnt changes
    // per pass the CTA lists the candidates among PS_THREADS positions
    // (ordered compaction), then each warp reduces one of them by the t
    // pivots and records its exact head
    int found = -1, fw = 0;
    for (int base = wlast + 1; base < m && cand > 0 && found < 0; base += PS_THREADS) {
      const int pos = base + tid;
      int r = -1, hr = HEAD_NONE;
      if (pos < m) {
        r = row_at(pos, p2r, stamp, epoch);
        hr = head[r];
      }
      const bool isc = hr <= col;
      const unsigned bal = __ballot_sync(FULL, isc);
      if (lane == 0) s_wcnt[wid] = __popc(bal);
      __syncthreads();
      int off = 0, ncand = 0;
      for (int k = 0; k < PS_FAST; ++k) {
        const int v = s_wcnt[k];
        off += k < wid ? v : 0;
        ncand += v;
      }
      if (isc) {
        const int o = off + __popc(bal & ((1u << lane) - 1u));
        s_list[o] = pos;
        s_lrow[o] = r;
        s_lhead[o] = hr;
      }
      __syncthreads();
      for (int j0 = 0; j0 < ncand && found < 0; j0 += PS_FAST) {
        const int j = j0 + wid;
        int hit_pos = 0x7fffffff;
        if (j < ncand) {
          const int rj = s_lrow[j], hrj = s_lhead[j];
          const uint32_t *v = D + (size_t)rj * ld + c0;
          V a0 = sa.load(lane < w ? v[lane] : 0u), a1 = sa.load(lane + 32 < w ? v[lane + 32] : 0u);
          for (int k = 0; k < t; ++k) {
            const int pc = s_piv[k].x;
            const V f = __shfl_sync(FULL, pc < 32 ? a0 : a1, pc & 31);
            // (left of pc PV is not kept up to date; a column there is not read again)
            const V u0 = !SA::NORM || lane >= pc ? PV[k][lane] : 0;
            const V u1 = !SA::NORM || lane + 32 >= pc ? PV[k][lane + 32] : 0;
            if constexpr (SA::NORM) {
              const V l = sa.plain(f, s_xi[k]);
              if (lane == 0) s_rl[wid][k] = l;
              a0 = sa.step(a0, l, u0);
              a1 = sa.step(a1, l, u1);
            } else {
              const V nf = sa.neg(f);
              if (lane == 0) s_rl[wid][k] = f;
              a0 = sa.upd(s_y[k], a0, nf, u0);
              a1 = sa.upd(s_y[k], a1, nf, u1);
            }
          }
          s_red[wid][lane] = a0;
          s_red[wid][lane + 32] = a1;
          const unsigned b0 = __ballot_sync(FULL, a0 != 0 && lane >= col);
          const unsigned b1 = __ballot_sync(FULL, a1 != 0 && lane + 32 >= col);
          const int hn = b0 ? __ffs(b0) - 1 : (b1 ? 32 + __ffs(b1) - 1 : HEAD_NONE);
          if (hn == col) hit_pos = s_list[j];
          if (lane == 0 && hn != hrj) {
            head[rj] = (uint8_t)hn;
            atomicSub(&s_cnt[hrj], 1);
            atomicAdd(&s_cnt[hn], 1);
          }
        }
        if (lane == 0) s_first[wid] = hit_pos;
        __syncthreads();
        for (int k = 0; k < PS_FAST; ++k)
          if (s_first[k] < (found < 0 ? 0x7fffffff : found)) {
            found = s_first[k];
            fw = k;
          }
        __syncthreads();  // s_first and s_red are rewritten by the next round
      }
      cand -= ncand;
    }
    if (found < 0) {
      __syncthreads();
      continue;
    }
    // the pivot comes from past the window; the row at position i goes to
    // position `found`: the first entry leaves the window (with the bound of
    // its values), a row outside it is recorded in p2r
    const V y = s_red[fw][col];
    if (wid == 0) {
      int ri = -1;
      if (z) {
        const int slot = s_ent[buf][0];
        const unsigned b0 = __ballot_sync(FULL, lane > col && Wv[slot][lane] != 0);
        const unsigned b1 = __ballot_sync(FULL, lane + 32 > col && Wv[slot][lane + 32] != 0);
        const int hd = b0 ? __ffs(b0) - 1 : (b1 ? 32 + __ffs(b1) - 1 : HEAD_NONE);
        ri = wrow[slot];
        if (lane == 0) {
          head[ri] = (uint8_t)hd;
          atomicAdd(&s_cnt[hd], 1);
        }
        // the other entries close up
        int en[PW_G], po[PW_G];
#pragma unroll
        for (int g = 0; g < PW_G; ++g) {
          const int e = lane + 32 * g + 1;
          en[g] = e < nl ? s_ent[buf][e] : 0;
          po[g] = e < nl ? s_epos[buf][e] : 0;
        }
        __syncwarp();
#pragma unroll
        for (int g = 0; g < PW_G; ++g) {
          const int e = lane + 32 * g + 1;
          if (e < nl) {
            s_ent[buf][e - 1] = en[g];
            s_epos[buf][e - 1] = po[g];
          }
        }
      }
      if (lane == 0) {
        const int rq = row_at(found, p2r, stamp, epoch);
        atomicSub(&s_cnt[head[rq]], 1);
        if (!z) ri = row_at(i, p2r, stamp, epoch);
        p2r[found] = ri;
        stamp[found] = epoch;
        s_piv[t] = make_int2(col, found);
        s_prow[t] = PW_R + t;
        s_y[t] = y;
        if constexpr (SA::NORM) {
          const int iv = sa.inverse_abs(s_inv, y);
          s_xi[t] = y < 0 ? -iv : iv;
        }
      }
      PV[t][lane] = s_red[fw][lane];
      PV[t][lane + 32] = s_red[fw][lane + 32];
      if (lane < t) Lm[PW_R + t][lane] = s_rl[fw][lane];
      if (lane + 32 < t) Lm[PW_R + t][lane + 32] = s_rl[fw][lane + 32];
    }
    if (z) --nl;
    __syncthreads();
    if (tid < nl) Lm[s_ent[buf][tid]][t] = 0;  // the window rows' multipliers of this pivot
    if constexpr (!SA::NORM) {
      // the window rows are zero in the column: they are scaled by y
      for (int e = wid; e < nl; e += PS_FAST) {
        V *row = Wv[s_ent[buf][e]];
        row[lane] = sa.mul(y, row[lane]);
        row[lane + 32] = sa.mul(y, row[lane + 32]);
      }
    }
    ++t;
    __syncthreads();
  }
  __syncthreads();

  // Division-free: the S_k, their inverses, the pivots x_k = y_k / S_k and the
  // pivots' inverses, by warp 0 (lane l: k = l and l + 32) from prefix and
  // suffix products: S_k is 1 times the product (mul) of y_0 .. y_{k-1}; with the
  // one inverse I = 1 / S_t, 1 / S_k is I times the product of y_k ..
  // y_{t-1}, and 1 / y_k = mul (S_k, 1 / S_{k+1}).  For p < 2^31 the
  // reference's inverse is the exact one, so it fails for some pivot
  // exactly when S_t, a product of all y_k, has no inverse.  For larger p
  // the reference's inverse of each x_k itself.
  const bool exact_inv = p < 0x80000000u;
  const auto word = [seq](uint32_t v) { return (uint64_t)seq << 32 | v; };
  if (wid == 0) {
    // last final position of a non-pivot row with a nonzero panel, here of
    // the window rows left
    for (int e = lane; e < nl; e += 32) atomicMax(&s_last, s_epos[buf][e]);
    const V unit = sa.load(1u % p);
    V x0 = unit, x1 = unit;
    if constexpr (SA::NORM) {
      const bool none = (lane < t && s_xi[lane] == 0) || (lane + 32 < t && s_xi[lane + 32] == 0);
      if (__any_sync(FULL, none) && lane == 0) s_err = 1;  // a pivot without an inverse
      if (lane < t) {
        x0 = s_y[lane];
        xinv_out[lane] = sa.canon(s_xi[lane]);
      }
      if (lane + 32 < t) {
        x1 = s_y[lane + 32];
        xinv_out[lane + 32] = sa.canon(s_xi[lane + 32]);
      }
    } else {
      const V e = sa.one();
      V y0 = lane < t ? s_y[lane] : e, y1 = lane + 32 < t ? s_y[lane + 32] : e;
      V f0 = y0, f1 = y1, b0 = y0, b1 = y1;  // prefix, suffix products
#pragma unroll 1
      for (int o = 1; o < 32; o <<= 1) {
        const V u0 = __shfl_up_sync(FULL, f0, o), u1 = __shfl_up_sync(FULL, f1, o);
        const V d0 = __shfl_down_sync(FULL, b0, o), d1 = __shfl_down_sync(FULL, b1, o);
        if (lane >= o) {
          f0 = sa.mul(u0, f0);
          f1 = sa.mul(u1, f1);
        }
        if (lane + o < 32) {
          b0 = sa.mul(b0, d0);
          b1 = sa.mul(b1, d1);
        }
      }
      f1 = sa.mul(__shfl_sync(FULL, f0, 31), f1);
      b0 = sa.mul(b0, __shfl_sync(FULL, b1, 0));
      V S0 = __shfl_up_sync(FULL, f0, 1), S1 = __shfl_up_sync(FULL, f1, 1);
      const V f31 = __shfl_sync(FULL, f0, 31);
      if (lane == 0) S1 = f31;
      S0 = lane == 0 ? unit : sa.mul(unit, S0);
      S1 = sa.mul(unit, S1);
      const V St = sa.mul(unit, __shfl_sync(FULL, f1, 31));
      uint32_t err = 0;
      V si0, si1;
      uint32_t xi0, xi1;
      if (exact_inv) {
        const uint32_t I = t > 0 ? inv_exact_i31(p, sa.canon(St)) : 1u % p;
        if (t > 0 && I == 0u) err = 1;
        const V vI = sa.load(I);
        si0 = sa.mul(vI, b0);
        si1 = sa.mul(vI, b1);
        V n0 = __shfl_down_sync(FULL, si0, 1), n1 = __shfl_down_sync(FULL, si1, 1);
        const V s32 = __shfl_sync(FULL, si1, 0);
        if (lane == 31) {
          n0 = s32;
          n1 = vI;
        }
        x0 = sa.plain(y0, si0);
        x1 = sa.plain(y1, si1);
        const V yi0 = sa.mul(S0, n0), yi1 = sa.mul(S1, n1);
        s_yinv[lane] = yi0;
        s_yinv[lane + 32] = yi1;
        xi0 = sa.canon(sa.plain(S0, yi0));
        xi1 = sa.canon(sa.plain(S1, yi1));
      } else {
        si0 = sa.load(inv_exact_u32(p, sa.canon(S0)));
        si1 = sa.load(inv_exact_u32(p, sa.canon(S1)));
        x0 = sa.plain(y0, si0);
        x1 = sa.plain(y1, si1);
        xi0 = lela_inv_u32(p, sa.canon(x0));
        xi1 = lela_inv_u32(p, sa.canon(x1));
        if (lane < t && (sa.canon(si0) == 0u || xi0 == 0u)) err = 1;
        if (lane + 32 < t && (sa.canon(si1) == 0u || xi1 == 0u)) err = 1;
      }
      if (lane < t) {
        s_sinv[lane] = si0;
        s_xi[lane] = (int)xi0;
        xinv_out[lane] = xi0;
      }
      if (lane + 32 < t) {
        s_sinv[lane + 32] = si1;
        s_xi[lane + 32] = (int)xi1;
        xinv_out[lane + 32] = xi1;
      }
      if (__any_sync(FULL, err != 0u) && lane == 0) s_err = 1;
    }
    // the panel's determinant factor: product of the x_k
    V dv = lane < t ? x0 : unit;
    if (lane + 32 < t) dv = sa.plain(dv, x1);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) dv = sa.plain(dv, __shfl_xor_sync(FULL, dv, o));
    if (lane == 0) s_det = sa.canon(dv);
  } else if (wid == 2 || wid == 3) {
    const int k = tid - 64;
    if (k < t) {
      const int2 pv = s_piv[k];
      pcol_out[k] = (uint32_t)pv.x;
      hout[PANEL_W_PIV + 2 * k] = word((uint32_t)pv.x);
      hout[PANEL_W_PIV + 2 * k + 1] = word((uint32_t)pv.y);
    }
  } else if (wid == 1) {
    // the largest transposition target; the positions past the window up to
    // it, through p2r (beyond it rows have not moved)
    const int i = i0 + t;
    int hi = i - 1;
    if (lane < t) hi = max(hi, s_piv[lane].y);
    if (lane + 32 < t) hi = max(hi, s_piv[lane + 32].y);
    hi = __reduce_max_sync(FULL, hi);
    int last = -1;
    for (int pos = max(wlast + 1, i) + lane; pos <= hi && pos < m; pos += 32)
      if (act[row_at(pos, p2r, stamp, epoch)]) last = pos;
    atomicMax(&s_last, last);
    if (lane == 0) s_hi = hi;
  }
  __syncthreads();
  if (tid == 0) {
    const int la = *last_act;
    int last = s_last;
    if (la > s_hi) last = max(last, la);
    const uint32_t uinv = exact_inv && t > 0;
    last = max(last, 0);
    hout[PANEL_W_T] = word((uint32_t)t | uinv << 8 | (uint32_t)s_err << 9);
    hout[PANEL_W_LAST] = word((uint32_t)last);
    hout[PANEL_W_DET] = word(s_det);
    s_uinv = (int)uinv;
    *last_act = -1;
  }
  // U_k (division-free: (S_k U_k) / S_k); entries left of the pivot column are
  // not kept up to date, and U_k is zero there
  auto u_at = [&](int k, int c) {
    if constexpr (SA::NORM) return sa.canon(PV[k][c]);
    else return sa.canon(sa.plain(PV[k][c], s_sinv[k]));
  };
  for (int e = tid; e < t * EW; e += PS_THREADS) {
    const int k = e / EW, c = e % EW;
    Uout[e] = c < s_piv[k].x ? 0u : u_at(k, c);
  }
  __syncthreads();
  // After the result is on its way to the host, for p < 2^31 (exact
  // pivot inverses): the inverses of U_P, the t x t upper triangular matrix of
  // the pivot rows at the pivot columns (U_P[k][j] = U_k[pcol_j], diagonal
  // x_k), and of L11, the unit lower triangle of the pivot rows' multipliers,
  // padded to 64 x 64 with the identity.  A row's multipliers are then
  // a_P U_P^-1 (a_P: its values at the pivot columns), all at once, and the pivot
  // rows' other columns U12 = L11^-1 A12.  In the
  // window's shared memory, now free.
  if (s_uinv) {
    uint32_t *X = dyn_w, *Y = X + INV_M, *T = Y + INV_M;
    for (int e = tid; e < EW * EW; e += PS_THREADS) {
      const int k = e / EW, j = e % EW;
      uint32_t u = k == j ? 1u : 0u, l = u;
      if (k < t && j < t) {
        if (j == k) u = SA::NORM ? sa.canon(s_xi[k]) : (uint32_t)s_xi[k];
        else if (j > k) u = u_at(k, s_piv[j].x);
        else if constexpr (SA::NORM) l = sa.canon(Lm[s_prow[k]][j]);
        else l = sa.canon(sa.plain(Lm[s_prow[k]][j], s_yinv[j]));
      }
      X[k * INV_LD + j] = u;
      Y[k * INV_LD + j] = l;
    }
    __syncthreads();
    const bool upper = tid < INV_THREADS;
    tri64_invert<A>(upper ? X : Y, upper ? T : T + INV_T, upper, ar, tid & (INV_THREADS - 1), t);
    for (int e = tid; e < t * EW; e += PS_THREADS) {
      Uinv_out[e] = X[e / EW * INV_LD + e % EW];
      Linv_out[e] = Y[e / EW * INV_LD + e % EW];
    }
  }
}

// Row permutation in one launch: each CTA takes a slice of PERM_COLS
// columns of every moved row.  Its threads load all their elements of the
// source rows at once (at most PERM_PER each, into registers), wait at the
// barrier, then store them to the destination rows; the CTAs own disjoint
// columns, so no grid-wide ordering is needed.  cnt <= 2 * EW rows.
constexpr int PERM_THREADS = 256, PERM_COLS = 32;
constexpr int PERM_PER = 2 * EW * PERM_COLS / PERM_THREADS;
__global__ void __launch_bounds__(PERM_THREADS)
    permute_rows_kernel(uint32_t *D, size_t ld, int n, const int *src,
                        const int *dst, int cnt) {
  pdl_enter();
  const int c0 = blockIdx.x * PERM_COLS, total = cnt * PERM_COLS;
  uint32_t v[PERM_PER];
#pragma unroll
  for (int u = 0; u < PERM_PER; ++u) {
    const int e = threadIdx.x + u * PERM_THREADS, c = c0 + e % PERM_COLS;
    v[u] = (e < total && c < n) ? D[(size_t)src[e / PERM_COLS] * ld + c] : 0u;
  }
  __syncthreads();
#pragma unroll
  for (int u = 0; u < PERM_PER; ++u) {
    const int e = threadIdx.x + u * PERM_THREADS, c = c0 + e % PERM_COLS;
    if (e < total && c < n) D[(size_t)dst[e / PERM_COLS] * ld + c] = v[u];
  }
}

// 4. Rows i0..r1 at their final positions, one warp per row: the
// reference's elimination steps on the panel part, pivot k applied with
// multiplier l_k = v[pcol_k] / x_k (v: the row's current value) and
// v -= l_k U_k.  Pivot row k takes the pivots before it (its L11 row, unit
// lower; its panel becomes U_k); rows below take all t (their L21 row; their
// panel becomes zero).  Row i0 + r of L = [L11; L21] goes to
// Lout[r * ldl + 0 .. t-1].
constexpr int SOLVE_THREADS = 256;
__global__ void __launch_bounds__(SOLVE_THREADS)
    panel_solve_kernel(uint32_t *__restrict__ D, size_t ld, int i0, int r1, int c0, int w, int t,
                       const uint32_t *__restrict__ pcol, const uint32_t *__restrict__ Uin,
                       const uint32_t *__restrict__ xinv, ArithWide ar,
                       uint32_t *__restrict__ Lout, size_t ldl) {
  __shared__ uint32_t sU[EW][EW];
  __shared__ uint32_t sX[EW];
  __shared__ int sP[EW];
  const int tid = threadIdx.x, lane = tid & 31;
  for (int e = tid; e < t * EW; e += SOLVE_THREADS) cp_async4(&sU[e / EW][e % EW], Uin + e, true);
  if (tid < EW) {
    sX[tid] = tid < t ? xinv[tid] : 0u;
    sP[tid] = tid < t ? (int)pcol[tid] : 0;
  }
  cp_async_wait_all();
  __syncthreads();
  const uint32_t p = ar.p;
  const int warps = (gridDim.x * SOLVE_THREADS) >> 5;
  for (int pos = i0 + ((blockIdx.x * SOLVE_THREADS + tid) >> 5); pos <= r1; pos += warps) {
    uint32_t *row = D + (size_t)pos * ld + c0;
    uint32_t a0 = lane < w ? row[lane] : 0u, a1 = lane + 32 < w ? row[lane + 32] : 0u;
    const int kk = pos - i0, lim = kk < t ? kk : t;
    uint32_t l0 = 0u, l1 = 0u;  // multipliers k = lane, lane + 32
    if (__any_sync(0xffffffffu, (a0 | a1) != 0u)) {
      for (int k = 0; k < lim; ++k) {
        const int pc = sP[k];
        const uint32_t f = __shfl_sync(0xffffffffu, pc < 32 ? a0 : a1, pc & 31);
        const uint32_t l = ar.mul(f, sX[k]);
        if (k == lane) l0 = l;
        if (k == lane + 32) l1 = l;
        const uint32_t nl = l ? p - l : 0u;
        a0 = ar.dot2(1u, a0, nl, sU[k][lane]);
        a1 = ar.dot2(1u, a1, nl, sU[k][lane + 32]);
      }
    }
    if (lane < w) row[lane] = a0;
    if (lane + 32 < w) row[lane + 32] = a1;
    uint32_t *lr = Lout + (size_t)kk * ldl;
    if (kk < t) {
      if (lane < t) lr[lane] = lane < kk ? l0 : (lane == kk ? 1u : 0u);
      if (lane + 32 < t) lr[lane + 32] = lane + 32 < kk ? l1 : (lane + 32 == kk ? 1u : 0u);
    } else {
      if (lane < t) lr[lane] = l0;
      if (lane + 32 < t) lr[lane + 32] = l1;
    }
  }
}

// The same results for p < 2^31 from the inverse of U_P (the search's
// Uinv, t x EW): a row's multipliers are l = a_P U_P^-1 (a_P: the row's
// values at the pivot columns), one dot product of length t per lane
// instead of t dependent elimination steps.  A pivot row k (position i0 +
// k) keeps multipliers l_j for j < k and 1 at k (a_P = sum_{j<k} l_j U_P[j] +
// U_P[k]), and its panel becomes U_k; every other row's panel becomes zero
// (each panel column either holds a pivot, eliminated from all rows below
// it, or was zero at and below the pivot row when it was reached).
template <class A>
__global__ void __launch_bounds__(SOLVE_THREADS)
    panel_solve_inv_kernel(uint32_t *D, size_t ld, int i0, int r1, int c0, int w,
                           int t, const uint32_t *pcol,
                           const uint32_t *Uin, const uint32_t *Uinv,
                           A ar, uint32_t *Lout, size_t ldl) {
  pdl_enter();
  __shared__ uint32_t sUi[EW][EW];
  __shared__ int sP[EW];
  const int tid = threadIdx.x, lane = tid & 31;
  for (int e = tid; e < t * EW; e += SOLVE_THREADS) cp_async4(&sUi[e / EW][e % EW], Uinv + e, true);
  if (tid < EW) sP[tid] = tid < t ? (int)pcol[tid] : 0;
  cp_async_wait_all();
  __syncthreads();
  const int pc0 = sP[lane], pc1 = sP[lane + 32];
  const int warps = (gridDim.x * SOLVE_THREADS) >> 5;
  for (int pos = i0 + ((blockIdx.x * SOLVE_THREADS + tid) >> 5); pos <= r1; pos += warps) {
    uint32_t *row = D + (size_t)pos * ld + c0;
    const uint32_t a0 = lane < w ? row[lane] : 0u, a1 = lane + 32 < w ? row[lane + 32] : 0u;
    // the row's values at the pivot columns: lane j holds a[pcol_j], a[pcol_{j+32}]
    const uint32_t x0 = __shfl_sync(0xffffffffu, a0, pc0 & 31);
    const uint32_t x1 = __shfl_sync(0xffffffffu, a1, pc0 & 31);
    const uint32_t y0 = __shfl_sync(0xffffffffu, a0, pc1 & 31);
    const uint32_t y1 = __shfl_sync(0xffffffffu, a1, pc1 & 31);
    const uint32_t ap0 = lane < t ? (pc0 < 32 ? x0 : x1) : 0u;
    const uint32_t ap1 = lane + 32 < t ? (pc1 < 32 ? y0 : y1) : 0u;
    uint32_t l0 = 0u, l1 = 0u;  // multipliers k = lane, lane + 32
    if (__any_sync(0xffffffffu, (ap0 | ap1) != 0u)) {
      typename A::Acc s0 = A::zero(), s1 = A::zero();
      for (int j = 0; j < t; ++j) {
        const uint32_t f = __shfl_sync(0xffffffffu, j < 32 ? ap0 : ap1, j & 31);
        ar.acc(s0, f, sUi[j][lane]);
        ar.acc(s1, f, sUi[j][lane + 32]);
      }
      l0 = ar.sum(s0);
      l1 = ar.sum(s1);
    }
    const int kk = pos - i0;
    uint32_t *lr = Lout + (size_t)kk * ldl;
    if (kk < t) {
      if (lane < w) row[lane] = Uin[(size_t)kk * EW + lane];
      if (lane + 32 < w) row[lane + 32] = Uin[(size_t)kk * EW + lane + 32];
      if (lane < t) lr[lane] = lane < kk ? l0 : (lane == kk ? 1u : 0u);
      if (lane + 32 < t) lr[lane + 32] = lane + 32 < kk ? l1 : (lane + 32 == kk ? 1u : 0u);
    } else {
      if (lane < w) row[lane] = 0u;
      if (lane + 32 < w) row[lane + 32] = 0u;
      if (lane < t) lr[lane] = l0;
      if (lane + 32 < t) lr[lane + 32] = l1;
    }
  }
}

// U12 = L11^-1 A12 for one panel, in place: forward substitution x_k = a_k -
// sum_{j<k} L11[k][j] x_j with the unit lower L11 (the panel's multipliers of
// its pivot rows, row stride ldl) in shared memory.  Four lanes per column
// of A12, lane l holding the column's entries j = l mod 4 in registers (the
// loops fully unrolled, so every register index is a constant): per k each
// lane sums its share of the products, two shuffles add the four shares, and
// the owner of entry k updates it.  The same field operations as any
// substitution with a unit diagonal.
constexpr int U12_THREADS = 128;
constexpr int U12_COLS = U12_THREADS / 4;
template <class A>
__global__ void __launch_bounds__(U12_THREADS)
    panel_u12_kernel(const uint32_t *__restrict__ L, size_t ldl, int t, uint32_t *__restrict__ B,
                     size_t ldb, int ncols, A ar) {
  __shared__ __align__(16) uint32_t sL[EW][EW];
  {
    constexpr int PER = EW * EW / U12_THREADS;
    uint32_t v[PER];
#pragma unroll
    for (int u = 0; u < PER; ++u) {
      const int e = threadIdx.x + u * U12_THREADS, k = e / EW, j = e % EW;
      v[u] = (k < t && j < k) ? L[(size_t)k * ldl + j] : 0u;
    }
#pragma unroll
    for (int u = 0; u < PER; ++u) {
      const int e = threadIdx.x + u * U12_THREADS;
      sL[e / EW][e % EW] = v[u];
    }
  }
  __syncthreads();
  const int l4 = threadIdx.x & 3;
  const int c = blockIdx.x * U12_COLS + (threadIdx.x >> 2);
  const bool valid = c < ncols;  // every lane stays for the shuffles
  const uint32_t p = ar.p;
  uint32_t x[EW / 4];  // x[i]: entry 4 i + l4
#pragma unroll
  for (int i = 0; i < EW / 4; ++i) {
    const int j = 4 * i + l4;
    x[i] = (valid && j < t) ? B[(size_t)j * ldb + c] : 0u;
  }
#pragma unroll
  for (int k = 1; k < EW; ++k) {
    if (k < t) {
      // entries j >= k still hold a_j, but L11[k][j] is zero there
      typename A::Acc acc = A::zero();
#pragma unroll
      for (int i = 0; i <= (k - 1) / 4; ++i) ar.acc(acc, sL[k][4 * i + l4], x[i]);
      uint32_t v = ar.sum(acc);
#pragma unroll
      for (int o = 1; o <= 2; o <<= 1) {  // v + w mod p without overflow (any p < 2^32)
        const uint32_t nw = p - __shfl_xor_sync(0xffffffffu, v, o);
        v = v >= nw ? v - nw : v + (p - nw);
      }
      if (l4 == (k & 3)) {
        const uint32_t a = x[k >> 2];
        x[k >> 2] = a >= v ? a - v : a + (p - v);
      }
    }
  }
#pragma unroll
  for (int i = 0; i < EW / 4; ++i) {
    const int j = 4 * i + l4;
    if (valid && j >= 1 && j < t) B[(size_t)j * ldb + c] = x[i];
  }
}

// Whether U12 is substituted column by column for p < 2^31, too: wide panels, whose product has
// many tiles of the same t <= 64 rows.  Measured with its launch (us, steps / product): p = 2^31
// - 1 t = 64 4000 columns 25 / 22, 8000 27 / 33, 32000 62 / 76, 300000 437 / 573, t = 8 16000 13 /
// 45, 300000 88 / 518; p = 65521 t = 64 32000 35 / 29, 300000 240 / 143, t = 32 32000 23 / 27, 300000
// 123 / 121, t = 16 32000 19 / 24, 300000 89 / 119, t = 2 300000 70 / 115; p = 251 t = 24 32000 21 /
// 22, 300000 105 / 96, t = 16 300000 88 / 94.  (Narrow panels of few pivots keep the product,
// whose launch starts early behind the solve: a 64 x 8000 form modulo 2^31 - 1 takes 107 us with
// it and 113 by steps, a 64 x 20000 one 130 and 121, 20 x 8000 74 and 63.)
static bool u12_by_steps(uint32_t p, int t, int rest) {
  if (p > 65536) return rest > (t <= 48 ? 6000 : 12000);
  return t <= 16 && rest > 16000;
}

int zp_echelon_dev(Ctx *c, int m, int n, uint32_t p, uint32_t *D, size_t ld, size_t *rank_out,
                   uint32_t *det_out, std::vector<int> *pivot_cols, EchelonKeep *keep) {
  if (p < 2) return ctx_fail(c, ST_ARG, "modulus must be at least 2");
  if (m < 0 || n < 0) return ctx_fail(c, ST_ARG, "negative dimension");
  if (m > 0 && n > 0 && ld < (size_t)n) return ctx_fail(c, ST_ARG, "leading dimension too small");
  if (pivot_cols) pivot_cols->clear();
  uint64_t det = 1 % p;
  size_t rank = 0;
  if (m == 0 || n == 0) {
    *rank_out = 0;
    *det_out = (uint32_t)det;
    return ST_OK;
  }

  // device scratch
  const size_t out_bytes = EW * sizeof(uint32_t);  // pivot columns
  // p2r, stamp (m each); permutation lists (4 EW); last row (1); histogram (EW + 1)
  const size_t i_bytes =
      (((size_t)2 * m + 4 * EW + 1 + EW + 1) * sizeof(int) + 255) & ~(size_t)255;
  const size_t h_bytes = ((size_t)2 * m + 255) & ~(size_t)255;
  const size_t sq_bytes = (size_t)EW * EW * 4;
  const size_t l_bytes = (size_t)m * EB * 4;
  void *base = nullptr;
  int st = ctx_buffer(c, BUF_ECH_0,
                      out_bytes + i_bytes + h_bytes + 4 * sq_bytes + l_bytes + 1024,
                      &base);
  if (st) return st;
  uint8_t *b8 = static_cast<uint8_t *>(base);
  uint32_t *d_pcol = reinterpret_cast<uint32_t *>(b8);
  int *d_p2r = reinterpret_cast<int *>(b8 + out_bytes);
  int *d_stamp = d_p2r + m;
  int *d_perm = d_stamp + m;      // 4*EW ints: src list, dst list
  int *d_last = d_perm + 4 * EW;  // largest row with a nonzero panel
  int *d_hist = d_last + 1;       // EW + 1 head counts
  uint8_t *d_head = b8 + out_bytes + i_bytes;
  uint8_t *d_act = d_head + m;
  uint32_t *d_U = reinterpret_cast<uint32_t *>(b8 + out_bytes + i_bytes + h_bytes);
  uint32_t *d_xinv = d_U + EW * EW;  // pivot inverses (EW)
  uint32_t *d_Uinv = d_xinv + EW * EW;  // U_P^-1 (t x EW), p < 2^31
  uint32_t *d_Linv = d_Uinv + EW * EW;  // L11^-1 (t x EW), p < 2^31
  uint32_t *d_L = d_Linv + EW * EW;  // the block's multipliers (m x EB)
  void *gws = nullptr;
  // one size for the panel and block updates and the block's trsm (which
  // takes the same workspace, so it must not grow it)
  st = ctx_workspace(c, std::max(zp_gemm_workspace_bytes(p, m, n, EB),
                                 zp_trsm_workspace_bytes(p, EB, n)),
                     &gws);
  if (st) return st;
  const WsHold hold(c);  // gws
  const bool small = p < (1u << 16);
  const uint16_t *inv_table = nullptr;
  if (SearchSmall::takes(p)) {
    void *tb = nullptr;
    if ((st = ctx_buffer(c, BUF_INV, PW_TABLE, &tb))) return st;
    if (c->inv_p != p) {
      c->inv_p = 0;  // p only when the first panel's result shows that the table is there
      inverse_table_kernel<<<((int)p / 2 + 261) / 256, 256, 0, c->stream>>>(p, static_cast<uint16_t *>(tb));
      ctx_launched(c);
      const cudaError_t ei = cudaGetLastError();
      if (ei != cudaSuccess) return ctx_cuda(c, ei, "echelon: inverses");
    }
    inv_table = static_cast<const uint16_t *>(tb);
  }
  const ArithSmall ars = ArithSmall::make(p);
  const ArithWide arw = ArithWide::make(p);
  void *mh = nullptr, *md = nullptr;
  if ((st = ctx_panel_map(c, &mh, &md))) return st;
  int *hperm = reinterpret_cast<int *>(static_cast<char *>(mh) + PANEL_PERM_OFF);
  static_assert(2 * (2 * EW) <= (int)PANEL_PERM_INTS, "staging layout");
  auto words = [](void *map) {
    return reinterpret_cast<volatile uint64_t *>(static_cast<char *>(map) + PANEL_WORDS_OFF);
  };
  volatile uint64_t *hwords = words(mh), *hwords_dev = words(md);
  cudaError_t e = cudaMemsetAsync(d_stamp, 0xff, (size_t)m * sizeof(int), c->stream);
  if (e == cudaSuccess && keep) {
    keep->swaps.clear();
    e = cudaMemsetAsync(keep->L, 0, (size_t)m * keep->ldL * 4, c->stream);
  }
  if (e == cudaSuccess) e = cudaMemsetAsync(d_last, 0xff, sizeof(int), c->stream);
  if (e == cudaSuccess) e = cudaMemsetAsync(d_hist, 0, (EW + 1) * sizeof(int), c->stream);
  if (e != cudaSuccess) return ctx_cuda(c, e, "echelon: scratch");

  struct {
    uint32_t t, uinv, err, last_pos, det;  // see the words' enum
    uint32_t pcol[EW], ti[EW], tq[EW];     // pivot columns; transposition k: (ti[k], tq[k])
  } h;
  std::vector<int> at, src, dst;
  int i = 0, epoch = 0;
  const int head_grid = std::max(1, std::min((m + 7) / 8, c->num_sms * 2));
  // Blocks of EB columns (delayed updates): a block's panels update only the
  // block's columns; the columns right of it are updated once per block,
  // U12 = L11^-1 A12 on the block's Tb pivot rows (from row ib) and
  // A22 -= L21 U12 on the rows below, down to R.  L = [L11; L21] holds the
  // block's multipliers: d_L row q (stride EB) belongs to the row at position
  // q, panel k of the block fills columns Tb_k .. Tb_k + t_k - 1, and later
  // panels' transpositions move d_L's rows with D's.  The result is the
  // panel-by-panel one: the multipliers are the same, and the delayed update
  // is the same Schur complement.  A block is delayed when the first panel
  // with pivots has at least DELAY_ROWS rows to update below them (dense
  // matrices); otherwise (staircase Schur complements, where few rows are
  // touched) each panel updates all columns at once and the block solve is
  // not paid.
  constexpr int DELAY_ROWS = 512;
  int ib = 0, Tb = 0, R = -1, b1 = 0, delayed = 0;
  auto flush = [&]() -> int {
    if (Tb == 0 || b1 >= n) return ST_OK;
    int s = zp_trsm_dev(c, false, true, Tb, n - b1, p, 1, d_L + (size_t)ib * EB, EB,
                        D + (size_t)ib * ld + b1, ld, nullptr);
    if (s) return s;
    const int rb = ib + Tb;
    if (R < rb) return ST_OK;
    int pi = prof_begin(c, "ech_block_update");
    s = zp_gemm_dev(c, GEMM_AUTO, R - rb + 1, n - b1, Tb, p, p - 1, d_L + (size_t)rb * EB, EB,
                    D + (size_t)ib * ld + b1, ld, 1, D + (size_t)rb * ld + b1, ld,
                    static_cast<uint8_t *>(gws));
    prof_end(c, pi);
    return s;
  };
  auto search = [&](auto sa, auto ar, int i, int c0, int w, uint32_t seq, int wcap) -> int {
    auto kern = panel_search_kernel<decltype(sa), decltype(ar)>;
    const size_t smem = PW_SMEM + (decltype(sa)::NORM ? PW_TABLE : 0);
    int s = ctx_smem_attr(c, (const void *)kern, (int)smem, "echelon: panel search attributes");
    if (s) return s;
    pdl_launch(kern, 1, PS_THREADS, smem, c->stream, D, ld, i, m, c0, w, sa, ar, d_head, d_act,
               d_hist, d_last, d_p2r, d_stamp, epoch, d_U, d_xinv, d_Uinv, d_Linv, d_pcol,
               hwords_dev, seq, wcap);
    return ST_OK;
  };
  // window rows of the search: the full PW_R, or 64 when the previous panel
  // had many rows below its pivots (dense matrices, where the first 64
  // active rows nearly always hold the panel's pivots; the rows past the
  // window stay reachable through the search's slower path)
  int wcap = PW_R;
  for (int c0 = 0; c0 < n && i < m; c0 += EW) {
    const int w = std::min(EW, n - c0);
    if (c0 % EB == 0) {
      if ((st = flush())) return st;
      ib = i;
      Tb = 0;
      R = -1;
      b1 = std::min(n, c0 + EB);
      delayed = -1;  // decided at the block's first panel with pivots
    }
    int pi = prof_begin(c, "ech_heads");
    pdl_launch(panel_heads_kernel, head_grid, HEADS_THREADS, 0, c->stream, D, ld, i, m, c0, w, p,
               d_head, d_act, d_hist, d_last);
    prof_end(c, pi);
    const uint32_t seq = ++c->panel_seq;
    pi = prof_begin(c, "ech_search");
    if (SearchSmall::takes(p))
      st = search(SearchSmall::make(p, inv_table), ars, i, c0, w, seq, wcap);
    else if (SearchMont::takes(p))
      st = search(SearchMont::make(p), arw, i, c0, w, seq, wcap);
    else if (small)
      st = search(SearchPlain<ArithSmall>::make(p), ars, i, c0, w, seq, wcap);
    else
      st = search(SearchPlain<ArithWide>::make(p), arw, i, c0, w, seq, wcap);
    if (st) return st;
    ++epoch;
    prof_end(c, pi);
    ctx_launched(c, 2);
    auto word = [&](int k, uint32_t *v) -> int {
      int s = ctx_wait_flag(c, reinterpret_cast<volatile uint32_t *>(hwords + k) + 1, seq,
                            "echelon: panel");
      if (s == ST_OK) *v = (uint32_t)hwords[k];
      return s;
    };
    uint32_t head_word = 0;
    if ((st = word(PANEL_W_T, &head_word)) || (st = word(PANEL_W_LAST, &h.last_pos)) ||
        (st = word(PANEL_W_DET, &h.det)))
      return st;
    if (inv_table) c->inv_p = p;
    h.t = std::min<uint32_t>(head_word & 0xffu, EW);
    h.uinv = head_word >> 8 & 1u;
    h.err = head_word >> 9 & 1u;
    for (uint32_t k = 0; k < h.t; ++k) {
      h.ti[k] = (uint32_t)i + k;
      if ((st = word(PANEL_W_PIV + 2 * (int)k, &h.pcol[k])) ||
          (st = word(PANEL_W_PIV + 2 * (int)k + 1, &h.tq[k])))
        return st;
    }
    if (h.err) return ctx_fail(c, ST_PIVOT, "Could not invert pivot-element in the ring");
    const int t = (int)h.t;
    if (t == 0) continue;
    // replay the transpositions on the positions they touch
    int hi = i;
    for (int k = 0; k < t; ++k) hi = std::max(hi, (int)h.tq[k]);
    at.resize(hi - i + 1);
    for (int q = i; q <= hi; ++q) at[q - i] = q;
    for (int k = 0; k < t; ++k) std::swap(at[h.ti[k] - i], at[h.tq[k] - i]);
    src.clear();
    dst.clear();
    for (int q = i; q <= hi; ++q)
      if (at[q - i] != q) {
        dst.push_back(q);
        src.push_back(at[q - i]);
      }
    const int cnt = (int)src.size();
    if (cnt > 2 * EW) return ctx_fail(c, ST_ARG, "echelon: permutation larger than expected");
    if (cnt > 0) {
      for (int k = 0; k < cnt; ++k) {
        hperm[k] = src[k];
        hperm[cnt + k] = dst[k];
      }
      e = cudaMemcpyAsync(d_perm, hperm, (size_t)2 * cnt * sizeof(int), cudaMemcpyHostToDevice,
                          c->stream);
      if (e != cudaSuccess) return ctx_cuda(c, e, "echelon: permutation");
      pdl_launch(permute_rows_kernel, (n + PERM_COLS - 1) / PERM_COLS, PERM_THREADS, 0, c->stream,
          D, ld, n, d_perm, d_perm + cnt, cnt);
      ctx_launched(c);
      if (Tb > 0) {  // the multipliers of the block's earlier panels move too
        pdl_launch(permute_rows_kernel, (EB + PERM_COLS - 1) / PERM_COLS, PERM_THREADS, 0, c->stream,
            d_L, EB, EB, d_perm, d_perm + cnt, cnt);
        ctx_launched(c);
      }
      if (keep && rank > 0) {  // and every earlier pivot's kept multipliers
        pdl_launch(permute_rows_kernel, ((int)rank + PERM_COLS - 1) / PERM_COLS, PERM_THREADS, 0,
                   c->stream, keep->L, keep->ldL, (int)rank, d_perm, d_perm + cnt, cnt);
        ctx_launched(c);
      }
    }
    // L11 / L21 and the panel's final values
    const int r0 = i + t;
    const int r1 = (h.last_pos >= (uint32_t)r0) ? (int)h.last_pos : r0 - 1;
    const int below = r1 - r0 + 1;
    wcap = below >= DELAY_ROWS ? EW : PW_R;
    if (delayed < 0) {
      delayed = below >= DELAY_ROWS;
      if (delayed) {  // rows a panel's solve does not reach hold zero multipliers
        e = cudaMemsetAsync(d_L + (size_t)i * EB, 0, (size_t)(m - i) * EB * 4, c->stream);
        if (e != cudaSuccess) return ctx_cuda(c, e, "echelon: multipliers");
      }
    }
    uint32_t *Lp = d_L + (size_t)i * EB + Tb;  // this panel's columns of L, from row i
    {
      const int groups = (r1 - i + 1 + SOLVE_THREADS / 32 - 1) / (SOLVE_THREADS / 32);
      pi = prof_begin(c, "ech_solve");
      const int sgrid = std::max(1, std::min(groups, c->num_sms * 8));
      // U_P^-1 when the search wrote it (p < 2^31: exact pivot inverses), else
      // the elimination steps
      if (h.uinv && small)
        pdl_launch(panel_solve_inv_kernel<ArithSmall>, sgrid, SOLVE_THREADS, 0, c->stream,
            D, ld, i, r1, c0, w, t, d_pcol, d_U, d_Uinv, ars, Lp, EB);
      else if (h.uinv)
        pdl_launch(panel_solve_inv_kernel<ArithWide>, sgrid, SOLVE_THREADS, 0, c->stream,
            D, ld, i, r1, c0, w, t, d_pcol, d_U, d_Uinv, arw, Lp, EB);
      else
        panel_solve_kernel<<<sgrid, SOLVE_THREADS, 0, c->stream>>>(D, ld, i, r1, c0, w, t, d_pcol,
                                                                   d_U, d_xinv, arw, Lp, EB);
      prof_end(c, pi);
      ctx_launched(c);
    }
    if (keep) {
      // this panel's multipliers (rows i..r1) into columns rank.. of L
      e = cudaMemcpy2DAsync(keep->L + (size_t)i * keep->ldL + rank, keep->ldL * 4, Lp, EB * 4,
                            (size_t)t * 4, (size_t)(r1 - i + 1), cudaMemcpyDeviceToDevice,
                            c->stream);
      if (e != cudaSuccess) return ctx_cuda(c, e, "pluq: multipliers");
      for (int k = 0; k < t; ++k) keep->swaps.emplace_back((int)h.ti[k], (int)h.tq[k]);
    }
    // the rest of the block's columns (delayed), or of all columns
    const int rest = (delayed ? b1 : n) - (c0 + w);
    if (rest > 0) {
      uint32_t *U12 = D + (size_t)i * ld + c0 + w;
      pi = prof_begin(c, "ech_u12");
      if (h.uinv && !u12_by_steps(p, t, rest)) {
        // U12 = L11^-1 A12 in place: one tile of rows, each CTA on its columns
        if ((st = zp_gemm_dev(c, GEMM_DIRECT, t, rest, t, p, 1, d_Linv, EW, U12, ld, 0, U12, ld,
                              static_cast<uint8_t *>(gws))))
          return st;
      } else {
        const int ugrid = (rest + U12_COLS - 1) / U12_COLS;
        if (small)
          panel_u12_kernel<<<ugrid, U12_THREADS, 0, c->stream>>>(Lp, EB, t, U12, ld, rest, ars);
        else
          panel_u12_kernel<<<ugrid, U12_THREADS, 0, c->stream>>>(Lp, EB, t, U12, ld, rest, arw);
        ctx_launched(c);
      }
      prof_end(c, pi);
      if (below > 0) {
        pi = prof_begin(c, "ech_update");
        st = zp_gemm_dev(c, GEMM_AUTO, below, rest, t, p, p - 1, Lp + (size_t)t * EB, EB, U12,
                         ld, 1, D + (size_t)r0 * ld + c0 + w, ld, static_cast<uint8_t *>(gws));
        prof_end(c, pi);
        if (st) return st;
      }
    }
    if (delayed) {
      // rows with multipliers: down to r1, and wherever a transposition moved one
      R = std::max(R, std::max(r1, hi));
      Tb += t;
    }
    det = (det * h.det) % p;
    if (pivot_cols)
      for (int k = 0; k < t; ++k) pivot_cols->push_back(c0 + (int)h.pcol[k]);
    rank += t;
    i += t;
  }
  if ((st = flush())) return st;
  *rank_out = rank;
  *det_out = (uint32_t)det;
  return ST_OK;
}

// ---------------------------------------------------------------- PLUQ
//
// Elimination::pluq (lela/algorithms/elimination.tcc:266-370) with
// DensePivotStrategy: at step i the first column, in the current column
// order, with a nonzero at or below row i, and its first such row, are
// swapped into place (transpositions (i, row) and (i, column)); det is
// multiplied by the pivot x; every row j below gets row_j - (a / x) row_i
// right of the pivot and keeps a / x below the diagonal.  A column passed
// over at step i is zero at and below row i and stays so, so the pivots are
// those of the non-reduced echelon form: the same rows, transpositions and
// values (the eliminations are the same field operations).  The echelon
// pipeline therefore runs with its multipliers kept (EchelonKeep); Q
// follows on the host from the pivot columns, and one gather writes L
// below the diagonal and U, its columns in Q's order, on and above it.

__global__ void pluq_assemble_kernel(const uint32_t *__restrict__ U, size_t ldu,
                                     const uint32_t *__restrict__ L, size_t ldl,
                                     const int *__restrict__ qcol, int m, int n, int r,
                                     uint32_t *__restrict__ out) {
  const size_t total = (size_t)m * n;
  for (size_t idx = blockIdx.x * (size_t)blockDim.x + threadIdx.x; idx < total;
       idx += (size_t)gridDim.x * blockDim.x) {
    const int q = (int)(idx / n), j = (int)(idx % n);
    out[idx] = j < min(q, r) ? L[(size_t)q * ldl + j] : U[(size_t)q * ldu + qcol[j]];
  }
}

int zp_pluq_dev(Ctx *c, int m, int n, uint32_t p, uint32_t *D, size_t ld,
                std::vector<std::pair<int, int>> *P, std::vector<std::pair<int, int>> *Q,
                size_t *rank, uint32_t *det) {
  P->clear();
  Q->clear();
  if (p < 2) return ctx_fail(c, ST_ARG, "modulus must be at least 2");
  if (m < 0 || n < 0) return ctx_fail(c, ST_ARG, "negative dimension");
  if (m == 0 || n == 0) {
    *rank = 0;
    *det = 1 % p;
    return ST_OK;
  }
  const int rmax = std::min(m, n);
  const size_t l_bytes = ((size_t)m * rmax * 4 + 255) & ~(size_t)255;
  const size_t o_bytes = ((size_t)m * n * 4 + 255) & ~(size_t)255;
  void *buf = nullptr;
  int st = ctx_buffer(c, BUF_PLUQ, l_bytes + o_bytes + (size_t)n * sizeof(int) + 256, &buf);
  if (st) return st;
  uint8_t *b8 = static_cast<uint8_t *>(buf);
  EchelonKeep keep;
  keep.L = reinterpret_cast<uint32_t *>(b8);
  keep.ldL = (size_t)rmax;
  uint32_t *out = reinterpret_cast<uint32_t *>(b8 + l_bytes);
  int *d_qcol = reinterpret_cast<int *>(b8 + l_bytes + o_bytes);
  std::vector<int> piv;
  if ((st = zp_echelon_dev(c, m, n, p, D, ld, rank, det, &piv, &keep))) return st;
  const int r = (int)*rank;
  for (const auto &sw : keep.swaps)
    if (sw.first != sw.second) P->push_back(sw);
  std::vector<int> qcol(n), where(n);  // position -> column, column -> position
  for (int j = 0; j < n; ++j) qcol[j] = where[j] = j;
  for (int i = 0; i < r; ++i) {
    const int pos = where[piv[i]];
    if (pos != i) {
      std::swap(qcol[i], qcol[pos]);
      where[qcol[i]] = i;
      where[qcol[pos]] = pos;
      Q->emplace_back(i, pos);
    }
  }
  std::reverse(P->begin(), P->end());  // the reference returns them reversed (:362-363)
  std::reverse(Q->begin(), Q->end());
  cudaError_t e = cudaMemcpyAsync(d_qcol, qcol.data(), (size_t)n * sizeof(int),
                                  cudaMemcpyHostToDevice, c->stream);
  if (e != cudaSuccess) return ctx_cuda(c, e, "pluq: column order");
  const size_t total = (size_t)m * n;
  const int grid = (int)std::min<size_t>((total + 255) / 256, (size_t)c->num_sms * 16);
  pluq_assemble_kernel<<<grid, 256, 0, c->stream>>>(D, ld, keep.L, keep.ldL, d_qcol, m, n, r, out);
  ctx_launched(c);
  e = cudaMemcpy2DAsync(D, ld * 4, out, (size_t)n * 4, (size_t)n * 4, (size_t)m,
                        cudaMemcpyDeviceToDevice, c->stream);
  if (e == cudaSuccess) e = cudaGetLastError();
  // the host vector qcol must outlive the copy above
  if (e == cudaSuccess) e = cudaStreamSynchronize(c->stream);
  return e == cudaSuccess ? ST_OK : ctx_cuda(c, e, "pluq: assembly");
}

// ---------------------------------------------------------------------------
// The standard method's reduced form with its transform:
// Elimination::echelonize_reduced (A, L, P, rank, det, true) (lela/
// algorithms/elimination.tcc:143-265).  There L starts as the identity and
// takes every row operation of A, with each transposition applied to its
// rows and columns, so that at the end R = L B with B = P A_in (the
// transpositions in the order they were applied).
//
// The pivots, the transpositions and the pivot values of that loop are those
// of the non-reduced form (the rows at and below the current one are the
// same in both loops), so the panel pipeline above gives them, together
// with the non-reduced rows U (r x n) and the multipliers Lk (m x r, unit
// lower trapezoidal) with B = Lk U.  Write Lk = [L1; L2] (r and m - r rows)
// and U_P for U at the pivot columns (upper triangular, the pivots on its
// diagonal).  Pivot rows only ever receive multiples of pivot rows, and the
// other rows keep their own unit entry, so L = [[X, 0], [Y, I]]; R's pivot
// rows have the identity at the pivot columns, and its other rows are zero.
// Hence X = U_P^-1 L1^-1, Y = -L2 L1^-1, and R's first r rows are
// U_P^-1 U:
//   1. Lout <- I (m x m), T <- L1 (unit lower), W <- U_P;
//   2. Lout[0:r, 0:r] <- T^-1             (trsm, unit lower: no inversions);
//   3. Lout[r:m, 0:r] <- -L2 Lout[0:r, 0:r]           (gemm, alpha = p - 1);
//   4. Lout[0:r, 0:r] <- W^-1 Lout[0:r, 0:r]      (trsm, upper: the pivots);
//   5. D[0:r, :] <- W^-1 D[0:r, :]; D's rows from r on are zero already.
// The only inversions are of the pivots, as in the reference, so a pivot it
// cannot invert fails here too (in the panel pipeline, before any solve).
// ---------------------------------------------------------------------------

// Step 1.  T (r x r) <- the unit lower triangle of Lk's first r rows; W
// (r x r) <- D's first r rows at the pivot columns piv (row i of D is zero
// left of piv[i], so W is upper triangular); Lout (m x m) <- the identity.
__global__ void transform_setup_kernel(const uint32_t *__restrict__ Lk, size_t ldk,
                                       const uint32_t *__restrict__ D, size_t ldd,
                                       const int *__restrict__ piv, int m, int r,
                                       uint32_t *__restrict__ T, uint32_t *__restrict__ W,
                                       uint32_t *__restrict__ Lout, size_t ldl) {
  const size_t mm = (size_t)m * m, rr = (size_t)r * r;
  for (size_t idx = blockIdx.x * (size_t)blockDim.x + threadIdx.x; idx < mm + 2 * rr;
       idx += (size_t)gridDim.x * blockDim.x) {
    if (idx < mm) {
      const size_t i = idx / m, j = idx % m;
      Lout[i * ldl + j] = i == j ? 1u : 0u;
    } else if (idx < mm + rr) {
      const size_t e = idx - mm, i = e / r, j = e % r;
      T[e] = j < i ? Lk[i * ldk + j] : (i == j ? 1u : 0u);
    } else {
      const size_t e = idx - mm - rr, i = e / r, j = e % r;
      W[e] = D[i * ldd + piv[j]];
    }
  }
}

int zp_echelon_transform_dev(Ctx *c, int m, int n, uint32_t p, uint32_t *D, size_t ld,
                             uint32_t *Lout, size_t ldl, std::vector<std::pair<int, int>> *P,
                             size_t *rank, uint32_t *det) {
  P->clear();
  if (p < 2) return ctx_fail(c, ST_ARG, "modulus must be at least 2");
  if (p >= 0x80000000u)
    return ctx_fail(c, ST_ARG,
                    "modulus must be below 2^31 (Modular<uint32>'s inverse wraps above it)");
  if (m < 0 || n < 0) return ctx_fail(c, ST_ARG, "negative dimension");
  if (m > 0 && ldl < (size_t)m) return ctx_fail(c, ST_ARG, "transform leading dimension too small");
  *rank = 0;
  *det = 1 % p;
  if (m == 0) return ST_OK;
  const int rmax = std::max(1, std::min(m, n));
  const size_t k_bytes = ((size_t)m * rmax * 4 + 255) & ~(size_t)255;
  const size_t sq_bytes = ((size_t)rmax * rmax * 4 + 255) & ~(size_t)255;
  void *buf = nullptr;
  int st = ctx_buffer(c, BUF_TRANSFORM, k_bytes + 2 * sq_bytes + (size_t)rmax * sizeof(int) + 256,
                      &buf);
  if (st) return st;
  uint8_t *b8 = static_cast<uint8_t *>(buf);
  uint32_t *Lk = reinterpret_cast<uint32_t *>(b8);
  uint32_t *T = reinterpret_cast<uint32_t *>(b8 + k_bytes);
  uint32_t *W = reinterpret_cast<uint32_t *>(b8 + k_bytes + sq_bytes);
  int *d_piv = reinterpret_cast<int *>(b8 + k_bytes + 2 * sq_bytes);
  std::vector<int> piv;
  if (n > 0) {
    EchelonKeep keep;
    keep.L = Lk;
    keep.ldL = (size_t)rmax;
    if ((st = zp_echelon_dev(c, m, n, p, D, ld, rank, det, &piv, &keep))) return st;
    for (const auto &sw : keep.swaps)
      if (sw.first != sw.second) P->push_back(sw);  // in the order applied
  }
  const int r = (int)*rank;
  cudaError_t e = cudaSuccess;
  if (r > 0)
    e = cudaMemcpyAsync(d_piv, piv.data(), (size_t)r * sizeof(int), cudaMemcpyHostToDevice,
                        c->stream);
  if (e != cudaSuccess) return ctx_cuda(c, e, "transform: pivot columns");
  {
    const size_t total = (size_t)m * m + 2 * (size_t)r * r;
    const int grid = (int)std::min<size_t>((total + 255) / 256, (size_t)c->num_sms * 16);
    transform_setup_kernel<<<grid, 256, 0, c->stream>>>(Lk, (size_t)rmax, D, ld, d_piv, m, r, T,
                                                        W, Lout, ldl);
    ctx_launched(c);
    if ((e = cudaGetLastError()) != cudaSuccess) return ctx_cuda(c, e, "transform: set-up");
  }
  if (r > 0) {
    size_t bad = 0;
    if ((st = zp_trsm_dev(c, false, true, r, r, p, 1u, T, (size_t)r, Lout, ldl, &bad))) return st;
    if (m > r &&
        (st = zp_gemm_dev(c, GEMM_AUTO, m - r, r, r, p, p - 1, Lk + (size_t)r * rmax, (size_t)rmax,
                          Lout, ldl, 0u, Lout + (size_t)r * ldl, ldl, nullptr)))
      return st;
    if ((st = zp_trsm_dev(c, true, false, r, r, p, 1u, W, (size_t)r, Lout, ldl, &bad))) return st;
    if ((st = zp_trsm_dev(c, true, false, r, n, p, 1u, W, (size_t)r, D, ld, &bad))) return st;
  }
  // the host vector piv must outlive the copy above
  e = cudaStreamSynchronize(c->stream);
  return e == cudaSuccess ? ST_OK : ctx_cuda(c, e, "transform");
}

}  // namespace lela

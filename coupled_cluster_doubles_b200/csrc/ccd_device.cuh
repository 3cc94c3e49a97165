// Device-side data structures and small helpers shared by the CCD kernels.
#pragma once

#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstdint>

namespace ccd {

// Packed amplitudes.  The amplitudes are antisymmetric, t_ab,ij = -t_ab,ji = -t_ba,ij = t_ba,ji,
// and so are V and D, so the solver iterates on one element in four: the quads (u, w) of a
// channel, u = strict particle pair a < b (pk of them), w = strict hole pair i < j (hk), row-major
// [u][w] with row stride hs.  T, V_hhpp and D use this layout (channel block at q_off, rows
// padded to a multiple of kBK with zeros).
//
// pp ladder.  D[ab,ij] = sum_{c<d} V[ab,cd] T[cd,ij] over the quads: V is the pk x pk packed
// matrix (1/4 of V_pppp), T the packed amplitudes themselves (16 consecutive rows are one
// contiguous B stage).  V is symmetric (<ab|v|cd> = <cd|v|ab>), so a channel with at most kSymHK
// strict hole pairs stores and streams only the blocks on and above the diagonal (blocks of
// kMaxBM rows and columns): each block above it serves its rows and, transposed, its columns.
// A stages are stored in HBM in their shared-memory image so that one bulk copy (TMA) moves each:
// [kBK][as] k-major, as = rows rounded up to 8, plus 4.  hs is 4 mod 8 beyond 4 hole pairs: with
// strides of 4 mod 8 doubles the 4 k-rows of an m16n8k16 fragment load fall on distinct banks.
// The last row tile of a channel is stored compact (only its real rows, rounded up to 8).
constexpr int kSMs = 148;      // SMs of a B200
constexpr int kBK = 16;        // K depth of one chunk
constexpr int kStages = 3;     // bulk-copy pipeline depth, stages of two chunks (one if hs > 20)
constexpr int kMaxHH = 72;     // hole pairs of a channel (ordered)
constexpr int kLadderConsumers = 256;                  // 8 warps of 16 rows
constexpr int kLadderThreads = kLadderConsumers + 32;  // + 1 producer warp
constexpr int kMaxBM = 128;    // rows per tile
constexpr int kBlkChunks = kMaxBM / kBK;  // K chunks of a block of columns
constexpr int kMaxNB = 36;     // largest row stride hs of the packed amplitudes
constexpr int kSymHK = 20;     // hole pairs up to which V's symmetry is used ...
constexpr int kSymHS = 20;     // ... and their largest hs
constexpr int kMaxAS = kMaxBM + 4;  // A stage row stride bound (doubles)

// Row stride of the packed layout for hk strict hole pairs.
__host__ __device__ inline int quad_hs(int hk) {
  return hk <= 2 ? hk : hk <= 4 ? 4 : 8 * ((hk + 3) / 8) + 4;
}
// Chunks of a pipeline stage.
__host__ __device__ inline int ladder_stage(int hs) { return hs <= 20 ? 2 : 1; }
constexpr int kStageA = 2 * kBK * (kMaxBM + 4), kStageB = 2 * kBK * 20;  // doubles; 2 * 20 >= 36
// Column classes: 0 thin, 1 mid (hs 12, 20), 2 wide (hs 28, 36).
__host__ __device__ inline int ladder_class(int hs) { return hs <= 4 ? 0 : hs <= 20 ? 1 : 2; }
// Doubles per k row of an A chunk for a tile of `rows` rows.
__host__ __device__ inline int ladder_as(int rows) { return ((rows + 7) & ~7) + 4; }
// First K chunk stored of row tile mt, and where K chunk kc of row tile mt (`rows` rows) starts in
// the channel's A image of nkc chunks a row.
__host__ __device__ inline int ladder_kc0(bool sym, int mt) { return sym ? kBlkChunks * mt : 0; }
__host__ __device__ inline int64_t ladder_chunk(bool sym, int nkc, int mt, int kc, int rows) {
  const int64_t before = (int64_t)mt * nkc - (sym ? kBlkChunks / 2 * mt * (mt - 1) : 0);
  return (before * kMaxAS + (int64_t)(kc - ladder_kc0(sym, mt)) * ladder_as(rows)) * kBK;
}

// Mixed-precision pp-ladder images (tensor-core operands, ccd_tc.cuh).  A K chunk of a
// 128-row tile holds kTcKC bf16 per row in 8 x 8 core matrices, K-major, no swizzle:
//   element (r, k) -> (r / 8) * kTcGroup + (k / 8) * 64 + (r % 8) * 8 + k % 8.
constexpr int kTcKC = 32;                    // K depth of one chunk (bf16 elements)
constexpr int kTcBM = 128;                   // rows per tile = UMMA M
constexpr int kTcMaxNB = 48;                 // padded columns = UMMA N (multiple of 16)
constexpr int kTcThreads = 192;
constexpr int kTcAPlane = kTcBM * kTcKC;     // bf16 elements of one A term per stage (8 KB)
constexpr int kTcBPlane = kTcMaxNB * kTcKC;  // one B term per stage (3 KB)
constexpr int kTcGroup = 8 * kTcKC;          // bf16 elements of one 8-row group of a chunk

// Padded UMMA N for hk columns.
__host__ __device__ inline int tc_nb(int hk) { return 16 * ((hk + 15) / 16); }
// Offset of element (r, k) inside a chunk image (bf16 units), 0 <= k < kTcKC: K-major core
// matrices (8 rows of 8 consecutive k), used for the A operand (V).
__host__ __device__ inline int tc_off(int r, int k) {
  return (r >> 3) * kTcGroup + (k >> 3) * 64 + (r & 7) * 8 + (k & 7);
}
// The B operand (T, N = hk columns) in MN-major core matrices (8 k-rows of 8 consecutive n):
// neighbouring columns are neighbouring bytes, as the assembly writes them.  Same
// 8 x 8 block positions as tc_off, so the shared-memory descriptors are the same.
__host__ __device__ inline int tc_off_mn(int n, int k) {
  return (n >> 3) * kTcGroup + (k >> 3) * 64 + (k & 7) * 8 + (n & 7);
}
// FP64 tensor-core MMA (mma.sync m8n8k4, the full-rate FP64 path of sm_100a): lane
// (g = lane / 4, t = lane % 4) supplies A[g][t] and B[t][g] and accumulates C[g][2t] and
// C[g][2t + 1].  One instruction does 256 multiply-adds, so the small channel GEMMs are no longer
// bound by instruction issue and shared-memory loads.
__device__ __forceinline__ void dmma_884(double (&c)[2], double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
      : "+d"(c[0]), "+d"(c[1])
      : "d"(a), "d"(b));
}

// C (16 x 8) += A (16 x 16) B (16 x 8) in FP64, lane layout (g = lane / 4, t = lane % 4):
// a[i] = A[g + 8 (i % 2)][t + 4 (i / 2)], b[i] = B[t + 4 i][g],
// c = {C[g][2t], C[g][2t + 1], C[g + 8][2t], C[g + 8][2t + 1]}.
__device__ __forceinline__ void dmma_16816(double (&c)[4], const double (&a)[8],
                                           const double (&b)[4]) {
  asm("mma.sync.aligned.m16n8k16.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, "
      "{%4,%5,%6,%7,%8,%9,%10,%11}, {%12,%13,%14,%15}, {%0,%1,%2,%3};"
      : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
      : "d"(a[0]), "d"(a[1]), "d"(a[2]), "d"(a[3]), "d"(a[4]), "d"(a[5]), "d"(a[6]), "d"(a[7]),
        "d"(b[0]), "d"(b[1]), "d"(b[2]), "d"(b[3]));
}

// x -> nt bf16 terms, each the round-to-nearest of what the previous ones leave (the
// remainders are exact in double).
// bf16 bits of a double h that has at most 8 significant bits: sign, exponent rebased from
// 1023 to 127, top 7 mantissa bits.  Zero and magnitudes below bf16's normal range (2^-126)
// give a signed zero; NaN stays NaN.
__device__ __forceinline__ __nv_bfloat16 bf16_of_short(double h) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(h);
  const unsigned short sign = (unsigned short)((b >> 48) & 0x8000u);
  const int e = (int)((b >> 52) & 0x7FF) - 1023 + 127;
  unsigned short bits;
  if (e <= 0) bits = sign;
  else if (e >= 255) bits = (unsigned short)(sign | 0x7F80u | ((b << 12) ? 0x40u : 0u));
  else bits = (unsigned short)(sign | (e << 7) | (unsigned)((b >> 45) & 0x7F));
  return __ushort_as_bfloat16(bits);
}

// x = t_0 + t_1 (+ t_2) + remainder, each t_p a bf16 (nt terms): t_p is the remainder rounded
// to 8 significant bits by Dekker's splitting (Dekker 1971: c = r (2^45 + 1), t = c - (c - r)),
// which is exact in bf16, and the next remainder r - t_p is exact in FP64.  Only FP64 and
// integer arithmetic, no conversion instructions.
__device__ __forceinline__ double split_bf16_step(double &x) {
  // Explicitly rounded operations: an FMA contraction of c - x would skip the rounding of c
  // that the splitting relies on.
  const double c = __dmul_rn(x, 35184372088833.0);  // 2^45 + 1
  double hi = __dsub_rn(c, __dsub_rn(c, x));
  if (fabs(hi) < 1.1754943508222875e-38) hi = 0.0;  // below bf16's normal range
  x = __dsub_rn(x, hi);
  return hi;
}
__device__ __forceinline__ void split_bf16(double x, __nv_bfloat16 *out, int nt) {
  for (int p = 0; p < nt; ++p) out[p] = bf16_of_short(split_bf16_step(x));
}
// The same with the term count known at compile time (the terms stay in registers).
template <int NT>
__device__ __forceinline__ void split_bf16_n(double x, __nv_bfloat16 (&out)[NT]) {
#pragma unroll
  for (int p = 0; p < NT; ++p) out[p] = bf16_of_short(split_bf16_step(x));
}

// One pp-ladder work tile: packed rows [128 mt, 128 mt + rows) of channel `ch`, K chunks
// [kc0, kc0 + nks).  Partial sums of D go to planes of one row tile each ([128][hs] doubles): the
// planes of row tile J lie together (LadderRows), in a symmetric channel first those of the
// transposed blocks of row tiles 0 .. J - 1, then one per K segment of its own.
struct LadderTile {
  int32_t ch, mt, kc0, nks;
  int32_t rows, hk, hs, nb;  // nb: UMMA N (tensor-core tiles)
  int32_t sym, nseg;         // nseg: K segments the channel's row tiles have room for
  int32_t pk, nkx;  // nkx: chunks of T X after the tile's own (tensor-core tiles)
  int64_t tmt_base, xt_base;
  int64_t a_base;   // first A chunk: + c * ladder_as(rows) * kBK (tensor core: see there)
  int64_t b_base;   // first B chunk: + c * kBK * hs
  int64_t ti_base;  // T of the tile's own rows (symmetric channels)
  int64_t out;      // D plane of the tile: + u_local * hs
  int64_t planes;   // planes of the channel
};
// First plane of row tile mt of a channel.
__host__ __device__ inline int ladder_plane(bool sym, int nseg, int mt) {
  return mt * nseg + (sym ? mt * (mt - 1) / 2 : 0);
}

// Where the ladder leaves D of a row tile: n planes of 128 * hs doubles from `base`; D is their sum
// in plane order.
struct LadderRows {
  int64_t base;
  int32_t n, stride;
};

// Per active regular channel.  A channel without quads (pk or hk zero) has no ladder tile, hh
// unit or assembly item: its amplitudes are zero.
struct ChanInfo {
  int32_t pp, hh, pk, hk;
  int32_t hs, nkc, nmt, nhht;  // packed row stride, K chunks, row tiles, hh-ladder slices
  // T X in the tensor-core ladder (small systems): its 32-deep K chunks (all hh columns), and where
  // its operands T (A, rows u) and X / 2 (B) are in the T image.
  int32_t nkx, pad_x;
  int64_t tmt_base, xt_base;
  int32_t sym, rt_off;  // V stored by its symmetry; first row tile among all channels'
  int64_t t_off;     // pphh block offset (reference t2 layout)
  int64_t pp_off;    // offset into pp_pairs / pp_swap / prow
  int64_t hh_off;    // offset into hh_pairs / hh_swap / hcol
  int64_t vhh_off;   // hh x hh block offset (V_hhhh)
  int64_t q_off;     // packed block: 16 nkc x hs doubles (T, V_hhpp)
  int64_t x_off;     // X: hk x hs
  int64_t part_off;  // partials of the hh ladder
  int32_t hh_first, tx_first;  // first of the channel's HHOut and TXTile records
  int32_t hht_first, hht_last;  // first of its full HHTile slices; the shorter one after them
  int64_t vkt_base;  // A tiles of V
  int64_t pk_off;    // strict particle pairs: offset into kcol / quad rows / r (pk entries)
  int64_t qcol_off;  // strict hole pairs: offset into quad columns / s (hk entries)
  // Mixed-precision operand images (bf16 terms, tensor-core layout; see ccd_tc.cuh):
  // nbt = UMMA N, nkct = 32-deep K chunks of V T.
  int32_t nbt, nkct;
  int64_t vtc_base, tkt_tc_base;
};

// hh-ladder unit: `rows` packed rows of a channel from row r0 of all channels', V and T at `base`,
// the partial of P at `part`.
struct __align__(16) HHTile {
  int32_t hk, hs, rows, r0;
  int64_t base, part;
};
// One element of X = V_hhhh + P: P's partials part[k * stride], k < nslices, where X goes (and the
// packed V_hhhh comes from) and, on the diagonal, s (s < 0: off the diagonal).
struct __align__(16) HHOut {
  int64_t part;
  int32_t nslices, stride, x, s;
  int32_t xt[2];  // X / 2 in the T image, rows kl and (negated) lk; -1: not there
};

// A warp's part of T X: `rows` rows, T and T X at `at`, X at `x`; from column j0 (hk > 8: 16 of them).
struct __align__(16) TXTile {
  int32_t hk, hs, rows, j0;
  int64_t at, x;
};

// Fused assembly, static data of strict packed row u (a < b) of a channel (index pk_off + u):
// particle indices a - np, b - np, e_a, e_b, and the offsets of rows ab and ba inside the
// channel block (ab * hh, ba * hh) ...
struct QuadRow {
  int32_t o_ab, o_ba;
  int32_t pa, pb;
  double ea, eb;
};
// ... and of strict hole pair w (i < j, index qcol_off + w): the columns ij and ji, the hole
// indices i, j and e_i + e_j.
struct QuadCol {
  int32_t c_ij, c_ji, i, j;
  double eij;
};
// Work item of the fused assembly: quads [q0, q1) (q = u * hk + w) of active channel ch, with
// what its threads need of the channel (so their table reads depend on the item alone).
struct QuadItem {
  int32_t ch, q0, q1, hk;
  int32_t hs, rt_off;
  int64_t q_off, pk_off, qcol_off;
};

// Per active modified channel (table path).
struct ModInfo {
  int32_t ph, hp;
  int64_t m_off;     // ph' x hp' block offset in the phhp slab (V_hpph uses the same size)
  int64_t y_off;     // hp' x hp' block offset (V_hphp)
};

// Fused-path ring: a modified channel and its transpose (the channel of the exchanged pairs),
// worked on in the layout of the first.  Set-up data of its operand images.
struct RingPair {
  int32_t ph, hp;
  int32_t ph_off, hp_off;  // the channel's ph' and hp' pairs
  int32_t other, self;     // channel slot of the transpose; self: it is the channel itself
  int64_t m_off;   // phhp block of the channel (V_hpph, quads of its elements)
  int64_t a_off;   // A: V_hphp of the channel (hp' x hp')
  int64_t b_src;   // V_hphp of the transpose (ph' x ph' in its order), the source of B
  int64_t c_src;   // V_hpph of the transpose, averaged with the channel's; -1: the same by the model
  int64_t tp, a_img, b_img, c_img, to_img;  // T' image; operands and destinations
  int32_t g, pad;  // warps of its units
};
// A pair and column tiles [n0, n0 + nt) of its S, with what its warps need of the pair.
struct RingUnit {
  int32_t ph, hp, n0, nt;
  int64_t tp, a_img, b_img, c_img, to_img;
};

// Contiguous element range [e0, e1) of one channel for the element-wise kernels.
struct ElemRange {
  int32_t ch;
  int32_t pad;
  int64_t e0, e1;
};

// Kernel ids of the start-time trace (Control::trace_*).  The FP64 ladder records every class
// under kTrLadderThin; LadderMid, LadderWide, Retile and Reduce are unused.
enum TraceKernel {
  kTrRingSmall = 0, kTrRingMid, kTrRingLarge, kTrHHSmall, kTrHHTiled, kTrOneBody, kTrLadderThin,
  kTrLadderMid, kTrLadderWide, kTrLadderTC, kTrAssemble, kTrLoopCtl, kTrEnergy, kTrRetile,
  kTrReduce, kTrHHReduce, kTrGather, kTraceKernels
};

// Device control block: iteration state of the solve loop lives on the device so that a
// captured iteration can be replayed without host round trips.
struct Control {
  double e_prev;         // corrEnergyPrev (starts at 100, main.cpp:494)
  double e_corr;         // corrCCD of the last iteration
  double e_diff;         // energyDiff
  double tol;
  double mixing;
  int64_t iterations;    // iterations performed
  int64_t max_iters;
  int32_t done;          // set when |dE| <= tol or the cap is reached; kernels then no-op
  int32_t parity;        // which t2 buffer holds the current amplitudes
  int32_t error;         // bit flags, see kErr*
  int32_t active;        // 1 while a solve is running (0: kernels run unconditionally)
  int32_t phase;         // mixed-precision solve: 1 = split-bf16 ladder, 2 = FP64 polish
  int32_t inject;        // test-only fault: 1 = the first FP64 pp-ladder CTA withholds its
                         // first stage (its bounded waits run out)
  double polish_rel;     // phase 1 -> 2 once |dE| <= max(tol, polish_rel * |E|)
  int64_t polish_iters;  // iterations run in phase 2
  int64_t stop_at;       // device solve loop: one graph launch runs while iterations < stop_at
  int64_t trace_iter;    // kernel trace: the iteration whose kernels record start times
  uint64_t trace_first[kTraceKernels];  // %globaltimer of the first / last CTA start
  uint64_t trace_last[kTraceKernels];
  uint64_t trace_end[kTraceKernels];    // %globaltimer when the last CTA finished
  double energies[128];  // corrCCD per iteration (first 128)
  int32_t err;           // kErrTimeout, kErrBadIndex, ... raised by kernels (never uploaded)
};

constexpr int32_t kErrNonFinite = 1;
constexpr int32_t kErrTimeout = 2;
constexpr int32_t kErrBadIndex = 4;
constexpr int32_t kErrAsym = 16;     // set-up: a channel's stored V is not symmetric
constexpr int32_t kErrRingLists = 32;  // ai_jb's rows and columns are not the ph' and hp' lists'
constexpr int32_t kErrRingMaps = 8;  // aj_ib / bi_ja / bj_ia are not ai_jb under the swaps

}  // namespace ccd

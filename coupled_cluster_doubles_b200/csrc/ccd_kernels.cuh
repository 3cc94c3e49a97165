// CCD iteration kernels for sm_100a (FP64 path).
//
// Reference correspondence (calc.cpp / Chain.hpp of justinlietz/coupled_cluster_doubles):
//   pp_ladder_kernel        V_pppp T part of D = 0.5 T X + 0.5 V T   calc.cpp:162-202
//                           (antisymmetry-packed; the assembly adds T X)
//   hh_slice, hh_reduce     X = V_hhhh + 0.5 V_hhpp T                calc.cpp:141-160
//   ring_small, ring16      Y = V_hphp + 0.5 V_hpph T'; R = T' Y     calc.cpp:264-313
//   ring_pair_kernel        the same for the fused path, T' from tp_gather_kernel
//   onebody_tables_kernel   calcChannelT2Diff_h2pp_h1 / _p2_p1hh     calc.cpp:9-25, 73-89
//   hh_post_kernel          the same dot products, read from the ladder intermediates, and T X
//   gather8_kernel          Chain::mapFromDistributed x 8            Chain.hpp:710-755
//   assemble_*_kernel       calcChannelT2_pphh                       calc.cpp:368-421
//   map_to_kernel           Chain::set + mapToDistributed x 5        Chain.hpp:503-527,757-802
//   energy_kernel           reduction(+:corr) + MPI_Allreduce + stop rule, main.cpp:511-519,668-670
#pragma once

#include <cstdint>

#include <cuda_bf16.h>

#include "ccd_device.cuh"

namespace ccd {

constexpr uint64_t kWaitLimitNs = 1000000000ull;  // bounded mbarrier waits: 1 s of globaltimer

__device__ __forceinline__ uint32_t smem_u32(const void *p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ uint64_t global_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
// Bounded wait on an mbarrier phase: try_wait suspends the thread in hardware until the phase
// completes or a short internal time limit passes; give up (false) after kWaitLimitNs.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity) {
  if (mbar_try_wait(bar, parity)) return true;
  const uint64_t t0 = global_ns();
  for (;;) {
#pragma unroll 1
    for (int i = 0; i < 256; ++i)
      if (mbar_try_wait(bar, parity)) return true;
    if (global_ns() - t0 > kWaitLimitNs) return false;
  }
}
// 1-D bulk copy global -> shared, completion counted on an mbarrier (TMA unit, no multicast).
__device__ __forceinline__ void bulk_g2s(uint32_t dst, const void *src, uint32_t bytes,
                                         uint32_t bar) {
  asm volatile(
      "cp.async.bulk.shared::cta.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
          dst),
      "l"(src), "r"(bytes), "r"(bar)
      : "memory");
}
// The same for data that an iteration reads once, and from HBM anyway if it is large (V): first to
// be evicted, so that it does not push out what other kernels read again.  In the FP64 iteration
// of EG N=54 |n|^2 <= 20 (V 50 MB) 55.0 -> 46.7 us, |n|^2 <= 36 (351 MB) 151.8 -> 148.6, PNM N=66
// 209.7 -> 206.4, and no change where everything fits (EG N=14).
__device__ __forceinline__ uint64_t l2_evict_first() {
  uint64_t p;
  asm("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
  return p;
}
__device__ __forceinline__ void bulk_g2s(uint32_t dst, const void *src, uint32_t bytes,
                                         uint32_t bar, uint64_t policy) {
  asm volatile(
      "cp.async.bulk.shared::cta.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1], "
      "%2, [%3], %4;" ::"r"(dst),
      "l"(src), "r"(bytes), "r"(bar), "l"(policy)
      : "memory");
}
// Programmatic dependent launch: wait until the preceding kernel of the stream has completed
// (its writes are visible), then allow the next kernel to begin launching once every CTA of
// this grid is resident.  Both are no-ops for kernels launched without the PDL attribute.
__device__ __forceinline__ void pdl_enter() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// gate 0: kernel of an FP64 iteration, gate 1: kernel of a mixed-precision iteration.  During
// a solve, an iteration whose precision does not match the phase is a no-op (a replayed batch
// can straddle the switch to the FP64 polish).
// The kernel id `tr` records its first and last CTA start in the trace of the armed iteration.
__device__ __forceinline__ void trace_start(const Control *ctl, int tr) {
  if (threadIdx.x == 0 && ctl->trace_iter == ctl->iterations) {
    Control *c = const_cast<Control *>(ctl);
    const unsigned long long t = global_ns();
    atomicMin(reinterpret_cast<unsigned long long *>(&c->trace_first[tr]), t);
    atomicMax(reinterpret_cast<unsigned long long *>(&c->trace_last[tr]), t);
  }
}
// Records, for the traced iteration, when a CTA of kernel `tr` finished (thread 0, after the
// CTA's work; the trace keeps the latest).
__device__ __forceinline__ void trace_end(const Control *ctl, int tr) {
  if (threadIdx.x == 0 && ctl->trace_iter == ctl->iterations) {
    Control *c = const_cast<Control *>(ctl);
    atomicMax(reinterpret_cast<unsigned long long *>(&c->trace_end[tr]),
              (unsigned long long)global_ns());
  }
}
__device__ __forceinline__ bool skip_iteration(const Control *ctl, int gate, int tr) {
  pdl_enter();
  trace_start(ctl, tr);
  // One round trip (the fields share a line), whatever the outcome.
  const int active = ctl->active, done = ctl->done, phase = ctl->phase;
  return active && (done || ((gate == 1) != (phase == 1)));
}

// ------------------------------------------------------------------------------------------
// pp ladder on the FP64 MMA over the packed quads:
//   D[u, w] = sum_c V[u, c] T[c, w]        (u = a<b, c = c<d, w = i<j)
// It needs only the amplitudes (T X is added later), so it starts at the head of an iteration
// beside the hh ladder and the ring.  Channels of up to kSymHK strict hole pairs stream the blocks
// of V on and above the diagonal alone: a block of rows I and columns J > I gives D_I += V_IJ T_J
// and D_J += V_IJ^T T_I.  EG N=54 |n|^2 <= 36: 559 MB of V become 351 (and 32 MB of D planes), in
// the iteration the ladder's 145 us become 111; PNM N=66: 716 MB to 457, 190 us to 142.  V in full
// is bound by HBM; halved, as much by each warp's chain of shared-memory loads, MMAs and barriers
// (the whole ladder alone: DRAM 53 %, FP64 MMA 51 % busy; thin class 54 and 41, mid 30 and 57).  Wider
// channels would need twice the FP64 MMA they already wait for, and more than 80 registers: FP64
// iterations with the half of V used up to 4, 12, 20 and 36 strict hole pairs, EG N=54
// |n|^2 <= 36 151.0, 150.1, 148.2, 155.9 us, N=38 105.5, 102.9, 103.5, 107.8, PNM N=66 206.6, 204.6,
// 205.3, 214.5.
// One CTA per SM, 80 registers, three 39 KB stages of two chunks: it leaves registers and shared
// memory for the other streams' kernels (at 94 registers its nine warps kept the ring's CTAs
// out; with a fourth stage the ladder alone is 5 % faster but the iteration slower, 64 for 56 us at
// EG N=54 |n|^2 <= 20).  Stages of one chunk, five deep: 51 and 66 us for the thin and the mid
// class alone at EG N=54 |n|^2 <= 36, 46 and 62 now.
// One producer warp: a lane claims tiles from a launch-wide counter (list sorted by class, wide
// first, then by decreasing work: longest-first list scheduling that adapts to CTAs starting
// late behind another stream's kernels) and streams pre-tiled A/B stages with bulk copies (TMA,
// no multicast) into a kStages-deep shared-memory ring guarded by mbarriers, across tile
// boundaries; beside a tile's first stage it leaves the tile's description for the consumers.
// T_I has a buffer of its own, filled once the previous tile's readers are done and needed only
// after the diagonal block's chunks.
// The 8 consumer warps: warp w owns rows [16w, 16w + 16) of the direct product; of the transposed
// product of chunk kc (16 columns, all 128 rows) warp kc % 8 does the whole, so nothing is reduced
// across warps.  (All warps sharing each chunk's transposed product, with a sum of eight parts
// through shared memory, was no faster for one column tile and slower for two.)
// ------------------------------------------------------------------------------------------

// What the consumers need of the tile a stage belongs to.
struct StageInfo {
  int64_t out, planes;
  int32_t rows, hk, hs, nks;  // nks: K chunks of the tile; 0: no more tiles
  int32_t kc0, mt, nseg, pk;  // nseg < 0: no transposed product
};

// The consumer side of one tile: its stages from the ring, then its D rows.  at: the next stage.
// FULL: a tile of 128 rows, whose A stride is a constant; only those have a transposed product.  A
// fragments (k-major, row stride ar) and B fragments (row stride hs) come from the stage
// conflict-free.  A warp whose lower 8-row half has no rows feeds zeros there instead of reading
// past the tile; columns past hk (the stage's next row, or stale) are not stored.  ti_bar,
// ti_parity: T_I's barrier.  False: a wait ran out (rows stay unwritten).
struct RingPos {  // a stage and the parity of its barriers
  int s = 0;
  uint32_t phase = 0;
  __device__ __forceinline__ void next() {
    if (++s == kStages) {
      s = 0;
      phase ^= 1;
    }
  }
};
template <int C, bool FULL>
__device__ __forceinline__ bool consume_mma(const StageInfo &ti, const double *As,
                                            const double *Bs, const double *Ti, uint64_t *bars,
                                            uint32_t ti_bar, uint32_t ti_parity, int tid,
                                            RingPos &at, double *__restrict__ d) {
  static_assert(kBK == 16, "one m16n8k16 K step per chunk");
  constexpr int kPer = C <= 3 ? 2 : 1;  // chunks of a stage
  const int warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int rows = FULL ? kMaxBM : ti.rows;
  const int ar = ladder_as(rows), hs = ti.hs;
  const int halves = FULL ? 2 : min(2, max(0, ((rows + 7) >> 3) - 2 * warp));  // 8-row halves
  // First chunk with a transposed product.
  const int off = FULL && ti.nseg >= 0 ? kBlkChunks * (ti.mt + 1) - ti.kc0 : ti.nks;
  bool have_ti = false;
  double acc[C][4];
#pragma unroll
  for (int j = 0; j < C; ++j) acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0.0;
  for (int c = 0; c < ti.nks; c += kPer) {
    const int s = at.s;
    if (!mbar_wait(smem_u32(&bars[s]), at.phase)) return false;
    at.next();
    const double *Ac = As + s * kStageA;
    const double *A0 = Ac + t * ar + 16 * warp + g, *B0 = Bs + s * kStageB + t * hs + g;
    auto direct = [&](const double *A, const double *B) {
      double a[8];
#pragma unroll
      for (int i = 0; i < 8; ++i)
        a[i] = (FULL || i % 2 == 0 || halves > 1) ? A[4 * (i / 2) * ar + 8 * (i % 2)] : 0.0;
#pragma unroll
      for (int j = 0; j < C; ++j) {
        double b[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) b[q] = B[4 * q * hs + 8 * j];
        dmma_16816(acc[j], a, b);
      }
    };
    if (FULL || halves > 0) {
      if (kPer == 2 && c + 1 < ti.nks) {
        direct(A0, B0);
        direct(A0 + kBK * ar, B0 + kBK * hs);
      } else {
        direct(A0, B0);
      }
    }
    if constexpr (FULL && C <= (kSymHK + 7) / 8) {
      const int u = (warp - ti.kc0 - c) & (kBlkChunks - 1);  // this warp's chunk of the stage
      if (c >= off && u < kPer && c + u < ti.nks) {
        if (!have_ti && !mbar_wait(ti_bar, ti_parity)) return false;
        have_ti = true;
        // D_J[16 columns of the chunk] = sum over the 128 rows, two column tiles at a time (a
        // lone one as two sums, of even and odd K steps: half the chain).
        const int kc = ti.kc0 + c + u, J = kc / kBlkChunks;
        const double *A = Ac + u * kBK * ar + g * ar + t;
        double *o = d + ti.planes +
                    (int64_t)(ladder_plane(true, ti.nseg, J) + ti.mt) * kMaxBM * hs +
                    (kc % kBlkChunks) * kBK * hs;
#pragma unroll
        for (int j0 = 0; j0 < C; j0 += 2) {
          constexpr int kHalf = C == 1 ? 2 : 1;
          double e[2][4] = {};
          const double *B = Ti + t * hs + g + 8 * j0;
#pragma unroll 2
          for (int k0 = 0; k0 < kMaxBM; k0 += 16 * kHalf) {
#pragma unroll
            for (int kk = 0; kk < kHalf; ++kk) {
              double a[8];
#pragma unroll
              for (int i = 0; i < 8; ++i)
                a[i] = A[8 * (i % 2) * ar + k0 + 16 * kk + 4 * (i / 2)];
#pragma unroll
              for (int j = 0; j < min(2, C - j0); ++j) {
                double b[4];
#pragma unroll
                for (int q = 0; q < 4; ++q) b[q] = B[(k0 + 16 * kk + 4 * q) * hs + 8 * j];
                dmma_16816(e[j + kk], a, b);
              }
            }
          }
#pragma unroll
          for (int j = 0; j < min(2, C - j0); ++j)
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              const int r = g + 8 * (q >> 1), col = 8 * (j0 + j) + 2 * t + (q & 1);
              if (kc * kBK + r < ti.pk && col < ti.hk)
                o[r * hs + col] = C == 1 ? e[0][q] + e[1][q] : e[j][q];
            }
        }
      }
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(smem_u32(&bars[kStages + s]));
  }
#pragma unroll
  for (int j = 0; j < C; ++j)
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int r = 16 * warp + g + 8 * (q >> 1), col = 8 * j + 2 * t + (q & 1);
      if (r < rows && col < ti.hk) d[ti.out + (int64_t)r * hs + col] = acc[j][q];
    }
  return true;
}

// Slack: fragment loads past hs in the last B stage and the last row of T_I.
constexpr size_t kLadderSmem =
    ((size_t)kStages * (kStageA + kStageB) + kMaxBM * kSymHS + 2 * kBK) * 8 +
    kStages * sizeof(StageInfo) + (2 * kStages + 2) * 8;
__global__ void __maxnreg__(80)
pp_ladder_kernel(const LadderTile *__restrict__ tiles, int n_tiles, int32_t *sched,
                 const double *__restrict__ v_t, const double *tq0, const double *tq1,
                 double *__restrict__ d, const Control *ctl, int32_t *err, int gate) {
  if (skip_iteration(ctl, gate, kTrLadderThin)) return;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  double *As = reinterpret_cast<double *>(smem_raw);
  double *Bs = As + kStages * kStageA;
  double *Ti = Bs + kStages * kStageB + kBK;
  StageInfo *info = reinterpret_cast<StageInfo *>(Ti + kMaxBM * kSymHS + kBK);
  uint64_t *bars = reinterpret_cast<uint64_t *>(info + kStages);  // full, then empty
  uint64_t *ti_full = bars + 2 * kStages, *ti_free = ti_full + 1;
  constexpr int kConsumerWarps = kLadderConsumers / 32;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(smem_u32(&bars[s]), 1);
      mbar_init(smem_u32(&bars[kStages + s]), kConsumerWarps);
    }
    mbar_init(smem_u32(ti_full), 1);
    mbar_init(smem_u32(ti_free), kConsumerWarps);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();

  if (warp == kConsumerWarps) {
    if (lane == 0) {
      const double *t_q = ctl->parity ? tq1 : tq0;
      const uint64_t v_policy = l2_evict_first();
      int gc = 0;   // stages issued by this CTA
      int nti = 0;  // tiles with a T_I so far
      bool stop = false;
      // Test-only fault (ccdgpu_inject_wait_timeout): CTA 0 never fills its first stage, so
      // its consumers' bounded waits run out, then this producer's wait for that stage does.
      const bool withhold = ctl->inject != 0 && blockIdx.x == 0;
      auto free_stage = [&]() {  // stage gc may be filled
        if (gc < kStages ||
            mbar_wait(smem_u32(&bars[kStages + gc % kStages]), ((gc / kStages) - 1) & 1))
          return true;
        atomicOr(err, kErrTimeout);
        return false;
      };
      int ti = blockIdx.x;  // the first tile needs no claim (grid <= n_tiles)
      while (ti < n_tiles && !stop) {
        const LadderTile tile = tiles[ti];
        // The next claim's latency hides behind this tile.
        ti = (int)gridDim.x + atomicAdd(&sched[0], 1);
        const uint32_t abytes = ladder_as(tile.rows) * kBK * 8;  // a chunk's
        const uint32_t bbytes = kBK * tile.hs * 8;
        const int per = ladder_stage(tile.hs);
        const double *asrc = v_t + tile.a_base, *bsrc = t_q + tile.b_base;
        // Chunks from diag_end on have a transposed product, which reads T_I.
        const int diag_end = kBlkChunks * (tile.mt + 1) - tile.kc0;
        bool need_ti = tile.sym && diag_end < tile.nks;
        const bool has_ti = need_ti;
        for (int c = 0; c < tile.nks; c += per, ++gc) {
          const int s = gc % kStages;
          if (need_ti) {
            // Once the previous tile's readers of the buffer are done; waited for only when the
            // next chunk needs it.
            bool ok = nti == 0 || mbar_try_wait(smem_u32(ti_free), (nti - 1) & 1);
            if (!ok && c + per > diag_end) ok = mbar_wait(smem_u32(ti_free), (nti - 1) & 1);
            if (ok) {
              const uint32_t bytes = kMaxBM * tile.hs * 8;
              mbar_expect_tx(smem_u32(ti_full), bytes);
              bulk_g2s(smem_u32(Ti), t_q + tile.ti_base, bytes, smem_u32(ti_full));
              need_ti = false;
            } else if (c + per > diag_end) {
              atomicOr(err, kErrTimeout);
              stop = true;
              break;
            }
          }
          if (!free_stage()) {
            stop = true;
            break;
          }
          if (withhold && gc == 0) continue;
          if (c == 0)
            info[s] = StageInfo{tile.out,  tile.planes, tile.rows, tile.hk, tile.hs, tile.nks,
                                tile.kc0, tile.mt, has_ti ? tile.nseg : -1, tile.pk};
          const uint32_t full = smem_u32(&bars[s]);
          const int n = min(per, tile.nks - c);
          mbar_expect_tx(full, n * (abytes + bbytes));
          bulk_g2s(smem_u32(As + s * kStageA), asrc + c * (abytes / 8), n * abytes, full,
                   v_policy);
          bulk_g2s(smem_u32(Bs + s * kStageB), bsrc + c * (bbytes / 8), n * bbytes, full);
        }
        nti += has_ti;
      }
      if (!stop && free_stage()) {  // the end marker
        info[gc % kStages].nks = 0;
        mbar_arrive(smem_u32(&bars[gc % kStages]));
      }
      // The last producer to finish (each has made its last claim) resets the counters for
      // the next launch.
      __threadfence();
      if (atomicAdd(&sched[1], 1) == (int)gridDim.x - 1) {
        sched[0] = 0;
        sched[1] = 0;
        __threadfence();
      }
    }
    return;
  }
  const int tid = threadIdx.x;
  RingPos at;
  int nti = 0;
  bool gave_up = false;
  for (;;) {
    // The first stage describes the tile.
    if (!mbar_wait(smem_u32(&bars[at.s]), at.phase)) {
      gave_up = true;
      break;
    }
    const StageInfo ti = info[at.s];
    if (ti.nks == 0) break;
    bool ok = true;
    const uint32_t tb = smem_u32(ti_full), tp = nti & 1;
    const bool full = ti.rows == kMaxBM;
    switch ((ti.hk + 7) / 8) {
      case 1:
        ok = full ? consume_mma<1, true>(ti, As, Bs, Ti, bars, tb, tp, tid, at, d)
                  : consume_mma<1, false>(ti, As, Bs, Ti, bars, tb, tp, tid, at, d);
        break;
      case 2:
        ok = full ? consume_mma<2, true>(ti, As, Bs, Ti, bars, tb, tp, tid, at, d)
                  : consume_mma<2, false>(ti, As, Bs, Ti, bars, tb, tp, tid, at, d);
        break;
      case 3:
        if (ti.hs <= kSymHS)
          ok = full ? consume_mma<3, true>(ti, As, Bs, Ti, bars, tb, tp, tid, at, d)
                    : consume_mma<3, false>(ti, As, Bs, Ti, bars, tb, tp, tid, at, d);
        else
          ok = consume_mma<4, false>(ti, As, Bs, Ti, bars, tb, tp, tid, at, d);
        break;
      case 4: ok = consume_mma<4, false>(ti, As, Bs, Ti, bars, tb, tp, tid, at, d); break;
      default: ok = consume_mma<5, false>(ti, As, Bs, Ti, bars, tb, tp, tid, at, d); break;
    }
    if (!ok) {  // a timed-out tile leaves its rows unfinished
      gave_up = true;
      break;
    }
    if (ti.nseg >= 0) {
      // A warp that had no turn passes T_I's phase all the same before it frees the buffer.
      if (!mbar_wait(tb, tp)) {
        gave_up = true;
        break;
      }
      ++nti;
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(ti_free));
    }
  }
  if (gave_up) {  // what the producer has issued lands before the CTA exits
    atomicOr(err, kErrTimeout);
    for (int s = 0; s < kStages; ++s, at.next()) mbar_wait(smem_u32(&bars[at.s]), at.phase);
    mbar_wait(smem_u32(ti_full), nti & 1);
  }
  trace_end(ctl, kTrLadderThin);
}

// cp.async (4-, 8- and 16-byte) global -> shared copies, committed and waited for by group.
__device__ __forceinline__ void cp_async8(void *dst, const void *src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_u32(dst)), "l"(src)
               : "memory");
}
__device__ __forceinline__ void cp_async4(void *dst, const void *src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(dst)), "l"(src)
               : "memory");
}
__device__ __forceinline__ void cp_async16(void *dst, const void *src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src)
               : "memory");
}
__device__ __forceinline__ void cp_async_commit() {
  asm volatile("cp.async.commit_group;" ::: "memory");
}
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// ------------------------------------------------------------------------------------------
// hh ladder intermediate (calc.cpp:141-160 and the one-body sums of calc.cpp:18-20, 82-84) over
// the packed quads:
//   X[kl, ij] = V_hhhh[kl, ij] + P[kl, ij],  P = sum_u V[u, kl] T[u, ij]   (k<l, i<j, u = a<b;
//               0.5 of the sum over all ordered pairs ab),
//   s[ij] = P[ij][ij],  r[u] = sum_ij V[u, ij] T[u, ij],
// a quarter of the reads and an eighth of the products of the ordered pairs.  V_hhpp is held in
// the packed layout of T, so a K slice of either is one contiguous range.
// hh_slice_kernel: units of two kinds in one launch.
//   hk <= 8: a warp per slice of kHHRows rows, its m8n8k4 fragments loaded straight from global
//   memory (8 consecutive columns of 4 rows a load, all loads of the slice in flight at once);
//   wider: a CTA per slice, both ranges copied to shared memory (16-byte cp.async; the row stride
//   hs is 4 mod 8 doubles, conflict-free for the fragments) and P on m16n8k16, warp w taking items
//   of one 16-row tile by kHHNC 8-column tiles.
// Both form the row dots r, and write the slice's partial P, which hh_reduce_kernel adds in a fixed order
// (deterministic).
// ------------------------------------------------------------------------------------------
constexpr int kHHThreads = 128;
constexpr int kHHRows = 32;  // packed rows of a slice
constexpr int kHHNC = 2;
// Slack: fragment loads of the rows and columns past hk in the last row.
constexpr size_t kHHSmem = (2 * (size_t)kHHRows * kMaxNB + 16) * sizeof(double);

__device__ __forceinline__ void hh_warp_unit(const HHTile &tt, const double *__restrict__ vq,
                                             const double *tq, double *__restrict__ part,
                                             double *__restrict__ r_out) {
  const int hk = tt.hk, hs = tt.hs, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int64_t base = tt.base + g;
  constexpr int kSteps = kHHRows / 4;
  double a[kSteps], b[kSteps], acc[2] = {0.0, 0.0};
#pragma unroll
  for (int k4 = 0; k4 < kSteps; ++k4) {
    const int k = 4 * k4 + t;
    const bool in = k < tt.rows && g < hk;
    a[k4] = in ? vq[base + k * hs] : 0.0;
    b[k4] = in ? tq[base + k * hs] : 0.0;
  }
#pragma unroll
  for (int k4 = 0; k4 < kSteps; ++k4) {
    dmma_884(acc, a[k4], b[k4]);
    double d = a[k4] * b[k4];  // row dot: a fixed butterfly over the columns
    d += __shfl_xor_sync(0xffffffffu, d, 4);
    d += __shfl_xor_sync(0xffffffffu, d, 8);
    d += __shfl_xor_sync(0xffffffffu, d, 16);
    if (g == 0 && 4 * k4 + t < tt.rows) r_out[tt.r0 + 4 * k4 + t] = d;
  }
#pragma unroll
  for (int q = 0; q < 2; ++q)
    if (g < hk && 2 * t + q < hk) part[g * hk + 2 * t + q] = acc[q];
}

__device__ __forceinline__ void hh_cta_unit(const HHTile &tt, const double *__restrict__ vq,
                                            const double *tq, double *__restrict__ part,
                                            double *__restrict__ r_out, double *sm) {
  const int hk = tt.hk, hs = tt.hs, rows = tt.rows, rows16 = (rows + 15) & ~15;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  double *Vs = sm, *Ts = sm + rows16 * hs;
  const int64_t base = tt.base;
  // Rows up to the next multiple of 16 are the block's zero padding, which is copied too.
  for (int e = 2 * threadIdx.x; e < rows16 * hs; e += 2 * kHHThreads) {
    cp_async16(Vs + e, vq + base + e);
    cp_async16(Ts + e, tq + base + e);
  }
  cp_async_commit();
  cp_async_wait<0>();
  __syncthreads();
  const int n8 = (hk + 7) >> 3, nch = (n8 + kHHNC - 1) / kHHNC, items = ((hk + 15) >> 4) * nch;
  for (int it = warp; it < items; it += kHHThreads / 32) {
    const int mt = it / nch, n0 = (it - mt * nch) * kHHNC;
    double acc[kHHNC][4];
#pragma unroll
    for (int n = 0; n < kHHNC; ++n) acc[n][0] = acc[n][1] = acc[n][2] = acc[n][3] = 0.0;
    for (int k16 = 0; k16 < rows16; k16 += 16) {
      double a[8];
#pragma unroll
      for (int i = 0; i < 8; ++i)  // A[kl][k] = V[k][kl]
        a[i] = Vs[(k16 + t + 4 * (i / 2)) * hs + 16 * mt + g + 8 * (i % 2)];
#pragma unroll
      for (int n = 0; n < kHHNC; ++n) {
        if (n0 + n >= n8) break;
        double b[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) b[q] = Ts[(k16 + t + 4 * q) * hs + 8 * (n0 + n) + g];
        dmma_16816(acc[n], a, b);
      }
    }
#pragma unroll
    for (int n = 0; n < kHHNC; ++n) {
      if (n0 + n >= n8) break;
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int kl = 16 * mt + g + 8 * (q >> 1), ij = 8 * (n0 + n) + 2 * t + (q & 1);
        if (kl < hk && ij < hk) part[kl * hk + ij] = acc[n][q];
      }
    }
  }
  for (int k = warp; k < rows; k += kHHThreads / 32) {
    double d = 0.0;
    for (int c = lane; c < hk; c += 32) d = fma(Vs[k * hs + c], Ts[k * hs + c], d);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) d += __shfl_xor_sync(0xffffffffu, d, o);
    if (lane == 0) r_out[tt.r0 + k] = d;
  }
}

// Units [0, n_cta) one per CTA, then n_warp units, one per warp of the following CTAs.
__global__ void __launch_bounds__(kHHThreads, 8)
hh_slice_kernel(const HHTile *__restrict__ tiles, int n_cta, int n_warp,
                const double *__restrict__ vq, const double *tq0, const double *tq1,
                double *__restrict__ part, double *__restrict__ r_out, const Control *ctl,
                int gate) {
  const bool wide = (int)blockIdx.x < n_cta;
  const int tr = wide ? kTrHHTiled : kTrHHSmall;
  const int w = ((int)blockIdx.x - n_cta) * (kHHThreads / 32) + (int)(threadIdx.x >> 5);
  // Static data, loaded beside the control block.
  const HHTile tt = tiles[wide ? (int)blockIdx.x : n_cta + min(w, n_warp - 1)];
  if (skip_iteration(ctl, gate, tr)) return;
  extern __shared__ __align__(16) double hh_smem[];
  if (!wide && w >= n_warp) return;
  const double *tq = ctl->parity ? tq1 : tq0;
  if (wide) hh_cta_unit(tt, vq, tq, part + tt.part, r_out, hh_smem);
  else hh_warp_unit(tt, vq, tq, part + tt.part, r_out);
  trace_end(ctl, tr);
}

// X and s: kHHLanes lanes per element of every channel's P (a flat list, so that channels of one
// hole pair do not take a CTA each), each adding every kHHLanes-th slice's partial with eight loads
// in flight, then a fixed shuffle tree.
constexpr int kHHLanes = 4;
// NT > 0: X / 2 also as NT bf16 terms, for the tensor-core ladder of a small system.
template <int NT>
__global__ void __launch_bounds__(128)
hh_reduce_kernel(const HHOut *__restrict__ outs, int n, const double *__restrict__ v_x,
                 const double *__restrict__ part, double *__restrict__ x,
                 double *__restrict__ s_out, __nv_bfloat16 *img, int64_t img_stride,
                 const Control *ctl, int gate) {
  const int i = (blockIdx.x * 128 + threadIdx.x) / kHHLanes, sub = threadIdx.x % kHHLanes;
  const HHOut o = outs[min(i, n - 1)];  // static data, loaded beside the control block
  const double vh = __ldg(v_x + o.x);
  if (skip_iteration(ctl, gate, kTrHHReduce)) return;
  const double *pb = part + o.part;
  double p = 0.0;
  for (int sl = sub; sl < o.nslices; sl += 8 * kHHLanes) {
    double y[8];
#pragma unroll
    for (int k = 0; k < 8; ++k)
      y[k] = sl + k * kHHLanes < o.nslices ? __ldcg(pb + (int64_t)(sl + k * kHHLanes) * o.stride)
                                           : 0.0;
#pragma unroll
    for (int k = 0; k < 8; ++k) p += y[k];
  }
#pragma unroll
  for (int m = kHHLanes / 2; m > 0; m >>= 1) p += __shfl_xor_sync(0xffffffffu, p, m);
  if (sub == 0 && i < n) {
    x[o.x] = vh + p;
    if (o.s >= 0) s_out[o.s] = p;
    if constexpr (NT > 0) {
      if (o.xt[0] >= 0) {
        __nv_bfloat16 a[NT], b[NT];
        split_bf16_n<NT>(0.5 * (vh + p), a);
        split_bf16_n<NT>(-0.5 * (vh + p), b);
#pragma unroll
        for (int q = 0; q < NT; ++q) {
          img[q * img_stride + o.xt[0]] = a[q];
          img[q * img_stride + o.xt[1]] = b[q];
        }
      }
    }
  }
  trace_end(ctl, kTrHHReduce);
}

// ------------------------------------------------------------------------------------------
// Ring term: Y = V_hphp + 0.5 V_hpph T', R = T' Y per modified channel (calc.cpp:264-313).
// Table path (ring_small_kernel, ring16_kernel): T' read from the phhp slab (t2Old_phhp), V_hpph
// held transposed per channel (Vt[k][i] = V_hpph[i][k], k < ph', i < hp'), R to t2Diff_phhp.
// Channels with ph', hp' <= kRingSmall run one per warp; larger ones one per CTA, grouped by
// padded size.
//
// Fused path (ring_pair_*): the channel of (a, i) and that of (i, a) together.  T' of the second
// is the transpose of the first's (t_ab,ij = t_ba,ji), and the assembly needs only the sums
//   S[ai, jb] = R[ai, jb] + R[bj, ia] = T' (A + C T') + B T'
// with A = V_hphp of the first channel, C = V_hpph (the same block for both, by the exchange of
// both pairs; of blocks that come from the host, their mean, which is exact for any) and
// B[ai, ck] = V_hphp[(k c), (i a)] of the second: three products instead of four and half of the
// amplitudes, of V_hpph and of the results (ring_unit, below).  Channels that do not pair up
// (tables from the host) run as on the table path, followed by ring_sums_kernel.
// ------------------------------------------------------------------------------------------
constexpr int kRingSmall = 16;
constexpr int kRingMax = 80;  // largest ph', hp'

// Quad of a phhp slab position: 4 * (packed position) + k, k = 0: (ab, ij), 1: (ab, ji),
// 2: (ba, ij), 3: (ba, ji); kNoQuad outside every quad.  The amplitude there is +t, -t, -t, +t.
constexpr uint32_t kNoQuad = ~0u;
__device__ __forceinline__ double ring_amplitude(const double *tq, uint32_t dst) {
  if (dst == kNoQuad) return 0.0;
  const double t = __ldcg(tq + (dst >> 2));
  return ((dst & 3) == 1 || (dst & 3) == 2) ? -t : t;
}

// The phhp slab (t2Old_phhp) of a fused handle from its packed amplitudes, for readers of the
// chain.
__global__ void __launch_bounds__(256)
phhp_gather_kernel(const uint32_t *__restrict__ dst, int64_t n, const double *tq0,
                   const double *tq1, double *__restrict__ phhp, const Control *ctl) {
  const double *__restrict__ t = ctl->parity ? tq1 : tq0;
  for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < n;
       p += (int64_t)gridDim.x * blockDim.x)
    phhp[p] = ring_amplitude(t, dst[p]);
}

// C (M8*8 x N8*8) = A B, K4*4 deep, on 8 x 8 tiles: warps warp, warp + nwarps, ... take items of
// one 8-row tile by NC column tiles (the A fragment is reused NC times).  A[m][k] =
// A[m * ars + k * aks], B[k][n] = B[k * ldb + n]; epi(row, col, value) stores each result.
template <int NC, class Epi>
__device__ __forceinline__ void warp_mma_gemm(const double *A, int ars, int aks, const double *B,
                                              int ldb, int M8, int N8, int K4, int warp,
                                              int nwarps, const Epi &epi) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int nch = (N8 + NC - 1) / NC;
  for (int it = warp; it < M8 * nch; it += nwarps) {
    const int mt = it / nch, n0 = (it - mt * nch) * NC, nn = min(NC, N8 - n0);
    double acc[NC][2];
#pragma unroll
    for (int n = 0; n < NC; ++n) acc[n][0] = acc[n][1] = 0.0;
    const double *ap = A + (mt * 8 + g) * ars + t * aks;
    const double *bp = B + t * ldb + n0 * 8 + g;
    const int astep = 4 * aks, bstep = 4 * ldb;
#pragma unroll 2
    for (int k4 = 0; k4 < K4; ++k4) {
      const double a = ap[k4 * astep];
#pragma unroll
      for (int n = 0; n < NC; ++n)
        if (n < nn) dmma_884(acc[n], a, bp[k4 * bstep + n * 8]);
    }
#pragma unroll
    for (int n = 0; n < NC; ++n)
      if (n < nn) {
        const int r = mt * 8 + g, c = (n0 + n) * 8 + 2 * t;
        epi(r, c, acc[n][0]);
        epi(r, c + 1, acc[n][1]);
      }
  }
}

__host__ __device__ inline int ring_pad8(int n) { return (n + 7) & ~7; }

// Channels with ph', hp' <= kRingSmall, one per warp (kRingSmallWarps per CTA), the same two
// products on the FP64 MMA: the warp's stage is padded to P, H in {8, 16} with zeros and a row
// stride of 20 doubles (4 mod 8: conflict-free fragment loads).
constexpr int kRingSmallWarps = 4;
constexpr int kRingSmallLd = kRingSmall + 4;
__global__ void __launch_bounds__(kRingSmallWarps * 32)
ring_small_kernel(const ModInfo *__restrict__ mods, int n, const double *__restrict__ v_hpph,
                  const double *__restrict__ v_hphp, const double *__restrict__ t_phhp,
                  double *__restrict__ out, const Control *ctl, int gate) {
  if (skip_iteration(ctl, gate, kTrRingSmall)) return;
  __shared__ __align__(16) double buf[kRingSmallWarps][3 * kRingSmall * kRingSmallLd];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int mi = blockIdx.x * kRingSmallWarps + w;
  if (mi >= n) return;  // whole warps: the MMAs below are warp-collective
  const ModInfo m = mods[mi];
  const int ph = m.ph, hp = m.hp, P = ring_pad8(ph), H = ring_pad8(hp), ld = kRingSmallLd;
  const int hs = H == 8 ? 3 : 4;  // log2 H
  double *Ts = buf[w], *Vt = Ts + kRingSmall * ld, *Ys = Vt + kRingSmall * ld;
  // Operands by cp.async (every load of the warp in flight at once), pad cells zeroed.
  for (int e = lane; e < P * H; e += 32) {
    const int r = e >> hs, c = e & (H - 1);
    if (r < ph && c < hp) {
      const int64_t src = m.m_off + r * hp + c;
      cp_async8(Ts + r * ld + c, t_phhp + src);
      cp_async8(Vt + r * ld + c, v_hpph + src);
    } else {
      Ts[r * ld + c] = 0.0;
      Vt[r * ld + c] = 0.0;
    }
  }
  for (int e = lane; e < H * H; e += 32) {
    const int r = e >> hs, c = e & (H - 1);
    if (r < hp && c < hp) cp_async8(Ys + r * ld + c, v_hphp + m.y_off + r * hp + c);
    else Ys[r * ld + c] = 0.0;
  }
  cp_async_commit();
  cp_async_wait<0>();
  __syncwarp();
  // A[i][k] = V_hpph[i][k] = Vt[k][i]; each Y element is read and written by its owner lane.
  warp_mma_gemm<2>(Vt, 1, ld, Ts, ld, H / 8, H / 8, P / 4, 0, 1,
                   [&](int r, int c, double v) { Ys[r * ld + c] = 0.5 * v + Ys[r * ld + c]; });
  __syncwarp();
  warp_mma_gemm<2>(Ts, ld, 1, Ys, ld, P / 8, H / 8, H / 4, 0, 1, [&](int r, int c, double v) {
    if (r < ph && c < hp) out[m.m_off + r * hp + c] = v;
  });
  trace_end(ctl, kTrRingSmall);
}

// Channels with ph', hp' > kRingSmall: one CTA per channel, the two products on the FP64
// m16n8k16 MMA (4 k-steps for a 64-wide channel instead of 14 with m8n8k4, so a warp's
// accumulator chains are short).  The channel is padded to PAD (a multiple of 16) with zeros
// in shared memory: T' [PAD][ld], Vt [PAD][ld], Y [PAD][ld] (V_hphp on arrival), ld = PAD + 4
// (4 mod 16 doubles: conflict-free fragment loads), all loaded with cp.async.  Warp w takes
// items of one 16-row tile by NC 8-column tiles.  Channels are grouped by PAD (32, 48, 64, 80),
// one launch per group, so a CTA's shared memory fits its channel and several CTAs share an SM.
constexpr int kRing16NC = 4;
__host__ __device__ constexpr int ring16_warps(int pad) {
  return (pad / 16) * ((pad / 8 + kRing16NC - 1) / kRing16NC);
}
// Operand buffers: the 32 group keeps two (T', V_hpph; Y replaces V_hpph, V_hphp is read into
// the accumulators), so that 8 CTAs share an SM; the wider groups three (T', V_hpph, V_hphp ->
// Y), which measured faster for them.
__host__ __device__ constexpr int ring16_bufs(int pad) { return pad <= 32 ? 2 : 3; }
__host__ __device__ constexpr size_t ring16_smem(int pad) {
  return (size_t)ring16_bufs(pad) * pad * (pad + 4) * sizeof(double);
}
// CTAs per SM that the shared memory allows (227 KB), kept by the register budget too.
__host__ __device__ constexpr int ring16_ctas(int pad) {
  return (int)((227 * 1024) / ring16_smem(pad)) > 8 ? 8 : (int)((227 * 1024) / ring16_smem(pad));
}
// init(slot, r, c) gives the starting accumulator of every output position of an item before
// its MMAs (it may also start loads that epi(r, c, v, slot) then uses: slot = n * 4 + the
// accumulator index).
template <int PAD, int MODE, class Init, class Epi>
__device__ __forceinline__ void ring16_gemm(const double *As, const double *Bs, int warp,
                                            const Init &init, const Epi &epi) {
  // MODE 0: A[m][k] = As[k][m] (k-major); MODE 1: A[m][k] = As[m][k].  B[k][n] = Bs[k][n].
  constexpr int ld = PAD + 4, N8 = PAD / 8, NCH = (N8 + kRing16NC - 1) / kRing16NC;
  constexpr int ITEMS = (PAD / 16) * NCH;
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  for (int it = warp; it < ITEMS; it += ring16_warps(PAD)) {
    const int mt = it / NCH, n0 = (it - mt * NCH) * kRing16NC;
    double acc[kRing16NC][4];
#pragma unroll
    for (int n = 0; n < kRing16NC; ++n) {
      const int r = 16 * mt + g, c = 8 * (n0 + n) + 2 * t;
      acc[n][0] = init(n * 4 + 0, r, c);
      acc[n][1] = init(n * 4 + 1, r, c + 1);
      acc[n][2] = init(n * 4 + 2, r + 8, c);
      acc[n][3] = init(n * 4 + 3, r + 8, c + 1);
    }
#pragma unroll
    for (int k16 = 0; k16 < PAD / 16; ++k16) {
      double a[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int m = 16 * mt + g + 8 * (i % 2), k = 16 * k16 + t + 4 * (i / 2);
        a[i] = MODE == 0 ? As[k * ld + m] : As[m * ld + k];
      }
#pragma unroll
      for (int n = 0; n < kRing16NC; ++n) {
        if (n0 + n >= N8) break;
        double b[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) b[q] = Bs[(16 * k16 + t + 4 * q) * ld + 8 * (n0 + n) + g];
        dmma_16816(acc[n], a, b);
      }
    }
#pragma unroll
    for (int n = 0; n < kRing16NC; ++n) {
      if (n0 + n >= N8) break;
      const int r = 16 * mt + g, c = 8 * (n0 + n) + 2 * t;
      epi(r, c, acc[n][0], n * 4 + 0);
      epi(r, c + 1, acc[n][1], n * 4 + 1);
      epi(r + 8, c, acc[n][2], n * 4 + 2);
      epi(r + 8, c + 1, acc[n][3], n * 4 + 3);
    }
  }
}
template <int PAD>
__global__ void __launch_bounds__(32 * ring16_warps(PAD), ring16_ctas(PAD))
ring16_kernel(const ModInfo *__restrict__ mods, const double *__restrict__ v_hpph,
              const double *__restrict__ v_hphp, const double *__restrict__ t_phhp,
              double *__restrict__ out, const Control *ctl, int gate) {
  if (skip_iteration(ctl, gate, PAD <= 32 ? kTrRingMid : kTrRingLarge)) return;
  extern __shared__ __align__(16) double r16[];
  constexpr int ld = PAD + 4, NT = 32 * ring16_warps(PAD), N8 = PAD / 8;
  constexpr int NCH = (N8 + kRing16NC - 1) / kRing16NC;
  constexpr bool TWO = ring16_bufs(PAD) == 2;
  static_assert((PAD / 16) * NCH == ring16_warps(PAD), "one GEMM item per warp");
  double *Ts = r16, *Vs = r16 + PAD * ld, *Ys = TWO ? Vs : r16 + 2 * PAD * ld;
  const ModInfo m = mods[blockIdx.x];
  const int ph = m.ph, hp = m.hp;
  for (int e = threadIdx.x; e < PAD * PAD; e += NT) {
    const int r = e / PAD, c = e - r * PAD;
    if (r < ph && c < hp) {
      const int64_t src = m.m_off + (int64_t)r * hp + c;
      cp_async8(Ts + r * ld + c, t_phhp + src);
      cp_async8(Vs + r * ld + c, v_hpph + src);
    } else {
      Ts[r * ld + c] = 0.0;
      Vs[r * ld + c] = 0.0;
    }
    if constexpr (!TWO) {
      if (r < hp && c < hp) cp_async8(Ys + r * ld + c, v_hphp + m.y_off + (int64_t)r * hp + c);
      else Ys[r * ld + c] = 0.0;
    }
  }
  cp_async_commit();
  const int warp = threadIdx.x >> 5;
  if constexpr (TWO) {
    // 2 Y = 2 V_hphp + V_hpph T' (V_hpph[i][k] = Vt[k][i]): the accumulators start from
    // 2 V_hphp (global loads issued while the stage lands) and are halved on the way into the
    // V_hpph buffer, once every warp is done reading it.
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int mt = warp / NCH, n0 = (warp - mt * NCH) * kRing16NC;
    double y[4 * kRing16NC];
    cp_async_wait<0>();
    __syncthreads();
    ring16_gemm<PAD, 0>(
        Vs, Ts, warp,
        [&](int, int r, int c) {
          return (r < hp && c < hp) ? 2.0 * __ldg(v_hphp + m.y_off + (int64_t)r * hp + c) : 0.0;
        },
        [&](int, int, double v, int slot) { y[slot] = 0.5 * v; });
    __syncthreads();
#pragma unroll
    for (int slot = 0; slot < 4 * kRing16NC; ++slot) {
      const int n = slot >> 2, q = slot & 3;
      if (n0 + n < N8)
        Ys[(16 * mt + g + 8 * (q >> 1)) * ld + 8 * (n0 + n) + 2 * t + (q & 1)] = y[slot];
    }
  } else {
    // Y = V_hphp + 0.5 V_hpph T' in the third buffer; each Y element has one owner lane.
    cp_async_wait<0>();
    __syncthreads();
    ring16_gemm<PAD, 0>(
        Vs, Ts, warp, [](int, int, int) { return 0.0; },
        [&](int r, int c, double v, int) { Ys[r * ld + c] = 0.5 * v + Ys[r * ld + c]; });
  }
  __syncthreads();
  // R = T' Y, stored for r < ph', c < hp'.
  ring16_gemm<PAD, 1>(
      Ts, Ys, warp, [](int, int, int) { return 0.0; },
      [&](int r, int c, double v, int) {
        if (r < ph && c < hp) out[m.m_off + (int64_t)r * hp + c] = v;
      });
  trace_end(ctl, PAD <= 32 ? kTrRingMid : kTrRingLarge);
}

// ---- Fused path: a channel and its transpose together ------------------------------------
// Units of one pair and a block of up to kPairNC 8-column tiles of S (columns of Y and S depend on
// the same columns of T' alone, so blocks share no product), on m16n8k16, by G = 1, 2 or 4 warps
// (ph', hp' <= 16, 32, 80), warp w on row tiles w, w + G, ...
// A, B, C and the destinations are stored in the order in which the lanes of a fragment take them,
// so every load of them is a 16-byte one, contiguous over the warp, straight into registers.  T'
// arrives as a stored shared-memory image (16-row, 16-column padding, row stride H16 + 4) by one
// bulk copy: a random 8-byte read of an amplitude costs the L2 a whole sector, and made by every
// column block they were half of the ring's time (61 -> 36 us without them at EG N=54
// |n|^2 <= 36), so tp_gather_kernel reads each amplitude once and writes the images.
constexpr int kPairNC = 4;
__host__ __device__ inline int pad16(int n) { return (n + 15) & ~15; }
__host__ __device__ inline int ring_group(int ph, int hp) {
  return (ph > hp ? ph : hp) <= 16 ? 1 : (ph > hp ? ph : hp) <= 32 ? 2 : 4;
}
// T' and Y of a unit (doubles): all of T' (row stride h + 4), or (COLS) the unit's columns alone,
// with Y's row stride 8 nt + 4.  Strides are 4 mod 8 doubles.  All of T' is 35 to 54 KB, which
// leaves room for one CTA of four warps beside the ladder; the columns leave room for two, and T' as
// the A operand then comes from L2.  Where those units are more than a CTA or two per SM the
// columns are the better choice.  All of T' and the columns, FP64 iterations by units, EG N=54: 160
// 36.7, 37.2 us; 322 58.5, 58.4; 448 91.6, 88.1; 600 118.4, 114.1; 732 156.1, 150.0; PNM N=66: 196
// 37.6, 39.4; 298 56.3, 55.0; 382 71.8, 71.9; 672 134.9, 132.0; 1218 220.5, 206.3.
__host__ __device__ inline bool ring_cols(int64_t units4) { return units4 > 2 * kSMs; }
__host__ __device__ constexpr int ring_ldy(int g, bool cols, int nt) {
  return g == 1 ? 20 : cols ? 8 * nt + 4 : 8 * kPairNC + 4;
}
__host__ __device__ constexpr int ring_unit_smem(int g, bool cols, int p, int h, int nt) {
  return p * (cols ? ring_ldy(g, cols, nt) : h + 4) + h * ring_ldy(g, cols, nt);
}
// Fragment-ordered A operand: [16-row tile][16-deep step][4][lane][2].
__device__ __forceinline__ void frag_load(double (&a)[8], const double *__restrict__ p) {
  const double2 *q = reinterpret_cast<const double2 *>(p) + (threadIdx.x & 31);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const double2 v = __ldg(q + 32 * j);
    a[2 * j] = v.x;
    a[2 * j + 1] = v.y;
  }
}
// acc += A B over K: A fragments from `frag`, two steps ahead of the products (f[0] and f[1] hold
// the first two on entry), B[k][n] = Bs[k * ldb + n], nt column tiles.
__device__ __forceinline__ void frag_start(double (&f)[2][8], const double *__restrict__ frag,
                                           int K) {
  frag_load(f[0], frag);
  if (K > 16) frag_load(f[1], frag + 256);
}
template <int NC>
__device__ __forceinline__ void mma_row(double (&acc)[NC][4], const double (&a)[8],
                                        const double *Bs, int ldb, int nt, int k0) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
#pragma unroll
  for (int n = 0; n < NC; ++n) {
    if (n >= nt) break;
    double b[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) b[q] = Bs[(k0 + t + 4 * q) * ldb + 8 * n + g];
    dmma_16816(acc[n], a, b);
  }
}
template <int NC>
__device__ __forceinline__ void frag_gemm(double (&acc)[NC][4], double (&f)[2][8],
                                          const double *__restrict__ frag, const double *Bs,
                                          int ldb, int nt, int K) {
  for (int k0 = 0; k0 < K; k0 += 32) {
    mma_row(acc, f[0], Bs, ldb, nt, k0);
    if (k0 + 32 < K) frag_load(f[0], frag + (k0 + 32) * 16);
    if (k0 + 16 < K) {
      mma_row(acc, f[1], Bs, ldb, nt, k0 + 16);
      if (k0 + 48 < K) frag_load(f[1], frag + (k0 + 48) * 16);
    }
  }
}
template <int G>
__device__ __forceinline__ void group_sync() {
  if constexpr (G == 1) __syncwarp();
  else if constexpr (G == 2)
    asm volatile("bar.sync %0, 64;" ::"r"(1 + (int)(threadIdx.x >> 6)) : "memory");
  else __syncthreads();
}
template <int G, bool COLS>
__device__ __forceinline__ void ring_unit(const RingUnit &m, const double *__restrict__ img,
                                          const int32_t *__restrict__ to_img, const double *tp,
                                          double *__restrict__ out, double *sm, uint32_t bar,
                                          uint32_t parity, int32_t *err) {
  constexpr int NC = G == 1 ? 2 : kPairNC;
  const int P = pad16(m.ph), H = pad16(m.hp), ldh = H + 4, n8 = (m.hp + 7) >> 3, nt = m.nt;
  const int w = (threadIdx.x >> 5) % G, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int ldy = ring_ldy(G, COLS, nt), ldt = COLS ? ldy : ldh;
  double *Ts = sm, *Ys = sm + P * ldt;
  if (COLS) {
    if (w == 0) {
      if (lane == 0) mbar_expect_tx(bar, P * nt * 64);
      __syncwarp();
      for (int r = lane; r < P; r += 32)
        bulk_g2s(smem_u32(Ts + r * ldt), tp + m.tp + (int64_t)r * ldh + 8 * m.n0, nt * 64, bar);
    }
  } else if (w == 0 && lane == 0) {
    mbar_expect_tx(bar, P * ldh * 8);
    bulk_g2s(smem_u32(Ts), tp + m.tp, P * ldh * 8, bar);
  }
  const double *Tj = COLS ? Ts : Ts + 8 * m.n0;  // this unit's columns of T'
  bool landed = false;
  auto wait = [&]() {
    if (!landed && !mbar_wait(bar, parity)) {
      atomicOr(err, kErrTimeout);
      mbar_wait(bar, parity);  // the copies land before the CTA exits
    }
    landed = true;
  };
  double f[2][8], acc[NC][4];
  for (int mt = w; 16 * mt < H; mt += G) {  // Y = A + C T'
    const double *c_frag = img + m.c_img + (int64_t)mt * P * 16;
    frag_start(f, c_frag, P);
    const double2 *ap =
        reinterpret_cast<const double2 *>(img + m.a_img) + ((int64_t)mt * n8 + m.n0) * 64 + lane;
#pragma unroll
    for (int n = 0; n < NC; ++n)
      if (n < nt) {
        const double2 lo = __ldg(ap + 64 * n), hi = __ldg(ap + 64 * n + 32);
        acc[n][0] = lo.x; acc[n][1] = lo.y; acc[n][2] = hi.x; acc[n][3] = hi.y;
      }
    wait();
    frag_gemm(acc, f, c_frag, Tj, ldt, nt, P);
#pragma unroll
    for (int n = 0; n < NC; ++n)
      if (n < nt)
#pragma unroll
        for (int q = 0; q < 4; ++q)
          Ys[(16 * mt + g + 8 * (q >> 1)) * ldy + 8 * n + 2 * t + (q & 1)] = acc[n][q];
  }
  const double *b_frag = img + m.b_img;
  if (16 * w < P) frag_start(f, b_frag + (int64_t)w * P * 16, P);
  wait();
  if (!COLS) group_sync<G>();
  for (int mt = w; 16 * mt < P; mt += G) {  // S = B T' + T' Y, to the quads
    const double *bf = b_frag + (int64_t)mt * P * 16;
    if (mt != w) frag_start(f, bf, P);
#pragma unroll
    for (int n = 0; n < NC; ++n) acc[n][0] = acc[n][1] = acc[n][2] = acc[n][3] = 0.0;
    frag_gemm(acc, f, bf, Tj, ldt, nt, P);
    const int4 *qp =
        reinterpret_cast<const int4 *>(to_img + m.to_img) + ((int64_t)mt * n8 + m.n0) * 32 + lane;
    int4 to[NC];
#pragma unroll
    for (int n = 0; n < NC; ++n)
      if (n < nt) to[n] = __ldg(qp + 32 * n);
    // T' as the A operand: from its image in shared memory, or (COLS) in global memory, 8 sectors
    // a load, all of them used, two steps ahead.
    const double *ta = COLS ? tp + m.tp + (int64_t)(16 * mt + g) * ldh + t
                             : Ts + (16 * mt + g) * ldh + t;
    auto t_load = [&](double (&a)[8], int k0) {
#pragma unroll
      for (int i = 0; i < 8; ++i) a[i] = ta[8 * (i % 2) * ldh + k0 + 4 * (i / 2)];
    };
    if constexpr (COLS) {
      t_load(f[0], 0);
      if (H > 16) t_load(f[1], 16);
      if (mt == w) group_sync<G>();  // Y is complete
      for (int k0 = 0; k0 < H; k0 += 32) {
        mma_row(acc, f[0], Ys, ldy, nt, k0);
        if (k0 + 32 < H) t_load(f[0], k0 + 32);
        if (k0 + 16 < H) {
          mma_row(acc, f[1], Ys, ldy, nt, k0 + 16);
          if (k0 + 48 < H) t_load(f[1], k0 + 48);
        }
      }
    } else {
      for (int k0 = 0; k0 < H; k0 += 16) {
        double a[8];
        t_load(a, k0);
        mma_row(acc, a, Ys, ldy, nt, k0);
      }
    }
#pragma unroll
    for (int n = 0; n < NC; ++n)
      if (n < nt) {
        if (to[n].x >= 0) out[to[n].x] = acc[n][0];
        if (to[n].y >= 0) out[to[n].y] = acc[n][1];
        if (to[n].z >= 0) out[to[n].z] = acc[n][2];
        if (to[n].w >= 0) out[to[n].w] = acc[n][3];
      }
  }
  if (COLS && 16 * w >= P) group_sync<G>();  // a warp without rows of S
}

template <int G, bool COLS = false>
__global__ void __launch_bounds__(G == 2 ? 64 : 128, G == 2 ? 8 : 4)
ring_pair_kernel(const RingUnit *__restrict__ units, int n, const double *__restrict__ img,
                 const int32_t *__restrict__ to_img, const double *tp, double *__restrict__ out,
                 const Control *ctl, int32_t *err, int gate) {
  constexpr int kTr = G == 1 ? kTrRingSmall : G == 2 ? kTrRingMid : kTrRingLarge;
  if (skip_iteration(ctl, gate, kTr)) return;
  extern __shared__ __align__(128) double rp_smem[];
  __shared__ uint64_t bars[G == 1 ? 4 : 1];
  constexpr int kPer = G == 1 ? 4 : 1;  // units per CTA
  const int sub = G == 1 ? threadIdx.x >> 5 : 0, u = blockIdx.x * kPer + sub;
  if (threadIdx.x == 0) {
    for (int i = 0; i < kPer; ++i) mbar_init(smem_u32(&bars[i]), 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  if (u < n)
    ring_unit<G, COLS>(units[u], img, to_img, tp, out, rp_smem + sub * ring_unit_smem(1, false, 16, 16, 2),
                 smem_u32(&bars[sub]), 0, err);
  trace_end(ctl, kTr);
}

// T' images: kGatherPer elements a thread, all their loads in flight together.  src: 2 x the packed
// position, + 1 where the amplitude is negated; -1 for the padding and outside every quad.
constexpr int kGatherThreads = 256;
constexpr int kGatherPer = 8;
__global__ void __launch_bounds__(kGatherThreads)
tp_gather_kernel(const int32_t *__restrict__ src, int64_t n, const double *tq0, const double *tq1,
                 double *__restrict__ tp, const Control *ctl, int gate) {
  if (skip_iteration(ctl, gate, kTrGather)) return;
  const double *__restrict__ tq = ctl->parity ? tq1 : tq0;
  const int64_t p0 = ((int64_t)blockIdx.x * kGatherThreads * (kGatherPer / 4) + threadIdx.x) * 4;
  int4 d[kGatherPer / 4];
  double v[kGatherPer];
  // A predicated load: a branch would leave one load in flight, and a common address for the
  // elements outside every quad would queue a request per warp at one L2 slice.
  auto pick = [&](int32_t k) {
    double t;
    asm("{ .reg .pred p; setp.ge.s32 p, %2, 0; mov.f64 %0, 0d0000000000000000; "
        "@p ld.global.cg.f64 %0, [%1]; }"
        : "=d"(t)
        : "l"(tq + (k >> 1)), "r"(k));
    return t;
  };
#pragma unroll
  for (int j = 0; j < kGatherPer / 4; ++j) {
    const int64_t p = p0 + (int64_t)j * 4 * kGatherThreads;
    d[j] = p < n ? __ldg(reinterpret_cast<const int4 *>(src + p)) : make_int4(-1, -1, -1, -1);
  }
#pragma unroll
  for (int j = 0; j < kGatherPer / 4; ++j) {
    v[4 * j] = pick(d[j].x);
    v[4 * j + 1] = pick(d[j].y);
    v[4 * j + 2] = pick(d[j].z);
    v[4 * j + 3] = pick(d[j].w);
  }
  auto sign = [](double t, int32_t k) { return (k & 1) ? -t : t; };
#pragma unroll
  for (int j = 0; j < kGatherPer / 4; ++j) {
    const int64_t p = p0 + (int64_t)j * 4 * kGatherThreads;
    if (p >= n) continue;
    double2 *o = reinterpret_cast<double2 *>(tp + p);
    o[0] = make_double2(sign(v[4 * j], d[j].x), sign(v[4 * j + 1], d[j].y));
    o[1] = make_double2(sign(v[4 * j + 2], d[j].z), sign(v[4 * j + 3], d[j].w));
  }
  trace_end(ctl, kTrGather);
}

// The two ring sums of every quad from R in the phhp slab, of a fused handle whose channels do not
// pair up (at: ai_jb, the phhp position of an amplitude).
constexpr int kAsmThreads = 256;
__global__ void __launch_bounds__(kAsmThreads)
ring_sums_kernel(const QuadItem *__restrict__ items, const ChanInfo *__restrict__ chans,
                 const QuadRow *__restrict__ qrows, const QuadCol *__restrict__ qcols,
                 const int32_t *__restrict__ at, const double *__restrict__ r,
                 double *__restrict__ r_quad) {
  const QuadItem item = items[blockIdx.x];
  const int q = item.q0 + threadIdx.x;
  if (q >= item.q1) return;
  const int u = q / item.hk, w = q - u * item.hk;
  const QuadRow rw = qrows[item.pk_off + u];
  const QuadCol cl = qcols[item.qcol_off + w];
  at += chans[item.ch].t_off;
  double *o = r_quad + 2 * (item.q_off + (int64_t)u * item.hs + w);
  o[0] = r[at[rw.o_ab + cl.c_ij]] + r[at[rw.o_ba + cl.c_ji]];
  o[1] = r[at[rw.o_ab + cl.c_ji]] + r[at[rw.o_ba + cl.c_ij]];
}

// Deterministic block reduction (fixed tree) of one double; result valid in thread 0.
template <int NT>
__device__ __forceinline__ double block_sum(double v, double *scratch) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  __syncthreads();
  if (lane == 0) scratch[warp] = v;
  __syncthreads();
  double r = 0.0;
  if (warp == 0) {
    r = lane < NT / 32 ? scratch[lane] : 0.0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) r += __shfl_down_sync(0xffffffffu, r, o);
  }
  return r;
}

// ------------------------------------------------------------------------------------------
// One-body terms through the 3-body chains (table path), one CTA per orbital:
//   hole k:     x = sum v_h_hpp * t2Old_h2pp_h1;  diff_h2pp_h1 = 0.5 x t2Old_h1pp_h2
//   particle a: y = sum t2Old_p1_p2hh * v_phh_p;  diff_p2_p1hh = -0.5 y t2Old_p2_p1hh
// (argument order of main.cpp:591-607).  Bound by latency: the few holes' blocks are long (18000
// elements at EG N=54 |n|^2 <= 20), so those CTAs have 1024 threads, the particles' 256, four
// elements each in flight: the call for the holes at EG N=38 |n|^2 <= 16 30 -> 17 us.
// ------------------------------------------------------------------------------------------
constexpr int kOBHoles = 1024, kOBParticles = 256, kOBPer = 4;
template <int NT>
__global__ void __launch_bounds__(NT)
onebody_tables_kernel(const int64_t *__restrict__ off, const double *__restrict__ va,
                      const double *__restrict__ vb, const double *__restrict__ t,
                      double *__restrict__ diff, double sign) {
  __shared__ double scratch[32];
  __shared__ double total;
  const int64_t lo = off[blockIdx.x], hi = off[blockIdx.x + 1];
  double part = 0.0;
  for (int64_t e0 = lo + threadIdx.x; e0 < hi; e0 += kOBPer * NT) {
    double a[kOBPer], b[kOBPer];
#pragma unroll
    for (int k = 0; k < kOBPer; ++k) {
      const int64_t e = e0 + k * NT;
      a[k] = e < hi ? va[e] : 0.0;
      b[k] = e < hi ? vb[e] : 0.0;
    }
#pragma unroll
    for (int k = 0; k < kOBPer; ++k) part += a[k] * b[k];
  }
  const double sum = block_sum<NT>(part, scratch);
  if (threadIdx.x == 0) total = sum;
  __syncthreads();
  const double f = sign * total;
#pragma unroll 4
  for (int64_t e = lo + threadIdx.x; e < hi; e += NT) diff[e] = f * t[e];
}

// What follows X and s, in one launch:
// - x_k and y_a as segmented sums of the hh ladder's by-products s and r over the strict pairs that
//   hold the orbital (twice, for the two orders of the summed pair), one warp per orbital (the
//   first n_ob CTAs), lane-strided partial sums and a fixed shuffle tree;
// - tx[u, w] = 0.5 T X = sum_{k<l} T[u, kl] X[kl, w] on the FP64 MMA (m8n8k4): a warp per unit of
//   tx_rows(hk) rows of a channel, T and X straight from global memory (X mostly from L1).  Here it
//   runs beside the ladder and the ring; in the assembly, which nothing overlaps, it took 6 of 34 us
//   at EG N=54 |n|^2 <= 36 (12 of 47 at PNM N=66).  Its CTAs queue before the ring's, and beside the
//   ladder an SM holds few, each for several times its time alone (dependent loads): one thread per
//   quad, 3051 CTAs of 256 threads, took from 51 to 81 us of the iteration, these 42 to 55.  (X's sum
//   over the slices done again by a CTA per row tile, without hh_reduce_kernel: 42 to 67.)
constexpr int kPostThreads = 128;
__host__ __device__ inline int tx_rows(int hk) { return hk <= 4 ? 128 : hk <= 8 ? 64 : 16; }

// Up to 8 hole pairs: X's fragments stay in registers (KS K steps of 4), rows by 8.
template <int KS>
__device__ __forceinline__ void tx_thin(const TXTile &tt, const double *__restrict__ tq,
                                        const double *__restrict__ x, double *__restrict__ tx) {
  const int lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3, hk = tt.hk, hs = tt.hs;
  double b[KS];
#pragma unroll
  for (int k = 0; k < KS; ++k)
    b[k] = q + 4 * k < hk && g < hk ? __ldcg(x + tt.x + (q + 4 * k) * hs + g) : 0.0;
  constexpr int kRows = 8 / KS;  // groups of 8 rows in flight
  for (int u0 = g; u0 - g < tt.rows; u0 += 8 * kRows) {
    double a[kRows][KS];
#pragma unroll
    for (int i = 0; i < kRows; ++i)
#pragma unroll
      for (int k = 0; k < KS; ++k)
        a[i][k] = u0 + 8 * i < tt.rows && q + 4 * k < hk
                      ? tq[tt.at + (u0 + 8 * i) * hs + q + 4 * k] : 0.0;
#pragma unroll
    for (int i = 0; i < kRows; ++i) {
      double c[2] = {0.0, 0.0};
#pragma unroll
      for (int k = 0; k < KS; ++k) dmma_884(c, a[i][k], b[k]);
#pragma unroll
      for (int e = 0; e < 2; ++e)
        if (u0 + 8 * i < tt.rows && 2 * q + e < hk)
          tx[tt.at + (u0 + 8 * i) * hs + 2 * q + e] = c[e];
    }
  }
}
// More: 16 rows and two 8-column tiles.
__device__ __forceinline__ void tx_wide(const TXTile &tt, const double *__restrict__ tq,
                                        const double *__restrict__ x, double *__restrict__ tx) {
  const int lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3, hk = tt.hk, hs = tt.hs;
  const bool in0 = g < tt.rows, in1 = g + 8 < tt.rows;
  const double *t0 = tq + tt.at + g * hs, *t1 = t0 + 8 * hs;
  const int j = tt.j0;
  const bool j0 = j + g < hk, j1 = j + 8 + g < hk;
  double c[4][2] = {};
#pragma unroll 4
  for (int k = q; k < hk + q; k += 4) {
    const bool in = k < hk;
    const double a0 = in0 && in ? t0[k] : 0.0, a1 = in1 && in ? t1[k] : 0.0;
    const double b0 = in && j0 ? x[tt.x + k * hs + j + g] : 0.0;
    const double b1 = in && j1 ? x[tt.x + k * hs + j + 8 + g] : 0.0;
    dmma_884(c[0], a0, b0);
    dmma_884(c[1], a1, b0);
    dmma_884(c[2], a0, b1);
    dmma_884(c[3], a1, b1);
  }
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int u = g + 8 * (i & 1), w = j + 8 * (i >> 1) + 2 * q + e;
      if (u < tt.rows && w < hk) tx[tt.at + (int64_t)u * hs + w] = c[i][e];
    }
}

__global__ void __launch_bounds__(kPostThreads, 8)
hh_post_kernel(int n_ob, int np, int nsp, const int64_t *__restrict__ list_off,
               const int32_t *__restrict__ list, const double *__restrict__ s,
               const double *__restrict__ r, double *__restrict__ xh, double *__restrict__ yp,
               const TXTile *__restrict__ tiles, int n_tx, const double *x, const double *tq0,
               const double *tq1, double *__restrict__ tx, const Control *ctl, int gate) {
  if ((int)blockIdx.x >= n_ob) {
    const int i = ((int)blockIdx.x - n_ob) * (kPostThreads / 32) + (int)(threadIdx.x >> 5);
    const TXTile tt = tiles[min(i, n_tx - 1)];  // static data, loaded beside the control block
    if (skip_iteration(ctl, gate, kTrOneBody)) return;
    if (i < n_tx) {
      const double *tq = ctl->parity ? tq1 : tq0;
      if (tt.hk <= 4) tx_thin<1>(tt, tq, x, tx);
      else if (tt.hk <= 8) tx_thin<2>(tt, tq, x, tx);
      else tx_wide(tt, tq, x, tx);
    }
    trace_end(ctl, kTrOneBody);
    return;
  }
  if (skip_iteration(ctl, gate, kTrOneBody)) return;
  const int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (w >= nsp) return;
  const bool hole = w < np;
  const double *src = hole ? s : r;
  // Eight lane-strided partial sums: the eight index loads of a round are issued together,
  // then the eight value loads, so a round costs two memory latencies; the last round of a
  // list is guarded (lists are mostly shorter than one round).
  double acc[8] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
  const int64_t hi = list_off[w + 1];
  for (int64_t e = list_off[w] + lane; e < hi; e += 256) {
    int32_t ix[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) ix[k] = e + 32 * k < hi ? __ldg(list + e + 32 * k) : -1;
#pragma unroll
    for (int k = 0; k < 8; ++k)
      if (ix[k] >= 0) acc[k] += __ldcg(src + ix[k]);
  }
  double v = ((acc[0] + acc[1]) + (acc[2] + acc[3])) + ((acc[4] + acc[5]) + (acc[6] + acc[7]));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  if (lane == 0) {
    if (hole) xh[w] = 2.0 * v;
    else yp[w - np] = 2.0 * v;
  }
  trace_end(ctl, kTrOneBody);
}

// One packed amplitude t of quad (u, w) into the mixed-precision operand image: nt bf16 terms
// of T as the B operand of V T in the tensor-core chunk layout (K = u).
template <int NT>
__device__ __forceinline__ void write_t_image_n(const ChanInfo &ch, int u, int w,
                                                const QuadCol &cl, double t, __nv_bfloat16 *img,
                                                int64_t stride) {
  __nv_bfloat16 hv[NT];
  split_bf16_n<NT>(t, hv);
  const int64_t o =
      ch.tkt_tc_base + (int64_t)(u >> 5) * (ch.nbt >> 3) * kTcGroup + tc_off_mn(w, u & 31);
#pragma unroll
  for (int p = 0; p < NT; ++p) img[p * stride + o] = hv[p];
  if (ch.nkx) {  // rows of T as the A operand of T X: columns ij and, negated, ji
    __nv_bfloat16 mv[NT];
    split_bf16_n<NT>(-t, mv);
    const int rg = (ch.pk + 7) >> 3;
    const int64_t oi = ch.tmt_base + (int64_t)(cl.c_ij >> 5) * rg * kTcGroup + tc_off(u, cl.c_ij & 31);
    const int64_t oj = ch.tmt_base + (int64_t)(cl.c_ji >> 5) * rg * kTcGroup + tc_off(u, cl.c_ji & 31);
#pragma unroll
    for (int p = 0; p < NT; ++p) {
      img[p * stride + oi] = hv[p];
      img[p * stride + oj] = mv[p];
    }
  }
}
__device__ __forceinline__ void write_t_image(const ChanInfo &ch, int u, int w, const QuadCol &cl,
                                              double t, int nt, __nv_bfloat16 *img,
                                              int64_t stride) {
  if (nt == 3) write_t_image_n<3>(ch, u, w, cl, t, img, stride);
  else write_t_image_n<2>(ch, u, w, cl, t, img, stride);
}

// ------------------------------------------------------------------------------------------
// Fused assembly (calc.cpp:384-418 plus the remaps folded in):
//   value = V + D + R_ai,jb - R_aj,ib - R_bi,ja + R_bj,ia          (ring: the two sums S, side by side)
//         + 0.5 x_i t_ab,ji - 0.5 x_j t_ab,ij                       (h2pp_h1 gathers, algebraically)
//         + (-0.5 y_b) t_ab,ij - (-0.5 y_a) t_ba,ij                 (p2_p1hh gathers, algebraically)
//   t_new = mixing value/(e_i+e_j-e_a-e_b) + (1-mixing) t_old;  E += V t_new
// with D = V_pppp T from the ladder's planes plus 0.5 T X from hh_post_kernel (a K extension of the
// ladder for T X would make it wait for the hh ladder).
// ------------------------------------------------------------------------------------------
constexpr int kAsmPerThread = 2;  // table path: elements per thread of an ElemRange
struct StopState {  // what decides whether the device solve loop goes on
  int64_t iterations, stop_at;
  int32_t done, phase;
};
__device__ __forceinline__ StopState energy_reduce(const double *epart, int n, Control *ctl,
                                                   int flags, double *e_out);
// Condition of the device solve loop's WHILE node after an iteration: another iteration while
// the stop rule has not fired, below the launch's iteration limit, and (body_mixed) in the
// mixed phase or (FP64 body) past it.
__device__ __forceinline__ void loop_set_condition(const StopState &st,
                                                   cudaGraphConditionalHandle cond,
                                                   bool body_mixed) {
  const bool more = !st.done && st.iterations < st.stop_at;
  const bool mixed_phase = st.phase == 1;
  cudaGraphSetConditional(cond, (more && (body_mixed ? mixed_phase : !mixed_phase)) ? 1u : 0u);
}

// Work is organised over quads (u, w); one thread computes one quad from V, D and t at its
// packed position and the two ring sums, and writes the new packed amplitude (and, in a mixed
// iteration, its bf16 terms).  The energy gains 4 V t_new per quad.  Persistent CTAs stride over
// work items of up to kQuadPerItem quads of one channel.  Bound by the latency of three dependent
// loads (item, table rows, operands), so by how many threads are resident.
constexpr int kQuadPerItem = kAsmThreads;  // one quad per thread and item
constexpr int kAsmCTAsPerSM = 5;

// D of quad (u, w) at packed position p: the planes of its row tile in order, then T X.
__device__ __forceinline__ double quad_d(const LadderRows *__restrict__ lrows, int rt_off,
                                         const double *__restrict__ dp,
                                         const double *__restrict__ tx, int u, int w, int hs,
                                         int64_t p) {
  const LadderRows lr = lrows[rt_off + (u >> 7)];
  const double *d = dp + lr.base + (u & 127) * hs + w;
  const double x = __ldcg(tx + p);
  double v = __ldcg(d);
#pragma unroll 4
  for (int s = 1; s < lr.n; ++s) v += __ldcg(d + (int64_t)s * lr.stride);
  return v + x;
}

// value of element (ab, ij) (calc.cpp:384-418) with t_ab,ji = -t and t_ba,ij = -t:
//   V + D + (R_ai,jb + R_bj,ia) - (R_aj,ib + R_bi,ja) + 0.5 x_i t_ab,ji - 0.5 x_j t_ab,ij
//     + (-0.5 y_b) t_ab,ij - (-0.5 y_a) t_ba,ij
__device__ __forceinline__ double quad_value(double v, double dm, double2 s, double t, double xi,
                                             double xj, double ya, double yb, double den,
                                             double mixing) {
  double value = v;
  value += dm;
  value += s.x;
  value -= s.y;
  value += (0.5 * xi) * (-t);
  value -= (0.5 * xj) * t;
  value += (-0.5 * yb) * t;
  value -= (-0.5 * ya) * (-t);
  value = value / den;
  return mixing * value + (1. - mixing) * t;
}

// LOOP: launched as the last kernel of a device-solve-loop body (sets the WHILE condition);
// the variant without it is the one profilers can replay.
template <bool LOOP>
__global__ void __launch_bounds__(kAsmThreads, kAsmCTAsPerSM)
assemble_fused_kernel(const QuadItem *__restrict__ items, int n_items,
                      const ChanInfo *__restrict__ chans, const LadderRows *__restrict__ lrows,
                      const QuadRow *__restrict__ qrows, const QuadCol *__restrict__ qcols,
                      const double *__restrict__ vq, const double *__restrict__ dp,
                      const double *__restrict__ tx, const double *__restrict__ r_quad,
                      const double *__restrict__ xh, const double *__restrict__ yp, double *tq0,
                      double *tq1, double *__restrict__ epart, int32_t *ticket, Control *ctl,
                      __nv_bfloat16 *__restrict__ tkt_tc, int64_t tkt_tc_stride, int nt,
                      cudaGraphConditionalHandle cond, int loop_body, int gate) {
  // loop_body: 0 outside the device solve loop, 1 / 2 last kernel of its FP64 / mixed body,
  // where the CTA that applies the stop rule also sets the loop condition.  A skipped body
  // (stop rule fired, or the other precision's phase) ends its loop.
  __shared__ double scratch[32];
  __shared__ int last;
  if (skip_iteration(ctl, gate, kTrAssemble)) {
    if constexpr (LOOP)
      if (blockIdx.x == 0 && threadIdx.x == 0) cudaGraphSetConditional(cond, 0u);
    return;
  }
  const double *__restrict__ t_old = ctl->parity ? tq1 : tq0;
  double *__restrict__ t_new = ctl->parity ? tq0 : tq1;
  const double mixing = ctl->mixing;
  double corr = 0.0;
  for (int it = blockIdx.x; it < n_items; it += gridDim.x) {
    const QuadItem item = items[it];
    const int q = item.q0 + threadIdx.x;
    if (q >= item.q1) continue;
    // q / hk as a multiply-high by ceil(2^32 / hk) (Granlund-Montgomery): exact for
    // q < 2^32 / hk (q < 2^21, hk < 2^11 here); hk = 1 has no 32-bit multiplier.
    const int hk = item.hk;
    const uint32_t magic = hk > 1 ? 0xFFFFFFFFu / (uint32_t)hk + 1u : 0u;
    const int u = hk > 1 ? (int)__umulhi((uint32_t)q, magic) : q, w = q - u * hk;
    const int64_t p = item.q_off + (int64_t)u * item.hs + w;
    const QuadRow rw = qrows[item.pk_off + u];
    const QuadCol cl = qcols[item.qcol_off + w];
    const double tv = t_old[p], vv = __ldg(vq + p);
    const double2 ring = __ldcg(reinterpret_cast<const double2 *>(r_quad + 2 * p));
    const double dv = quad_d(lrows, item.rt_off, dp, tx, u, w, item.hs, p);
    // The one-body sums are small arrays every quad reads: through L1 (an L2-only load
    // would send every warp to the same few L2 slices).
    const double t1 = quad_value(vv, dv, ring, tv, xh[cl.i], xh[cl.j], yp[rw.pa], yp[rw.pb],
                                 cl.eij - rw.ea - rw.eb, mixing);
    t_new[p] = t1;
    if (nt) write_t_image(chans[item.ch], u, w, cl, t1, nt, tkt_tc, tkt_tc_stride);
    corr += 4.0 * (vv * t1);
  }
  const double sum = block_sum<kAsmThreads>(corr, scratch);
  trace_end(ctl, kTrAssemble);
  // The last CTA to finish sums the partials and applies the stop rule (no extra launch).
  if (threadIdx.x == 0) {
    epart[blockIdx.x] = sum;
    __threadfence();
    last = (atomicAdd(ticket, 1) == (int)gridDim.x - 1);
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  const StopState st = energy_reduce(epart, gridDim.x, ctl, 3, nullptr);
  if (threadIdx.x == 0) {
    *ticket = 0;
    if constexpr (LOOP) loop_set_condition(st, cond, loop_body == 2);
  }
}

// ---- Between the packed amplitudes and the reference's layout ----------------------------

// D of the ladder in the reference layout (t2Diff_pphh), from the ladder's planes and T X: a quad's
// four elements as +D, -D, -D, +D; rows a = b and columns i = j stay zero.
__global__ void __launch_bounds__(kAsmThreads)
expand_d_kernel(const QuadItem *__restrict__ items, const ChanInfo *__restrict__ chans,
                const LadderRows *__restrict__ lrows, const QuadRow *__restrict__ qrows,
                const QuadCol *__restrict__ qcols, const double *__restrict__ dp,
                const double *__restrict__ tx, double *__restrict__ d) {
  const QuadItem item = items[blockIdx.x];
  const int q = item.q0 + threadIdx.x;
  if (q >= item.q1) return;
  const int u = q / item.hk, w = q - u * item.hk;
  const double v = quad_d(lrows, item.rt_off, dp, tx, u, w, item.hs,
                          item.q_off + (int64_t)u * item.hs + w);
  const QuadRow rw = qrows[item.pk_off + u];
  const QuadCol cl = qcols[item.qcol_off + w];
  double *o = d + chans[item.ch].t_off;
  o[rw.o_ab + cl.c_ij] = v;
  o[rw.o_ab + cl.c_ji] = -v;
  o[rw.o_ba + cl.c_ij] = -v;
  o[rw.o_ba + cl.c_ji] = v;
}

// Quad of element (ab, ij): prow[ab] = 2 u (a < b), 2 u + 1 (a > b) or -1 (a = b), hcol[ij]
// alike; sign flips once per exchanged pair.  False: in no quad.
__device__ __forceinline__ bool quad_of(const ChanInfo &ch, const int32_t *__restrict__ prow,
                                        const int32_t *__restrict__ hcol, int ab, int ij, int &u,
                                        int &w, bool &neg) {
  const int r = prow[ch.pp_off + ab], c = hcol[ch.hh_off + ij];
  u = r >> 1;
  w = c >> 1;
  neg = ((r ^ c) & 1) != 0;
  return r >= 0 && c >= 0;
}

// Packed amplitudes -> t2_pphh in the reference's order (coalesced stores).
__global__ void __launch_bounds__(256)
expand_t_kernel(const ElemRange *__restrict__ ranges, const ChanInfo *__restrict__ chans,
                const int32_t *__restrict__ prow, const int32_t *__restrict__ hcol,
                const double *tq0, const double *tq1, const Control *ctl,
                double *__restrict__ t2) {
  const ElemRange rg = ranges[blockIdx.x];
  const ChanInfo &ch = chans[rg.ch];
  const double *t = ctl->parity ? tq1 : tq0;
  for (int64_t e = rg.e0 + threadIdx.x; e < rg.e1; e += blockDim.x) {
    const int64_t loc = e - ch.t_off;
    const int ab = (int)(loc / ch.hh), ij = (int)(loc - (int64_t)ab * ch.hh);
    int u, w;
    bool neg;
    double v = 0.0;
    if (quad_of(ch, prow, hcol, ab, ij, u, w, neg)) {
      v = t[ch.q_off + (int64_t)u * ch.hs + w];
      if (neg) v = -v;
    }
    t2[e] = v;
  }
}

// A value of the packed layout from its (ab, ij) elements of the reference layout (V_hhpp).
__global__ void __launch_bounds__(kAsmThreads)
pack_quads_kernel(const QuadItem *__restrict__ items, const ChanInfo *__restrict__ chans,
                  const QuadRow *__restrict__ qrows, const QuadCol *__restrict__ qcols,
                  const double *__restrict__ src, double *__restrict__ out) {
  const QuadItem item = items[blockIdx.x];
  const int q = item.q0 + threadIdx.x;
  if (q >= item.q1) return;
  const int u = q / item.hk, w = q - u * item.hk;
  out[item.q_off + (int64_t)u * item.hs + w] =
      src[chans[item.ch].t_off + qrows[item.pk_off + u].o_ab + qcols[item.qcol_off + w].c_ij];
}

// The bf16 operand image of a mixed handle's tensor-core ladder from the packed amplitudes,
// before a mixed iteration that follows something other than a mixed iteration.
__global__ void __launch_bounds__(kAsmThreads)
t_image_kernel(const QuadItem *__restrict__ items, const ChanInfo *__restrict__ chans,
               const QuadCol *__restrict__ qcols, const double *tq0, const double *tq1, const Control *ctl,
               __nv_bfloat16 *__restrict__ img, int64_t stride, int nt) {
  const QuadItem item = items[blockIdx.x];
  const int q = item.q0 + threadIdx.x;
  if (q >= item.q1) return;
  const int u = q / item.hk, w = q - u * item.hk;
  const double *t = ctl->parity ? tq1 : tq0;
  write_t_image(chans[item.ch], u, w, qcols[item.qcol_off + w],
                t[item.q_off + (int64_t)u * item.hs + w], nt, img, stride);
}

// Table path assembly: exactly calcChannelT2_pphh over the eight gathered chains.
__global__ void __launch_bounds__(kAsmThreads)
assemble_tables_kernel(const ElemRange *__restrict__ ranges, const ChanInfo *__restrict__ chans,
                       const int2 *__restrict__ pp_pairs, const int2 *__restrict__ hh_pairs,
                       const double *__restrict__ v_pphh, const double *__restrict__ dmat,
                       const double *__restrict__ gath, int64_t n_t,
                       const double *__restrict__ eps, const double *__restrict__ t_old,
                       double *__restrict__ t_new, double *__restrict__ epart, double mixing) {
  __shared__ double scratch[32];
  const ElemRange rg = ranges[blockIdx.x];
  const ChanInfo ch = chans[rg.ch];
  const int hh = ch.hh;
  double corr = 0.0;
  for (int64_t e = rg.e0 + threadIdx.x; e < rg.e1; e += kAsmThreads) {
    const int64_t loc = e - ch.t_off;
    const int ab = (int)(loc / hh), ij = (int)(loc - (int64_t)ab * hh);
    const int2 pab = pp_pairs[ch.pp_off + ab], pij = hh_pairs[ch.hh_off + ij];
    const double v = v_pphh[e];
    double value = v;
    value += dmat[e];
    value += gath[4 * n_t + e];  // ai_jb
    value -= gath[5 * n_t + e];  // aj_ib
    value -= gath[6 * n_t + e];  // bi_ja
    value += gath[7 * n_t + e];  // bj_ia
    value += gath[1 * n_t + e];  // jab_i
    value -= gath[0 * n_t + e];  // iab_j
    value += gath[3 * n_t + e];  // b_aij
    value -= gath[2 * n_t + e];  // a_bij
    value = value / (eps[pij.x] + eps[pij.y] - eps[pab.x] - eps[pab.y]);
    value = mixing * value + (1. - mixing) * t_old[e];
    t_new[e] = value;
    corr += v * value;
  }
  const double sum = block_sum<kAsmThreads>(corr, scratch);
  if (threadIdx.x == 0) epart[blockIdx.x] = sum;
}

// The eight mapFromDistributed gathers: out_k[e] = src_k[flat_k[e]].
__global__ void gather8_kernel(int64_t n_t, const int32_t *__restrict__ flat,
                               const double *__restrict__ hpp, const double *__restrict__ phh,
                               const double *__restrict__ phhp, double *__restrict__ out) {
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < n_t;
       e += (int64_t)gridDim.x * blockDim.x) {
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const double *src = k < 2 ? hpp : (k < 4 ? phh : phhp);
      out[k * n_t + e] = src[flat[k * n_t + e]];
    }
  }
}

// Chain::set + the five mapToDistributed scatters, plus the packed amplitudes (buffer `parity`
// of the control block).  An element that is not a number or infinite anywhere (also where no
// quad reads it) makes its quad, or the first quad of all, not a number, so that the next
// iteration reports it: `mark` is that second pass, launched after the first.
__global__ void map_to_kernel(const ElemRange *__restrict__ ranges, const ChanInfo *__restrict__ chans,
                              const int32_t *__restrict__ prow, const int32_t *__restrict__ hcol,
                              const int32_t *__restrict__ flat, int64_t n_t,
                              const double *__restrict__ t2, double *__restrict__ t2_old,
                              double *__restrict__ old_h2pp_h1, double *__restrict__ old_h1pp_h2,
                              double *__restrict__ old_p1_p2hh, double *__restrict__ old_p2_p1hh,
                              double *__restrict__ old_phhp, double *tq0, double *tq1,
                              int with_3body, const Control *ctl, int mark) {
  const ElemRange rg = ranges[blockIdx.x];
  const ChanInfo &ch = chans[rg.ch];
  double *tq = ctl->parity ? tq1 : tq0;
  for (int64_t e = rg.e0 + threadIdx.x; e < rg.e1; e += blockDim.x) {
    const double t = t2[e];
    if (mark && isfinite(t)) continue;
    const int64_t loc = e - ch.t_off;
    const int ab = (int)(loc / ch.hh), ij = (int)(loc - (int64_t)ab * ch.hh);
    int u, w;
    bool neg;
    const bool in = quad_of(ch, prow, hcol, ab, ij, u, w, neg);
    if (mark) {
      tq[in ? ch.q_off + (int64_t)u * ch.hs + w : 0] = __longlong_as_double(0x7ff8000000000000ll);
      continue;
    }
    if (t2_old != t2) t2_old[e] = t;
    if (with_3body) {
      old_h2pp_h1[flat[1 * n_t + e]] = t;  // jab_i
      old_h1pp_h2[flat[0 * n_t + e]] = t;  // iab_j
      old_p1_p2hh[flat[2 * n_t + e]] = t;  // a_bij
      old_p2_p1hh[flat[3 * n_t + e]] = t;  // b_aij
    }
    old_phhp[flat[4 * n_t + e]] = t;       // ai_jb
    if (in && prow[ch.pp_off + ab] == 2 * u && hcol[ch.hh_off + ij] == 2 * w)
      tq[ch.q_off + (int64_t)u * ch.hs + w] = t;
  }
}

// Sum of the per-CTA energy partials (Neumaier-compensated, fixed order) by one block of
// kEnergyThreads threads, then the reference's stop rule on the device.  flags: 1 = flip the
// amplitude buffer parity, 2 = count this as an iteration of the solve loop.
// Nothing overlaps it at the end of an iteration, so every memory round trip counts: the control
// block's fields are read together, beside the partial sums.  The state is thread 0's.
constexpr int kEnergyThreads = 256;
__device__ __forceinline__ void neumaier_add(double &s, double &c, double x) {
  const double t = s + x;
  c += fabs(s) >= fabs(x) ? (s - t) + x : (x - t) + s;
  s = t;
}
__device__ __forceinline__ StopState energy_reduce(const double *epart, int n, Control *ctl,
                                                   int flags, double *e_out) {
  constexpr int kWarps = kEnergyThreads / 32;
  __shared__ double ss[kWarps], cs[kWarps];
  Control c0;
  if (threadIdx.x == 0) {
    c0.e_prev = ctl->e_prev;
    c0.e_diff = ctl->e_diff;
    c0.tol = ctl->tol;
    c0.polish_rel = ctl->polish_rel;
    c0.iterations = ctl->iterations;
    c0.max_iters = ctl->max_iters;
    c0.polish_iters = ctl->polish_iters;
    c0.stop_at = ctl->stop_at;
    c0.active = ctl->active;
    c0.phase = ctl->phase;
    c0.done = ctl->done;
    c0.error = ctl->error;
    c0.parity = ctl->parity;
  }
  double s = 0.0, c = 0.0;
  for (int i = threadIdx.x; i < n; i += kEnergyThreads) neumaier_add(s, c, __ldcg(epart + i));
  // (s, c) pairs: within a warp by a fixed tree, then the warps' likewise.
#pragma unroll
  for (int w = 16; w > 0; w >>= 1) {
    c += __shfl_down_sync(0xffffffffu, c, w);
    neumaier_add(s, c, __shfl_down_sync(0xffffffffu, s, w));
  }
  if (threadIdx.x % 32 == 0) {
    ss[threadIdx.x / 32] = s;
    cs[threadIdx.x / 32] = c;
  }
  __syncthreads();
  if (threadIdx.x >= 32) return StopState{};
  s = threadIdx.x < kWarps ? ss[threadIdx.x] : 0.0;
  c = threadIdx.x < kWarps ? cs[threadIdx.x] : 0.0;
#pragma unroll
  for (int w = kWarps / 2; w > 0; w >>= 1) {
    c += __shfl_down_sync(0xffffffffu, c, w);
    neumaier_add(s, c, __shfl_down_sync(0xffffffffu, s, w));
  }
  StopState st{};
  if (threadIdx.x == 0) {
    const double corr = 0.25 * (s + c);
    if (e_out) *e_out = corr;
    if (flags & 2) {
      const double diff = corr - c0.e_prev;
      ctl->e_prev = corr;
      ctl->e_corr = corr;
      ctl->e_diff = diff;
      if (c0.iterations < 128) ctl->energies[c0.iterations] = corr;
      ctl->iterations = ++c0.iterations;
      if (c0.active && c0.phase == 2) ctl->polish_iters = c0.polish_iters + 1;
      if (!isfinite(corr)) {
        ctl->error = c0.error | kErrNonFinite;
        c0.done = 1;
      }
      if (c0.active && c0.phase == 1) {
        // Mixed phase: hand over to FP64 iterations once the energy change reaches the
        // rounding floor of the split-bf16 ladder, or stops shrinking.
        if (fabs(diff) <= fmax(c0.tol, c0.polish_rel * fabs(corr)) ||
            (c0.iterations > 2 && fabs(diff) >= fabs(c0.e_diff)))
          ctl->phase = c0.phase = 2;
        if (c0.iterations > c0.max_iters) c0.done = 1;
      } else if (fabs(diff) <= c0.tol || c0.iterations > c0.max_iters) {
        c0.done = 1;
      }
      if (c0.done) ctl->done = 1;
    }
    if (flags & 1) ctl->parity = c0.parity ^ 1;
    st = StopState{c0.iterations, c0.stop_at, c0.done, c0.phase};
  }
  return st;
}

// Last node of an iteration body of the device solve loop (a CUDA graph with WHILE conditional
// nodes) when the system has no assembly blocks: decides from the control block whether the
// loop runs another iteration.  body_mixed: the mixed-precision loop continues in phase 1 only;
// the FP64 loop never runs in phase 1.  Otherwise the fused assembly, the last kernel of every
// body, sets the condition (also when it skipped), so no loop can spin without progress: a
// body either advances `iterations` or clears its condition.
__global__ void loop_ctl_kernel(const Control *ctl, cudaGraphConditionalHandle cond,
                                int body_mixed) {
  pdl_enter();
  trace_start(ctl, kTrLoopCtl);
  if (threadIdx.x != 0) return;
  loop_set_condition(StopState{ctl->iterations, ctl->stop_at, ctl->done, ctl->phase}, cond,
                     body_mixed != 0);
}

// MBPT2 (MBPT2Corr.cpp:6-38) over the elements of the active channels, one CTA per range:
// epart[range] = sum <ij|v|ab>^2 / (e_i + e_j - e_a - e_b) (energy_reduce applies the 1/4), and
// with t_out the first-order amplitudes t_ab,ij = <ab|v|ij> / (e_i + e_j - e_a - e_b).
__global__ void __launch_bounds__(256)
mbpt2_kernel(const ElemRange *__restrict__ ranges, const ChanInfo *__restrict__ chans,
             const int2 *__restrict__ pp_pairs, const int2 *__restrict__ hh_pairs,
             const double *__restrict__ v_pphh, const double *__restrict__ eps,
             double *__restrict__ t_out, double *__restrict__ epart) {
  __shared__ double scratch[32];
  const ElemRange rg = ranges[blockIdx.x];
  const ChanInfo ch = chans[rg.ch];
  double acc = 0.0;
  for (int64_t e = rg.e0 + threadIdx.x; e < rg.e1; e += blockDim.x) {
    const int64_t loc = e - ch.t_off;
    const int ab = (int)(loc / ch.hh), ij = (int)(loc - (int64_t)ab * ch.hh);
    const int2 pab = pp_pairs[ch.pp_off + ab], pij = hh_pairs[ch.hh_off + ij];
    const double den = eps[pij.x] + eps[pij.y] - eps[pab.x] - eps[pab.y];
    const double v = v_pphh[e];
    acc += v * v / den;
    if (t_out) t_out[e] = v / den;
  }
  const double sum = block_sum<256>(acc, scratch);
  if (threadIdx.x == 0) epart[blockIdx.x] = sum;
}

__global__ void __launch_bounds__(kEnergyThreads)
energy_kernel(const double *__restrict__ epart, int n, Control *ctl, int flags, double *e_out,
              int gate) {
  if (skip_iteration(ctl, gate, kTrEnergy)) return;
  energy_reduce(epart, n, ctl, flags, e_out);
}

}  // namespace ccd

// t2Diff_pphh without the antisymmetry of T2, V_hhpp and V_hhhh that the packed kernels rely on
// (calc.cpp:141-202 element by element), for the stage calls and the table path, and the check that
// tells when it is needed.
#pragma once

#include "ccd_kernels.cuh"
#include "ccd_setup.cuh"

namespace ccd {

// Largest |src|, as bits (non-negative doubles order as integers; a NaN is above them all).
__global__ void __launch_bounds__(256)
max_abs_kernel(const double *__restrict__ src, int64_t n, unsigned long long *__restrict__ out) {
  unsigned long long m = 0;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < n;
       e += (int64_t)gridDim.x * blockDim.x)
    m = max(m, (unsigned long long)__double_as_longlong(fabs(src[e])));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0) atomicMax(out, m);
}

// Sets *flag where src (t2_pphh layout) is not antisymmetric in (a, b) or in (i, j).  Amplitudes of
// the table path are antisymmetric but for the rounding of their sums, hence the bound, far above
// that and as far below what the iteration's results are compared at.
constexpr double kAntisymmetry = 1e-12;  // of the largest element
__global__ void __launch_bounds__(256)
antisymmetry_kernel(const ElemRange *__restrict__ ranges, const ChanInfo *__restrict__ chans,
                    const int32_t *__restrict__ pp_swap, const int32_t *__restrict__ hh_swap,
                    const double *__restrict__ src, const unsigned long long *__restrict__ largest,
                    unsigned long long *__restrict__ flag) {
  const ElemRange rg = ranges[blockIdx.x];
  const ChanInfo &ch = chans[rg.ch];
  const double bound = kAntisymmetry * __longlong_as_double((long long)*largest);
  bool differs = false;
  for (int64_t e = rg.e0 + threadIdx.x; e < rg.e1; e += blockDim.x) {
    const int64_t loc = e - ch.t_off;
    const int ab = (int)(loc / ch.hh), ij = (int)(loc - (int64_t)ab * ch.hh);
    const int ba = pp_swap[ch.pp_off + ab], ji = hh_swap[ch.hh_off + ij];
    const double v = src[e];
    differs |= fabs(v + src[ch.t_off + (int64_t)ba * ch.hh + ij]) > bound ||
               fabs(v + src[ch.t_off + (int64_t)ab * ch.hh + ji]) > bound;
  }
  if (differs) *flag = 1;
}
// The same for the columns of V_hhhh, against the largest element of the channel (one CTA each; its
// rows need not be antisymmetric, see hh_records_kernel).
__global__ void __launch_bounds__(256)
antisymmetry_hhhh_kernel(const ChanInfo *__restrict__ chans, const int32_t *__restrict__ hh_swap,
                         const double *__restrict__ v_hhhh,
                         unsigned long long *__restrict__ flag) {
  __shared__ unsigned long long largest;
  const ChanInfo ch = chans[blockIdx.x];
  const double *v = v_hhhh + ch.vhh_off;
  if (threadIdx.x == 0) largest = 0;
  __syncthreads();
  unsigned long long m = 0;
  for (int e = threadIdx.x; e < ch.hh * ch.hh; e += blockDim.x)
    m = max(m, (unsigned long long)__double_as_longlong(fabs(v[e])));
  atomicMax(&largest, m);
  __syncthreads();
  const double bound = kAntisymmetry * __longlong_as_double((long long)largest);
  for (int e = threadIdx.x; e < ch.hh * ch.hh; e += blockDim.x) {
    const int kl = e / ch.hh, ij = e - kl * ch.hh;
    if (fabs(v[e] + v[kl * ch.hh + hh_swap[ch.hh_off + ij]]) > bound) *flag = 1;
  }
}

// X = V_hhhh + 0.5 V_hhpp T, hh x hh: a thread per element, blockIdx.x the channel.
__global__ void __launch_bounds__(256)
general_x_kernel(const ChanInfo *__restrict__ chans, const double *__restrict__ v_pphh,
                 const double *__restrict__ v_hhhh, const double *__restrict__ t,
                 double *__restrict__ x) {
  const ChanInfo &ch = chans[blockIdx.x];
  const int hh = ch.hh;
  for (int e = blockIdx.y * blockDim.x + threadIdx.x; e < hh * hh; e += gridDim.y * blockDim.x) {
    const int kl = e / hh, ij = e - kl * hh;
    const double *v = v_pphh + ch.t_off + kl, *tt = t + ch.t_off + ij;
    double p = 0.0;
    for (int64_t ab = 0; ab < ch.pp; ++ab) p = fma(v[ab * hh], tt[ab * hh], p);
    x[ch.vhh_off + e] = v_hhhh[ch.vhh_off + e] + 0.5 * p;
  }
}

// Element (u, w), u = a<b and w = c<d, of a channel's packed V: from the pp ladder's tiles (a
// symmetric channel's hold those on and above the diagonal blocks); a channel without strict hole
// pairs has no tiles: row-major where V came from the host, else from the model.
__device__ __forceinline__ double packed_v(const ChanInfo &ch, const double *__restrict__ v_t,
                                           const ModelDev &m, bool generated,
                                           const int32_t *__restrict__ kcol,
                                           const int2 *__restrict__ pp_pairs, int u, int w) {
  if (!ch.hk) {
    if (!generated) return v_t[ch.vkt_base + (int64_t)u * ch.pk + w];
    const int2 ab = pp_pairs[ch.pp_off + kcol[ch.pk_off + u]];
    const int2 cd = pp_pairs[ch.pp_off + kcol[ch.pk_off + w]];
    return tbme_dev(m, ab.x, ab.y, cd.x, cd.y);
  }
  if (ch.sym && w < kMaxBM * (u / kMaxBM)) {
    const int r = u;
    u = w;
    w = r;
  }
  const int mt = u / kMaxBM, rows = min(kMaxBM, ch.pk - mt * kMaxBM);
  return v_t[ch.vkt_base + ladder_chunk(ch.sym, ch.nkc, mt, w / kBK, rows) +
             (w % kBK) * ladder_as(rows) + u % kMaxBM];
}

// D = 0.5 V_pppp T + 0.5 T X, a thread per element: sum over c<d of V (T[cd] - T[dc]).  Only V_pppp
// is taken as antisymmetric.  A path for inputs that no solve produces: plain loads, whose V
// is one broadcast and T one coalesced read per warp and row.
__global__ void __launch_bounds__(256)
general_d_kernel(const ElemRange *__restrict__ ranges, const ChanInfo *__restrict__ chans,
                 const int32_t *__restrict__ prow, const int32_t *__restrict__ kcol,
                 const int32_t *__restrict__ pp_swap, const int2 *__restrict__ pp_pairs,
                 const double *__restrict__ v_t, ModelDev m, bool generated,
                 const double *__restrict__ x, const double *__restrict__ t,
                 double *__restrict__ d) {
  const ElemRange rg = ranges[blockIdx.x];
  const ChanInfo &ch = chans[rg.ch];
  const int hh = ch.hh;
  for (int64_t e = rg.e0 + threadIdx.x; e < rg.e1; e += blockDim.x) {
    const int64_t loc = e - ch.t_off;
    const int ab = (int)(loc / hh), ij = (int)(loc - (int64_t)ab * hh);
    const int r = prow[ch.pp_off + ab];
    const double *tt = t + ch.t_off;
    double vt = 0.0, tx = 0.0;
    for (int w = 0; r >= 0 && w < ch.pk; ++w) {
      const int cd = kcol[ch.pk_off + w], dc = pp_swap[ch.pp_off + cd];
      vt = fma(packed_v(ch, v_t, m, generated, kcol, pp_pairs, r >> 1, w),
               tt[(int64_t)cd * hh + ij] - tt[(int64_t)dc * hh + ij], vt);
    }
    if (r & 1) vt = -vt;  // row ba (r >= 0; rows a = b have vt = 0)
    for (int kl = 0; kl < hh; ++kl)
      tx = fma(tt[(int64_t)ab * hh + kl], x[ch.vhh_off + kl * hh + ij], tx);
    d[e] = 0.5 * vt + 0.5 * tx;
  }
}

}  // namespace ccd

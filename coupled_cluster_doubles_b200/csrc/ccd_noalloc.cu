// ccdgpu_calc_channel_t2diff_pphh_noalloc: the ladder term of one regular channel,
// computed without allocating any memory.
//
// Some callers cannot call cudaMalloc: a host that owns every byte of device memory through
// its own pool or budget and forbids a library to take more, or code that must not perturb
// the allocator state between calls.  This entry point serves them.  The caller passes all
// inputs and outputs as device buffers, and the split-K intermediate lives in a fixed
// file-scope device array that the library carries (kNoAllocScratchDoubles doubles, 2 MiB per
// GPU that loads the library, held until the process exits).
//
// Scratch layout (doubles): [0, 32) unused, [32, 32 + hh^2) X, then nslices * hh^2 partial
// products, nslices = ceil(pp / 64).
#include <cuda_runtime.h>

#include <cstdint>
#include <mutex>

#include "ccd_device.cuh"
#include "ccdgpu.h"

namespace {

using ccd::dmma_16816;

constexpr int64_t kNoAllocScratchDoubles = int64_t(1) << 18;  // 2 MiB
constexpr int kSliceRows = 64;
constexpr int kThreads = 256;
constexpr int kMaxDevices = 64;
constexpr int kMaxHH = 72;

static __device__ __align__(256) double g_noalloc_scratch[kNoAllocScratchDoubles];

double *g_scratch_ptr[kMaxDevices] = {};
std::mutex g_setup_mutex;

// Partial products of X over 64-row slices of the pp index, one CTA per slice: the slice's part
// of V_hhpp and T goes to shared memory once (K-major, row stride hh rounded up to 16 plus 4
// doubles: conflict-free fragment loads; zero past hh and past the slice) and each warp takes
// 16 x 8 tiles of the hh x hh product on the FP64 MMA (m16n8k16, at most four steps).  A channel
// of one slice has its X finished here; the others are summed by noalloc_x_sum_kernel.
// At hh = 54 a thread-per-element loop over shared memory spent 2 * 64 loads an element and was
// as long as the rest of the call.
__host__ __device__ inline int x_ld(int hh) { return ((hh + 15) & ~15) + 4; }
__global__ void __launch_bounds__(kThreads)
noalloc_x_kernel(const double *__restrict__ v_hhpp, const double *__restrict__ t2,
                 const double *__restrict__ v_hhhh, int pp, int hh, double *scratch) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  extern __shared__ double sm[];
  const int slice = blockIdx.x, k0 = slice * kSliceRows, ld = x_ld(hh), hp = ld - 4;
  const int rows = min(kSliceRows, pp - k0), rows16 = (rows + 15) & ~15, nout = hh * hh;
  double *Vs = sm, *Ts = sm + kSliceRows * ld;  // Vs[k][kl] = V_hhpp[kl][k0+k], Ts[k][ij]
  for (int e = threadIdx.x; e < kSliceRows * hp; e += kThreads) {
    const int k = e & (kSliceRows - 1), c = e / kSliceRows;  // V: coalesced over k
    if (k < rows16) Vs[k * ld + c] = (k < rows && c < hh) ? v_hhpp[(int64_t)c * pp + k0 + k] : 0.0;
  }
  for (int e = threadIdx.x; e < rows16 * hp; e += kThreads) {
    const int k = e / hp, c = e - k * hp;  // T: coalesced over the columns
    Ts[k * ld + c] = (k < rows && c < hh) ? t2[(int64_t)(k0 + k) * hh + c] : 0.0;
  }
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int n8 = (hh + 7) >> 3, items = (hp >> 4) * n8;
  const bool whole = gridDim.x == 1;
  double *x = scratch + 32, *part = x + nout + (int64_t)slice * nout;
  for (int it = warp; it < items; it += kThreads / 32) {
    const int mt = it / n8, nt = it - mt * n8;
    double acc[4] = {0.0, 0.0, 0.0, 0.0};
    for (int k16 = 0; k16 < rows16; k16 += 16) {
      double a[8], b[4];
#pragma unroll
      for (int i = 0; i < 8; ++i)
        a[i] = Vs[(k16 + t + 4 * (i / 2)) * ld + 16 * mt + g + 8 * (i % 2)];
#pragma unroll
      for (int q = 0; q < 4; ++q) b[q] = Ts[(k16 + t + 4 * q) * ld + 8 * nt + g];
      dmma_16816(acc, a, b);
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int kl = 16 * mt + g + 8 * (q >> 1), ij = 8 * nt + 2 * t + (q & 1);
      if (kl < hh && ij < hh) {
        const int idx = kl * hh + ij;
        if (whole) x[idx] = 0.5 * acc[q] + v_hhhh[idx];
        else part[idx] = acc[q];
      }
    }
  }
}

// X = V_hhhh + 0.5 * sum of the slices in slice order, one element per thread, a block of
// slices' loads in flight ahead of their additions.  (The last CTA of the product kernel did
// this alone: hh^2 / 256 elements per thread, one after another.)
__global__ void __launch_bounds__(kThreads)
noalloc_x_sum_kernel(const double *__restrict__ v_hhhh, int hh, int nslices, double *scratch) {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const int nout = hh * hh, idx = blockIdx.x * kThreads + threadIdx.x;
  if (idx >= nout) return;
  double *x = scratch + 32;
  const double *part = x + nout + idx;
  double p = 0.0;
  int s = 0;
  for (; s + 16 <= nslices; s += 16) {
    double v[16];
#pragma unroll
    for (int k = 0; k < 16; ++k) v[k] = __ldcg(part + (int64_t)(s + k) * nout);
#pragma unroll
    for (int k = 0; k < 16; ++k) p += v[k];
  }
  for (; s < nslices; ++s) p += __ldcg(part + (int64_t)s * nout);
  x[idx] = 0.5 * p + v_hhhh[idx];
}

// D = 0.5 V_pppp T + 0.5 T X (the two dgemm calls of calc.cpp:167-201) on the FP64 MMA: one CTA
// per 16 rows, so that a channel of some hundred rows already reaches most SMs without partial
// sums in global memory; its warps (16, or 8 where the accumulators need their registers) split
// K (pp, then hh) in steps of 16 and their partial tiles are added in a fixed order through
// shared memory.  C = 8-column tiles.  Operands come
// straight from global memory: a step reads V once (8 rows of 32 contiguous bytes per load)
// and T, which all CTAs share, from L2.  Launched programmatically: V T, which needs no X, starts
// with the X kernel in a channel of one slice, else beside the sum of the slices (which waits for
// the products before it lets this kernel start).  The whole call at pp = 1796, hh = 54 (369
// MFLOP, 28 MB): 37 us, 211 us with one thread per element (two loads a multiply-add); bound by
// the FP64 MMA of the 113 CTAs (13 us) and the L1 path of their fragment loads.
__host__ __device__ constexpr int d_warps(int c) { return c <= 4 ? 16 : 8; }
template <int C>
__global__ void __launch_bounds__(d_warps(C) * 32)
noalloc_d_kernel(const double *__restrict__ v_pppp, const double *__restrict__ t2, int pp, int hh,
                 const double *scratch, double *__restrict__ d) {
  constexpr int kDWarps = d_warps(C);
  __shared__ double red[kDWarps / 2][16 * 8 * C];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int64_t r0 = (int64_t)blockIdx.x * 16;
  double acc[C][4];
#pragma unroll
  for (int c = 0; c < C; ++c) acc[c][0] = acc[c][1] = acc[c][2] = acc[c][3] = 0.0;
  // acc += A[r0 + 16 rows][K] B[K][hh], this warp's steps of 16.
  auto gemm = [&](const double *A, const double *B, int K) {
    const double *a0 = A + (r0 + g) * K, *a1 = a0 + (int64_t)8 * K;
    const bool in0 = r0 + g < pp, in1 = r0 + g + 8 < pp;
#pragma unroll 2
    for (int k0 = 16 * warp; k0 < K; k0 += 16 * kDWarps) {
      double a[8];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int k = k0 + t + 4 * i;
        a[2 * i] = (in0 && k < K) ? a0[k] : 0.0;
        a[2 * i + 1] = (in1 && k < K) ? a1[k] : 0.0;
      }
#pragma unroll
      for (int c = 0; c < C; ++c) {
        double b[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const int k = k0 + t + 4 * q, col = 8 * c + g;
          b[q] = (k < K && col < hh) ? B[(int64_t)k * hh + col] : 0.0;
        }
        dmma_16816(acc[c], a, b);
      }
    }
  };
  gemm(v_pppp, t2, pp);
  asm volatile("griddepcontrol.wait;" ::: "memory");
  gemm(t2, scratch + 32, hh);
  // Partial tiles of the upper half of the warps onto the lower half, halving each round.
  double *mine = red[warp % (kDWarps / 2)] + lane * 4 * C;
#pragma unroll
  for (int h = kDWarps / 2; h >= 1; h >>= 1) {
    if (warp >= h && warp < 2 * h)
#pragma unroll
      for (int c = 0; c < C; ++c)
#pragma unroll
        for (int q = 0; q < 4; ++q) red[warp - h][lane * 4 * C + 4 * c + q] = acc[c][q];
    __syncthreads();
    if (warp < h)
#pragma unroll
      for (int c = 0; c < C; ++c)
#pragma unroll
        for (int q = 0; q < 4; ++q) acc[c][q] += mine[4 * c + q];
    __syncthreads();
  }
  if (warp) return;
#pragma unroll
  for (int c = 0; c < C; ++c)
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int64_t row = r0 + g + 8 * (q >> 1);
      const int col = 8 * c + 2 * t + (q & 1);
      if (row < pp && col < hh) d[row * hh + col] = 0.5 * acc[c][q];
    }
}

using DKernel = void (*)(const double *, const double *, int, int, const double *, double *);
DKernel d_kernel_of(int hh) {
  static const DKernel k[] = {noalloc_d_kernel<1>, noalloc_d_kernel<2>, noalloc_d_kernel<3>,
                              noalloc_d_kernel<4>, noalloc_d_kernel<5>, noalloc_d_kernel<6>,
                              noalloc_d_kernel<7>, noalloc_d_kernel<8>, noalloc_d_kernel<9>};
  return k[(hh - 1) / 8];
}

// Launch that may begin before the stream's previous kernel has finished (both wait in
// griddepcontrol.wait before they read its results).
template <typename... KArgs, typename... Args>
cudaError_t launch_dependent(void (*kernel)(KArgs...), unsigned grid, unsigned block,
                             cudaStream_t st, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(block);
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
}

// Device address of the scratch array for the current device, looked up once per device.
int scratch_for_current_device(double **out) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) {
    (void)cudaGetLastError();
    return CCDGPU_ERR_NO_DEVICE;
  }
  if (dev < 0 || dev >= kMaxDevices) return CCDGPU_ERR_UNSUPPORTED;
  std::lock_guard<std::mutex> lock(g_setup_mutex);
  if (!g_scratch_ptr[dev]) {
    double *p = nullptr;
    const cudaError_t e = cudaGetSymbolAddress(reinterpret_cast<void **>(&p), g_noalloc_scratch);
    if (e != cudaSuccess || !p) {
      (void)cudaGetLastError();
      return CCDGPU_ERR_CUDA;
    }
    // Dynamic shared memory of the X kernel at the largest supported hh (72).
    if (cudaFuncSetAttribute(noalloc_x_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             2 * kSliceRows * x_ld(kMaxHH) * (int)sizeof(double)) !=
        cudaSuccess) {
      (void)cudaGetLastError();
      return CCDGPU_ERR_CUDA;
    }
    g_scratch_ptr[dev] = p;
  }
  *out = g_scratch_ptr[dev];
  return CCDGPU_OK;
}

}  // namespace

extern "C" int ccdgpu_calc_channel_t2diff_pphh_noalloc(const double *v_pppp, const double *v_hhpp,
                                                       const double *v_hhhh, const double *t2,
                                                       double *d, int64_t pp, int64_t hh,
                                                       void *stream) {
  if (!v_pppp || !v_hhpp || !v_hhhh || !t2 || !d || pp < 1 || hh < 1)
    return CCDGPU_ERR_INVALID_ARGUMENT;
  const int64_t nslices = (pp + kSliceRows - 1) / kSliceRows;
  if (hh > kMaxHH || pp > (int64_t(1) << 20) || 32 + (nslices + 1) * hh * hh > kNoAllocScratchDoubles)
    return CCDGPU_ERR_UNSUPPORTED;  // beyond the fixed scratch capacity
  double *scratch = nullptr;
  int rc = scratch_for_current_device(&scratch);
  if (rc) return rc;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const size_t smem = (size_t)2 * kSliceRows * x_ld((int)hh) * sizeof(double);
  noalloc_x_kernel<<<(unsigned)nslices, kThreads, smem, st>>>(v_hhpp, t2, v_hhhh, (int)pp,
                                                              (int)hh, scratch);
  cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess && nslices > 1)
    e = launch_dependent(noalloc_x_sum_kernel, (unsigned)((hh * hh + kThreads - 1) / kThreads),
                         kThreads, st, v_hhhh, (int)hh, (int)nslices, scratch);
  if (e == cudaSuccess)
    e = launch_dependent(d_kernel_of((int)hh), (unsigned)((pp + 15) / 16), 32 * d_warps((int)(hh + 7) / 8), st,
                         v_pppp, t2, (int)pp, (int)hh, (const double *)scratch, d);
  if (e != cudaSuccess) {
    (void)cudaGetLastError();
    return e == cudaErrorMemoryAllocation ? CCDGPU_ERR_OUT_OF_MEMORY : CCDGPU_ERR_CUDA;
  }
  return CCDGPU_OK;
}

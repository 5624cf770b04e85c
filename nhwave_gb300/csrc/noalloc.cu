// noalloc.cu -- nhw_estimate_dt_noalloc: the Courant time step of
// estimate_dt computed on device arrays that the caller owns, with the
// reduction's scratch in a fixed device array of this library instead of
// memory that the library allocates.
//
// Who needs it: a host model that keeps its fields in device memory that it
// does not get from cudaMalloc -- a Fortran code whose arrays belong to the
// OpenACC or CUDA Fortran runtime, a framework whose caching allocator owns
// the GPU -- and that cannot let a library call cudaMalloc/cudaFree behind
// its back: those calls synchronise the device, stalling the caller's other
// streams, and they draw on a memory budget that such callers fix up front.
// The handle-based entry points allocate a scenario arena at nhw_create; this
// one allocates nothing and keeps no per-call state on the host.
#include <cuda_runtime.h>

#include <algorithm>
#include <mutex>
#include <string>

#include "../../include/nhwave_gb300.h"
#include "state.h"

namespace nhw {

void set_last_error(const std::string& s);

namespace {

constexpr int kNaThreads = 256;
constexpr int kNaMaxBlocks = 8192;                                                   // partial minima held
constexpr long long kNaMaxCells = 16777216;
constexpr int kNaCounter = kNaMaxBlocks;                                             // counter slot

// The scratch: one partial minimum per block, then a 256-byte line whose
// first word counts the blocks that have finished.  65,792 bytes, held on
// every device that loads the library until the process exits.  Host code
// must not use this name as an address; it takes the address from
// cudaGetSymbolAddress (scratch_on_current_device).
static __device__ __align__(256) double g_dt_scratch[kNaMaxBlocks + 32];

// Running minimum m updated by a candidate x the way the reference does
// (src/nhwave.F:3730-3746, `if(dxonu<tmp2) tmp2=dxonu`): a NaN candidate fails
// the comparison and leaves m as it was.
__device__ __forceinline__ double na_min(double m, double x) { return x < m ? x : m; }
__device__ __forceinline__ double na_max(double a, double b) { return a > b ? a : b; }

// |x| of a finite or infinite x as an integer that orders as |x| does (the
// bit patterns of non-negative doubles are ordered); -1 for NaN, which every
// other value exceeds, so that a maximum skips it
__device__ __forceinline__ long long abs_bits(double x) {
  const long long b = __double_as_longlong(x) & 0x7fffffffffffffffll;
  return b > 0x7ff0000000000000ll ? -1ll : b;
}
__device__ __forceinline__ long long max_ll(long long a, long long b) { return a > b ? a : b; }

// a double as an integer of the same order (no NaN), and back: the minima are
// reduced without the FP64 pipe, whose latency is most of a small grid's time
__device__ __forceinline__ long long order_key(double x) {
  const long long b = __double_as_longlong(x);
  return b ^ ((b >> 63) & 0x7fffffffffffffffll);
}
__device__ __forceinline__ double from_key(long long k) {
  return __longlong_as_double(k ^ ((k >> 63) & 0x7fffffffffffffffll));
}

// a >= b where b is a normal number that no rounding to zero or infinity made
__device__ __forceinline__ bool above(double a, double b) {
  const unsigned long long lo = 0x0010000000000000ull, hi = 0x7ff0000000000000ull;   // bits of 2^-1022 and infinity
  return a >= b && (unsigned long long)__double_as_longlong(b) - lo < hi - lo;
}

// the block's minimum of m and, with kAll, maxima of u and v, valid in thread 0
template <bool kAll>
__device__ __forceinline__ void block_reduce(long long& m, long long& u, long long& v) {
  __shared__ long long sh[3][kNaThreads / 32];
  for (int o = 16; o > 0; o >>= 1) {
    m = min(m, __shfl_down_sync(0xffffffffu, m, o));
    if (kAll) {
      u = max_ll(u, __shfl_down_sync(0xffffffffu, u, o));
      v = max_ll(v, __shfl_down_sync(0xffffffffu, v, o));
    }
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  __syncthreads();   // sh may still be read from the call before
  if (lane == 0) {
    sh[0][warp] = m;
    if (kAll) {
      sh[1][warp] = u;
      sh[2][warp] = v;
    }
  }
  __syncthreads();
  if (threadIdx.x == 0)
    for (int w = 1; w < kNaThreads / 32; ++w) {
      m = min(m, sh[0][w]);
      if (kAll) {
        u = max_ll(u, sh[1][w]);
        v = max_ll(v, sh[2][w]);
      }
    }
}

// Same values as the handle's estimate_dt (src/nhwave.F:3694-3874 with
// viscous and slide limits off): tmp2 = min over interior cells of
// dx/max(|U|+sqrt(g D), Small), dy/max(|V|+sqrt(g D), Small) and
// dsig(k) D/max(|W|, Small); dt = min(1.05 dt_old, CFL tmp2, Large, DT_MAX).
// Arrays are the reference's ghosted Fortran ones: U(Mloc,Nloc,Kloc),
// D(Mloc,Nloc), dsig(Kloc) with Mloc = Mglob+4 (two ghost cells a side).
//
// A thread takes kc levels of a column.  Rounded sums and quotients are
// monotone, so the smallest dx/(|U| + sqrt(g D)) of a block is that of the
// column whose max |U| + sqrt(g D) is largest: one square root a thread and two
// divisions a block instead of two and three a cell, the maxima kept in
// integers off the FP64 pipe (1.2 TFLOP/s on GB300).  The dsig D / |W| of the
// levels are divided only where products, with a margin far above their
// rounding, do not show the smallest of them to be above dx/(|U| + sqrt(g D))
// or its y counterpart; products out of range and negative dsig show nothing.  Read once, coalesced along i: bound by the launch on
// small grids and by HBM on large ones (GB300, a call in a graph with its
// memset: 256 x 8 x 10 33.1 -> 10.4 us, 1024 x 64 x 20 129 -> 18.6 us,
// 600 x 300 x 24 348 -> 30.9 us, whose bytes alone take 0.1, 5 and 15 us).
__global__ void __launch_bounds__(kNaThreads)
k_dt_min_noalloc(const double* __restrict__ U, const double* __restrict__ V, const double* __restrict__ W,
                 const double* __restrict__ D, const double* __restrict__ dsig, int M, int N, int K, int kc,
                 double dx, double dy, double cfl, double dt_old, double dt_max, double* __restrict__ dt_out,
                 double* __restrict__ scratch) {
  const long long Ml = M + 2 * NG, lev = Ml * (N + 2 * NG);
  const unsigned cols = (unsigned)M * (unsigned)N;
  const unsigned items = cols * (unsigned)((K + kc - 1) / kc);   // at most kNaMaxCells
  double m = kLarge;
  long long bu = -1ll, bv = -1ll;   // largest |U| + sqrt(g D), |V| + sqrt(g D) so far
  for (unsigned t = blockIdx.x * kNaThreads + threadIdx.x; t < items; t += gridDim.x * kNaThreads) {
    const unsigned ch = t / cols, col = t - ch * cols, jj = col / (unsigned)M;
    const long long c2 = NG + (int)(col - jj * (unsigned)M) + Ml * (NG + (int)jj);
    const int k0 = (int)ch * kc, k1 = min(K, k0 + kc);
    const double Dq = D[c2];
    long long u = -1ll, v = -1ll, w = -1ll, sg = 0x7fffffffffffffffll;
    const long long c3 = c2 + lev * (NG + k0);
#pragma unroll 4
    for (int k = k0; k < k1; ++k) {
      const long long c = c3 + lev * (k - k0);
      u = max_ll(u, abs_bits(U[c]));
      v = max_ll(v, abs_bits(V[c]));
      w = max_ll(w, abs_bits(W[c]));
      sg = min(sg, __double_as_longlong(dsig[NG + k]));   // as integers: a negative one comes first
    }
    const double s = sqrt(kGrav * Dq);
    const double tu = u < 0 ? kSmall : na_max(__longlong_as_double(u) + s, kSmall);
    const double tv = v < 0 ? kSmall : na_max(__longlong_as_double(v) + s, kSmall);
    bu = max_ll(bu, __double_as_longlong(tu));
    bv = max_ll(bv, __double_as_longlong(tv));
    const double a = __longlong_as_double(sg) * Dq, wm = w < 0 ? kSmall : na_max(__longlong_as_double(w), kSmall);
    const double wf = wm * 1.0000001;
    if (sg < 0 || !(above(a * tu, dx * wf) || above(a * tv, dy * wf)))
      for (int k = k0; k < k1; ++k) m = na_min(m, dsig[NG + k] * Dq / na_max(fabs(W[c3 + lev * (k - k0)]), kSmall));
  }
  long long key = order_key(m);
  block_reduce<true>(key, bu, bv);
  __shared__ bool last;
  if (threadIdx.x == 0) {
    m = from_key(key);
    if (bu >= 0) m = na_min(m, dx / __longlong_as_double(bu));
    if (bv >= 0) m = na_min(m, dy / __longlong_as_double(bv));
    scratch[blockIdx.x] = m;
    __threadfence();
    const unsigned prev = atomicAdd(reinterpret_cast<unsigned*>(scratch + kNaCounter), 1u);
    last = prev == gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  key = order_key(kLarge);
  for (unsigned b = threadIdx.x; b < gridDim.x; b += kNaThreads)
    key = min(key, order_key(reinterpret_cast<volatile double*>(scratch)[b]));
  block_reduce<false>(key, bu, bv);
  if (threadIdx.x == 0) {
    const double dt_growth = (double)1.05f * dt_old;
    dt_out[0] = na_min(na_min(na_min(dt_growth, cfl * from_key(key)), kLarge), dt_max);
  }
}

constexpr int kNaDevices = 64;
std::mutex g_na_mu;
double* g_na_ptr[kNaDevices] = {};

// Device address of g_dt_scratch on the current device, looked up once per
// device (the first call on a device does this set-up).
int scratch_on_current_device(double** out) {
  int dev = -1;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) {
    set_last_error(std::string("nhw_estimate_dt_noalloc: cudaGetDevice: ") + cudaGetErrorString(e));
    return NHW_ERR_CUDA;
  }
  std::lock_guard<std::mutex> g(g_na_mu);
  if (dev >= 0 && dev < kNaDevices && g_na_ptr[dev]) {
    *out = g_na_ptr[dev];
    return NHW_OK;
  }
  void* p = nullptr;
  e = cudaGetSymbolAddress(&p, g_dt_scratch);
  if (e != cudaSuccess || !p) {
    set_last_error(std::string("nhw_estimate_dt_noalloc: cudaGetSymbolAddress: ") + cudaGetErrorString(e));
    return NHW_ERR_CUDA;
  }
  if (dev >= 0 && dev < kNaDevices) g_na_ptr[dev] = static_cast<double*>(p);
  *out = static_cast<double*>(p);
  return NHW_OK;
}

// Device memory of the current device, or managed memory.  Device memory of
// another GPU is refused: without peer access the kernel's loads would fault.
bool on_device(const void* p, int dev) {
  cudaPointerAttributes a{};
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  if (a.type == cudaMemoryTypeManaged) return true;
  return a.type == cudaMemoryTypeDevice && a.device == dev;
}

}  // namespace
}  // namespace nhw

extern "C" int nhw_estimate_dt_noalloc(const double* U, const double* V, const double* W, const double* D,
                                       const double* dsig, int32_t Mglob, int32_t Nglob, int32_t Kglob,
                                       double dx, double dy, double cfl, double dt_old, double dt_max,
                                       double* dt_out, void* stream) {
  using namespace nhw;
  if (!U || !V || !W || !D || !dsig || !dt_out) {
    set_last_error("nhw_estimate_dt_noalloc: null array");
    return NHW_ERR_ARG;
  }
  if (Mglob < 1 || Nglob < 1 || Kglob < 1 || !(dx > 0.0) || !(dy > 0.0)) {
    set_last_error("nhw_estimate_dt_noalloc: grid sizes and dx, dy must be positive");
    return NHW_ERR_ARG;
  }
  const long long n = (long long)Mglob * Nglob * Kglob;
  if (n > kNaMaxCells) {
    set_last_error("nhw_estimate_dt_noalloc: Mglob*Nglob*Kglob = " + std::to_string(n) +
                   " interior cells exceeds the limit of " + std::to_string(kNaMaxCells) +
                   " that its static device scratch holds");
    return NHW_ERR_ARG;
  }
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess) {
    cudaGetLastError();
    set_last_error("nhw_estimate_dt_noalloc: no current CUDA device");
    return NHW_ERR_CUDA;
  }
  for (const void* p : {(const void*)U, (const void*)V, (const void*)W, (const void*)D, (const void*)dsig,
                        (const void*)dt_out})
    if (!on_device(p, dev)) {
      set_last_error("nhw_estimate_dt_noalloc: every array must be device memory of the current device "
                     "(device " + std::to_string(dev) + ") or managed memory");
      return NHW_ERR_ARG;
    }
  double* scratch = nullptr;
  int rc = scratch_on_current_device(&scratch);
  if (rc) return rc;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  // the blocks-done counter must start at zero; partial minima are all rewritten
  cudaError_t e = cudaMemsetAsync(scratch + kNaCounter, 0, sizeof(unsigned), s);
  if (e != cudaSuccess) {
    set_last_error(std::string("nhw_estimate_dt_noalloc: cudaMemsetAsync: ") + cudaGetErrorString(e));
    return NHW_ERR_CUDA;
  }
  // whole columns where there are enough of them to fill the GPU's 152 SMs
  // (one square root a column), else as many chunks of levels as fill it
  const long long cols = (long long)Mglob * Nglob, fill = 152 * 512;
  const long long chunks = std::min<long long>(Kglob, (fill + cols - 1) / cols);
  const int kc = (int)((Kglob + chunks - 1) / chunks);
  const long long items = (long long)Mglob * Nglob * ((Kglob + kc - 1) / kc);
  const unsigned nb = (unsigned)std::min<long long>(kNaMaxBlocks, (items + kNaThreads - 1) / kNaThreads);
  k_dt_min_noalloc<<<nb, kNaThreads, 0, s>>>(U, V, W, D, dsig, Mglob, Nglob, Kglob, kc, dx, dy, cfl, dt_old, dt_max,
                                             dt_out, scratch);
  e = cudaGetLastError();
  if (e != cudaSuccess) {
    set_last_error(std::string("nhw_estimate_dt_noalloc: launch: ") + cudaGetErrorString(e));
    return NHW_ERR_CUDA;
  }
  return NHW_OK;
}

// Binned power spectrum on the device, the estimator of flowpm/pk.py:7-103
// (_initialize_pk / power_spectrum):
//   P[b] = (sum_{modes in bin b} W |F(k)|^2) / (sum_{modes in bin b} W)
//          * prod(boxsize) / (nx ny nz)^2,     b = 1 .. nedges - 1
// where F is the unnormalised FFT of the field, the bin of a mode is
// numpy.digitize(|k|, edges) with edges = kmin + n dk (n < nedges) and
// |k| = sqrt(sum_d (2 pi i_d / L_d)^2), and W is the reference's weight on
// the full spectrum: 1 on the z planes 0 and nz - 1, 2 elsewhere.  The sums
// run over the half spectrum of an R2C transform, each mode standing for
// itself and its Hermitian mirror (full-spectrum z index nz - l).
#include <cufft.h>

#include <atomic>
#include <map>
#include <mutex>
#include <tuple>

#include "fpm_kernels.cuh"

namespace fpm {

struct PkGeom {
  int nx, ny, nz, nzh;
  double vx, vy, vz;  // 2 pi / L_d: k_d = i_d * v_d
  double kmin, dk;
  int nedges;
};

__device__ __forceinline__ double pk_edge(const PkGeom& g, int n) {
  return g.kmin + (double)n * g.dk;  // numpy.arange(kmin, kmax, dk)[n]
}

// numpy.digitize(x, edges): number of edges <= x.
__device__ __forceinline__ int pk_bin(const PkGeom& g, double x) {
  int b = (int)floor((x - g.kmin) / g.dk) + 1;
  b = b < 0 ? 0 : (b > g.nedges ? g.nedges : b);
  while (b > 0 && x < pk_edge(g, b - 1)) --b;
  while (b < g.nedges && x >= pk_edge(g, b)) ++b;
  return b;
}

__device__ __forceinline__ int signed_freq(int i, int n) {
  return i < (n - 1) / 2 + 1 ? i : i - n;
}

// Full-spectrum weight W of z index l (flowpm/pk.py:12-15).
__device__ __forceinline__ double pk_w(int l, int nz) {
  return (l == 0 || l == nz - 1) ? 1.0 : 2.0;
}

// pk_bin for k^2 = kk with less FP64: the bin from a float square root,
// and the exact comparison with the edges (of kmag() in double, as
// numpy.digitize sees it) only for modes within the float's error of one.
// rdk = 1 / dk, off = kmin / dk.
struct PkFast {
  float rdk, off;
};

__device__ __forceinline__ int pk_bin_fast(const PkGeom& g, const PkFast& q,
                                           double kxy, double kx, double ky,
                                           double kz) {
  const float x = sqrtf((float)(kxy + kz * kz)) * q.rdk;
  const float t = x - q.off;
  const float f = floorf(t);
  // x carries a relative error under 3 ulps (conversion, root, product with
  // the rounded 1 / dk), off and the difference one each
  const float eps = 5e-7f * (x + fabsf(q.off) + 1.f);
  const float r = t - f;
  if (r < eps || r > 1.f - eps)
    return pk_bin(g, sqrt(kx * kx + ky * ky + kz * kz));
  return f < 0.f ? 0 : (f >= (float)g.nedges ? g.nedges : (int)f + 1);
}

// Where the sums of a block go before scratch.
enum PkHist {
  kPkWarp = 0,    // a histogram per warp in shared memory, no atomics
  kPkBlock = 1,   // one per block in shared memory
  kPkGlobal = 2   // straight into scratch
};
constexpr int kPkWarps = 8;

// Adds psum[b][bin] += w |F|^2 and nsum[b][bin] += w of every batch entry b
// to scratch (2 (nedges + 1) doubles per entry, zeroed by the caller).
//
// The modes (+-i, +-j, l) have the same |k|, bit for bit, so a warp takes
// the up to four rows (i, j) together, lanes on consecutive l: one bin and
// one weight per lane for four modes.  |k| does not decrease along l, so
// the lanes of a bin are contiguous: their sums are formed with segmented
// shuffles and the first lane of each run adds them to the histogram, each
// bin once.  Measured at 256^3 (67 MB of spectrum, 10 us to read): one double
// atomic per mode on the block's histogram, most of them to the same few
// bins, 535 us; this 37 us, bound by the FP64 work and shuffles per warp.
template <int HIST>
__global__ void __launch_bounds__(32 * kPkWarps)
k_pk_accumulate(const float2* __restrict__ dk, int batch, PkGeom g, PkFast q,
                double* __restrict__ scratch) {
  extern __shared__ double sh_[];
  const int nb = g.nedges + 1;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  constexpr int NH = HIST == kPkWarp ? kPkWarps : HIST == kPkBlock ? 1 : 0;
  unsigned* cnt = reinterpret_cast<unsigned*>(sh_ + NH * nb);
  double* hs = sh_ + (HIST == kPkWarp ? warp * nb : 0);
  unsigned* hc = cnt + (HIST == kPkWarp ? warp * nb : 0);
  const int nj = g.ny / 2 + 1, nl = (g.nzh + 31) / 32;
  // one entry's modes are numbered in 32 bits
  const unsigned items = (unsigned)(g.nx / 2 + 1) * nj * nl;
  const unsigned unj = nj, unl = nl, nzh = g.nzh;
  for (int b = blockIdx.y; b < batch; b += gridDim.y) {
    double* out = scratch + (int64_t)b * 2 * nb;
    if (HIST != kPkGlobal) {
      for (int t = threadIdx.x; t < NH * nb; t += blockDim.x) {
        sh_[t] = 0.0;
        cnt[t] = 0;
      }
      __syncthreads();
    }
    const float2* f = dk + (int64_t)b * g.nx * g.ny * g.nzh;
    for (unsigned e = blockIdx.x * kPkWarps + warp; e < items;
         e += gridDim.x * kPkWarps) {
      const unsigned row = e / unl;
      const int l = (int)(e - row * unl) * 32 + lane;
      const int i = (int)(row / unj), j = (int)(row - (unsigned)i * unj);
      const int i2 = i ? g.nx - i : 0, j2 = j ? g.ny - j : 0;
      const bool two_i = i2 != i, two_j = j2 != j;
      const bool valid = l < g.nzh;
      double p2 = 0.0;
      unsigned c = 0;
      int bin = -1 - lane;  // a run of its own past the row's end
      if (valid) {
        const float2 zero = make_float2(0.f, 0.f);
        auto mode = [&](int a, int b) {
          return f[((unsigned)a * (unsigned)g.ny + (unsigned)b) * nzh +
                   (unsigned)l];
        };
        const float2 v0 = mode(i, j), v1 = two_j ? mode(i, j2) : zero;
        const float2 v2 = two_i ? mode(i2, j) : zero;
        const float2 v3 = two_i && two_j ? mode(i2, j2) : zero;
        const double kx = signed_freq(i, g.nx) * g.vx;
        const double ky = signed_freq(j, g.ny) * g.vy;
        const double kz = signed_freq(l, g.nz) * g.vz;
        bin = pk_bin_fast(g, q, kx * kx + ky * ky, kx, ky, kz);
        const int w = (int)pk_w(l, g.nz) +
                      (l != 0 && 2 * l != g.nz ? (int)pk_w(g.nz - l, g.nz) : 0);
        p2 = ((double)v0.x * v0.x + (double)v0.y * v0.y) +
             ((double)v1.x * v1.x + (double)v1.y * v1.y);
        p2 += ((double)v2.x * v2.x + (double)v2.y * v2.y) +
              ((double)v3.x * v3.x + (double)v3.y * v3.y);
        p2 *= w;
        c = (unsigned)w * (two_i ? 2u : 1u) * (two_j ? 2u : 1u);
      }
      const unsigned heads = run_heads((uint32_t)bin, lane);
      const bool head = (heads >> lane) & 1u;
      const int longest = (int)__reduce_max_sync(
          0xffffffffu, head ? (unsigned)run_length(heads, lane) : 1u);
      for (int o = 1; o < longest; o <<= 1) {
        // lane + o is in this lane's run when no run starts in (lane, lane + o]
        const bool same =
            lane + o < 32 &&
            ((unsigned long long)heads >> (lane + 1) & ((1ull << o) - 1)) == 0;
        const double tp = __shfl_down_sync(0xffffffffu, p2, o);
        const unsigned tc = __shfl_down_sync(0xffffffffu, c, o);
        if (same) {
          p2 += tp;
          c += tc;
        }
      }
      if (valid && head) {
        if (HIST == kPkWarp) {
          hs[bin] += p2;
          hc[bin] += c;
        } else if (HIST == kPkBlock) {
          atomicAdd(&hs[bin], p2);
          atomicAdd(&hc[bin], c);
        } else {
          atomicAdd(&out[bin], p2);
          atomicAdd(&out[nb + bin], (double)c);
        }
      }
      __syncwarp();  // the warp's next adds come after these
    }
    if (HIST != kPkGlobal) {
      __syncthreads();
      for (int t = threadIdx.x; t < nb; t += blockDim.x) {
        double p2 = 0.0, c = 0.0;
#pragma unroll
        for (int h = 0; h < NH; ++h) {
          p2 += sh_[h * nb + t];
          c += cnt[h * nb + t];
        }
        if (c != 0.0) {
          atomicAdd(&out[t], p2);
          atomicAdd(&out[nb + t], c);
        }
      }
    }
    if (HIST != kPkGlobal) __syncthreads();  // the next entry clears them
  }
}

// power[b][i] = psum[b][i+1] / nsum[b][i+1] * vol / ncell^2, i < nedges - 1.
__global__ void k_pk_finalize(const double* __restrict__ scratch, int batch,
                              int nedges, double scale,
                              float* __restrict__ power) {
  const int nb = nedges + 1, nout = nedges - 1;
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < batch * nout;
       t += gridDim.x * blockDim.x) {
    const int b = t / nout, i = t - b * nout;
    const double* s = scratch + (int64_t)b * 2 * nb;
    power[t] = (float)(s[i + 1] / s[nb + i + 1] * scale);
  }
}

int pk_check(const void* dk, int batch, int nx, int ny, int nz,
             const double* boxsize, double dkw, int nedges, const float* power) {
  if (!dk || !power || !boxsize || batch < 1 || nx < 1 || ny < 1 || nz < 1 ||
      nedges < 2 || !(dkw > 0) || !(boxsize[0] > 0) || !(boxsize[1] > 0) ||
      !(boxsize[2] > 0))
    return FPM_ERR_ARG;
  return FPM_OK;
}

PkGeom pk_geom(int nx, int ny, int nz, const double* boxsize, double kmin,
               double dkw, int nedges) {
  PkGeom g;
  g.nx = nx;
  g.ny = ny;
  g.nz = nz;
  g.nzh = nz / 2 + 1;
  // numpy.fft.fftfreq(N, 1 / (N 2 pi / L)) = i * (1 / (N d))
  const double dx = 1. / (nx * 2 * M_PI / boxsize[0]);
  const double dy = 1. / (ny * 2 * M_PI / boxsize[1]);
  const double dz = 1. / (nz * 2 * M_PI / boxsize[2]);
  g.vx = 1.0 / (nx * dx);
  g.vy = 1.0 / (ny * dy);
  g.vz = 1.0 / (nz * dz);
  g.kmin = kmin;
  g.dk = dkw;
  g.nedges = nedges;
  return g;
}

// Launch the accumulate + finalize pair on zeroed scratch.
int pk_launch(const float2* dk, int batch, const PkGeom& g, double* scratch,
              double vol, float* power, cudaStream_t st) {
  // Histograms per warp while eight of them (12 bytes a bin) fit the default
  // 48 KiB of shared memory, 511 edges; then one per block, 4095 edges; then
  // none.
  const size_t hist = (sizeof(double) + sizeof(unsigned)) * (g.nedges + 1);
  const int mode = kPkWarps * hist <= 48 * 1024 ? kPkWarp
                   : hist <= 48 * 1024          ? kPkBlock
                                                : kPkGlobal;
  const int64_t items = (int64_t)(g.nx / 2 + 1) * (g.ny / 2 + 1) *
                        ((g.nzh + 31) / 32);
  int64_t blocks = (items + kPkWarps - 1) / kPkWarps;
  if (blocks > kNumSMs * 8) blocks = kNumSMs * 8;
  const dim3 grid((unsigned)blocks, (unsigned)(batch < 65535 ? batch : 65535));
  const PkFast q = {(float)(1.0 / g.dk), (float)(g.kmin / g.dk)};
  g_launches.fetch_add(2, std::memory_order_relaxed);
  if (mode == kPkWarp)
    k_pk_accumulate<kPkWarp>
        <<<grid, 32 * kPkWarps, kPkWarps * hist, st>>>(dk, batch, g, q, scratch);
  else if (mode == kPkBlock)
    k_pk_accumulate<kPkBlock>
        <<<grid, 32 * kPkWarps, hist, st>>>(dk, batch, g, q, scratch);
  else
    k_pk_accumulate<kPkGlobal>
        <<<grid, 32 * kPkWarps, 0, st>>>(dk, batch, g, q, scratch);
  const double ncell = (double)g.nx * g.ny * g.nz;
  const int nout = batch * (g.nedges - 1);
  k_pk_finalize<<<(nout + 255) / 256, 256, 0, st>>>(
      scratch, batch, g.nedges, vol / (ncell * ncell), power);
  return cudaGetLastError() == cudaSuccess ? FPM_OK : FPM_ERR_CUDA;
}

}  // namespace fpm

using namespace fpm;

extern "C" int fpm_pk_bin(const void* delta_k, int batch, int nx, int ny,
                          int nz, const double* boxsize, double kmin,
                          double dk, int nedges, float* power, void* stream) {
  int rc = pk_check(delta_k, batch, nx, ny, nz, boxsize, dk, nedges, power);
  if (rc != FPM_OK) return rc;
  cudaStream_t st = (cudaStream_t)stream;
  const PkGeom g = pk_geom(nx, ny, nz, boxsize, kmin, dk, nedges);
  const size_t n = 2 * (size_t)batch * (nedges + 1);
  double* scratch = nullptr;
  if (cudaMallocAsync((void**)&scratch, n * sizeof(double), st) != cudaSuccess) {
    cudaGetLastError();
    return FPM_ERR_OOM;
  }
  rc = cudaMemsetAsync(scratch, 0, n * sizeof(double), st) == cudaSuccess
           ? FPM_OK
           : FPM_ERR_CUDA;
  if (rc == FPM_OK)
    rc = pk_launch((const float2*)delta_k, batch, g, scratch,
                   boxsize[0] * boxsize[1] * boxsize[2], power, st);
  cudaFreeAsync(scratch, st);
  return rc;
}

namespace {
// R2C plans of fpm_power_spectrum per (device, batch, nx, ny, nz), at most
// kMaxPkPlans of them: past that the least recently used one is destroyed
// (cufftDestroy frees its work area with cudaFree, which waits for the work
// already queued on the device).  The lock is held while a plan is bound to
// the caller's stream and its transform is queued.
constexpr size_t kMaxPkPlans = 8;
struct PkPlan {
  cufftHandle h;
  uint64_t used;
};
std::mutex g_pk_mu;
std::map<std::tuple<int, int, int, int, int>, PkPlan> g_pk_plans;
uint64_t g_pk_tick = 0;
}  // namespace

extern "C" int fpm_power_spectrum_work(int batch, int nx, int ny, int nz,
                                       int nedges, int64_t* bytes) {
  if (batch < 1 || nx < 1 || ny < 1 || nz < 1 || nedges < 2 || !bytes)
    return FPM_ERR_ARG;
  // the spectrum, then the bin sums on a multiple of 16 bytes
  const int64_t spec = (int64_t)sizeof(float2) * batch * nx * ny * (nz / 2 + 1);
  *bytes = (spec + 15) / 16 * 16 +
           2 * (int64_t)sizeof(double) * batch * (nedges + 1);
  return FPM_OK;
}

extern "C" int fpm_power_spectrum_ws(const float* field, int batch, int nx,
                                     int ny, int nz, const double* boxsize,
                                     double kmin, double dk, int nedges,
                                     float* power, void* work,
                                     int64_t work_bytes, void* stream) {
  if (!field || !work) return FPM_ERR_ARG;
  int rc = pk_check(field, batch, nx, ny, nz, boxsize, dk, nedges, power);
  if (rc != FPM_OK) return rc;
  int64_t need = 0;
  fpm_power_spectrum_work(batch, nx, ny, nz, nedges, &need);
  if (work_bytes < need) return FPM_ERR_ARG;
  if ((uintptr_t)work % 16 != 0) return FPM_ERR_ALIGN;
  cudaStream_t st = (cudaStream_t)stream;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return FPM_ERR_CUDA;
  float2* spec = (float2*)work;
  const size_t sums = 2 * sizeof(double) * (size_t)batch * (nedges + 1);
  double* scratch = (double*)((char*)work + need - sums);
  {
    std::lock_guard<std::mutex> lk(g_pk_mu);
    const auto key = std::make_tuple(dev, batch, nx, ny, nz);
    auto it = g_pk_plans.find(key);
    if (it == g_pk_plans.end()) {
      if (g_pk_plans.size() >= kMaxPkPlans) {
        auto old = g_pk_plans.begin();
        for (auto j = g_pk_plans.begin(); j != g_pk_plans.end(); ++j)
          if (j->second.used < old->second.used) old = j;
        cufftDestroy(old->second.h);
        g_pk_plans.erase(old);
      }
      int n[3] = {nx, ny, nz};
      cufftHandle h;
      if (cufftPlanMany(&h, 3, n, nullptr, 1, 0, nullptr, 1, 0, CUFFT_R2C,
                        batch) != CUFFT_SUCCESS)
        return FPM_ERR_CUFFT;
      it = g_pk_plans.emplace(key, PkPlan{h, 0}).first;
    }
    it->second.used = ++g_pk_tick;
    if (cufftSetStream(it->second.h, st) != CUFFT_SUCCESS ||
        cufftExecR2C(it->second.h, (cufftReal*)field, (cufftComplex*)spec) !=
            CUFFT_SUCCESS)
      return FPM_ERR_CUFFT;
  }
  if (cudaMemsetAsync(scratch, 0, sums, st) != cudaSuccess)
    return FPM_ERR_CUDA;
  return pk_launch(spec, batch, pk_geom(nx, ny, nz, boxsize, kmin, dk, nedges),
                   scratch, boxsize[0] * boxsize[1] * boxsize[2], power, st);
}

extern "C" int fpm_power_spectrum(const float* field, int batch, int nx,
                                  int ny, int nz, const double* boxsize,
                                  double kmin, double dk, int nedges,
                                  float* power, void* stream) {
  int64_t bytes = 0;
  if (!field ||
      fpm_power_spectrum_work(batch, nx, ny, nz, nedges, &bytes) != FPM_OK)
    return FPM_ERR_ARG;
  cudaStream_t st = (cudaStream_t)stream;
  void* work = nullptr;
  if (cudaMallocAsync(&work, bytes, st) != cudaSuccess) {
    cudaGetLastError();
    return FPM_ERR_OOM;
  }
  const int rc = fpm_power_spectrum_ws(field, batch, nx, ny, nz, boxsize,
                                       kmin, dk, nedges, power, work, bytes,
                                       stream);
  cudaFreeAsync(work, st);
  return rc;
}

// ---------------------------------------------------------------------------
// Allocation-free variant of fpm_pk_bin.
//
// Some callers cannot let a library allocate device memory: applications
// that hand all of a GPU's memory to their own pool or arena (where a
// cudaMalloc / cudaMallocAsync from a library fails or fragments it), and
// latency-critical loops that forbid allocation after start-up because an
// allocation can synchronise the device.  For them the bin accumulators of
// the power spectrum live in a fixed file-scope device array instead of
// stream-ordered scratch.  The array is part of this library's module, so
// every GPU that loads the library holds it (128 KiB) until the process
// exits.
// ---------------------------------------------------------------------------
static __device__ __align__(256) double
    g_pk_static_scratch[FPM_PK_NOALLOC_MAX_DOUBLES];

namespace {

constexpr int kMaxDevices = 64;
std::mutex g_static_mu;
double* g_static_ptr[kMaxDevices] = {};

// Device address of g_pk_static_scratch on the current device.  On host,
// the name g_pk_static_scratch is only a stand-in for the device symbol,
// so its device address is looked up once per device (with that device
// current) and cached for the life of the process: a cudaDeviceReset,
// which unloads the module, is not supported in between.
int static_scratch(double** out) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return FPM_ERR_CUDA;
  if (dev < 0 || dev >= kMaxDevices) return FPM_ERR_UNSUPPORTED;
  std::lock_guard<std::mutex> lk(g_static_mu);
  if (!g_static_ptr[dev]) {
    void* p = nullptr;
    if (cudaGetSymbolAddress(&p, g_pk_static_scratch) != cudaSuccess ||
        !p) {
      cudaGetLastError();
      return FPM_ERR_CUDA;
    }
    g_static_ptr[dev] = (double*)p;
  }
  *out = g_static_ptr[dev];
  return FPM_OK;
}

}  // namespace

extern "C" int fpm_pk_bin_noalloc(const void* delta_k, int batch, int nx,
                                  int ny, int nz, const double* boxsize,
                                  double kmin, double dk, int nedges,
                                  float* power, void* stream) {
  int rc = pk_check(delta_k, batch, nx, ny, nz, boxsize, dk, nedges, power);
  if (rc != FPM_OK) return rc;
  const int64_t n = 2 * (int64_t)batch * (nedges + 1);
  if (n > FPM_PK_NOALLOC_MAX_DOUBLES) return FPM_ERR_LIMIT;
  double* scratch = nullptr;
  rc = static_scratch(&scratch);
  if (rc != FPM_OK) return rc;
  cudaStream_t st = (cudaStream_t)stream;
  // The array keeps the previous call's sums: clear the part this call uses.
  if (cudaMemsetAsync(scratch, 0, n * sizeof(double), st) != cudaSuccess)
    return FPM_ERR_CUDA;
  const PkGeom g = pk_geom(nx, ny, nz, boxsize, kmin, dk, nedges);
  return pk_launch((const float2*)delta_k, batch, g, scratch,
                   boxsize[0] * boxsize[1] * boxsize[2], power, st);
}

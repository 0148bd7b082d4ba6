// Stand-alone CIC paint / readout / neighbour kernels (the operators of
// flowpm/utils.py:32-91 cic_paint and :163-210 cic_readout) and their C ABI.
#include <atomic>

#include "fpm_kernels.cuh"

namespace fpm {

// The operators on caller's catalogues, whose particles come in any order:
// every (x, y) row of a particle's neighbours is its own L2 sector, and a
// warp-wide access costs the L1 one cycle per sector.  The two z neighbours
// of a row are consecutive floats, and three times out of four lie in one
// aligned group of four, so they are one 16-byte access of that group (the
// other cells of the group read and ignored, or incremented by zero).
// Measured on B200, 4 M particles on 256^3: paint 175 us a cell, 137 us as
// aligned pairs, 120 us in groups; 2 M on 200 x 180 x 150: paint 87 -> 55 us,
// readout 46 -> 41, readout adjoint 125 -> 86, paint adjoint 100 -> 50 (a
// division per particle and per corner accesses before).
struct CatPos {
  Axis ax, ay, az;
  int64_t row[4];  // (x, y) rows, neighbour (cx, cy) at row[cx + 2 cy]
};

__device__ __forceinline__ CatPos cat_pos(const float* __restrict__ part,
                                          int64_t g, int nx, int ny, int nz) {
  CatPos c;
  cic_axes(ld3(part, g), nx, ny, nz, c.ax, c.ay, c.az);
  const int64_t x0 = (int64_t)c.ax.i0 * ny, x1 = (int64_t)c.ax.i1 * ny;
  c.row[0] = (x0 + c.ay.i0) * nz;
  c.row[1] = (x1 + c.ay.i0) * nz;
  c.row[2] = (x0 + c.ay.i1) * nz;
  c.row[3] = (x1 + c.ay.i1) * nz;
  return c;
}

// A mesh (all batch entries), so that a group does not leave it.
struct CatMesh {
  const float *begin, *end;
};

// The place of a cell in its aligned group of four, or 3 when the group does
// not hold its z neighbour too (the last place, a row's wrap) or leaves the
// mesh.
__device__ __forceinline__ int group_place(const CatMesh& M, const float* p,
                                           const CatPos& c) {
  const int o = (int)((uintptr_t)p >> 2 & 3);
  return c.az.i1 == c.az.i0 + 1 && p - o >= M.begin && p - o + 4 <= M.end ? o
                                                                          : 3;
}

// The values of a row's z neighbours; m: the batch entry.
__device__ __forceinline__ float2 cat_pair(const CatMesh& M,
                                           const float* __restrict__ m,
                                           const CatPos& c, int q) {
  const float* p = m + c.row[q] + c.az.i0;
  const int o = group_place(M, p, c);
  if (o == 3)
    return make_float2(__ldg(p), __ldg(m + c.row[q] + c.az.i1));
  const float4 v = __ldg(reinterpret_cast<const float4*>(p - o));
  return o == 0 ? make_float2(v.x, v.y)
                : o == 1 ? make_float2(v.y, v.z) : make_float2(v.z, v.w);
}

// m[row] += (a, b) at the z neighbours.
__device__ __forceinline__ void cat_add(const CatMesh& M,
                                        float* __restrict__ m,
                                        const CatPos& c, int q, float a,
                                        float b) {
  float* p = m + c.row[q] + c.az.i0;
  const int o = group_place(M, p, c);
  if (o == 3) {
    red_add(p, a);
    red_add(m + c.row[q] + c.az.i1, b);
  } else {
    red_add_f4(p - o,
               make_float4(o == 0 ? a : 0.f, o == 0 ? b : o == 1 ? a : 0.f,
                           o == 1 ? b : o == 2 ? a : 0.f, o == 2 ? b : 0.f));
  }
}

__device__ __forceinline__ float row_weight(const CatPos& c, int q) {
  return __fmul_rn((q & 1) ? c.ax.w1 : c.ax.w0, (q >> 1) ? c.ay.w1 : c.ay.w0);
}

// mesh[b] += sum_c w_c * weight at the 8 neighbours of each particle of batch
// entry b = blockIdx.y (+ gridDim.y ...).  One thread per particle.
__global__ void __launch_bounds__(kThreads)
k_cic_paint(float* __restrict__ mesh, int nx, int ny, int nz,
            const float* __restrict__ part, int64_t npart, int batch,
            const float* __restrict__ weight) {
  const int64_t ncell = (int64_t)nx * ny * nz;
  const CatMesh M = {mesh, mesh + batch * ncell};
  for (int b = blockIdx.y; b < batch; b += gridDim.y) {
    float* m = mesh + b * ncell;
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
         t < npart; t += (int64_t)gridDim.x * blockDim.x) {
      const int64_t g = b * npart + t;
      const CatPos c = cat_pos(part, g, nx, ny, nz);
      const float wt = weight ? weight[g] : 1.0f;
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const float w = row_weight(c, q);
        float w0 = __fmul_rn(w, c.az.w0), w1 = __fmul_rn(w, c.az.w1);
        if (weight) {
          w0 = __fmul_rn(wt, w0);
          w1 = __fmul_rn(wt, w1);
        }
        cat_add(M, m, c, q, w0, w1);
      }
    }
  }
}

__global__ void __launch_bounds__(kThreads)
k_cic_readout(const float* __restrict__ mesh, int nx, int ny, int nz,
              const float* __restrict__ part, int64_t npart, int batch,
              float* __restrict__ out) {
  const int64_t ncell = (int64_t)nx * ny * nz;
  const CatMesh M = {mesh, mesh + batch * ncell};
  for (int b = blockIdx.y; b < batch; b += gridDim.y) {
    const float* m = mesh + b * ncell;
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
         t < npart; t += (int64_t)gridDim.x * blockDim.x) {
      const int64_t g = b * npart + t;
      const CatPos c = cat_pos(part, g, nx, ny, nz);
      float2 v[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) v[q] = cat_pair(M, m, c, q);
      float acc = 0.0f;
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const float w = row_weight(c, q);
        acc = __fmaf_rn(v[q].x, __fmul_rn(w, c.az.w0), acc);
        acc = __fmaf_rn(v[q].y, __fmul_rn(w, c.az.w1), acc);
      }
      out[g] = acc;
    }
  }
}

// sum_c v[c] W and sum_c v[c] grad W (dW/dy of an axis: -sign(y - n), with
// sign(0) = 0: -1 for the lower neighbour when y is not on its face, 0 when
// it is, 1 for the upper).
__device__ __forceinline__ void cat_sums(const CatPos& c, const float2* v,
                                         float3 y, float& sum, float3& grad) {
  const float dx = y.x - floorf(y.x) > 0.f ? -1.f : 0.f,
              dy = y.y - floorf(y.y) > 0.f ? -1.f : 0.f,
              dz = y.z - floorf(y.z) > 0.f ? -1.f : 0.f;
  float s[4], t[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    s[q] = v[q].x * c.az.w0 + v[q].y * c.az.w1;
    t[q] = v[q].x * dz + v[q].y;
  }
  const float a0 = s[0] * c.ay.w0 + s[2] * c.ay.w1,
              a1 = s[1] * c.ay.w0 + s[3] * c.ay.w1;
  const float b0 = s[0] * dy + s[2], b1 = s[1] * dy + s[3];
  const float e0 = t[0] * c.ay.w0 + t[2] * c.ay.w1,
              e1 = t[1] * c.ay.w0 + t[3] * c.ay.w1;
  sum = a0 * c.ax.w0 + a1 * c.ax.w1;
  grad = make_float3(a0 * dx + a1, b0 * c.ax.w0 + b1 * c.ax.w1,
                     e0 * c.ax.w0 + e1 * c.ax.w1);
}

__global__ void __launch_bounds__(kThreads)
k_cic_paint_adjoint(const float* __restrict__ lmesh, int nx, int ny, int nz,
                    const float* __restrict__ part, int64_t npart, int batch,
                    const float* __restrict__ weight,
                    float* __restrict__ lpart, float* __restrict__ lweight) {
  const int64_t ncell = (int64_t)nx * ny * nz;
  const CatMesh M = {lmesh, lmesh + batch * ncell};
  for (int b = blockIdx.y; b < batch; b += gridDim.y) {
    const float* m = lmesh + b * ncell;
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
         t < npart; t += (int64_t)gridDim.x * blockDim.x) {
      const int64_t g = b * npart + t;
      const CatPos c = cat_pos(part, g, nx, ny, nz);
      float2 v[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) v[q] = cat_pair(M, m, c, q);
      float sum;
      float3 gr;
      cat_sums(c, v, ld3(part, g), sum, gr);
      const float wt = weight ? weight[g] : 1.f;
      if (lpart) st3(lpart, g, make_float3(wt * gr.x, wt * gr.y, wt * gr.z));
      if (lweight) lweight[g] = sum;
    }
  }
}

__global__ void __launch_bounds__(kThreads)
k_cic_readout_adjoint(const float* __restrict__ mesh, int nx, int ny, int nz,
                      const float* __restrict__ part, int64_t npart,
                      int batch, const float* __restrict__ lout,
                      float* __restrict__ lmesh, float* __restrict__ lpart) {
  const int64_t ncell = (int64_t)nx * ny * nz;
  for (int b = blockIdx.y; b < batch; b += gridDim.y) {
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
         t < npart; t += (int64_t)gridDim.x * blockDim.x) {
      const int64_t g = b * npart + t;
      const CatPos c = cat_pos(part, g, nx, ny, nz);
      const float lo = lout[g];
      if (lpart) {
        const float* m = mesh + b * ncell;
        const CatMesh M = {mesh, mesh + batch * ncell};
        float2 v[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) v[q] = cat_pair(M, m, c, q);
        float sum;
        float3 gr;
        cat_sums(c, v, ld3(part, g), sum, gr);
        st3(lpart, g, make_float3(lo * gr.x, lo * gr.y, lo * gr.z));
      }
      if (lmesh) {
        float* m = lmesh + b * ncell;
        const CatMesh M = {lmesh, lmesh + batch * ncell};
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const float w = row_weight(c, q);
          cat_add(M, m, c, q, __fmul_rn(lo, __fmul_rn(w, c.az.w0)),
                  __fmul_rn(lo, __fmul_rn(w, c.az.w1)));
        }
      }
    }
  }
}

__global__ void __launch_bounds__(kThreads)
k_cic_neighbours(int nx, int ny, int nz, const float* __restrict__ part,
                 int64_t n, int32_t* __restrict__ idx, float* __restrict__ w) {
  for (int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; g < n;
       g += (int64_t)gridDim.x * blockDim.x) {
    const float x = part[3 * g + 0], y = part[3 * g + 1], z = part[3 * g + 2];
    Axis ax = cic_axis(x, nx), ay = cic_axis(y, ny), az = cic_axis(z, nz);
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      const int cx = conn_x(c), cy = conn_y(c), cz = conn_z(c);
      const int ix = cx ? ax.i1 : ax.i0, iy = cy ? ay.i1 : ay.i0,
                iz = cz ? az.i1 : az.i0;
      idx[8 * g + c] = (ix * ny + iy) * nz + iz;
      w[8 * g + c] = cic_w(ax, ay, az, cx, cy, cz);
    }
  }
}

static unsigned grid_elems(int64_t n) {
  int64_t blocks = (n + kThreads - 1) / kThreads;
  const int64_t cap = (int64_t)kNumSMs * 32;
  if (blocks < 1) blocks = 1;
  return (unsigned)(blocks < cap ? blocks : cap);
}

static bool bad_dims(int batch, int nx, int ny, int nz) {
  return batch < 1 || nx < 1 || ny < 1 || nz < 1 ||
         (int64_t)nx * ny * nz > (int64_t)1 << 31;
}

}  // namespace fpm

using namespace fpm;

namespace {

dim3 cat_grid(int64_t npart, int batch) {
  const unsigned x = grid_elems(npart);
  const int y = (int)(batch < 65535 ? batch : 65535);
  return dim3(x, (unsigned)y);
}

int launched() {
  g_launches.fetch_add(1, std::memory_order_relaxed);
  return cudaGetLastError() == cudaSuccess ? FPM_OK : FPM_ERR_CUDA;
}

}  // namespace

extern "C" int fpm_cic_paint(float* mesh, int batch, int nx, int ny, int nz,
                             const float* part, int64_t npart,
                             const float* weight, void* stream) {
  if (!mesh || (!part && npart > 0) || npart < 0 || bad_dims(batch, nx, ny, nz))
    return FPM_ERR_ARG;
  if (npart == 0) return FPM_OK;
  k_cic_paint<<<cat_grid(npart, batch), kThreads, 0,
                (cudaStream_t)stream>>>(
      mesh, nx, ny, nz, part, npart, batch, weight);
  return launched();
}

extern "C" int fpm_cic_readout(const float* mesh, int batch, int nx, int ny,
                               int nz, const float* part, int64_t npart,
                               float* out, void* stream) {
  if (!mesh || ((!part || !out) && npart > 0) || npart < 0 ||
      bad_dims(batch, nx, ny, nz))
    return FPM_ERR_ARG;
  if (npart == 0) return FPM_OK;
  k_cic_readout<<<cat_grid(npart, batch), kThreads, 0,
                  (cudaStream_t)stream>>>(
      mesh, nx, ny, nz, part, npart, batch, out);
  return launched();
}

extern "C" int fpm_cic_paint_adjoint(const float* lam_mesh, int batch, int nx,
                                     int ny, int nz, const float* part,
                                     int64_t npart, const float* weight,
                                     float* lam_part, float* lam_weight,
                                     void* stream) {
  if (!lam_mesh || batch < 1 || nx < 1 || ny < 1 || nz < 1 || npart < 0 ||
      (npart > 0 && !part) || (!lam_part && !lam_weight))
    return FPM_ERR_ARG;
  if (npart == 0) return FPM_OK;
  k_cic_paint_adjoint<<<cat_grid(npart, batch), kThreads, 0,
                        (cudaStream_t)stream>>>(
      lam_mesh, nx, ny, nz, part, npart, batch, weight, lam_part, lam_weight);
  return launched();
}

extern "C" int fpm_cic_readout_adjoint(const float* mesh, int batch, int nx,
                                       int ny, int nz, const float* part,
                                       int64_t npart, const float* lam_out,
                                       float* lam_mesh, float* lam_part,
                                       void* stream) {
  if (batch < 1 || nx < 1 || ny < 1 || nz < 1 || npart < 0 ||
      (npart > 0 && (!part || !lam_out)) || (!lam_mesh && !lam_part) ||
      (lam_part && !mesh))
    return FPM_ERR_ARG;
  if (npart == 0) return FPM_OK;
  k_cic_readout_adjoint<<<cat_grid(npart, batch), kThreads, 0,
                          (cudaStream_t)stream>>>(
      mesh, nx, ny, nz, part, npart, batch, lam_out, lam_mesh, lam_part);
  return launched();
}

extern "C" int fpm_cic_neighbours(int nx, int ny, int nz, const float* part,
                                  int64_t npart, int32_t* idx, float* w,
                                  void* stream) {
  if (npart < 0 || bad_dims(1, nx, ny, nz) ||
      (npart > 0 && (!part || !idx || !w)))
    return FPM_ERR_ARG;
  if (npart == 0) return FPM_OK;
  k_cic_neighbours<<<grid_elems(npart), kThreads, 0, (cudaStream_t)stream>>>(
      nx, ny, nz, part, npart, idx, w);
  return cudaGetLastError() == cudaSuccess ? FPM_OK : FPM_ERR_CUDA;
}

namespace fpm {

__global__ void __launch_bounds__(kThreads)
k_lattice_shift(const float* __restrict__ in, float* __restrict__ out,
                int64_t np, int64_t total, int ny, int nz, float sign) {
  for (int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; g < total;
       g += (int64_t)gridDim.x * blockDim.x) {
    const int64_t local = g % np;
    const int64_t t = local / nz;
    const int k = (int)(local - t * nz);
    const int i = (int)(t / ny);
    const int j = (int)(t - (int64_t)i * ny);
    out[3 * g + 0] = __fadd_rn(in[3 * g + 0], sign * (float)i);
    out[3 * g + 1] = __fadd_rn(in[3 * g + 1], sign * (float)j);
    out[3 * g + 2] = __fadd_rn(in[3 * g + 2], sign * (float)k);
  }
}

// k_lattice_shift for nz % 4 == 0 and 16-byte aligned arrays, one float4 per
// thread: four particles of one row are three of them, so a thread needs one
// pair of 32-bit divisions.  3.2 GB (512^3) take 0.52 ms against 0.75 ms
// with a particle and four 64-bit divisions per thread.
__global__ void __launch_bounds__(kThreads)
k_lattice_shift4(const float4* __restrict__ in, float4* __restrict__ out,
                 unsigned quads, int64_t total, unsigned ny, unsigned nz,
                 float sign) {
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < total;
       t += (int64_t)gridDim.x * blockDim.x) {
    const int64_t a = t / 3;                    // group of four particles
    const int r = (int)(t - 3 * a);
    const unsigned k4 = (unsigned)(a % quads);  // of its simulation
    const unsigned row = k4 / (nz / 4);
    const unsigned iu = row / ny;
    const float i = sign * (float)iu, j = sign * (float)(row - iu * ny);
    const unsigned k0 = 4 * (k4 - row * (nz / 4));
    float4 v = in[t];
    if (r == 0) {
      v.x = __fadd_rn(v.x, i);
      v.y = __fadd_rn(v.y, j);
      v.z = __fadd_rn(v.z, sign * (float)k0);
      v.w = __fadd_rn(v.w, i);
    } else if (r == 1) {
      v.x = __fadd_rn(v.x, j);
      v.y = __fadd_rn(v.y, sign * (float)(k0 + 1));
      v.z = __fadd_rn(v.z, i);
      v.w = __fadd_rn(v.w, j);
    } else {
      v.x = __fadd_rn(v.x, sign * (float)(k0 + 2));
      v.y = __fadd_rn(v.y, i);
      v.z = __fadd_rn(v.z, j);
      v.w = __fadd_rn(v.w, sign * (float)(k0 + 3));
    }
    out[t] = v;
  }
}

__global__ void __launch_bounds__(kThreads)
k_saxpy(float* __restrict__ y, const float* __restrict__ x, float a,
        int64_t n) {
  for (int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; g < n;
       g += (int64_t)gridDim.x * blockDim.x)
    y[g] = __fadd_rn(y[g], __fmul_rn(a, x[g]));
}

}  // namespace fpm

extern "C" int fpm_lattice_shift(const float* in, float* out, int batch,
                                 int nx, int ny, int nz, int sign,
                                 void* stream) {
  if (!in || !out || bad_dims(batch, nx, ny, nz) || (sign != 1 && sign != -1))
    return FPM_ERR_ARG;
  const int64_t np = (int64_t)nx * ny * nz;
  const int64_t total = (int64_t)batch * np;
  if (nz % 4 == 0 && (uintptr_t)in % 16 == 0 && (uintptr_t)out % 16 == 0) {
    const int64_t n4 = total / 4 * 3;
    k_lattice_shift4<<<grid_elems(n4), kThreads, 0, (cudaStream_t)stream>>>(
        (const float4*)in, (float4*)out, (unsigned)(np / 4), n4, (unsigned)ny,
        (unsigned)nz, (float)sign);
    return launched();
  }
  k_lattice_shift<<<grid_elems(total), kThreads, 0, (cudaStream_t)stream>>>(
      in, out, np, total, ny, nz, (float)sign);
  return cudaGetLastError() == cudaSuccess ? FPM_OK : FPM_ERR_CUDA;
}

extern "C" int fpm_saxpy(float* y, const float* x, float a, int64_t n,
                         void* stream) {
  if (n < 0 || (n > 0 && (!x || !y))) return FPM_ERR_ARG;
  if (n == 0) return FPM_OK;
  k_saxpy<<<grid_elems(n), kThreads, 0, (cudaStream_t)stream>>>(y, x, a, n);
  return cudaGetLastError() == cudaSuccess ? FPM_OK : FPM_ERR_CUDA;
}

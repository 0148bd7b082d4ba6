// Fused Fourier solve of the force meshes for power-of-two meshes of 16 to
// 128 cells per axis: density -> three force meshes in three kernels,
// without cuFFT and without intermediate passes over HBM.
//
//   k_fft_plane_fwd  (one CTA per x plane)  rho(x, y, z) -> S(x, ky, kz)
//       real-to-complex DFT along z, complex DFT along y; also zeroes rho
//       for the next paint.
//   k_fft_x          (one CTA per 16 (ky, kz) columns)
//       DFT along x, the transfer function (flowpm/tfpm.py:199-215
//       apply_longrange), inverse DFT along x; also for meshes of 256 or 512
//       along x.  k_fft_x_grad3: with the order-0 gradient, the three force
//       spectra instead of the potential.
//   k_fft_plane_inv  (one CTA per x plane, and component for order 0)
//       inverse DFT along y, complex-to-real along z, y and z components of
//       the force by the stencil; k_fft_stencil_x takes the x component.
//
// Meshes of 256 or 512 take each axis as its own pass (k_fft_z_fwd, k_fft_y,
// k_fft_x, k_fft_z_inv), and the 2LPT of power-of-two lattices passes shared by
// its outputs (k_lpt_*).
//
// The transforms are unnormalised in both directions, as cuFFT's, so the
// spectra have cuFFT's R2C layout (x, y, z/2 + 1) and the results match
// the cuFFT path to rounding.  Every length-N DFT runs as N = N1 * N2 (the
// "four-step" split): a group of N2 threads, each holding N1 values in
// registers, does N1-point DFTs, a twiddle, one exchange through shared
// memory and N2-point DFTs.  Twiddles come from tables of exp(-2 pi i m / 128)
// and exp(-2 pi i m / 512) computed in double on the host.
#include <cmath>
#include <mutex>

#include "fpm_kernels.cuh"

namespace fpm {

namespace {

constexpr int kFftThreads = 256;

__constant__ float2 c_w128[128];  // exp(-2 pi i m / 128), m = 0..127
__constant__ float2 c_w512[512];  // exp(-2 pi i m / 512), m = 0..511
__device__ float2 g_w512[512];    // the same, for lane-dependent indices

__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
  return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
// a * conj(b)
__device__ __forceinline__ float2 cmulc(float2 a, float2 b) {
  return make_float2(a.x * b.x + a.y * b.y, a.y * b.x - a.x * b.y);
}

template <int N>
struct Split;
template <>
struct Split<8> {
  static constexpr int N1 = 4, N2 = 2;
};
template <>
struct Split<16> {
  static constexpr int N1 = 4, N2 = 4;
};
template <>
struct Split<32> {
  static constexpr int N1 = 8, N2 = 4;
};
template <>
struct Split<64> {
  static constexpr int N1 = 8, N2 = 8;
};
template <>
struct Split<128> {
  static constexpr int N1 = 16, N2 = 8;
};
template <>
struct Split<256> {
  static constexpr int N1 = 16, N2 = 16;
};
template <>
struct Split<512> {
  static constexpr int N1 = 32, N2 = 16;
};

// In-register DFT of N (2 to 32) values by even/odd (radix-2, decimation
// in time) recursion, every index a compile-time constant: forward
// X[k] = sum_j x[j] exp(-2 pi i jk / N), inverse with +i.
template <int N, bool INV>
struct Dft {
  static __device__ __forceinline__ void run(float2 (&a)[N]) {
    constexpr int H = N / 2;
    float2 e[H], o[H];
#pragma unroll
    for (int j = 0; j < H; ++j) {
      e[j] = a[2 * j];
      o[j] = a[2 * j + 1];
    }
    Dft<H, INV>::run(e);
    Dft<H, INV>::run(o);
#pragma unroll
    for (int k = 0; k < H; ++k) {
      float2 v = o[k];
      if (k != 0) {
        if (4 * k == N) {  // exp(-+ i pi / 2) = -+ i
          v = INV ? make_float2(-v.y, v.x) : make_float2(v.y, -v.x);
        } else {
          const float2 w = c_w128[k * (128 / N)];
          v = INV ? cmulc(v, w) : cmul(v, w);
        }
      }
      a[k] = make_float2(e[k].x + v.x, e[k].y + v.y);
      a[k + H] = make_float2(e[k].x - v.x, e[k].y - v.y);
    }
  }
};
template <bool INV>
struct Dft<1, INV> {
  static __device__ __forceinline__ void run(float2 (&)[1]) {}
};

template <int N, bool INV>
__device__ __forceinline__ void dft(float2 (&a)[N]) {
  Dft<N, INV>::run(a);
}

// ---------------------------------------------------------------------------
// Rows of real values, a group of N2 lanes per row (M complex values)
// ---------------------------------------------------------------------------

// Twiddles of a lane's row transform: t[k1] = W_M^(g k1) and w[e] =
// W_2M^(k) of its element e = u N2 + k2, k = g + N2 u + N1 k2.
//
// Rows of more than 64 values would keep 64 registers of them: their w[e] is
// read from the table where it is used.
template <int M>
struct RowTw {
  static constexpr int N1 = Split<M>::N1, N2 = Split<M>::N2;
  static constexpr bool kKeep = M <= 64;
  float2 t[N1], w[kKeep ? N1 : 1];
  int g;
  static __device__ __forceinline__ float2 table(int g, int e) {
    const int k = g + N2 * (e / N2) + N1 * (e % N2);
    return __ldg(&g_w512[k * (256 / M)]);
  }
  __device__ __forceinline__ void load(int lane_g) {
    g = lane_g;
#pragma unroll
    for (int k1 = 0; k1 < N1; ++k1)
      t[k1] = __ldg(&g_w512[((g * k1) & (M - 1)) * (512 / M)]);
    if (kKeep) {
#pragma unroll
      for (int e = 0; e < N1; ++e) w[kKeep ? e : 0] = table(g, e);
    }
  }
  __device__ __forceinline__ float2 at(int e) const {
    return kKeep ? w[kKeep ? e : 0] : table(g, e);
  }
};

// Slot of (k1, j) in a row's exchange: lanes of a group write one k1 at
// consecutive j and read consecutive k1 at one j; the exclusive or spreads
// the latter over the banks.
template <int N2>
__device__ __forceinline__ int ex_slot(int k1, int j) {
  return k1 * N2 + (j ^ (k1 & (N2 - 1)));
}

// Element (u, k2) of the lane that holds M - k for this lane's k = g + N2 u
// + N1 k2, fetched from it (lane g = 0 is its own partner).
template <int M>
__device__ __forceinline__ void row_partner(
    const float2 (&a)[Split<M>::N1], int g, int lane,
    float2 (&m)[Split<M>::N1]) {
  constexpr int N1 = Split<M>::N1, N2 = Split<M>::N2, U = N1 / N2;
  const int src = (lane & ~(N2 - 1)) | ((N2 - g) & (N2 - 1));
#pragma unroll
  for (int u = 0; u < U; ++u)
#pragma unroll
    for (int k2 = 0; k2 < N2; ++k2) {
      const float2 v = a[(U - 1 - u) * N2 + (N2 - 1 - k2)];
      const float2 t = make_float2(__shfl_sync(0xffffffffu, v.x, src),
                                   __shfl_sync(0xffffffffu, v.y, src));
      const float2 own = u == 0 ? a[(N2 - k2) & (N2 - 1)]
                                : a[(U - u) * N2 + (N2 - 1 - k2)];
      m[u * N2 + k2] = g ? t : own;
    }
}

// Real-to-complex DFT of a row: on entry a[j1] = x[2m] + i x[2m + 1] of
// element m = N2 j1 + g; on exit a[u N2 + k2] = X[k], k = g + N2 u + N1 k2,
// except X[0], which is X[0] + i X[M] (both real).  X[k] = E + W_2M^k O with
// E = (Z[k] + conj Z[M-k]) / 2 and O = (Z[k] - conj Z[M-k]) / 2i.  ex: M
// slots of shared memory of the row's own; every lane of the warp takes
// part.
template <int M>
__device__ __forceinline__ void row_r2c(float2 (&a)[Split<M>::N1], float2* ex,
                                        int g, int lane, const RowTw<M>& tw) {
  constexpr int N1 = Split<M>::N1, N2 = Split<M>::N2;
  dft<N1, false>(a);
  __syncwarp();  // the row's slots are free
#pragma unroll
  for (int k1 = 0; k1 < N1; ++k1)
    ex[ex_slot<N2>(k1, g)] = k1 ? cmul(a[k1], tw.t[k1]) : a[0];
  __syncwarp();
#pragma unroll
  for (int u = 0; u < N1 / N2; ++u) {
    float2 b[N2];
#pragma unroll
    for (int j = 0; j < N2; ++j) b[j] = ex[ex_slot<N2>(g + N2 * u, j)];
    dft<N2, false>(b);
#pragma unroll
    for (int k2 = 0; k2 < N2; ++k2) a[u * N2 + k2] = b[k2];
  }
  float2 m[N1];
  row_partner<M>(a, g, lane, m);
#pragma unroll
  for (int e = 0; e < N1; ++e) {
    const float2 zk = a[e], zm = m[e];
    const float2 E = make_float2(0.5f * (zk.x + zm.x), 0.5f * (zk.y - zm.y));
    const float2 O = make_float2(0.5f * (zk.y + zm.y), -0.5f * (zk.x - zm.x));
    const float2 W = cmul(tw.at(e), O);
    a[e] = make_float2(E.x + W.x, E.y + W.y);
    if (e == 0 && g == 0) a[e] = make_float2(zk.x + zk.y, zk.x - zk.y);
  }
}

// The converse (unnormalised): on entry a[u N2 + k2] = X[k] with X[0] + i
// X[M] in the place of X[0]; on exit a[j1] = x[2m] + i x[2m + 1].
template <int M>
__device__ __forceinline__ void row_c2r(float2 (&a)[Split<M>::N1], float2* ex,
                                        int g, int lane, const RowTw<M>& tw) {
  constexpr int N1 = Split<M>::N1, N2 = Split<M>::N2;
  float2 m[N1];
  row_partner<M>(a, g, lane, m);
#pragma unroll
  for (int e = 0; e < N1; ++e) {
    const float2 xk = a[e], xm = m[e];
    const float2 A = make_float2(xk.x + xm.x, xk.y - xm.y);
    const float2 B = make_float2(xk.x - xm.x, xk.y + xm.y);
    const float2 cb = cmulc(B, tw.at(e));
    a[e] = make_float2(A.x - cb.y, A.y + cb.x);  // A + i conj(W^k) B
    if (e == 0 && g == 0) a[e] = make_float2(xk.x + xk.y, xk.x - xk.y);
  }
  __syncwarp();  // the row's slots are free
#pragma unroll
  for (int u = 0; u < N1 / N2; ++u) {
    const int k1 = g + N2 * u;
    float2 b[N2];
#pragma unroll
    for (int k2 = 0; k2 < N2; ++k2) b[k2] = a[u * N2 + k2];
    dft<N2, true>(b);
#pragma unroll
    for (int j2 = 0; j2 < N2; ++j2) ex[ex_slot<N2>(k1, j2)] = b[j2];
  }
  __syncwarp();
#pragma unroll
  for (int k1 = 0; k1 < N1; ++k1) {
    const float2 v = ex[ex_slot<N2>(k1, g)];
    a[k1] = k1 ? cmulc(v, tw.t[k1]) : v;
  }
  dft<N1, true>(a);
}

// The element before (element m - 1 of the row, periodic) of each element of
// the lane, and the one after: v[j1] of lane g is element N2 j1 + g.
template <int N1, int N2>
__device__ __forceinline__ float row_prev(const float (&v)[N1], int j1, int g,
                                          int lane) {
  const float s = g == N2 - 1 ? v[(j1 + N1 - 1) % N1] : v[j1];
  return __shfl_sync(0xffffffffu, s,
                     (lane & ~(N2 - 1)) | ((g + N2 - 1) & (N2 - 1)));
}
template <int N1, int N2>
__device__ __forceinline__ float row_next(const float (&v)[N1], int j1, int g,
                                          int lane) {
  const float s = g == 0 ? v[(j1 + 1) % N1] : v[j1];
  return __shfl_sync(0xffffffffu, s,
                     (lane & ~(N2 - 1)) | ((g + 1) & (N2 - 1)));
}

// One row loaded as the a[] of row_r2c from the painted density P (PAIRS: z
// pairs, one float4 per element, see paint_rows) or a plain mesh; zero: the
// row is cleared (a lane clears what it alone has read).
template <int M, bool PAIRS>
__device__ __forceinline__ void row_load(float2 (&a)[Split<M>::N1], float* P,
                                         int zero, int g, int lane) {
  constexpr int N1 = Split<M>::N1, N2 = Split<M>::N2;
  if (PAIRS) {
    float4* p4 = reinterpret_cast<float4*>(P);
    float4 v[N1];
    float y[N1];
#pragma unroll
    for (int j1 = 0; j1 < N1; ++j1) v[j1] = p4[N2 * j1 + g];
#pragma unroll
    for (int j1 = 0; j1 < N1; ++j1) y[j1] = v[j1].w;
#pragma unroll
    for (int j1 = 0; j1 < N1; ++j1)
      a[j1] = make_float2(
          __fadd_rn(v[j1].x, row_prev<N1, N2>(y, j1, g, lane)),
          __fadd_rn(v[j1].z, v[j1].y));
    if (zero) {
#pragma unroll
      for (int j1 = 0; j1 < N1; ++j1)
        p4[N2 * j1 + g] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
  } else {
    float2* p2 = reinterpret_cast<float2*>(P);
#pragma unroll
    for (int j1 = 0; j1 < N1; ++j1) a[j1] = p2[N2 * j1 + g];
    if (zero) {
#pragma unroll
      for (int j1 = 0; j1 < N1; ++j1)
        p2[N2 * j1 + g] = make_float2(0.f, 0.f);
    }
  }
}

// 4-point central difference with periodic wrap, the arithmetic of
// k_stencil_grad: (8 (f[+1] - f[-1]) - (f[+2] - f[-2])) / 12.
__device__ __forceinline__ float stencil4f(float m2, float m1, float p1,
                                           float p2) {
  return __fmul_rn(__fsub_rn(__fmul_rn(8.f, __fsub_rn(p1, m1)),
                             __fsub_rn(p2, m2)),
                   1.0f / 12.0f);
}

// z component of the 4-point gradient of the lane's elements (x[2m], x[2m +
// 1]) of a row.
template <int N1, int N2>
__device__ __forceinline__ void row_grad(const float2 (&a)[N1],
                                         float2 (&f)[N1], int g, int lane) {
  float x[N1], y[N1];
#pragma unroll
  for (int j = 0; j < N1; ++j) {
    x[j] = a[j].x;
    y[j] = a[j].y;
  }
#pragma unroll
  for (int j = 0; j < N1; ++j) {
    const float px = row_prev<N1, N2>(x, j, g, lane),
                py = row_prev<N1, N2>(y, j, g, lane),
                nx = row_next<N1, N2>(x, j, g, lane),
                ny = row_next<N1, N2>(y, j, g, lane);
    f[j] = make_float2(stencil4f(px, py, y[j], nx),
                       stencil4f(py, x[j], nx, ny));
  }
}

// ---------------------------------------------------------------------------
// Columns, N2 threads per column, each holding N1 values
// ---------------------------------------------------------------------------

// First half of a forward DFT of N values by thread g of its column: on
// entry a[j1] = x[N2 j1 + g]; the N1-point DFTs, the twiddle and the write
// to the exchange ex (slot q of the column at ex[q * cs]).
template <int N>
__device__ __forceinline__ void col_fwd_put(float2 (&a)[Split<N>::N1],
                                            float2* ex, int cs, int g) {
  constexpr int N1 = Split<N>::N1, N2 = Split<N>::N2;
  dft<N1, false>(a);
#pragma unroll
  for (int k1 = 0; k1 < N1; ++k1)
    ex[(k1 * N2 + g) * cs] =
        k1 ? cmul(a[k1], c_w512[((g * k1) & (N - 1)) * (512 / N)]) : a[0];
}
// Second half, after a barrier: b[k2] = X[g + N2 u + N1 k2].  The slots read
// are this thread's alone.
template <int N>
__device__ __forceinline__ void col_fwd_get(float2 (&b)[Split<N>::N2],
                                            const float2* ex, int cs, int g,
                                            int u) {
  constexpr int N2 = Split<N>::N2;
#pragma unroll
  for (int j = 0; j < N2; ++j) b[j] = ex[((g + N2 * u) * N2 + j) * cs];
  dft<N2, false>(b);
}
// The converse (unnormalised): b[k2] = X[g + N2 u + N1 k2] into this
// thread's slots; after a barrier, a[j1] = x[N2 j1 + g].
template <int N>
__device__ __forceinline__ void col_inv_put(float2 (&b)[Split<N>::N2],
                                            float2* ex, int cs, int g, int u) {
  constexpr int N2 = Split<N>::N2;
  const int k1 = g + N2 * u;
  dft<N2, true>(b);
#pragma unroll
  for (int j2 = 0; j2 < N2; ++j2)
    ex[(k1 * N2 + j2) * cs] =
        j2 ? cmulc(b[j2], c_w512[((j2 * k1) & (N - 1)) * (512 / N)]) : b[0];
}
template <int N>
__device__ __forceinline__ void col_inv_get(float2 (&a)[Split<N>::N1],
                                            const float2* ex, int cs, int g) {
  constexpr int N1 = Split<N>::N1, N2 = Split<N>::N2;
#pragma unroll
  for (int k1 = 0; k1 < N1; ++k1) a[k1] = ex[(k1 * N2 + g) * cs];
  dft<N1, true>(a);
}

// ---------------------------------------------------------------------------
// Kernels
// ---------------------------------------------------------------------------

// Threads of the plane kernels: one per column and exchange group, at least
// four warps for the rows.
template <int NY, int M>
__host__ __device__ constexpr int plane_threads() {
  return M * Split<NY>::N2 > 128 ? M * Split<NY>::N2 : 128;
}
// Row pitch of the plane in shared memory (float2): the rows that a half
// warp touches together fall on different banks, and rows stay 16-byte
// aligned.
template <int M>
__host__ __device__ constexpr int plane_pitch() {
  return M + 8;
}
template <int NY, int M>
__host__ __device__ constexpr size_t plane_smem() {
  return (size_t)NY * (plane_pitch<M>() + M) * sizeof(float2);
}

// One x plane of one simulation of the run: rho -> S.  A warp transforms
// 32 / N2 rows at a time from global memory in registers (exchanges within
// the warp), then the block transforms the M columns (kz = 0 and kz = M are
// real and go through the y DFT together as column 0 = X[.][0] + i X[.][M],
// separated on the way out: Y0 = (C[ky] + conj C[-ky]) / 2, YM = (C[ky] -
// conj C[-ky]) / 2i), one exchange through shared memory, results straight
// to global memory.  Three block barriers; the same transform with the plane
// in shared memory between every stage and a barrier around each took 14.6
// us at 128^3 (25 MB read or cleared, 8 MB written, all in L2); this 10.5, the
// inverse 13.7 and 11.0.  zero_rho: clears rho for the next paint.
template <int NY, int M, bool PAIRS>
__global__ void __launch_bounds__(plane_threads<NY, M>())
k_fft_plane_fwd(const SimDev* __restrict__ sims, int first, int nx,
                float* __restrict__ rho, float2* __restrict__ dk,
                int painted, int zero_rho) {
  extern __shared__ __align__(16) float2 smem[];
  constexpr int T = plane_threads<NY, M>(), PP = plane_pitch<M>();
  constexpr int R1 = Split<M>::N1, R2 = Split<M>::N2, RW = 32 / R2;
  constexpr int N1 = Split<NY>::N1, N2 = Split<NY>::N2;
  constexpr int NZH = M + 1;
  float2* P = smem;            // NY rows of PP
  float2* Q = smem + NY * PP;  // the columns' exchange
  const int lane = threadIdx.x & 31, g = lane % R2;
  RowTw<M> tw;
  tw.load(g);
  pdl_wait();  // the density painted before
  const int s = first + blockIdx.x / nx;
  const int x = blockIdx.x % nx;
  const SimDev& S = sims[s];
  constexpr int NF = PAIRS ? 2 : 1;  // floats per cell
  float* plane = rho + (painted ? S.r_off : S.m_off) +
                 (int64_t)x * NY * NF * 2 * M;
  float2* dst = dk + S.s_off + (int64_t)x * NY * NZH;
#pragma unroll 1
  for (int r0 = (threadIdx.x >> 5) * RW; r0 < NY; r0 += T / 32 * RW) {
    const int r = r0 + lane / R2;  // NY is a multiple of RW
    float2 a[R1];
    row_load<M, PAIRS>(a, plane + r * NF * 2 * M, zero_rho, g, lane);
    float2* row = P + r * PP;
    row_r2c<M>(a, row, g, lane, tw);
    __syncwarp();  // the exchange has been read
#pragma unroll
    for (int u = 0; u < R1 / R2; ++u)
#pragma unroll
      for (int k2 = 0; k2 < R2; ++k2)
        row[g + R2 * u + R1 * k2] = a[u * R2 + k2];
  }
  __syncthreads();
  const int c = threadIdx.x % M, gc = threadIdx.x / M;
  const bool col = T == M * N2 || gc < N2;
  if (col) {
    float2 a[N1];
#pragma unroll
    for (int j1 = 0; j1 < N1; ++j1) a[j1] = P[(N2 * j1 + gc) * PP + c];
    col_fwd_put<NY>(a, Q + c, M, gc);
  }
  __syncthreads();
  float2* col0 = P;  // the plane has been read
  if (col) {
#pragma unroll
    for (int u = 0; u < N1 / N2; ++u) {
      float2 b[N2];
      col_fwd_get<NY>(b, Q + c, M, gc, u);
#pragma unroll
      for (int k2 = 0; k2 < N2; ++k2) {
        const int ky = gc + N2 * u + N1 * k2;
        if (c == 0)
          col0[ky] = b[k2];
        else
          dst[ky * NZH + c] = b[k2];
      }
    }
  }
  __syncthreads();
  for (int ky = threadIdx.x; ky < NY; ky += T) {
    const float2 v = col0[ky], vm = col0[(NY - ky) & (NY - 1)];
    dst[ky * NZH] = make_float2(0.5f * (v.x + vm.x), 0.5f * (v.y - vm.y));
    dst[ky * NZH + M] = make_float2(0.5f * (v.y + vm.y), -0.5f * (v.x - vm.x));
  }
}

// The x pass: out = inverse-DFT_x(pre * w(k) * DFT_x(in)) for kXCols
// consecutive (ky, kz) columns of one simulation per block (spectra in the
// R2C layout (x, y, z/2 + 1), unnormalised): the potential of
// k_fourier_potential, the same arithmetic per mode.  N2 threads per column
// hold N1 values each in registers from global memory and back, with one
// exchange through shared memory each way: the slots that a thread reads
// between the two are its own, so there are two barriers in all.  With zero,
// the block also zeroes its share of that buffer: zmul floats per cell of the
// sim (1: the painted density, from r_off; 4: the interleaved adjoint force
// mesh).
// Measured on B200 against a block that moved its columns through shared
// memory in 64-point sub-lines (about 20 barriers) and divided in double:
// 13.5 -> 7.2 us at 128^3, 0.47 -> 0.33 ms at 512^3 (1.08 GB, 3.2 TB/s), and
// with the density's clearing 69 -> 47 us at 256^3.  The new exchange with the
// double division took 13.0, 0.58 and 74: that division was the bound.
constexpr int kXCols = 16;
template <int NX>
__host__ __device__ constexpr int x_threads() {
  return kXCols * Split<NX>::N2;
}

// Blocks of the x pass that the registers of an SM hold.
template <int NX>
__host__ __device__ constexpr int x_blocks() {
  return NX == 512 ? 2 : NX == 256 ? 3 : NX == 128 ? 6 : 8;
}

// PLAIN: the transfer function is the Green's function alone.
template <int NX, bool PLAIN>
__global__ void __launch_bounds__(x_threads<NX>(), x_blocks<NX>())
k_fft_x(const SimDev* __restrict__ sims, int first, int nblk,
        const float2* in, float2* out, float* __restrict__ zero, int zmul,
        AxisTabs tabs, Green G, const int32_t* __restrict__ nsteps, int pos) {
  constexpr int N1 = Split<NX>::N1, N2 = Split<NX>::N2, C = kXCols;
  extern __shared__ __align__(16) float2 smem[];
  pdl_wait();  // the spectrum written before
  const int s = first + blockIdx.x / nblk;
  if (nsteps && pos > nsteps[s]) return;  // finished simulation
  const int blk = blockIdx.x % nblk;
  const SimDev& S = sims[s];
  const unsigned ncols = (unsigned)S.my * (unsigned)S.mzh;
  const int cl = threadIdx.x % C, g = threadIdx.x / C;
  const unsigned c = blk * C + cl;  // my is a multiple of 16
  float2* ex = smem + cl;
  const float2* src = in + S.s_off + c + (size_t)g * ncols;
  float2 a[N1];
#pragma unroll
  for (int j1 = 0; j1 < N1; ++j1) a[j1] = src[(size_t)(N2 * j1) * ncols];
  if (zero) {  // this block's share, in float4
    const int64_t q4 = (int64_t)zmul * S.mx * S.my * S.mz / 4;
    const int64_t per = (q4 + nblk - 1) / nblk;
    float4* r4 = reinterpret_cast<float4*>(
        zero + (zmul == 1 ? S.r_off : zmul * S.m_off));
    const int64_t e1 = min(q4, (blk + 1) * per);
    for (int64_t e = blk * per + threadIdx.x; e < e1; e += C * N2)
      r4[e] = make_float4(0.f, 0.f, 0.f, 0.f);
  }
  // potential spectrum delta * pre * w(k), w the transfer function G
  const unsigned ky = c / (unsigned)S.mzh, kz = c - ky * (unsigned)S.mzh;
  const float pre = (float)((double)S.bf * S.bf * S.bf /
                            ((double)S.mx * S.my * S.mz));
  const double* kkx = tabs.kk + S.tab;
  const float2* kk2 = tabs.kk2 + S.tab;
  const float* wx = tabs.win + S.tab;
  double kyz = 0.0;
  float2 kyz2 = make_float2(0.f, 0.f);
  float wyv = 1.f, wzv = 1.f;
  if (PLAIN) {
    kyz2 = two_add(kk2[S.mx + ky], kk2[S.mx + S.my + kz]);
  } else {
    kyz = kkx[S.mx + ky] + kkx[S.mx + S.my + kz];
    // the CIC windows only enter with deconvolution
    if (G.deconv) {
      wyv = wx[S.mx + ky];
      wzv = wx[S.mx + S.my + kz];
    }
  }
  col_fwd_put<NX>(a, ex, C, g);
  __syncthreads();
#pragma unroll
  for (int u = 0; u < N1 / N2; ++u) {
    float2 b[N2];
    col_fwd_get<NX>(b, ex, C, g, u);
#pragma unroll
    for (int k2 = 0; k2 < N2; ++k2) {
      const int kx = g + N2 * u + N1 * k2;
      const float w =
          PLAIN ? green_inv(kk2[kx], kyz2)
                : green_w(G, s, kkx[kx] + kyz, G.deconv ? wx[kx] : 1.f, wyv,
                          wzv);
      b[k2].x = __fmul_rn(__fmul_rn(b[k2].x, pre), w);
      b[k2].y = __fmul_rn(__fmul_rn(b[k2].y, pre), w);
    }
    col_inv_put<NX>(b, ex, C, g, u);
  }
  __syncthreads();
  col_inv_get<NX>(a, ex, C, g);
  float2* dst = out + S.s_off + c + (size_t)g * ncols;
#pragma unroll
  for (int j1 = 0; j1 < N1; ++j1) dst[(size_t)(N2 * j1) * ncols] = a[j1];
}

// Order-0 gradient: DFT along x, the three force spectra, inverse DFT along
// x of each.
template <int NX>
__global__ void __launch_bounds__(x_threads<NX>())
k_fft_x_grad3(const SimDev* __restrict__ sims, int first, int nblk,
              const float2* __restrict__ dk, float2* __restrict__ fk,
              AxisTabs tabs, Green G) {
  constexpr int N1 = Split<NX>::N1, N2 = Split<NX>::N2, C = kXCols;
  extern __shared__ __align__(16) float2 smem[];
  pdl_wait();
  const int s = first + blockIdx.x / nblk;
  const SimDev& S = sims[s];
  const unsigned ncols = (unsigned)S.my * (unsigned)S.mzh;
  const int cl = threadIdx.x % C, g = threadIdx.x / C;
  const unsigned c = (blockIdx.x % nblk) * C + cl;
  const int64_t nmodes = (int64_t)NX * ncols;
  float2* ex = smem + cl;
  const float2* src = dk + S.s_off + c + (size_t)g * ncols;
  float2 a[N1];
#pragma unroll
  for (int j1 = 0; j1 < N1; ++j1) a[j1] = src[(size_t)(N2 * j1) * ncols];
  const unsigned ky = c / (unsigned)S.mzh, kz = c - ky * (unsigned)S.mzh;
  const float pre = (float)((double)S.bf * S.bf * S.bf /
                            ((double)S.mx * S.my * S.mz));
  const double* kkx = tabs.kk + S.tab;
  const double kyz = kkx[S.mx + ky] + kkx[S.mx + S.my + kz];
  const float* wx = tabs.win + S.tab;
  const float* gx = tabs.grad + S.tab;
  const float gyv = gx[S.mx + ky], gzv = gx[S.mx + S.my + kz];
  col_fwd_put<NX>(a, ex, C, g);
  __syncthreads();
#pragma unroll
  for (int u = 0; u < N1 / N2; ++u) {
    float2 b[N2];
    col_fwd_get<NX>(b, ex, C, g, u);
#pragma unroll
    for (int k2 = 0; k2 < N2; ++k2) {
      const int kx = g + N2 * u + N1 * k2;
      const float w = green_w(G, s, kkx[kx] + kyz, wx[kx], wx[S.mx + ky],
                              wx[S.mx + S.my + kz]);
      a[u * N2 + k2] = make_float2(__fmul_rn(__fmul_rn(b[k2].x, pre), w),
                                   __fmul_rn(__fmul_rn(b[k2].y, pre), w));
    }
  }
#pragma unroll 1
  for (int d = 0; d < 3; ++d) {
#pragma unroll
    for (int u = 0; u < N1 / N2; ++u) {
      float2 b[N2];
#pragma unroll
      for (int k2 = 0; k2 < N2; ++k2) {
        const int kx = g + N2 * u + N1 * k2;
        const float gd = d == 0 ? gx[kx] : (d == 1 ? gyv : gzv);
        const float2 v = a[u * N2 + k2];
        b[k2] = make_float2(-__fmul_rn(v.y, gd), __fmul_rn(v.x, gd));
      }
      col_inv_put<NX>(b, ex, C, g, u);
    }
    __syncthreads();
    float2 f[N1];
    col_inv_get<NX>(f, ex, C, g);
    __syncthreads();  // the next component overwrites the exchange
    float2* o = fk + 3 * S.s_off + d * nmodes + c + (size_t)g * ncols;
#pragma unroll
    for (int j1 = 0; j1 < N1; ++j1) o[(size_t)(N2 * j1) * ncols] = f[j1];
  }
}

// ---------------------------------------------------------------------------
// z and y passes of meshes whose planes do not fit one block (ny and nz of
// 256 or 512): rows along z by warps in registers, columns along y as the x
// pass.  Each is one read and one write of the mesh or spectrum, the density
// formed from its z pairs and cleared in the first, the z component of the
// force taken in the last.  Measured against the library's plane transforms
// with a kernel for the pairs before and the whole stencil after: at 512^3
// 0.40 + 0.33 + 0.24 -> 0.41 + 0.27 ms forward, 0.24 + 0.34 + 0.41 -> 0.24 +
// 0.28 + 0.29 ms back; at 256^3, 35 + 27 -> 33 + 30 us and 27 + 34 + 55 -> 30
// + 42 + 41.  A plain density of 256^3 is better cleared by the x pass (6 us
// there) than here: rows of 8 bytes a lane read and cleared in one pass took
// 83 us.
// ---------------------------------------------------------------------------
constexpr int kZThreads = 256;

template <int M, bool PAIRS>
__global__ void __launch_bounds__(kZThreads, 2)
k_fft_z_fwd(const SimDev* __restrict__ sims, int first, int nrows,
            float* __restrict__ rho, float2* __restrict__ dk, int painted,
            int zero, const int32_t* __restrict__ nsteps, int pos) {
  constexpr int N1 = Split<M>::N1, N2 = Split<M>::N2, RW = 32 / N2;
  constexpr int PP = M + 8;  // rows of a half warp on different banks
  __shared__ float2 ex_[kZThreads / N2][PP];
  const int s = first + blockIdx.y;
  if (nsteps && pos > nsteps[s]) return;  // finished simulation
  const int lane = threadIdx.x & 31, g = lane % N2;
  RowTw<M> tw;
  tw.load(g);
  constexpr int NF = PAIRS ? 2 : 1;
  float* in = rho + (painted ? sims[s].r_off : sims[s].m_off);
  float2* out = dk + sims[s].s_off;
  float2* ex = ex_[threadIdx.x / N2];
  const int wpb = kZThreads / 32;
  for (int r0 = (blockIdx.x * wpb + (threadIdx.x >> 5)) * RW; r0 < nrows;
       r0 += gridDim.x * wpb * RW) {  // nrows is a multiple of RW
    const int r = r0 + lane / N2;
    float2 a[N1];
    row_load<M, PAIRS>(a, in + (size_t)r * NF * 2 * M, zero, g, lane);
    row_r2c<M>(a, ex, g, lane, tw);
    float2* o = out + (size_t)r * (M + 1);
#pragma unroll
    for (int e = 0; e < N1; ++e) {
      float2 v = a[e];
      if (e == 0 && g == 0) {  // X[0] and X[M], both real
        o[M] = make_float2(v.y, 0.f);
        v.y = 0.f;
      }
      o[g + N2 * (e / N2) + N1 * (e % N2)] = v;
    }
  }
}

// GRAD: also the z component of the force of each row.
template <int M, bool GRAD>
__global__ void __launch_bounds__(kZThreads, 2)
k_fft_z_inv(const SimDev* __restrict__ sims, int first, int nrows,
            const float2* __restrict__ spec, float* __restrict__ phi,
            float* __restrict__ fmesh, const int32_t* __restrict__ nsteps,
            int pos) {
  constexpr int N1 = Split<M>::N1, N2 = Split<M>::N2, RW = 32 / N2;
  constexpr int PP = M + 8;
  __shared__ float2 ex_[kZThreads / N2][PP];
  const int s = first + blockIdx.y;
  if (nsteps && pos > nsteps[s]) return;
  const int lane = threadIdx.x & 31, g = lane % N2;
  RowTw<M> tw;
  tw.load(g);
  const SimDev& S = sims[s];
  const float2* in = spec + S.s_off;
  float2* out = reinterpret_cast<float2*>(phi + S.m_off);
  float2* fz = reinterpret_cast<float2*>(
      fmesh + 3 * S.m_off + 2 * (int64_t)S.mx * S.my * S.mz);
  float2* ex = ex_[threadIdx.x / N2];
  const int wpb = kZThreads / 32;
  for (int r0 = (blockIdx.x * wpb + (threadIdx.x >> 5)) * RW; r0 < nrows;
       r0 += gridDim.x * wpb * RW) {
    const int r = r0 + lane / N2;
    const float2* x = in + (size_t)r * (M + 1);
    float2 a[N1];
#pragma unroll
    for (int e = 0; e < N1; ++e) a[e] = x[g + N2 * (e / N2) + N1 * (e % N2)];
    if (g == 0) a[0].y = x[M].x;  // both real
    row_c2r<M>(a, ex, g, lane, tw);
    const size_t o = (size_t)r * M + g;
#pragma unroll
    for (int j1 = 0; j1 < N1; ++j1) out[o + N2 * j1] = a[j1];
    if (GRAD) {
      float2 f[N1];
      row_grad<N1, N2>(a, f, g, lane);
#pragma unroll
      for (int j1 = 0; j1 < N1; ++j1) fz[o + N2 * j1] = f[j1];
    }
  }
}

// DFT along y of kXCols consecutive columns (x, kz) per block, in place.
template <int NY, bool INV>
__global__ void __launch_bounds__(x_threads<NY>(), x_blocks<NY>())
k_fft_y(const SimDev* __restrict__ sims, int first, float2* __restrict__ dk,
        const int32_t* __restrict__ nsteps, int pos) {
  constexpr int N1 = Split<NY>::N1, N2 = Split<NY>::N2, C = kXCols;
  extern __shared__ __align__(16) float2 smem[];
  const int s = first + blockIdx.y;
  if (nsteps && pos > nsteps[s]) return;
  const SimDev& S = sims[s];
  const unsigned nzh = S.mzh;
  const int cl = threadIdx.x % C, g = threadIdx.x / C;
  const unsigned q = blockIdx.x * C + cl;  // mx is a multiple of 16
  const unsigned x = q / nzh, kz = q - x * nzh;
  float2* col = dk + S.s_off + (size_t)x * NY * nzh + kz;
  float2* ex = smem + cl;
  if (!INV) {
    float2 a[N1];
#pragma unroll
    for (int j1 = 0; j1 < N1; ++j1) a[j1] = col[(N2 * j1 + g) * nzh];
    col_fwd_put<NY>(a, ex, C, g);
    __syncthreads();
#pragma unroll
    for (int u = 0; u < N1 / N2; ++u) {
      float2 b[N2];
      col_fwd_get<NY>(b, ex, C, g, u);
#pragma unroll
      for (int k2 = 0; k2 < N2; ++k2)
        col[(g + N2 * u + N1 * k2) * nzh] = b[k2];
    }
  } else {
#pragma unroll
    for (int u = 0; u < N1 / N2; ++u) {
      float2 b[N2];
#pragma unroll
      for (int k2 = 0; k2 < N2; ++k2)
        b[k2] = col[(g + N2 * u + N1 * k2) * nzh];
      col_inv_put<NY>(b, ex, C, g, u);
    }
    __syncthreads();
    float2 a[N1];
    col_inv_get<NY>(a, ex, C, g);
#pragma unroll
    for (int j1 = 0; j1 < N1; ++j1) col[(N2 * j1 + g) * nzh] = a[j1];
  }
}

// ---------------------------------------------------------------------------
// 2LPT on the particle lattice (flowpm/tfpm.py:148-180 lpt_init) for
// power-of-two axes of 16 to 512.  A displacement or a second derivative of
// the potential is the Laplacian's inverse T times a factor per axis and a
// power of i, so the factor of an axis is applied where that axis is
// transformed back and the outputs share the passes before it:
//
//   rows forward, k_lpt_y_fwd     linear field -> spectrum along (y, z)
//   k_lpt_x       forward and back along x of T, gx T, gx^2 T
//   k_lpt_y_inv   back along y of gy^b (gx^a T), a + b <= 2: six spectra
//   k_lpt_rows_source  back along z of the six second derivatives of a row,
//                 the second-order source, and its row forward again
//   k_lpt_y_fwd, k_lpt_x, k_lpt_y_inv  of the source: three spectra
//   k_lpt_rows_out  back along z of both displacements; disp, mom and force
//
// Bound by memory: 49 passes over a field of 4 bytes per cell, against 98 of
// one transform per output (library transforms of three passes each, a
// kernel for the spectra, the source and the particles).  Measured on B200,
// 256^3 to second order with positions: 1.82 -> 0.85 ms (3.3 GB, 3.9 TB/s;
// y back 117 us a pass, rows out 229, source 156, x 66).
// ---------------------------------------------------------------------------

// Spectrum row <-> the lane's elements k = g + N2 u + N1 k2, X[0] and X[M]
// (both real) in one.
template <int M>
__device__ __forceinline__ int row_k(int g, int e) {
  constexpr int N1 = Split<M>::N1, N2 = Split<M>::N2;
  return g + N2 * (e / N2) + N1 * (e % N2);
}

template <int M>
__device__ __forceinline__ void spec_put(const float2 (&a)[Split<M>::N1],
                                         float2* o, int g) {
#pragma unroll
  for (int e = 0; e < Split<M>::N1; ++e) {
    float2 v = a[e];
    if (e == 0 && g == 0) {
      o[M] = make_float2(v.y, 0.f);
      v.y = 0.f;
    }
    o[row_k<M>(g, e)] = v;
  }
}

// The row x as stored; mid: X[M] (lane g = 0).
template <int M>
__device__ __forceinline__ void spec_get(float2 (&a)[Split<M>::N1],
                                         float2& mid, const float2* x, int g) {
#pragma unroll
  for (int e = 0; e < Split<M>::N1; ++e) a[e] = x[row_k<M>(g, e)];
  mid = g ? make_float2(0.f, 0.f) : x[M];
}

// Times gz^p and, with I, times i; then packed for row_c2r.
template <int M, bool I>
__device__ __forceinline__ void spec_factor(float2 (&a)[Split<M>::N1],
                                            float2 mid, const float* gz, int p,
                                            int g) {
  if (p > 0) {
    const float gm = __ldg(gz + M);
#pragma unroll
    for (int e = 0; e < Split<M>::N1; ++e) {
      const float f = __ldg(gz + row_k<M>(g, e));
      a[e].x *= f;
      a[e].y *= f;
      if (p > 1) {
        a[e].x *= f;
        a[e].y *= f;
      }
    }
    mid.x *= gm;
    mid.y *= gm;
    if (p > 1) {
      mid.x *= gm;
      mid.y *= gm;
    }
  }
  if (I) {
#pragma unroll
    for (int e = 0; e < Split<M>::N1; ++e) a[e] = make_float2(-a[e].y, a[e].x);
    mid.x = -mid.y;
  }
  if (g == 0) a[0].y = mid.x;
}

// Pitch of the rows of M + 1 modes: whole sectors, so that 16 consecutive
// columns are four of them.  The columns of the padding are transformed too
// (nothing reads them).  A pitch of whole lines (M + 16) was no faster.
template <int M>
__host__ __device__ constexpr int lpt_pitch() {
  return M + 4;
}

constexpr int kLptZThreads = 128;  // row kernels of one row at a time
constexpr int kLptOutThreads = 96;

// nrows (all simulations of the run) is a multiple of the rows of a warp.
template <int M>
__global__ void __launch_bounds__(kLptZThreads, 4)
k_lpt_rows_fwd(const float* __restrict__ in, float2* __restrict__ out,
               int nrows) {
  constexpr int N1 = Split<M>::N1, N2 = Split<M>::N2, RW = 32 / N2;
  __shared__ float2 ex_[kLptZThreads / N2][M + 8];
  const int lane = threadIdx.x & 31, g = lane % N2, wpb = kLptZThreads / 32;
  RowTw<M> tw;
  tw.load(g);
  for (int r0 = (blockIdx.x * wpb + (threadIdx.x >> 5)) * RW; r0 < nrows;
       r0 += gridDim.x * wpb * RW) {
    const int r = r0 + lane / N2;
    const float2* p = reinterpret_cast<const float2*>(in) + (size_t)r * M;
    float2 a[N1];
#pragma unroll
    for (int j1 = 0; j1 < N1; ++j1) a[j1] = p[N2 * j1 + g];
    row_r2c<M>(a, ex_[threadIdx.x / N2], g, lane, tw);
    spec_put<M>(a, out + (size_t)r * lpt_pitch<M>(), g);
  }
}

// Forward along y, in place; columns (x, kz) of all simulations of the run.
template <int NY>
__global__ void __launch_bounds__(x_threads<NY>(), x_blocks<NY>())
k_lpt_y_fwd(float2* __restrict__ dk, unsigned nzh) {
  constexpr int N1 = Split<NY>::N1, N2 = Split<NY>::N2, C = kXCols;
  extern __shared__ __align__(16) float2 smem[];
  const int cl = threadIdx.x % C, g = threadIdx.x / C;
  const unsigned q = blockIdx.x * C + cl;  // nx is a multiple of 16
  const unsigned x = q / nzh, kz = q - x * nzh;
  float2* col = dk + (size_t)x * NY * nzh + kz;
  float2* ex = smem + cl;
  float2 a[N1];
#pragma unroll
  for (int j1 = 0; j1 < N1; ++j1) a[j1] = col[(N2 * j1 + g) * nzh];
  col_fwd_put<NY>(a, ex, C, g);
  __syncthreads();
#pragma unroll
  for (int u = 0; u < N1 / N2; ++u) {
    float2 b[N2];
    col_fwd_get<NY>(b, ex, C, g, u);
#pragma unroll
    for (int k2 = 0; k2 < N2; ++k2) col[(g + N2 * u + N1 * k2) * nzh] = b[k2];
  }
}

// Blocks of the kernels below that the registers of an SM should hold (at 256
// unbounded, one: the y pass back 166 against 126 us; three spill and gain
// nothing).
template <int N>
__host__ __device__ constexpr int lpt_blocks() {
  return N == 512 ? 1 : N == 256 ? 2 : N == 128 ? 4 : 8;
}

// Column v (in kx or ky order of the transform) back along its axis, n times:
// as it is, then times the axis factor each.  Output d goes to o + slot[d].
template <int N>
__device__ __forceinline__ void lpt_outputs(float2 (&v)[Split<N>::N1],
                                            float2* ex, int g, int n,
                                            const float* gr, float2* o,
                                            size_t stride, longlong3 slot) {
  constexpr int N1 = Split<N>::N1, N2 = Split<N>::N2, C = kXCols;
#pragma unroll 1
  for (int d = 0; d < n; ++d) {
    if (d > 0) {
#pragma unroll
      for (int e = 0; e < N1; ++e) {
        const float f = __ldg(gr + g + N2 * (e / N2) + N1 * (e % N2));
        v[e].x *= f;
        v[e].y *= f;
      }
    }
    __syncthreads();  // the exchange is free
#pragma unroll
    for (int u = 0; u < N1 / N2; ++u) {
      float2 b[N2];
#pragma unroll
      for (int k2 = 0; k2 < N2; ++k2) b[k2] = v[u * N2 + k2];
      col_inv_put<N>(b, ex, C, g, u);
    }
    __syncthreads();
    float2 f[N1];
    col_inv_get<N>(f, ex, C, g);
    float2* w = o + (d == 0 ? slot.x : d == 1 ? slot.y : slot.z);
#pragma unroll
    for (int j1 = 0; j1 < N1; ++j1) w[(N2 * j1 + g) * stride] = f[j1];
  }
}

// Forward along x, the inverse Laplacian, back along x: nout of T, gx T and
// gx^2 T.  kk2, gx: the lattice's axis tables.
template <int NX>
__global__ void __launch_bounds__(x_threads<NX>(), lpt_blocks<NX>())
k_lpt_x(const float2* __restrict__ in, float2* __restrict__ out,
        int64_t slot, int nblk, unsigned ny, unsigned nzh,
        const float2* __restrict__ kk2, const float* __restrict__ gx,
        int nout) {
  constexpr int N1 = Split<NX>::N1, N2 = Split<NX>::N2, C = kXCols;
  extern __shared__ __align__(16) float2 smem[];
  const unsigned ncols = ny * nzh;
  const int cl = threadIdx.x % C, g = threadIdx.x / C;
  const int b0 = blockIdx.x / nblk;
  const unsigned c = (blockIdx.x - b0 * nblk) * C + cl;  // ny % 16 == 0
  const size_t at = (size_t)b0 * NX * ncols + c;
  float2* ex = smem + cl;
  const float2* src = in + at + (size_t)g * ncols;
  float2 v[N1];
#pragma unroll
  for (int j1 = 0; j1 < N1; ++j1) v[j1] = src[(size_t)(N2 * j1) * ncols];
  const unsigned ky = c / nzh, kz = c - ky * nzh;
  const unsigned nz = 2 * (nzh - 4);
  const float pre = (float)(1.0 / ((double)NX * ny * nz));
  const float2 kyz = two_add(kk2[NX + ky], kk2[NX + ny + min(kz, nz / 2)]);
  col_fwd_put<NX>(v, ex, C, g);
  __syncthreads();
#pragma unroll
  for (int u = 0; u < N1 / N2; ++u) {
    float2 b[N2];
    col_fwd_get<NX>(b, ex, C, g, u);
#pragma unroll
    for (int k2 = 0; k2 < N2; ++k2) {
      // 0 at k = 0, where the reference's 1 meets a gradient of 0
      const float w = green_inv(kk2[g + N2 * u + N1 * k2], kyz);
      v[u * N2 + k2] = make_float2(__fmul_rn(__fmul_rn(b[k2].x, pre), w),
                                   __fmul_rn(__fmul_rn(b[k2].y, pre), w));
    }
  }
  lpt_outputs<NX>(v, ex, g, nout, gx, out + at, ncols,
                  longlong3{0, slot, 2 * slot});
}

// Back along y of gy^b t[a], b <= nout - 1 - a for the nout spectra t of
// k_lpt_x, into the slots o[] in the order (a, b) = (0, 0), (0, 1), ...
struct LptSlots {
  int o[6];
};
template <int NY>
__global__ void __launch_bounds__(x_threads<NY>(), lpt_blocks<NY>())
k_lpt_y_inv(const float2* __restrict__ t, float2* __restrict__ u,
            int64_t slot, unsigned nzh, const float* __restrict__ gy, int nout,
            const __grid_constant__ LptSlots S) {
  constexpr int N1 = Split<NY>::N1, N2 = Split<NY>::N2, C = kXCols;
  extern __shared__ __align__(16) float2 smem[];
  const int cl = threadIdx.x % C, g = threadIdx.x / C;
  const unsigned q = blockIdx.x * C + cl;
  const unsigned x = q / nzh, kz = q - x * nzh;
  const size_t at = (size_t)x * NY * nzh + kz;
  int k = 0;
#pragma unroll 1
  for (int a = 0; a < nout; ++a) {
    const float2* col = t + a * slot + at;
    float2 v[N1];
#pragma unroll
    for (int e = 0; e < N1; ++e)
      v[e] = col[(size_t)(g + N2 * (e / N2) + N1 * (e % N2)) * nzh];
    const int n = nout - a;
    lpt_outputs<NY>(v, smem + cl, g, n, gy, u + at, nzh,
                    longlong3{S.o[k] * slot, n > 1 ? S.o[k + 1] * slot : 0,
                              n > 2 ? S.o[k + 2] * slot : 0});
    k += n;
  }
}

// Rows of the six spectra u -> second derivatives (their common sign dropped,
// as the source is quadratic) -> source, forward along z.
template <int M>
__global__ void __launch_bounds__(kLptZThreads, 3)
k_lpt_rows_source(const float2* __restrict__ u, int64_t slot,
                  float2* __restrict__ out, int nrows,
                  const float* __restrict__ gz) {
  constexpr int N1 = Split<M>::N1, N2 = Split<M>::N2, RW = 32 / N2;
  __shared__ float2 ex_[kLptZThreads / N2][M + 8];
  const int lane = threadIdx.x & 31, g = lane % N2, wpb = kLptZThreads / 32;
  float2* ex = ex_[threadIdx.x / N2];
  RowTw<M> tw;
  tw.load(g);
  const float c37 = (float)(3.0 / 7.0);
  for (int r0 = (blockIdx.x * wpb + (threadIdx.x >> 5)) * RW; r0 < nrows;
       r0 += gridDim.x * wpb * RW) {
    const size_t at = (size_t)(r0 + lane / N2) * lpt_pitch<M>();
    float2 s[N1], t[N1];
#pragma unroll 1
    for (int d = 0; d < 6; ++d) {
      // xx, yy, zz, yz, zx, xy = slots 5, 2, 0, 1, 3, 4 times gz^p
      const int from = d == 0 ? 5 : d == 1 ? 2 : d == 2 ? 0 : d == 3 ? 1
                                                      : d == 4 ? 3 : 4;
      const int p = d == 2 ? 2 : d == 3 || d == 4 ? 1 : 0;
      float2 a[N1], mid;
      spec_get<M>(a, mid, u + from * slot + at, g);
      spec_factor<M, false>(a, mid, gz, p, g);
      row_c2r<M>(a, ex, g, lane, tw);
#pragma unroll
      for (int j = 0; j < N1; ++j) {
        if (d == 0) {
          s[j] = a[j];
        } else if (d == 1) {
          t[j] = make_float2(__fadd_rn(s[j].x, a[j].x),
                             __fadd_rn(s[j].y, a[j].y));
          s[j] = make_float2(__fmul_rn(s[j].x, a[j].x),
                             __fmul_rn(s[j].y, a[j].y));
        } else if (d == 2) {
          s[j].x = __fmaf_rn(t[j].x, a[j].x, s[j].x);
          s[j].y = __fmaf_rn(t[j].y, a[j].y, s[j].y);
        } else {
          s[j].x = __fmaf_rn(-a[j].x, a[j].x, s[j].x);
          s[j].y = __fmaf_rn(-a[j].y, a[j].y, s[j].y);
        }
      }
    }
#pragma unroll
    for (int j = 0; j < N1; ++j)
      s[j] = make_float2(__fmul_rn(s[j].x, c37), __fmul_rn(s[j].y, c37));
    row_r2c<M>(s, ex, g, lane, tw);
    spec_put<M>(s, out + at, g);
  }
}

// Rows of the displacement spectra -> disp (positions with shift), mom and
// force of the row's particles.  Warp d of a block takes component d of the
// same rows, the first-order displacement from slot 3, 1 or 0 and the second
// (order 2) from 5, 4 or 2, both in registers; the arrays, interleaved x, y, z,
// go through shared memory one after the other, through two buffers in turn.
template <int M>
__global__ void __launch_bounds__(kLptOutThreads, 4)
k_lpt_rows_out(const float2* __restrict__ u, int64_t slot, int order,
               const float* __restrict__ gz, const float* __restrict__ coef,
               int nrows, unsigned nx, unsigned ny, int shift,
               float* __restrict__ disp, float* __restrict__ mom,
               float* __restrict__ force) {
  constexpr int N1 = Split<M>::N1, N2 = Split<M>::N2, RW = 32 / N2;
  constexpr int NZ = 2 * M, P = 3 * NZ + 16;  // rows on different banks
  __shared__ float2 ex_[kLptOutThreads / N2][M + 8];
  __shared__ __align__(16) float stage[2][RW * P];
  const int lane = threadIdx.x & 31, g = lane % N2, d = threadIdx.x >> 5;
  float2* ex = ex_[threadIdx.x / N2];
  RowTw<M> tw;
  tw.load(g);
  int buf = 0;
  for (int r0 = blockIdx.x * RW; r0 < nrows; r0 += gridDim.x * RW) {
    const unsigned r = r0 + lane / N2;
    const size_t at = (size_t)r * lpt_pitch<M>();
    const unsigned x = r / ny, b = x / nx;  // one b for the rows of a block
    const float* c = coef + 6 * b;
    float2 p1[N1], p2[N1], mid;
    spec_get<M>(p1, mid, u + (d == 0 ? 3 : d == 1 ? 1 : 0) * slot + at, g);
    spec_factor<M, true>(p1, mid, gz, d == 2, g);
    row_c2r<M>(p1, ex, g, lane, tw);
    const float c0 = c[0], c1 = c[1];
    if (order == 2) {
      spec_get<M>(p2, mid, u + (d == 0 ? 5 : d == 1 ? 4 : 2) * slot + at, g);
      spec_factor<M, true>(p2, mid, gz, d == 2, g);
      row_c2r<M>(p2, ex, g, lane, tw);
#pragma unroll
      for (int j = 0; j < N1; ++j)
        p2[j] = make_float2(__fmul_rn(c1, p2[j].x), __fmul_rn(c1, p2[j].y));
    }
#pragma unroll
    for (int j = 0; j < N1; ++j)
      p1[j] = make_float2(__fmul_rn(c0, p1[j].x), __fmul_rn(c0, p1[j].y));
    const float q = d == 0 ? (float)(x - b * nx) : (float)(r - x * ny);
#pragma unroll 1
    for (int w = 0; w < 3; ++w) {  // disp, mom, force
      float* st = stage[buf] + (lane / N2) * P + d;
      const float f1 = w ? c[2 * w] : 1.f, f2 = w ? c[2 * w + 1] : 1.f;
#pragma unroll
      for (int j = 0; j < N1; ++j) {
        const int k = 2 * (N2 * j + g);
        float2 v = make_float2(__fmul_rn(f1, p1[j].x), __fmul_rn(f1, p1[j].y));
        if (order == 2) {
          v.x = __fadd_rn(v.x, __fmul_rn(f2, p2[j].x));
          v.y = __fadd_rn(v.y, __fmul_rn(f2, p2[j].y));
        }
        if (w == 0 && shift) {
          v.x = __fadd_rn(v.x, d == 2 ? (float)k : q);
          v.y = __fadd_rn(v.y, d == 2 ? (float)(k + 1) : q);
        }
        // lanes alternate between the two cells: odd and even banks
        st[3 * k + 3 * (g & 1)] = g & 1 ? v.y : v.x;
        st[3 * k + 3 - 3 * (g & 1)] = g & 1 ? v.x : v.y;
      }
      __syncthreads();
      float4* o = reinterpret_cast<float4*>(w == 0 ? disp : w == 1 ? mom
                                                                   : force) +
                  (size_t)r0 * (3 * NZ / 4);
      // the block leaves this buffer alone until the barrier after next
#pragma unroll 4
      for (int e = threadIdx.x; e < RW * (3 * NZ / 4); e += kLptOutThreads) {
        const int row = e / (3 * NZ / 4), t = e - row * (3 * NZ / 4);
        o[e] = *reinterpret_cast<const float4*>(stage[buf] + row * P + 4 * t);
      }
      buf ^= 1;
    }
  }
}

// Output modes of k_fft_plane_inv.
enum PlaneOut {
  kOutStencil = 0,  // potential -> phi, force y and z by the 4-point stencil
  kOutGrad3 = 1,    // three force spectra -> the three force meshes
  kOutReal = 2      // one spectrum -> one real mesh (phi)
};

// One x plane of one spectrum: inverse DFT along y from global memory (one
// exchange), complex-to-real along z by warps in registers: Zc[k] = A + i
// conj(W^k) B with A = X[k] + conj X[M-k], B = X[k] - conj X[M-k], and the
// inverse M-point DFT of Zc gives x[2m] + i x[2m+1].  The columns kz = 0 and
// kz = M, real after the y inverse, share one complex column (X[.][0] + i
// X[.][M]).  With the stencil, the z component comes from the row in
// registers, the y component from the plane in shared memory, each thread
// walking along y with a window of five rows.
template <int NY, int M, int MODE>
__global__ void __launch_bounds__(plane_threads<NY, M>())
k_fft_plane_inv(const SimDev* __restrict__ sims, int first, int nx,
                const float2* __restrict__ spec, float* __restrict__ fmesh,
                float* __restrict__ phi) {
  extern __shared__ __align__(16) float2 smem[];
  constexpr bool GRAD3 = MODE == kOutGrad3;
  constexpr int T = plane_threads<NY, M>(), PP = plane_pitch<M>();
  constexpr int R1 = Split<M>::N1, R2 = Split<M>::N2, RW = 32 / R2;
  constexpr int N1 = Split<NY>::N1, N2 = Split<NY>::N2;
  constexpr int NZH = M + 1;
  float2* P = smem;
  float2* Q = smem + NY * PP;
  const int lane = threadIdx.x & 31, g = lane % R2;
  RowTw<M> tw;
  tw.load(g);
  pdl_wait();
  const int d = GRAD3 ? blockIdx.x % 3 : 0;
  const int rest = GRAD3 ? blockIdx.x / 3 : blockIdx.x;
  const int x = rest % nx;
  const int s = first + rest / nx;
  const SimDev& S = sims[s];
  const int64_t nmodes = (int64_t)nx * NY * NZH;
  const int64_t mcells = (int64_t)nx * NY * 2 * M;
  const int64_t plane = (int64_t)x * NY * 2 * M;
  const float2* src = spec + (GRAD3 ? 3 * S.s_off + d * nmodes : S.s_off) +
                      (int64_t)x * NY * NZH;
  const int c = threadIdx.x % M, gc = threadIdx.x / M;
  const bool col = T == M * N2 || gc < N2;
  if (col) {
#pragma unroll
    for (int u = 0; u < N1 / N2; ++u) {
      float2 b[N2];
#pragma unroll
      for (int k2 = 0; k2 < N2; ++k2) {
        const float2* row = src + (gc + N2 * u + N1 * k2) * NZH;
        b[k2] = row[c];
        if (c == 0) {
          const float2 xm = row[M];
          b[k2] = make_float2(b[k2].x - xm.y, b[k2].y + xm.x);
        }
      }
      col_inv_put<NY>(b, Q + c, M, gc, u);
    }
  }
  __syncthreads();
  if (col) {
    float2 a[N1];
    col_inv_get<NY>(a, Q + c, M, gc);
#pragma unroll
    for (int j1 = 0; j1 < N1; ++j1) P[(N2 * j1 + gc) * PP + c] = a[j1];
  }
  __syncthreads();
  float2* out = reinterpret_cast<float2*>(
      GRAD3 ? fmesh + 3 * S.m_off + d * mcells + plane : phi + S.m_off + plane);
  float2* fz = reinterpret_cast<float2*>(fmesh + 3 * S.m_off + 2 * mcells +
                                         plane);
#pragma unroll 1
  for (int r0 = (threadIdx.x >> 5) * RW; r0 < NY; r0 += T / 32 * RW) {
    const int r = r0 + lane / R2;
    float2* row = P + r * PP;
    float2 a[R1];
#pragma unroll
    for (int u = 0; u < R1 / R2; ++u)
#pragma unroll
      for (int k2 = 0; k2 < R2; ++k2)
        a[u * R2 + k2] = row[g + R2 * u + R1 * k2];
    row_c2r<M>(a, row, g, lane, tw);
#pragma unroll
    for (int j1 = 0; j1 < R1; ++j1) out[r * M + R2 * j1 + g] = a[j1];
    if (MODE == kOutStencil) {
      float2 f[R1];
      row_grad<R1, R2>(a, f, g, lane);
#pragma unroll
      for (int j1 = 0; j1 < R1; ++j1) fz[r * M + R2 * j1 + g] = f[j1];
      __syncwarp();  // the exchange has been read
#pragma unroll
      for (int j1 = 0; j1 < R1; ++j1) row[R2 * j1 + g] = a[j1];
    }
  }
  if (MODE != kOutStencil) return;
  __syncthreads();
  // y component: four z cells per thread, YL rows of them
  constexpr int NQ = M / 2;                        // float4 per row
  constexpr int NT = T / NQ < NY ? T / NQ : NY;    // threads along y
  constexpr int YL = NY / NT;
  const int q = threadIdx.x % NQ, t = threadIdx.x / NQ;
  if (t >= NT) return;
  float4* fy = reinterpret_cast<float4*>(fmesh + 3 * S.m_off + mcells + plane);
  auto at = [&](int y) {
    return reinterpret_cast<const float4*>(P + (y & (NY - 1)) * PP)[q];
  };
  const int y0 = t * YL;
  float4 m2 = at(y0 - 2), m1 = at(y0 - 1), z = at(y0), p1 = at(y0 + 1);
#pragma unroll
  for (int i = 0; i < YL; ++i) {
    const float4 p2 = at(y0 + i + 2);
    fy[(y0 + i) * NQ + q] = make_float4(
        stencil4f(m2.x, m1.x, p1.x, p2.x), stencil4f(m2.y, m1.y, p1.y, p2.y),
        stencil4f(m2.z, m1.z, p1.z, p2.z), stencil4f(m2.w, m1.w, p1.w, p2.w));
    m2 = m1;
    m1 = z;
    z = p1;
    p1 = p2;
  }
}

// x component of the force from the potential planes x - 2 .. x + 2
// (periodic), four z cells per thread.
template <int NY, int NZ>
__global__ void __launch_bounds__(kFftThreads)
k_fft_stencil_x(const SimDev* __restrict__ sims, int first, int nx,
                const float* __restrict__ phi, float* __restrict__ fmesh) {
  pdl_wait();
  constexpr int PL = NY * NZ / 4;  // float4 per plane
  const int64_t total = (int64_t)nx * PL;
  const int s = first + blockIdx.y;
  const SimDev& S = sims[s];
  const float4* p = reinterpret_cast<const float4*>(phi + S.m_off);
  float4* o = reinterpret_cast<float4*>(fmesh + 3 * S.m_off);
  for (int64_t e = (int64_t)blockIdx.x * kFftThreads + threadIdx.x; e < total;
       e += (int64_t)gridDim.x * kFftThreads) {
    const int x = (int)(e / PL);
    const int r = (int)(e - (int64_t)x * PL);
    const float4 m2 = p[(int64_t)((x - 2 + nx) % nx) * PL + r];
    const float4 m1 = p[(int64_t)((x - 1 + nx) % nx) * PL + r];
    const float4 p1 = p[(int64_t)((x + 1) % nx) * PL + r];
    const float4 p2 = p[(int64_t)((x + 2) % nx) * PL + r];
    o[e] = make_float4(stencil4f(m2.x, m1.x, p1.x, p2.x),
                       stencil4f(m2.y, m1.y, p1.y, p2.y),
                       stencil4f(m2.z, m1.z, p1.z, p2.z),
                       stencil4f(m2.w, m1.w, p1.w, p2.w));
  }
}

// ---------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------

std::mutex g_tw_mu;
bool g_tw_ready[64] = {};

int allow_smem(const void* k, size_t bytes) {
  if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)bytes) != cudaSuccess) {
    cudaGetLastError();
    return FPM_ERR_CUDA;
  }
  return FPM_OK;
}

template <int NY, int M>
int set_plane_smem() {
  constexpr size_t b = plane_smem<NY, M>();
  for (const void* k : {(const void*)k_fft_plane_fwd<NY, M, true>,
                        (const void*)k_fft_plane_fwd<NY, M, false>,
                        (const void*)k_fft_plane_inv<NY, M, kOutStencil>,
                        (const void*)k_fft_plane_inv<NY, M, kOutGrad3>,
                        (const void*)k_fft_plane_inv<NY, M, kOutReal>})
    if (allow_smem(k, b) != FPM_OK) return FPM_ERR_CUDA;
  return FPM_OK;
}

template <int NX>
__host__ __device__ constexpr size_t x_smem() {
  return (size_t)NX * kXCols * sizeof(float2);
}

#define FPM_FFT_SIZES(X) X(16) X(32) X(64) X(128)
#define FPM_FFT_HALF(X) X(8) X(16) X(32) X(64)

bool pow2_in_range(int n) { return n >= 16 && n <= 128 && (n & (n - 1)) == 0; }

template <int NY>
int prepare_ny(int M) {
  switch (M) {
#define FPM_PREP_M(MM) \
  case MM: return set_plane_smem<NY, MM>();
    FPM_FFT_HALF(FPM_PREP_M)
#undef FPM_PREP_M
  }
  return FPM_ERR_UNSUPPORTED;
}

// The kernels of one mesh shape (NY, M = nz / 2).  rho: the painted density
// (pairs: z pairs), or with real_out a plain mesh.
template <int NY, int M>
void launch_shape(const SimDev* sims, int first, int n, int nx, float* rho,
                  bool pairs, int zero_rho, float2* dk, float2* fk, float* fmesh,
                  float* phi, AxisTabs tabs, const Green& G, bool grad3,
                  bool real_out, cudaStream_t st) {
  constexpr size_t smem = plane_smem<NY, M>();
  constexpr int T = plane_threads<NY, M>();
  auto fwd = pairs ? k_fft_plane_fwd<NY, M, true>
                   : k_fft_plane_fwd<NY, M, false>;
  launch_pdl(fwd, dim3(n * nx), dim3(T), smem, st, sims, first, nx, rho, dk,
             real_out ? 0 : 1, zero_rho);
  const int nblk = NY * (M + 1) / kXCols;  // NY is a multiple of 16
  const bool plain = green_plain(G);
  switch (nx) {
#define FPM_X_CASE(NN)                                                       \
  case NN:                                                                   \
    if (grad3)                                                               \
      launch_pdl(k_fft_x_grad3<NN>, dim3(n * nblk), dim3(x_threads<NN>()),   \
                 x_smem<NN>(), st, sims, first, nblk, (const float2*)dk, fk, \
                 tabs, G);                                                   \
    else                                                                     \
      launch_pdl(plain ? k_fft_x<NN, true> : k_fft_x<NN, false>,             \
                 dim3(n * nblk), dim3(x_threads<NN>()), x_smem<NN>(), st,    \
                 sims, first, nblk, (const float2*)dk, dk,                   \
                 (float*)nullptr, 1, tabs, G, (const int32_t*)nullptr, 0);   \
    break;
    FPM_FFT_SIZES(FPM_X_CASE)
#undef FPM_X_CASE
  }
  if (grad3) {
    k_fft_plane_inv<NY, M, kOutGrad3><<<n * nx * 3, T, smem, st>>>(
        sims, first, nx, fk, fmesh, phi);
    return;
  }
  if (real_out) {  // potential of `rho` -> phi
    k_fft_plane_inv<NY, M, kOutReal><<<n * nx, T, smem, st>>>(
        sims, first, nx, dk, nullptr, phi);
    return;
  }
  launch_pdl(k_fft_plane_inv<NY, M, kOutStencil>, dim3(n * nx),
             dim3(T), smem, st, sims, first, nx, (const float2*)dk, fmesh,
             phi);
  const int64_t quads = (int64_t)nx * NY * 2 * M / 4;
  int64_t bx = (quads + kFftThreads - 1) / kFftThreads;
  const int64_t cap = (int64_t)kNumSMs * 8 / (n < 1 ? 1 : n) + 1;
  if (bx > cap) bx = cap;
  launch_pdl(k_fft_stencil_x<NY, 2 * M>, dim3((unsigned)bx, (unsigned)n),
             dim3(kFftThreads), 0, st, sims, first, nx, (const float*)phi,
             fmesh);
}

template <int NY>
void launch_ny(int M, const SimDev* sims, int first, int n, int nx,
               float* rho, bool pairs, int zero_rho, float2* dk, float2* fk,
               float* fmesh, float* phi, AxisTabs tabs, const Green& G, bool grad3,
               bool real_out, cudaStream_t st) {
  switch (M) {
#define FPM_SHAPE_CASE(MM)                                                  \
  case MM:                                                                  \
    launch_shape<NY, MM>(sims, first, n, nx, rho, pairs, zero_rho, dk, fk,  \
                         fmesh, phi, tabs, G, grad3, real_out, st);         \
    break;
    FPM_FFT_HALF(FPM_SHAPE_CASE)
#undef FPM_SHAPE_CASE
  }
}

}  // namespace

bool fft_fused_supported(int nx, int ny, int nz) {
  return pow2_in_range(nx) && pow2_in_range(ny) && pow2_in_range(nz);
}

namespace {

// Twiddle tables and shared-memory limits of the x pass, once per device.
int prepare_device() {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) {
    cudaGetLastError();
    return FPM_ERR_CUDA;
  }
  std::lock_guard<std::mutex> lock(g_tw_mu);
  if (g_tw_ready[dev]) return FPM_OK;
  float2 w[512], w128[128];
  for (int m = 0; m < 512; ++m) {
    const double t = -2.0 * 3.14159265358979323846 * m / 512.0;
    w[m] = make_float2((float)std::cos(t), (float)std::sin(t));
  }
  for (int m = 0; m < 128; ++m) w128[m] = w[4 * m];
  if (cudaMemcpyToSymbol(c_w512, w, sizeof(w)) != cudaSuccess ||
      cudaMemcpyToSymbol(g_w512, w, sizeof(w)) != cudaSuccess ||
      cudaMemcpyToSymbol(c_w128, w128, sizeof(w128)) != cudaSuccess) {
    cudaGetLastError();
    return FPM_ERR_CUDA;
  }
  for (const void* k : {(const void*)k_fft_x<512, true>,
                        (const void*)k_fft_x<512, false>,
                        (const void*)k_fft_y<512, true>,
                        (const void*)k_fft_y<512, false>})
    if (allow_smem(k, x_smem<512>()) != FPM_OK) return FPM_ERR_CUDA;
  g_tw_ready[dev] = true;
  return FPM_OK;
}

}  // namespace

int fft_fused_prepare(int nx, int ny, int nz) {
  if (!fft_fused_supported(nx, ny, nz)) return FPM_ERR_UNSUPPORTED;
  if (prepare_device() != FPM_OK) return FPM_ERR_CUDA;
  const int M = nz / 2;
  switch (ny) {
#define FPM_PREP_CASE(NN) \
  case NN: return prepare_ny<NN>(M);
    FPM_FFT_SIZES(FPM_PREP_CASE)
#undef FPM_PREP_CASE
  }
  return FPM_ERR_UNSUPPORTED;
}

void launch_fft_force(const SimDev* sims, int first, int n, int nx, int ny,
                      int nz, float* rho, bool pairs, int zero_rho,
                      float2* dk, float2* fk, float* fmesh, float* phi, AxisTabs tabs,
                      const Green& G, bool grad3, cudaStream_t st) {
  if (n <= 0) return;
  g_launches.fetch_add(grad3 ? 3 : 4, std::memory_order_relaxed);
  switch (ny) {
#define FPM_NY_CASE(NN)                                                      \
  case NN:                                                                   \
    launch_ny<NN>(nz / 2, sims, first, n, nx, rho, pairs, zero_rho, dk, fk,  \
                  fmesh, phi, tabs, G, grad3, false, st);                    \
    break;
    FPM_FFT_SIZES(FPM_NY_CASE)
#undef FPM_NY_CASE
  }
}

void launch_fft_potential(const SimDev* sims, int first, int n, int nx,
                          int ny, int nz, const float* in, float2* dk,
                          float* out, AxisTabs tabs, const Green& G,
                          cudaStream_t st) {
  if (n <= 0) return;
  g_launches.fetch_add(3, std::memory_order_relaxed);
  float* src = const_cast<float*>(in);  // read only (zero_rho = 0)
  switch (ny) {
#define FPM_NY_CASE(NN)                                                   \
  case NN:                                                                \
    launch_ny<NN>(nz / 2, sims, first, n, nx, src, false, 0, dk, nullptr, \
                  nullptr, out, tabs, G, false, true, st);                \
    break;
    FPM_FFT_SIZES(FPM_NY_CASE)
#undef FPM_NY_CASE
  }
}

bool fft_xpass_supported(int nx, int ny, int nz) {
  return (nx == 256 || nx == 512) && ny % kXCols == 0 && nz % 2 == 0;
}

int fft_xpass_prepare() { return prepare_device(); }

void launch_fft_xpass(const SimDev* sims, int first, int n, int nx, int ny,
                      int nzh, const float2* in, float2* out, float* zero,
                      int zmul, AxisTabs tabs, const Green& G,
                      const int32_t* nsteps, int pos, cudaStream_t st) {
  if (n <= 0) return;
  g_launches.fetch_add(1, std::memory_order_relaxed);
  const int nblk = ny * nzh / kXCols;
  const unsigned grid = (unsigned)(n * nblk);
  const bool plain = green_plain(G);
  if (nx == 512) {
    auto k = plain ? k_fft_x<512, true> : k_fft_x<512, false>;
    k<<<grid, x_threads<512>(), x_smem<512>(), st>>>(
        sims, first, nblk, in, out, zero, zmul, tabs, G, nsteps, pos);
  } else {
    auto k = plain ? k_fft_x<256, true> : k_fft_x<256, false>;
    k<<<grid, x_threads<256>(), x_smem<256>(), st>>>(
        sims, first, nblk, in, out, zero, zmul, tabs, G, nsteps, pos);
  }
}

bool fft_zy_supported(int ny, int nz) {
  return (ny == 256 || ny == 512) && (nz == 256 || nz == 512);
}

namespace {

// Blocks of the row kernels: every SM full twice over.
dim3 z_grid(int nx, int ny, int M, int n) {
  const int rows = nx * ny, per = kZThreads / (M == 256 ? 16 : 8);
  const int blocks = rows / per, cap = kNumSMs * 8;
  return dim3((unsigned)(blocks < cap ? blocks : cap), (unsigned)n);
}

template <bool INV>
void launch_y(const SimDev* sims, int first, int n, int nx, int ny, int nz,
              float2* dk, const int32_t* nsteps, int pos, cudaStream_t st) {
  const dim3 grid((unsigned)(nx * (nz / 2 + 1) / kXCols), (unsigned)n);
  if (ny == 512)
    k_fft_y<512, INV><<<grid, x_threads<512>(), x_smem<512>(), st>>>(
        sims, first, dk, nsteps, pos);
  else
    k_fft_y<256, INV><<<grid, x_threads<256>(), x_smem<256>(), st>>>(
        sims, first, dk, nsteps, pos);
}

}  // namespace

void launch_fft_zy_fwd(const SimDev* sims, int first, int n, int nx, int ny,
                       int nz, float* rho, bool painted, bool pairs, int zero,
                       float2* dk, const int32_t* nsteps, int pos,
                       cudaStream_t st) {
  if (n <= 0) return;
  g_launches.fetch_add(2, std::memory_order_relaxed);
  const int M = nz / 2;
  auto k = M == 256 ? (pairs ? k_fft_z_fwd<256, true> : k_fft_z_fwd<256, false>)
                    : (pairs ? k_fft_z_fwd<128, true>
                             : k_fft_z_fwd<128, false>);
  k<<<z_grid(nx, ny, M, n), kZThreads, 0, st>>>(
      sims, first, nx * ny, rho, dk, painted ? 1 : 0, zero, nsteps, pos);
  launch_y<false>(sims, first, n, nx, ny, nz, dk, nsteps, pos, st);
}

void launch_fft_zy_inv(const SimDev* sims, int first, int n, int nx, int ny,
                       int nz, float2* spec, float* phi, float* fmesh,
                       const int32_t* nsteps, int pos, cudaStream_t st) {
  if (n <= 0) return;
  g_launches.fetch_add(2, std::memory_order_relaxed);
  launch_y<true>(sims, first, n, nx, ny, nz, spec, nsteps, pos, st);
  const int M = nz / 2;
  auto k = M == 256 ? (fmesh ? k_fft_z_inv<256, true> : k_fft_z_inv<256, false>)
                    : (fmesh ? k_fft_z_inv<128, true>
                             : k_fft_z_inv<128, false>);
  k<<<z_grid(nx, ny, M, n), kZThreads, 0, st>>>(sims, first, nx * ny, spec,
                                                phi, fmesh, nsteps, pos);
}

// ---------------------------------------------------------------------------
// 2LPT passes
// ---------------------------------------------------------------------------
bool lpt_fused_supported(int nx, int ny, int nz) {
  const auto ok = [](int n) {
    return n >= 16 && n <= 512 && (n & (n - 1)) == 0;
  };
  return ok(nx) && ok(ny) && ok(nz);
}

namespace {

#define FPM_LPT_SIZES(X) X(16) X(32) X(64) X(128) X(256) X(512)
#define FPM_LPT_HALF(X) X(8) X(16) X(32) X(64) X(128) X(256)

int row_blocks(int nrows, int M, int threads, int per_sm) {
  int n2 = 2;  // Split<M>::N2
  if (M >= 16) n2 = 4;
  if (M >= 64) n2 = 8;
  if (M >= 256) n2 = 16;
  const int per = threads / n2, blocks = (nrows + per - 1) / per;
  return blocks < kNumSMs * per_sm ? blocks : kNumSMs * per_sm;
}

}  // namespace

int lpt_fused_prepare() {
  if (prepare_device() != FPM_OK) return FPM_ERR_CUDA;
  for (const void* k :
       {(const void*)k_lpt_x<512>, (const void*)k_lpt_y_fwd<512>,
        (const void*)k_lpt_y_inv<512>})
    if (allow_smem(k, x_smem<512>()) != FPM_OK) return FPM_ERR_CUDA;
  return FPM_OK;
}

void launch_lpt_fused(const LptRun& R, cudaStream_t st) {
  g_launches.fetch_add(R.order == 2 ? 9 : 5, std::memory_order_relaxed);
  const int M = R.nz / 2, nrows = R.count * R.nx * R.ny;
  const unsigned nzh = M + 4;  // lpt_pitch
  const int64_t slot = (int64_t)nrows * nzh;
  const unsigned ygrid = (unsigned)((int64_t)R.count * R.nx * nzh / kXCols);
  const int nblk = (int)(R.ny * nzh / kXCols);
  const float* gy = R.grad + R.nx;
  const float* gz = gy + R.ny;
  float2 *u = R.six, *t = R.four, *sp = t + 3 * slot;
  switch (M) {
#define FPM_LPT_ROWS(MM)                                                  \
  case MM:                                                                \
    k_lpt_rows_fwd<MM><<<row_blocks(nrows, MM, kLptZThreads, 16),         \
                         kLptZThreads, 0, st>>>(R.linear, sp, nrows); \
    break;
    FPM_LPT_HALF(FPM_LPT_ROWS)
#undef FPM_LPT_ROWS
  }
  for (int pass = 1; pass <= R.order; ++pass) {
    const int nout = pass == 1 && R.order == 2 ? 3 : 2;
    const LptSlots S = nout == 3   ? LptSlots{{0, 1, 2, 3, 4, 5}}
                       : pass == 1 ? LptSlots{{0, 1, 3}}
                                   : LptSlots{{2, 4, 5}};
    switch (R.ny) {
#define FPM_LPT_Y(N)                                                     \
  case N:                                                                \
    k_lpt_y_fwd<N><<<ygrid, x_threads<N>(), x_smem<N>(), st>>>(sp, nzh); \
    break;
      FPM_LPT_SIZES(FPM_LPT_Y)
#undef FPM_LPT_Y
    }
    switch (R.nx) {
#define FPM_LPT_X(N)                                                         \
  case N:                                                                    \
    k_lpt_x<N><<<(unsigned)(R.count * nblk), x_threads<N>(), x_smem<N>(),    \
                 st>>>(sp, t, slot, nblk, R.ny, nzh, R.kk2, R.grad, nout); \
    break;
      FPM_LPT_SIZES(FPM_LPT_X)
#undef FPM_LPT_X
    }
    switch (R.ny) {
#define FPM_LPT_Y(N)                                                       \
  case N:                                                                  \
    k_lpt_y_inv<N><<<ygrid, x_threads<N>(), x_smem<N>(), st>>>(t, u, slot, \
                                                               nzh, gy, nout, S); \
    break;
      FPM_LPT_SIZES(FPM_LPT_Y)
#undef FPM_LPT_Y
    }
    if (pass == 1 && R.order == 2) {
      switch (M) {
#define FPM_LPT_ROWS(MM)                                                  \
  case MM:                                                                \
    k_lpt_rows_source<MM><<<row_blocks(nrows, MM, kLptZThreads, 12),      \
                            kLptZThreads, 0, st>>>(u, slot, sp, nrows, gz); \
    break;
        FPM_LPT_HALF(FPM_LPT_ROWS)
#undef FPM_LPT_ROWS
      }
    }
  }
  switch (M) {
#define FPM_LPT_ROWS(MM)                                                   \
  case MM:                                                                 \
    k_lpt_rows_out<MM><<<row_blocks(nrows, MM, 32, 16), kLptOutThreads, 0, \
                         st>>>(                                            \
        u, slot, R.order, gz, R.coef, nrows, R.nx, R.ny, R.shift, R.disp,  \
        R.mom, R.force);                                                   \
    break;
    FPM_LPT_HALF(FPM_LPT_ROWS)
#undef FPM_LPT_ROWS
  }
}

}  // namespace fpm

// lorenzo.cu -- the multidimensional Lorenzo variant's own passes for sm_103a.
//
// A field of nx*ny*nz floats (x fastest) is stored as the fastmode1 stream
// (blockSize 32) of the int32 codes
//     r = q - q[j-1] - q[k-1] + q[j-1][k-1]      (neighbours outside are 0)
// where q are fastmode1's quantization codes; the 1-D delta fastmode1 takes
// along x makes the packed values the 3-D Lorenzo residual.  The stream starts
// with [nx][ny][nz] as u32 little-endian.  This file holds the passes around
// the fastmode1 pipelines (which pack and unpack r as codes):
//   lorenzo_codes_kernel  x -> r, and the 12-byte dims header
//   lorenzo_zsum_kernel   r -> r summed along z, in place
//   lorenzo_ysum_kernel   ... summed along y and dequantized, in place
// The reference predicts along the flattened array only; this variant has no
// reference code and is checked against the oracle's restatement.
#include <cstring>
#include <type_traits>

#include "szp_device.cuh"
#include "szp_kernels.h"

namespace szp {

// (float)q * eb with the x86 NaN rule when eb is not finite (szpd_float.cc:67,86,112);
// the same arithmetic as the decode pipelines'.
__device__ __forceinline__ float x86_dequant(uint32_t q, float eb, bool special) {
  const float f = __int2float_rn((int32_t)q);
  const float r = __fmul_rn(f, eb);
  return special ? x86_nan_fix(r, f, eb) : r;
}

// x -> r.  A thread takes V neighbouring values of kCodeRows rows (and the row
// above them) through `kz` planes, so that a value is quantized 5/4 times
// instead of once for each of the four codes it enters: the differences along
// y are taken in registers, and those along z against the plane before, which
// the thread still holds.  V = 4 (16-byte loads and stores) where rows are
// multiples of 4 values and x and r 16-byte aligned, else 1.
// F2I runs at 16 lanes per clock and SM, an eighth of an add, and bound the
// version that quantized each value's three neighbours again: 49 M values
// (500 x 384 x 256) took 0.153 ms.  A field of one row (ny == 1) has no rows to
// share: R = 1, one quantization a value (2^24 values, a call: 154 us with R = 4,
// 95 so).
constexpr int kCodeRows = 4;

template <int V, int R>
__global__ void __launch_bounds__(256) lorenzo_codes_kernel(const LorenzoArgs a, uint32_t kz) {
  const float eb = a.eb_dev ? *a.eb_dev : a.eb;
  const float inv = __fdiv_rn(1.0f, eb);  // fastmode1's float inverse (szp_float.cc:185)
  uint32_t flags = 0;
  using XV = typename std::conditional<V == 4, float4, float>::type;
  const uint32_t nxv = a.nx / V, ny = a.ny, nz = a.nz;
  constexpr int TOP = R > 1 ? 0 : 1;  // x[0] is the row above, which a field of one row has not
  const uint64_t njb = (ny + R - 1) / R, nkc = (nz + kz - 1) / kz;
  const uint64_t items = nxv * njb * nkc, plane = (uint64_t)nxv * ny;
  const XV* __restrict__ xs = reinterpret_cast<const XV*>(a.x);
  for (uint64_t it = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; it < items;
       it += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t i = (uint32_t)(it % nxv);
    const uint64_t rest = it / nxv;
    const uint32_t j0 = (uint32_t)(rest % njb) * R, k0 = (uint32_t)(rest / njb) * kz;
    const uint32_t k1 = (uint32_t)min((uint64_t)nz, (uint64_t)k0 + kz), rows = min((uint32_t)R, ny - j0);
    uint32_t wp[R][V];  // y differences of the plane before
#pragma unroll
    for (int r = 0; r < R; r++)
#pragma unroll
      for (int v = 0; v < V; v++) wp[r][v] = 0;
    for (uint32_t k = k0 ? k0 - 1 : 0; k < k1; k++) {
      const uint64_t at = k * plane + (uint64_t)j0 * nxv + i;
      float x[R + 1][V];
#pragma unroll
      for (int r = TOP; r <= R; r++) {
        XV t{};  // row j0 - 1 + r
        if (r ? (uint32_t)r <= rows : j0 > 0) t = __ldg(xs + at + (int64_t)(r - 1) * nxv);
        memcpy(x[r], &t, sizeof t);
      }
      uint32_t q[R + 1][V];
      float pm = 0.0f;
#pragma unroll
      for (int r = TOP; r <= R; r++)
#pragma unroll
        for (int v = 0; v < V; v++) {
          const float p = __fmul_rz(x[r][v], inv);
          pm = maxabs_nan(pm, p);
          q[r][v] = (uint32_t)__float2int_rz(p);
        }
      if (!(pm < 16777216.0f)) {  // a value whose float product is not exact, or NaN
#pragma unroll
        for (int r = TOP; r <= R; r++)
#pragma unroll
          for (int v = 0; v < V; v++)
            if (r ? (uint32_t)r <= rows : j0 > 0) q[r][v] = (uint32_t)quantize(x[r][v], inv, flags);
      }
      if (TOP || j0 == 0) {
#pragma unroll
        for (int v = 0; v < V; v++) q[0][v] = 0;
      }
#pragma unroll
      for (int r = 0; r < R; r++) {
        int32_t o[V];
#pragma unroll
        for (int v = 0; v < V; v++) {
          const uint32_t w = q[r + 1][v] - q[r][v];
          o[v] = (int32_t)(w - wp[r][v]);
          wp[r][v] = w;
        }
        if (k >= k0 && (uint32_t)r < rows) {
          int32_t* dst = a.r + (at + (uint64_t)r * nxv) * V;
          if constexpr (V == 4) {
            *reinterpret_cast<int4*>(dst) = make_int4(o[0], o[1], o[2], o[3]);
          } else {
            dst[0] = o[0];
          }
        }
      }
    }
  }
  if (blockIdx.x == 0 && threadIdx.x < 12) {
    const uint32_t d[3] = {a.nx, a.ny, a.nz};
    a.head[threadIdx.x] = (uint8_t)(d[threadIdx.x >> 2] >> (8 * (threadIdx.x & 3)));
  }
  if (__any_sync(0xffffffffu, flags != 0) && (threadIdx.x & 31) == 0) atomicOr(a.err, kErrQuantRange);
}

// In-place running sums of q along a line of `len` elements `stride` apart,
// starting at p; U = 16 loads in flight before their sums are stored (8 left a
// third of the bandwidth unused: a column per thread is all the parallelism a
// field has), and for lines shorter than that 4, with twice the threads on an SM
// (1,000,000 x 5 x 3 values, both passes: 63 us with 16, 37 so).  DEQ: the sums are dequantized ((float)q * eb,
// szpd_float.cc:67,86,112) and stored as floats.
template <bool DEQ, int U>
__device__ __forceinline__ void lorenzo_line(int32_t* __restrict__ p, uint64_t stride, uint32_t len, float eb,
                                             bool special) {
  uint32_t run = 0;
  auto put = [&](uint64_t at) {
    if (DEQ) {
      reinterpret_cast<float*>(p)[at] = x86_dequant(run, eb, special);
    } else {
      p[at] = (int32_t)run;
    }
  };
  uint32_t j = 0;
  for (; j + U <= len; j += U) {
    uint32_t v[U];
#pragma unroll
    for (int u = 0; u < U; u++) v[u] = (uint32_t)p[(j + u) * stride];
#pragma unroll
    for (int u = 0; u < U; u++) {
      run += v[u];
      put((j + u) * stride);
    }
  }
  for (; j < len; j += 4) {  // the line's end
    uint32_t v[4];
#pragma unroll
    for (int u = 0; u < 4; u++) v[u] = j + u < len ? (uint32_t)p[(j + u) * stride] : 0u;
#pragma unroll
    for (int u = 0; u < 4; u++) {
      run += v[u];
      if (j + u < len) put((j + u) * stride);
    }
  }
}

// One thread per (j, i): sums along z.
template <int U>
__global__ void __launch_bounds__(64, U == 4 ? 32 : 1) lorenzo_zsum_kernel(const LorenzoArgs a) {
  const uint64_t cols = (uint64_t)a.nx * a.ny;
  for (uint64_t c = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; c < cols; c += (uint64_t)gridDim.x * blockDim.x)
    lorenzo_line<false, U>(a.q + c, cols, a.nz, 0.0f, false);
}

// One thread per (k, i): sums along y, then dequantizes in place; the last
// planes first, whose sums along z are still in L2 (of 126 MB).
template <int U>
__global__ void __launch_bounds__(64, U == 4 ? 32 : 1) lorenzo_ysum_kernel(const LorenzoArgs a) {
  const float eb = *a.eb_dev;
  const bool special = !isfinite(eb);
  const uint64_t cols = (uint64_t)a.nx * a.nz, plane = (uint64_t)a.nx * a.ny;
  for (uint64_t c = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; c < cols; c += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t i = c % a.nx, k = a.nz - 1 - c / a.nx;
    lorenzo_line<true, U>(a.q + k * plane + i, a.nx, a.ny, eb, special);
  }
}

static uint32_t lorenzo_grid(uint64_t items, uint32_t per_cta, uint32_t cap) {
  const uint64_t g = (items + per_cta - 1) / per_cta;
  return (uint32_t)(g < 1 ? 1 : (g > cap ? cap : g));
}

cudaError_t launch_lorenzo_codes(const LorenzoArgs& a, uint32_t sm_count, cudaStream_t st) {
  const bool v4 = (a.nx & 3) == 0 && ((uintptr_t)a.x & 15) == 0 && ((uintptr_t)a.r & 15) == 0;
  // columns of R rows; planes are split among threads until there are 1024 threads
  // per SM, but not below 5 (the plane before the first is read too)
  const uint32_t R = a.ny == 1 ? 1 : kCodeRows;
  const uint64_t cols = (uint64_t)(v4 ? a.nx / 4 : a.nx) * ((a.ny + R - 1) / R);
  uint32_t kz = a.nz ? a.nz : 1;
  while (kz > 8 && cols * ((a.nz + kz - 1) / kz) < 1024ull * sm_count) kz = (kz + 1) / 2;
  const uint64_t items = cols * ((a.nz + kz - 1) / kz);
  auto k = R == 1 ? (v4 ? lorenzo_codes_kernel<4, 1> : lorenzo_codes_kernel<1, 1>)
                  : (v4 ? lorenzo_codes_kernel<4, kCodeRows> : lorenzo_codes_kernel<1, kCodeRows>);
  k<<<lorenzo_grid(items, 256, 1u << 30), 256, 0, st>>>(a, kz);
  return cudaGetLastError();
}

cudaError_t launch_lorenzo_inverse(const LorenzoArgs& a, uint32_t sm_count, cudaStream_t st) {
  if ((uint64_t)a.nx * a.ny * a.nz == 0) return cudaSuccess;
  if (a.nz > 1) {  // one plane is its own sum along z
    auto k = a.nz < 16 ? lorenzo_zsum_kernel<4> : lorenzo_zsum_kernel<16>;
    k<<<lorenzo_grid((uint64_t)a.nx * a.ny, 64, 32 * sm_count), 64, 0, st>>>(a);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  auto k = a.ny < 16 ? lorenzo_ysum_kernel<4> : lorenzo_ysum_kernel<16>;
  k<<<lorenzo_grid((uint64_t)a.nx * a.nz, 64, 32 * sm_count), 64, 0, st>>>(a);
  return cudaGetLastError();
}

}  // namespace szp

// layout.cu -- population initialisation, conversion between the device
// A-A storage and the reference's FP64 array-of-structures layout, and the
// FP64 global mass/momentum/finite check.
//
// Post-stream population q of node x (what the reference holds in f_curr
// after a step) lives, after an even step, in the opposite slot of the
// upstream node x - e_q, and after an odd step in slot q of x itself.  When
// the upstream node does not exist (array boundary of a non-periodic axis)
// the reference never writes that entry and it keeps the initial
// equilibrium w_q (src/LBM_PSM_BGK_dynamics.cpp:94-99 skips targets outside
// the array).
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <algorithm>

#include "lbmpsm_internal.cuh"

namespace lbmpsm {

template <typename T>
__device__ __forceinline__ double load_pop(const void* f, long long loc, int storage, float scale,
                                           double w) {
  (void)sizeof(T);
  if (storage == 0) return static_cast<const double*>(f)[loc];
  if (storage == 1) return w + (double)static_cast<const float*>(f)[loc];
  if (storage == 3) return w + (double)__bfloat162float(static_cast<const __nv_bfloat16*>(f)[loc]);
  return w + (double)(__half2float(static_cast<const __half*>(f)[loc]) / scale);
}

__device__ __forceinline__ void store_pop(void* f, long long loc, int storage, float scale,
                                          double w, double v) {
  if (storage == 0)
    static_cast<double*>(f)[loc] = v;
  else if (storage == 1)
    static_cast<float*>(f)[loc] = (float)(v - w);
  else if (storage == 3)
    static_cast<__nv_bfloat16*>(f)[loc] = __float2bfloat16_rn((float)(v - w));
  else
    static_cast<__half*>(f)[loc] = __float2half_rn((float)(v - w) * scale);
}

template <class L>
__device__ __forceinline__ long long loc_of(const Geom& g, const Nbr& nb, long long n, int q,
                                            int after_odd) {
  const int cx = L::ex(q), cy = L::ey(q), cz = L::ez(q);
  if (!nbr_ok(nb, -cx, -cy, -cz)) return -1;
  if (after_odd) return (long long)q * g.Np + n;
  return (long long)L::opp(q) * g.Np + n + nbr_off(nb, -cx, -cy, -cz);
}

template <class L>
__global__ void init_kernel(Geom g, void* f, int storage, float scale) {
  const long long n = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= g.Np) return;
  for (int q = 0; q < L::Q; ++q) {
    const long long loc = (long long)q * g.Np + n;
    if (storage == 0)
      static_cast<double*>(f)[loc] = L::w(q);  // feq(rho = 1, u = 0) = w_q
    else if (storage == 1)
      static_cast<float*>(f)[loc] = 0.0f;
    else if (storage == 3)
      static_cast<__nv_bfloat16*>(f)[loc] = __float2bfloat16_rn(0.0f);
    else
      static_cast<__half*>(f)[loc] = __float2half_rn(0.0f);
  }
}

cudaError_t launch_init_populations(const Geom& g, void* f, int storage, float scale16,
                                    cudaStream_t st) {
  const unsigned blocks = (unsigned)((g.Np + 255) / 256);
  if (g.dim == 2)
    init_kernel<D2Q9><<<blocks, 256, 0, st>>>(g, f, storage, scale16);
  else
    init_kernel<D3Q19><<<blocks, 256, 0, st>>>(g, f, storage, scale16);
  return cudaGetLastError();
}

// Populations between the A-A storage (x fastest, one array per direction) and
// the reference's array f[node*q + iq], node = (i*ny + j)*nz + k (halo
// included): a transposition.  Block (bi, bm) takes 32 nodes along i and POP_M
// consecutive (j, k) pairs, which are POP_M*Q consecutive doubles of the
// reference array for each i; both sides are then read and written in runs (one
// thread per node moved 19 doubles 8 bytes at a time at strides of the whole
// y-z plane).  Coherent host memory (NVLink-C2C) takes the same runs, so there
// the kernels work on the caller's array: 96x80x70 (83 MB), 766 -> 454 us in and
// 840 -> 610 us out against a staged device copy.
//
// Periodic halo nodes read their periodic twin, as after the reference's
// exchange, and are ignored on input.
constexpr int POP_I = 32, POP_M = 8, POP_THREADS = 256;

template <class L>
__device__ __forceinline__ bool pop_node(const Geom& g, int i, long long m, int (&s)[3], bool& halo) {
  const int j = (int)(m / g.L[2]), k = (int)(m - (long long)j * g.L[2]);
  const int h[3] = {i, j, k};
  halo = false;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    s[d] = h[d];
    if (g.off[d] == 1) {
      s[d] = h[d] - 1;
      if (s[d] < 0 || s[d] >= g.S[d]) halo = true;
      if (s[d] < 0) s[d] = g.S[d] - 1;
      if (s[d] >= g.S[d]) s[d] = 0;
    }
  }
  return i < g.L[0] && j < g.L[1];
}

template <class L>
__global__ void __launch_bounds__(POP_THREADS) get_pop_kernel(Geom g, const void* f, int storage,
                                                              int after_odd, float scale, double* out,
                                                              long long mfirst) {
  constexpr int Q = L::Q, RUN = POP_M * Q, PITCH = RUN + (RUN % 2 == 0 ? 1 : 0);
  __shared__ double tile[POP_I * PITCH];
  const int i0 = (int)blockIdx.x * POP_I;
  const long long M = (long long)g.L[1] * g.L[2], m0 = mfirst + (long long)blockIdx.y * POP_M;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int mm = warp; mm < POP_M; mm += POP_THREADS / 32) {
    int s[3];
    bool halo;
    if (m0 + mm >= M || !pop_node<L>(g, i0 + lane, m0 + mm, s, halo)) continue;
    const long long n = node_index(g, s[0], s[1], s[2]);
    const Nbr nb = make_nbr(g, s[0], s[1], s[2]);
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      const long long loc = loc_of<L>(g, nb, n, q, after_odd);
      tile[lane * PITCH + mm * Q + q] =
          loc >= 0 ? load_pop<int>(f, loc, storage, scale, L::w(q)) : L::w(q);
    }
  }
  __syncthreads();
  const int run = (int)min((long long)POP_M, M - m0) * Q;
  for (int ii = warp; ii < POP_I && i0 + ii < g.L[0]; ii += POP_THREADS / 32) {
    double* dst = out + ((long long)(i0 + ii) * M + m0) * Q;
    for (int t = lane; t < run; t += 32) dst[t] = tile[ii * PITCH + t];
  }
}

template <class L>
__global__ void __launch_bounds__(POP_THREADS) set_pop_kernel(Geom g, void* f, int storage,
                                                              int after_odd, float scale, const double* in,
                                                              long long mfirst) {
  constexpr int Q = L::Q, RUN = POP_M * Q, PITCH = RUN + (RUN % 2 == 0 ? 1 : 0);
  __shared__ double tile[POP_I * PITCH];
  const int i0 = (int)blockIdx.x * POP_I;
  const long long M = (long long)g.L[1] * g.L[2], m0 = mfirst + (long long)blockIdx.y * POP_M;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int run = (int)min((long long)POP_M, M - m0) * Q;
  for (int ii = warp; ii < POP_I && i0 + ii < g.L[0]; ii += POP_THREADS / 32) {
    const double* src = in + ((long long)(i0 + ii) * M + m0) * Q;
    for (int t = lane; t < run; t += 32) tile[ii * PITCH + t] = src[t];
  }
  __syncthreads();
  for (int mm = warp; mm < POP_M; mm += POP_THREADS / 32) {
    int s[3];
    bool halo;
    if (m0 + mm >= M || !pop_node<L>(g, i0 + lane, m0 + mm, s, halo) || halo) continue;
    const long long n = node_index(g, s[0], s[1], s[2]);
    const Nbr nb = make_nbr(g, s[0], s[1], s[2]);
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      const long long loc = loc_of<L>(g, nb, n, q, after_odd);
      if (loc >= 0) store_pop(f, loc, storage, scale, L::w(q), tile[lane * PITCH + mm * Q + q]);
    }
  }
}

// The tiles of rows (j, k) go through blockIdx.y (65535 at most) in turns.
template <class Fn>
static cudaError_t pop_launch(const Geom& g, Fn fn) {
  const long long M = (long long)g.L[1] * g.L[2], tiles = (M + POP_M - 1) / POP_M;
  for (long long t0 = 0; t0 < tiles; t0 += 65535)
    fn(dim3((unsigned)((g.L[0] + POP_I - 1) / POP_I), (unsigned)std::min<long long>(tiles - t0, 65535)), t0 * POP_M);
  return cudaGetLastError();
}

cudaError_t launch_get_populations(const Geom& g, const void* f, int storage, int after_odd,
                                   float scale16, double* out_ref, cudaStream_t st) {
  return pop_launch(g, [&](dim3 grid, long long m0) {
    if (g.dim == 2)
      get_pop_kernel<D2Q9><<<grid, POP_THREADS, 0, st>>>(g, f, storage, after_odd, scale16, out_ref, m0);
    else
      get_pop_kernel<D3Q19><<<grid, POP_THREADS, 0, st>>>(g, f, storage, after_odd, scale16, out_ref, m0);
  });
}

cudaError_t launch_set_populations(const Geom& g, void* f, int storage, int after_odd,
                                   float scale16, const double* in_ref, cudaStream_t st) {
  return pop_launch(g, [&](dim3 grid, long long m0) {
    if (g.dim == 2)
      set_pop_kernel<D2Q9><<<grid, POP_THREADS, 0, st>>>(g, f, storage, after_odd, scale16, in_ref, m0);
    else
      set_pop_kernel<D3Q19><<<grid, POP_THREADS, 0, st>>>(g, f, storage, after_odd, scale16, in_ref, m0);
  });
}

// ------------------------------------------------------------------ check
constexpr int CHECK_THREADS = 256;
constexpr int CHECK_BLOCKS = 1024;

// Error-free transformation a + b = s + e (Knuth's TwoSum, no contraction).
__device__ __forceinline__ void two_sum_f(float a, float b, float& s, float& e) {
  s = __fadd_rn(a, b);
  const float bb = __fadd_rn(s, -a);
  e = __fadd_rn(__fadd_rn(a, -__fadd_rn(s, -bb)), __fadd_rn(b, -bb));
}

// Blocks walk x-rows with 32-bit index arithmetic (64-bit integer division
// is emulated and slow).  FP64 storage sums the populations in FP64.  FP32 /
// FP16 / BF16 storage sums each node's deviations g = f - w in FP32 and adds the
// node sums into double-float accumulators on the FP32 pipe; the weights add
// up to exactly 1 per node (mass = nodes + sum g) and to 0 in every momentum
// component.
template <class L, bool F64>
__global__ void __launch_bounds__(CHECK_THREADS) check_partial_kernel(Geom g, const void* f,
                                                                       int storage, int after_odd,
                                                                       float scale, double* partial,
                                                                       int* status) {
  double acc[4] = {0.0, 0.0, 0.0, 0.0};
  float hi[4] = {0.f, 0.f, 0.f, 0.f}, lo[4] = {0.f, 0.f, 0.f, 0.f};
  unsigned nodes = 0;
  bool bad = false;
  const float inv_scale = 1.0f / scale;
  const int R = g.S[1] * g.S[2];
  for (int r = blockIdx.x; r < R; r += gridDim.x) {
    const int sy = r % g.S[1], sz = r / g.S[1];
    for (int sx = threadIdx.x; sx < g.S[0]; sx += blockDim.x) {
      const long long n = node_index(g, sx, sy, sz);
      const Nbr nb = make_nbr(g, sx, sy, sz);
      if (F64) {
        for (int q = 0; q < L::Q; ++q) {
          const long long loc = loc_of<L>(g, nb, n, q, after_odd);
          const double v = loc >= 0 ? static_cast<const double*>(f)[loc] : L::w(q);
          if (!isfinite(v)) bad = true;
          acc[0] += v;
          acc[1] += v * L::ex(q);
          acc[2] += v * L::ey(q);
          acc[3] += v * L::ez(q);
        }
      } else {
        float ns[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int q = 0; q < L::Q; ++q) {
          const long long loc = loc_of<L>(g, nb, n, q, after_odd);
          float v = 0.0f;
          if (loc >= 0)
            v = storage == 1   ? static_cast<const float*>(f)[loc]
                : storage == 3 ? __bfloat162float(static_cast<const __nv_bfloat16*>(f)[loc])
                               : __half2float(static_cast<const __half*>(f)[loc]) * inv_scale;
          if (!isfinite(v)) bad = true;
          ns[0] += v;
          if (L::ex(q)) ns[1] += L::ex(q) > 0 ? v : -v;
          if (L::ey(q)) ns[2] += L::ey(q) > 0 ? v : -v;
          if (L::ez(q)) ns[3] += L::ez(q) > 0 ? v : -v;
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          float sv, e;
          two_sum_f(hi[k], ns[k], sv, e);
          hi[k] = sv;
          lo[k] = __fadd_rn(lo[k], e);
        }
        ++nodes;
      }
    }
  }
  if (!F64) {
    acc[0] = (double)hi[0] + (double)lo[0] + (double)nodes;
    for (int k = 1; k < 4; ++k) acc[k] = (double)hi[k] + (double)lo[k];
  }
  if (bad) atomicOr(status, STATUS_NONFINITE);
  for (int k = 0; k < 4; ++k)
    for (int o = 16; o > 0; o >>= 1) acc[k] += __shfl_xor_sync(0xffffffffu, acc[k], o);
  __shared__ double part[CHECK_THREADS / 32][4];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0)
    for (int k = 0; k < 4; ++k) part[warp][k] = acc[k];
  __syncthreads();
  if (threadIdx.x < 4) {
    double s = 0.0;
    for (int w = 0; w < CHECK_THREADS / 32; ++w) s += part[w][threadIdx.x];
    partial[4 * blockIdx.x + threadIdx.x] = s;
  }
}

__global__ void check_final_kernel(const double* partial, int nblocks, double* acc4) {
  if (threadIdx.x < 4) {
    double s = 0.0;
    for (int b = 0; b < nblocks; ++b) s += partial[4 * b + threadIdx.x];
    acc4[threadIdx.x] = s;
  }
}

// acc4 must have room for 4 + 4*CHECK_BLOCKS doubles (partials after the sums).
cudaError_t launch_check(const Geom& g, const void* f, int storage, int after_odd, float scale16,
                         double* acc4, int* status, cudaStream_t st) {
  double* partial = acc4 + 4;
  if (g.dim == 2) {
    if (storage == 0)
      check_partial_kernel<D2Q9, true><<<CHECK_BLOCKS, CHECK_THREADS, 0, st>>>(
          g, f, storage, after_odd, scale16, partial, status);
    else
      check_partial_kernel<D2Q9, false><<<CHECK_BLOCKS, CHECK_THREADS, 0, st>>>(
          g, f, storage, after_odd, scale16, partial, status);
  } else {
    if (storage == 0)
      check_partial_kernel<D3Q19, true><<<CHECK_BLOCKS, CHECK_THREADS, 0, st>>>(
          g, f, storage, after_odd, scale16, partial, status);
    else
      check_partial_kernel<D3Q19, false><<<CHECK_BLOCKS, CHECK_THREADS, 0, st>>>(
          g, f, storage, after_odd, scale16, partial, status);
  }
  check_final_kernel<<<1, 32, 0, st>>>(partial, CHECK_BLOCKS, acc4);
  return cudaGetLastError();
}

}  // namespace lbmpsm

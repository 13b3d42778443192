// Abs-max reduction, fp32 -> int8 quantisation and the one-off weight conversion.
// All three are plain HBM-bound streaming kernels: 16-byte loads, several in flight per thread,
// grids sized from the SM count.
#include "mi8_internal.h"
#include "mi8_ptx.cuh"

namespace mi8 {

namespace {

constexpr int kBlock = 256;

__device__ __forceinline__ unsigned abs_bits(float v) { return __float_as_uint(v) & 0x7fffffffu; }

__device__ __forceinline__ unsigned max4(unsigned m, const float4& v) {
  m = max(m, abs_bits(v.x));
  m = max(m, abs_bits(v.y));
  m = max(m, abs_bits(v.z));
  m = max(m, abs_bits(v.w));
  return m;
}

// Block-wide maximum of an unsigned value; result valid in thread 0.
__device__ __forceinline__ unsigned block_max(unsigned m, unsigned* smem) {
  m = __reduce_max_sync(0xffffffffu, m);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if(lane == 0)
    smem[warp] = m;
  __syncthreads();
  if(warp == 0) {
    m = lane < (kBlock / 32) ? smem[lane] : 0u;
    m = __reduce_max_sync(0xffffffffu, m);
  }
  return m;
}

// |x| of non-negative IEEE floats orders like the unsigned integer of its bits, and Inf/NaN sort
// above every finite value, so one unsigned max finds both the maximum and non-finite input.
// Every block parks its maximum in `partials`; the last block to arrive reduces them, writes the
// results and resets the arrival counter.
__global__ void __launch_bounds__(kBlock)
mi8_absmax_kernel(const float* __restrict__ x, size_t n, unsigned* partials, unsigned* counter, float* d_absmax,
                  float* d_quant_mult, int* status) {
  pdl_launch_dependents();
  const TraceHandles th = trace_open_all();
  unsigned long long* const tb = th.first;
  pdl_wait();
  trace_stamp_start(th, kTrAbsmax);
  __shared__ unsigned red[kBlock / 32];
  __shared__ int is_last;
  unsigned m = 0u;
  const size_t n4 = n / 4;
  const float4* x4 = reinterpret_cast<const float4*>(x);
  const size_t stride = static_cast<size_t>(gridDim.x) * kBlock;
  size_t i = static_cast<size_t>(blockIdx.x) * kBlock + threadIdx.x;
  for(; i + 3 * stride < n4; i += 4 * stride) {
    const float4 a = __ldg(x4 + i);
    const float4 b = __ldg(x4 + i + stride);
    const float4 c = __ldg(x4 + i + 2 * stride);
    const float4 d = __ldg(x4 + i + 3 * stride);
    m = max4(max4(max4(max4(m, a), b), c), d);
  }
  for(; i < n4; i += stride)
    m = max4(m, __ldg(x4 + i));
  if(blockIdx.x == 0 && threadIdx.x < (n & 3))
    m = max(m, abs_bits(x[n4 * 4 + threadIdx.x]));

  m = block_max(m, red);
  if(threadIdx.x == 0) {
    partials[blockIdx.x] = m;
    __threadfence();
    const unsigned old = atomicAdd(counter, 1u);
    is_last = (old == gridDim.x - 1) ? 1 : 0;
  }
  __syncthreads();
  if(!is_last) {
    trace_stamp(tb, kTrAbsmax, 2);
    trace_stamp(th.last, kTrAbsmax, 3);
    return;
  }
  __threadfence();
  m = 0u;
  for(unsigned b = threadIdx.x; b < gridDim.x; b += kBlock)
    m = max(m, __ldcg(partials + b));
  __syncthreads();  // `red` is reused
  m = block_max(m, red);
  if(threadIdx.x == 0) {
    *counter = 0u;  // leave the workspace zeroed for the next call
    if(m >= 0x7f800000u)
      atomicMax(status, static_cast<int>(kDevNonFinite));
    const float mx = __uint_as_float(m);
    if(d_absmax != nullptr)
      *d_absmax = mx;
    if(d_quant_mult != nullptr)
      *d_quant_mult = (m == 0u) ? 1.0f : __fdiv_rn(127.0f, mx);
  }
  trace_stamp(tb, kTrAbsmax, 2);
  trace_stamp(th.last, kTrAbsmax, 3);
}

__device__ __forceinline__ int quantize_one(float v, float qm) {
  int r = __float2int_rn(__fmul_rn(v, qm));  // round half to even; NaN -> 0
  return max(-127, min(127, r));              // -128 is never produced
}

__device__ __forceinline__ unsigned pack4(const float4& v, float qm) {
  return (static_cast<unsigned>(quantize_one(v.x, qm)) & 0xffu) | ((static_cast<unsigned>(quantize_one(v.y, qm)) & 0xffu) << 8) |
         ((static_cast<unsigned>(quantize_one(v.z, qm)) & 0xffu) << 16) | ((static_cast<unsigned>(quantize_one(v.w, qm)) & 0xffu) << 24);
}

// 16 floats per thread and iteration: four 16-byte loads, the lanes of a warp side by side in each, and four bytes out for each (64 consecutive bytes per
// thread before: affine 3937 x 1024 x 4096 34.3 -> 33.8 us; the cluster below likewise, 250 x 1024 x 32000 21.03 -> 20.72).  Vectors beyond the end are the
// last one once more (the same four bytes to the same place): with a guard at every load and store launches of up to 300000 floats, back to back, were slower
// than with 64 consecutive bytes (65536 floats 1.34 us then, 1.43 with guards, 1.17 so; 1 M 2.6, 2.24, 2.17; only 1024 floats 0.97, 1.09, 1.01).
__global__ void __launch_bounds__(kBlock)
mi8_quantize_kernel(const float* __restrict__ x, size_t n, const float* __restrict__ d_quant_mult, int8_t* __restrict__ q) {
  pdl_launch_dependents();
  const TraceHandles th = trace_open_all();
  unsigned long long* const tb = th.first;
  pdl_wait();
  trace_stamp_start(th, kTrQuantize);
  const float qm = *d_quant_mult;
  const size_t n4 = n / 4;
  const float4* x4 = reinterpret_cast<const float4*>(x);
  unsigned* q4 = reinterpret_cast<unsigned*>(q);
  for(size_t i = static_cast<size_t>(blockIdx.x) * (4 * kBlock) + threadIdx.x; i < n4; i += static_cast<size_t>(gridDim.x) * (4 * kBlock)) {
    float4 v[4];
#pragma unroll
    for(int e = 0; e < 4; ++e)
      v[e] = __ldg(x4 + min(i + e * kBlock, n4 - 1));
#pragma unroll
    for(int e = 0; e < 4; ++e)
      q4[min(i + e * kBlock, n4 - 1)] = pack4(v[e], qm);
  }
  if(blockIdx.x == 0 && threadIdx.x < (n & 3))
    q[n4 * 4 + threadIdx.x] = static_cast<int8_t>(quantize_one(x[n4 * 4 + threadIdx.x], qm));
  trace_stamp(tb, kTrQuantize, 2);
  trace_stamp(th.last, kTrQuantize, 3);
}

// Abs-max and quantisation of a small tensor in one launch: a cluster of kCtas CTAs reads the tensor once into registers (kChunks x 16
// consecutive floats per thread), reduces its maximum through the CTAs' shared memory and quantises what it holds.
// Such a tensor's cost is launches and round trips, not bytes: two kernels read it twice with a grid-wide reduction at the end of the
// first and a launch boundary between them.  Both kernels against this one, back to back: 131072 and 262144 floats 7.3 -> 5.4 us;
// affine 256 x 512 x 2048 10.9 -> 7.9 us, 250 x 1024 x 32000 24.2 -> 21.1 us, 4 x 256 x 1536 8.8 -> 6.8 us.
template <int kCtas, int kChunks>
__global__ void __cluster_dims__(kCtas, 1, 1) __launch_bounds__(1024)
mi8_prepare_cluster_kernel(const float* __restrict__ x, int n16, float* d_quant_mult, int8_t* __restrict__ q, int* status) {
  pdl_launch_dependents();
  const TraceHandles th = trace_open_all();
  unsigned long long* const tb = th.first;
  __shared__ unsigned red[32];
  __shared__ unsigned cta_max[kCtas];
  if(kCtas > 1)
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");   // (this CTA runs: the others may write to cta_max)
  pdl_wait();
  trace_stamp_start(th, kTrQuantize);
  const int rank = kCtas > 1 ? static_cast<int>(blockIdx.x) : 0;
  const float4* x4 = reinterpret_cast<const float4*>(x);
  float4 v[kChunks][4];
  unsigned m = 0u;
  // (the lanes of a warp side by side in each load; beyond the end the last vector once more, which leaves the maximum as it is.  Guards at every load and
  // store cost up to 0.1 us: 1024 floats 1.06 with 64 consecutive bytes per thread, 1.17 with guards, 1.02 so; 8448 1.62, 1.74, 1.58; 256000 5.2, 4.04, 3.91)
#pragma unroll
  for(int c = 0; c < kChunks; ++c) {
    const int i = (c * kCtas + rank) * 4 * static_cast<int>(blockDim.x) + static_cast<int>(threadIdx.x);
#pragma unroll
    for(int e = 0; e < 4; ++e)
      v[c][e] = __ldg(x4 + min(i + e * static_cast<int>(blockDim.x), 4 * n16 - 1));
  }
#pragma unroll
  for(int c = 0; c < kChunks; ++c)
#pragma unroll
    for(int e = 0; e < 4; ++e)
      m = max4(m, v[c][e]);
  m = __reduce_max_sync(0xffffffffu, m);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = static_cast<int>(blockDim.x) >> 5;
  if(lane == 0)
    red[warp] = m;
  __syncthreads();
  m = __reduce_max_sync(0xffffffffu, lane < warps ? red[lane] : 0u);
  if(kCtas > 1) {
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    if(threadIdx.x < kCtas)
      st_cluster_u32(mapa_shared(smem_u32(&cta_max[rank]), threadIdx.x), m);
    cluster_sync_all();
    m = cta_max[0];
#pragma unroll
    for(int c = 1; c < kCtas; ++c)
      m = max(m, cta_max[c]);
  }
  const float qm = m == 0u ? 1.0f : __fdiv_rn(127.0f, __uint_as_float(m));
  if(rank == 0 && threadIdx.x == 0) {
    *d_quant_mult = qm;
    if(m >= 0x7f800000u)
      atomicMax(status, static_cast<int>(kDevNonFinite));
  }
#pragma unroll
  for(int c = 0; c < kChunks; ++c) {
    const int i = (c * kCtas + rank) * 4 * static_cast<int>(blockDim.x) + static_cast<int>(threadIdx.x);
    unsigned* const q4 = reinterpret_cast<unsigned*>(q) + i;
    if((c * kCtas + rank + 1) * static_cast<int>(blockDim.x) <= n16) {
#pragma unroll
      for(int e = 0; e < 4; ++e)
        q4[e * static_cast<int>(blockDim.x)] = pack4(v[c][e], qm);
    } else {
#pragma unroll
      for(int e = 0; e < 4; ++e)
        if(i + e * static_cast<int>(blockDim.x) < 4 * n16)
          q4[e * static_cast<int>(blockDim.x)] = pack4(v[c][e], qm);
    }
  }
  trace_stamp(tb, kTrQuantize, 2);
  trace_stamp(th.last, kTrQuantize, 3);
}
constexpr int kPrepareCtas = 8;
constexpr size_t kOneCtaMaxN = 512 * 16;
constexpr size_t kClusterMaxN = static_cast<size_t>(kPrepareCtas) * 1024 * 16 * 2;

// W fp32 [K,N] row-major -> Bt int8 [N,K] row-major.  A block moves a 128(k) x 32(n) tile: a thread reads a 4 x 4 part of it, four columns of four rows (a
// warp four times 128 bytes with each load), packs every column's four values into a word and parks it in shared memory (no bank conflicts), and a
// warp stores 128 consecutive bytes of a row of Bt.  Where rows of W are not 16-byte aligned (`vec` 0) it reads value by value, a column per lane.
// Bound by the read of W (from L2 behind the abs-max while W fits there).  Conversion of 1024 x 4096: 9.68 us with sixteen 4-byte loads per thread, 8.94 with
// four 16-byte ones; of 4096 x 8192: 81 us with 32 x 32 tiles and a byte per store, 53 us with the loads of before.
__global__ void __launch_bounds__(256)
mi8_transpose_quantize_kernel(const float* __restrict__ w, int K, int N, const float* __restrict__ d_quant_mult,
                              int8_t* __restrict__ bt, int words, int vec) {
  pdl_launch_dependents();
  pdl_wait();
  __shared__ unsigned tile[32][33];   // [n][k / 4]
  const float qm = *d_quant_mult;
  const int n0 = blockIdx.x * 32, k0 = blockIdx.y * 128;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if(vec) {
    const int n = 4 * (lane & 7), q = 4 * warp + (lane >> 3);   // four columns, four rows from 4 q on
    float4 v[4];
#pragma unroll
    for(int i = 0; i < 4; ++i)
      v[i] = k0 + 4 * q + i < K && n0 + n < N ? __ldg(reinterpret_cast<const float4*>(w + static_cast<size_t>(k0 + 4 * q + i) * N + n0 + n))
                                              : make_float4(0.f, 0.f, 0.f, 0.f);
    tile[n][q] = pack4(make_float4(v[0].x, v[1].x, v[2].x, v[3].x), qm);
    tile[n + 1][q] = pack4(make_float4(v[0].y, v[1].y, v[2].y, v[3].y), qm);
    tile[n + 2][q] = pack4(make_float4(v[0].z, v[1].z, v[2].z, v[3].z), qm);
    tile[n + 3][q] = pack4(make_float4(v[0].w, v[1].w, v[2].w, v[3].w), qm);
  } else {
    const int n = n0 + lane;
    float4 v[4];
#pragma unroll
    for(int i = 0; i < 4; ++i) {
      const int k = k0 + 4 * (warp + 8 * i);
      const float* src = w + static_cast<size_t>(k) * N + n;
      v[i].x = (k < K && n < N) ? __ldg(src) : 0.0f;
      v[i].y = (k + 1 < K && n < N) ? __ldg(src + N) : 0.0f;
      v[i].z = (k + 2 < K && n < N) ? __ldg(src + 2 * static_cast<size_t>(N)) : 0.0f;
      v[i].w = (k + 3 < K && n < N) ? __ldg(src + 3 * static_cast<size_t>(N)) : 0.0f;
    }
#pragma unroll
    for(int i = 0; i < 4; ++i)
      tile[lane][warp + 8 * i] = pack4(v[i], qm);
  }
  __syncthreads();
#pragma unroll
  for(int i = 0; i < 4; ++i) {
    const int r = warp + 8 * i, k = k0 + 4 * lane;
    if(n0 + r < N && k < K) {
      int8_t* dst = bt + static_cast<size_t>(n0 + r) * K + k;
      const unsigned o = tile[r][lane];
      if(words) {   // K is a multiple of four and Bt 4-byte aligned
        *reinterpret_cast<unsigned*>(dst) = o;
      } else {
        for(int e = 0; e < 4 && k + e < K; ++e)
          dst[e] = static_cast<int8_t>(o >> (8 * e));
      }
    }
  }
}

// out[b][c][r] = in[b][r][c]: the last two axes of a float tensor swapped, 32 x 32 tiles through shared memory so that
// reads and writes are both contiguous.  (Serves affine / dot with transA, which the reference resolves by a transpose
// node in front of the quantisation, src/tensors/cpu/intgemm_interface.h:52.)
__global__ void __launch_bounds__(256)
mi8_transpose_f32_kernel(const float* __restrict__ in, int rows, int cols, float* __restrict__ out) {
  pdl_launch_dependents();
  pdl_wait();
  __shared__ float tile[32][33];
  const size_t plane = static_cast<size_t>(rows) * cols;
  const float* src = in + blockIdx.z * plane;
  float* dst = out + blockIdx.z * plane;
  const int c0 = blockIdx.x * 32, r0 = blockIdx.y * 32;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
#pragma unroll
  for(int i = 0; i < 32; i += 8) {
    const int r = r0 + ty + i, c = c0 + tx;
    tile[ty + i][tx] = (r < rows && c < cols) ? src[static_cast<size_t>(r) * cols + c] : 0.0f;
  }
  __syncthreads();
#pragma unroll
  for(int i = 0; i < 32; i += 8) {
    const int c = c0 + ty + i, r = r0 + tx;
    if(c < cols && r < rows)
      dst[static_cast<size_t>(c) * rows + r] = tile[tx][ty + i];
  }
}

int stream_grid(size_t work_items) {
  const size_t per_block = static_cast<size_t>(kBlock) * 4;
  size_t blocks = (work_items + per_block - 1) / per_block;
  const size_t cap = static_cast<size_t>(sm_count()) * 8;
  if(blocks > cap)
    blocks = cap;
  if(blocks < 1)
    blocks = 1;
  return static_cast<int>(blocks);
}

}  // namespace

MI8_DEFINE_TRACE_SETTER(trace_set_quant)

int launch_max_absolute(const float* x, size_t n, float* d_absmax, float* d_quant_mult, void* ws, size_t ws_bytes,
                        cudaStream_t stream) {
  if(x == nullptr || n == 0)
    return MI8_ERR_BAD_ARG;
  if(ws == nullptr || ws_bytes < kWsHeaderBytes)
    return MI8_ERR_WORKSPACE;
  if(reinterpret_cast<uintptr_t>(x) & 15u)
    return MI8_ERR_MISALIGNED;
  int* status = device_status_ptr();
  if(status == nullptr)
    return MI8_ERR_LAUNCH;
  uint8_t* wsb = static_cast<uint8_t*>(ws);
  int grid = stream_grid(n / 4 + 1);
  if(grid > kWsMaxAbsmaxBlocks)
    grid = kWsMaxAbsmaxBlocks;
  launch_kernel(mi8_absmax_kernel, dim3(grid), dim3(kBlock), 0, stream, x, n, reinterpret_cast<unsigned*>(wsb + kWsOffAbsmaxPartials),
                                                 reinterpret_cast<unsigned*>(wsb + kWsOffAbsmaxCounter), d_absmax,
                                                 d_quant_mult, status);
  count_launch();
  return check_launch();
}

int launch_quantize(const float* x, size_t n, const float* d_quant_mult, int8_t* q, cudaStream_t stream) {
  if(x == nullptr || q == nullptr || d_quant_mult == nullptr || n == 0)
    return MI8_ERR_BAD_ARG;
  if((reinterpret_cast<uintptr_t>(x) & 15u) || (reinterpret_cast<uintptr_t>(q) & 15u))
    return MI8_ERR_MISALIGNED;
  // A chunk of 16 floats per thread until the SMs are full: with four in turn, 4 M floats were 246 blocks, 13 warps per SM
  // (affine 3937 x 1024 x 4096 41.3 -> 34.3 us, 2000 x 4096 x 1024 35.2 -> 30.0, 4096 x 1024 x 32000 134.8 -> 130.6).
  const size_t want = (n / 16 + kBlock) / kBlock, cap = static_cast<size_t>(sm_count()) * 8;
  const int grid = static_cast<int>(want < cap ? want : cap);
  launch_kernel(mi8_quantize_kernel, dim3(grid), dim3(kBlock), 0, stream, x, n, d_quant_mult, q);
  count_launch();
  return check_launch();
}

int launch_prepare(const float* x, size_t n, float* d_quant_mult, int8_t* q, void* ws, size_t ws_bytes, cudaStream_t stream) {
  // Up to kOneCtaMaxN floats one CTA, up to kClusterMaxN the cluster (beyond, eight SMs read for longer than the other launch costs).
  // Launches back to back, in us: one CTA 1.23 at 4096 floats, 1.51 at 8192; cluster 1.57 at 8448, 1.75 at 32768, 3.91 at 256000; the two kernels
  // 4.51 at 307200 (and 5.2 to 5.7 from 8208 to 262160 when the lines were drawn).
  if(n == 0 || n % 16 != 0 || n > kClusterMaxN) {
    const int rc = launch_max_absolute(x, n, nullptr, d_quant_mult, ws, ws_bytes, stream);
    return rc != MI8_OK ? rc : launch_quantize(x, n, d_quant_mult, q, stream);
  }
  if(x == nullptr)
    return MI8_ERR_BAD_ARG;
  if(ws == nullptr || ws_bytes < kWsHeaderBytes)   // (not needed here; the same arguments are refused as for larger tensors)
    return MI8_ERR_WORKSPACE;
  if(reinterpret_cast<uintptr_t>(x) & 15u)
    return MI8_ERR_MISALIGNED;
  if(q == nullptr || d_quant_mult == nullptr)
    return MI8_ERR_BAD_ARG;
  if(reinterpret_cast<uintptr_t>(q) & 15u)
    return MI8_ERR_MISALIGNED;
  int* status = device_status_ptr();
  if(status == nullptr)
    return MI8_ERR_LAUNCH;
  const int n16 = static_cast<int>(n / 16);
  if(n <= kOneCtaMaxN)
    launch_kernel(mi8_prepare_cluster_kernel<1, 1>, dim3(1), dim3((n16 + 31) / 32 * 32), 0, stream, x, n16, d_quant_mult, q, status);
  else if(n16 <= kPrepareCtas * 1024)
    launch_kernel(mi8_prepare_cluster_kernel<kPrepareCtas, 1>, dim3(kPrepareCtas), dim3(((n16 + kPrepareCtas - 1) / kPrepareCtas + 31) / 32 * 32), 0, stream,
                  x, n16, d_quant_mult, q, status);
  else
    launch_kernel(mi8_prepare_cluster_kernel<kPrepareCtas, 2>, dim3(kPrepareCtas), dim3(1024), 0, stream, x, n16, d_quant_mult, q, status);
  count_launch();
  return check_launch();
}

int launch_transpose_quantize(const float* w, int K, int N, const float* d_quant_mult, int8_t* bt, cudaStream_t stream) {
  if(w == nullptr || bt == nullptr || d_quant_mult == nullptr || K <= 0 || N <= 0)
    return MI8_ERR_BAD_ARG;
  if((K + 31) / 32 > 65535)
    return MI8_ERR_UNSUPPORTED;
  const int words = K % 4 == 0 && (reinterpret_cast<uintptr_t>(bt) & 3u) == 0 ? 1 : 0;
  const int vec = N % 4 == 0 && (reinterpret_cast<uintptr_t>(w) & 15u) == 0 ? 1 : 0;
  launch_kernel(mi8_transpose_quantize_kernel, dim3((N + 31) / 32, (K + 127) / 128), dim3(256), 0, stream, w, K, N, d_quant_mult, bt, words, vec);
  count_launch();
  return check_launch();
}

int launch_transpose_f32(const float* in, int batch, int rows, int cols, float* out, cudaStream_t stream) {
  if(in == nullptr || out == nullptr || batch <= 0 || rows <= 0 || cols <= 0)
    return MI8_ERR_BAD_ARG;
  dim3 grid((cols + 31) / 32, (rows + 31) / 32, batch);
  if(grid.y > 65535 || grid.z > 65535)
    return MI8_ERR_UNSUPPORTED;
  launch_kernel(mi8_transpose_f32_kernel, grid, dim3(256), 0, stream, in, rows, cols, out);
  count_launch();
  return check_launch();
}

}  // namespace mi8

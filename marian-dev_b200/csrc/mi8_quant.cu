// Abs-max reduction, fp32 -> int8 quantisation and the one-off weight conversion.
// All three are plain HBM-bound streaming kernels: 16-byte loads, several in flight per thread,
// grids sized from the SM count.
#include <algorithm>
#include <atomic>

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

// Larger tensors take two launches that overlap.  mi8_absmax_kernel_parts lets the next kernel start once its own wait is over - what was in front of it has
// then completed - and every block leaves its maximum in `partials`; the kernel behind it (mi8_quantize_kernel_held, mi8_convert_kernel) fetches its share
// of the tensor into registers in front of its own wait, beside the search for the maximum, and then needs the blocks' maxima only.  The search is bound by
// the L2's reads beside those of the other kernel, whose blocks have to fit on the SMs with it: a block of 256 threads per SM leaves most registers to them;
// where that takes more than a few turns, more threads gain more than they displace (both launches back to back, 256 / 512 / 1024 threads, in us: 1 M
// floats 3.86 / 4.03 / 4.23, 1.4 M 5.05 / 4.23 / 6.28, 2 M 5.39 / 4.64 / 6.86, 3.5 M 6.89 / 6.76 / 7.27, 4 M 9.42 / 9.04 / 7.34, 16 M 32.0 / 24.7 / 22.8).
// Against a search that also reduces its blocks' maxima and a quantisation that waits for it before it reads: 256 K floats 5.36 -> 3.45 us,
// 512 K 5.50 -> 3.52, 1 M 7.5 -> 3.86, 2 M 7.8 -> 4.64, 4 M 8.5 -> 7.3, 8 M 12.0 -> 11.9, 16 M 24.2 -> 22.8.
template <int kThreads>
__global__ void __launch_bounds__(kThreads)
mi8_absmax_kernel_parts(const float* __restrict__ x, size_t n, unsigned* partials) {
  const TraceHandles th = trace_open_all();
  pdl_wait();
  pdl_launch_dependents();   // (behind the wait: the next kernel reads `x` in front of its own)
  trace_stamp_start(th, kTrAbsmax);
  constexpr int kLoads = 8;
  __shared__ unsigned red[kThreads / 32];
  const size_t n4 = n / 4, stride = static_cast<size_t>(gridDim.x) * kThreads;
  const float4* x4 = reinterpret_cast<const float4*>(x);
  unsigned m = 0u;
  for(size_t i = static_cast<size_t>(blockIdx.x) * kThreads + threadIdx.x; i < n4; i += kLoads * stride) {
    float4 v[kLoads];
#pragma unroll
    for(int e = 0; e < kLoads; ++e)
      v[e] = __ldg(x4 + min(i + e * stride, n4 - 1));
#pragma unroll
    for(int e = 0; e < kLoads; ++e)
      m = max4(m, v[e]);
  }
  if(blockIdx.x == 0 && threadIdx.x < (n & 3))
    m = max(m, abs_bits(x[n4 * 4 + threadIdx.x]));
  m = __reduce_max_sync(0xffffffffu, m);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if(lane == 0)
    red[warp] = m;
  __syncthreads();
  if(warp == 0) {
    m = __reduce_max_sync(0xffffffffu, lane < kThreads / 32 ? red[lane] : 0u);
    if(lane == 0)
      partials[blockIdx.x] = m;
  }
  trace_stamp(th.first, kTrAbsmax, 2);
  trace_stamp(th.last, kTrAbsmax, 3);
}

// The multiplier from the maxima that mi8_absmax_kernel_parts left, for every thread of a block of kBlock; block (0, 0) also stores it.
__device__ __forceinline__ float parts_multiplier(const unsigned* partials, int n_partials, unsigned* red, float* d_quant_mult, int* status) {
  unsigned m = 0u;
  for(int i = threadIdx.x; i < n_partials; i += kBlock)
    m = max(m, __ldcg(partials + i));
  m = __reduce_max_sync(0xffffffffu, m);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if(lane == 0)
    red[warp] = m;
  __syncthreads();
  m = __reduce_max_sync(0xffffffffu, lane < kBlock / 32 ? red[lane] : 0u);
  const float qm = m == 0u ? 1.0f : __fdiv_rn(127.0f, __uint_as_float(m));
  if(blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) {
    *d_quant_mult = qm;
    if(m >= 0x7f800000u)
      atomicMax(status, static_cast<int>(kDevNonFinite));
  }
  return qm;
}

// kHeld 16-byte vectors per thread, a warp's lanes side by side in each (beyond the end the last one once more).  Three blocks per SM are resident beside
// the search for the maximum, so kHeld is the smallest that puts the tensor into so many; beyond eight there are more blocks, whose turn comes later.
// `early`: the next kernel may begin beside this one; not behind a conversion, which is not part of a chain.
template <int kHeld>
__global__ void __launch_bounds__(kBlock)
mi8_quantize_kernel_held(const float* __restrict__ x, size_t n, const unsigned* partials, int n_partials, float* d_quant_mult, int8_t* __restrict__ q,
                         int* status, int early) {
  if(early)
    pdl_launch_dependents();
  const TraceHandles th = trace_open_all();
  __shared__ unsigned red[kBlock / 32];
  const size_t n4 = n / 4, i = static_cast<size_t>(blockIdx.x) * (kHeld * kBlock) + threadIdx.x;
  const float4* x4 = reinterpret_cast<const float4*>(x);
  unsigned* q4 = reinterpret_cast<unsigned*>(q);
  float4 v[kHeld];
#pragma unroll
  for(int e = 0; e < kHeld; ++e)
    v[e] = __ldcg(x4 + min(i + e * kBlock, n4 - 1));
  pdl_wait();
  trace_stamp_start(th, kTrQuantize);
  const float qm = parts_multiplier(partials, n_partials, red, d_quant_mult, status);
#pragma unroll
  for(int e = 0; e < kHeld; ++e)
    q4[min(i + e * kBlock, n4 - 1)] = pack4(v[e], qm);
  if(blockIdx.x == 0 && threadIdx.x < (n & 3))
    q[n4 * 4 + threadIdx.x] = static_cast<int8_t>(quantize_one(x[n4 * 4 + threadIdx.x], qm));
  trace_stamp(th.first, kTrQuantize, 2);
  trace_stamp(th.last, kTrQuantize, 3);
}

// Abs-max and quantisation of a small tensor in one launch: a cluster of kCtas CTAs reads the tensor once into registers (16
// floats per thread), reduces its maximum through the CTAs' shared memory and quantises what it holds.
// Such a tensor's cost is launches and round trips, not bytes: two kernels read it twice with a grid-wide reduction at the end of the
// first and a launch boundary between them.  Both kernels against this one, back to back: 131072 and 262144 floats 7.3 -> 5.4 us;
// affine 256 x 512 x 2048 10.9 -> 7.9 us, 250 x 1024 x 32000 24.2 -> 21.1 us, 4 x 256 x 1536 8.8 -> 6.8 us.
template <int kCtas>
__global__ void __cluster_dims__(kCtas, 1, 1) __launch_bounds__(1024)
mi8_prepare_cluster_kernel(const float* __restrict__ x, int n16, float* d_quant_mult, int8_t* __restrict__ q, int* status, Trigger trigger) {
  const TraceHandles th = trace_open_all();
  unsigned long long* const tb = th.first;
  __shared__ unsigned red[32];
  __shared__ unsigned cta_max[kCtas];
  if(kCtas > 1)
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");   // (this CTA runs: the others may write to cta_max)
  if(trigger == Trigger::kAtStart)
    pdl_launch_dependents();
  pdl_wait();
  if(trigger == Trigger::kBehindWait)
    pdl_launch_dependents();
  trace_stamp_start(th, kTrQuantize);
  const int rank = kCtas > 1 ? static_cast<int>(blockIdx.x) : 0;
  const float4* x4 = reinterpret_cast<const float4*>(x);
  float4 v[4];
  unsigned m = 0u;
  // (the lanes of a warp side by side in each load; beyond the end the last vector once more, which leaves the maximum as it is.  Guards at every load and
  // store cost up to 0.1 us: 1024 floats 1.06 with 64 consecutive bytes per thread, 1.17 with guards, 1.02 so; 8448 1.62, 1.74, 1.58; 256000 5.2, 4.04, 3.91)
  const int i = rank * 4 * static_cast<int>(blockDim.x) + static_cast<int>(threadIdx.x);
#pragma unroll
  for(int e = 0; e < 4; ++e)
    v[e] = __ldg(x4 + min(i + e * static_cast<int>(blockDim.x), 4 * n16 - 1));
#pragma unroll
  for(int e = 0; e < 4; ++e)
    m = max4(m, v[e]);
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
  unsigned* const q4 = reinterpret_cast<unsigned*>(q) + i;
  if((rank + 1) * static_cast<int>(blockDim.x) <= n16) {
#pragma unroll
    for(int e = 0; e < 4; ++e)
      q4[e * static_cast<int>(blockDim.x)] = pack4(v[e], qm);
  } else {
#pragma unroll
    for(int e = 0; e < 4; ++e)
      if(i + e * static_cast<int>(blockDim.x) < 4 * n16)
        q4[e * static_cast<int>(blockDim.x)] = pack4(v[e], qm);
  }
  trace_stamp(tb, kTrQuantize, 2);
  trace_stamp(th.last, kTrQuantize, 3);
}
constexpr int kPrepareCtas = 8, kWideCtas = 16;
constexpr size_t kOneCtaMaxN = 512 * 16;
constexpr size_t kWideMinN = 32768;
constexpr size_t kNarrowMaxN = static_cast<size_t>(kPrepareCtas) * 1024 * 16, kClusterMaxN = static_cast<size_t>(kWideCtas) * 1024 * 16;

// W fp32 [K,N] row-major -> Bt int8 [N,K] row-major.  A block moves a 128(k) x 32(n) tile: a thread reads a 4 x 4 part of it, four columns of four rows (a
// warp four times 128 bytes with each load), packs every column's four values into a word and parks it in shared memory (no bank conflicts), and a
// warp stores 128 consecutive bytes of a row of Bt.  Where rows of W are not 16-byte aligned (`vec` 0) it reads value by value, a column per lane.
// Bound by the read of W beside mi8_absmax_kernel_parts (see there), which this kernel's own reads overlap.  Conversion of 512 x 2048: 7.6 -> 3.8 us back to back
// against reads behind the maximum, 1024 x 4096 9.2 -> 7.1, 2048 x 4096 15.6 -> 14.5, 4096 x 8192 50.6 -> 49.0 (from the first row on 51.2).
__global__ void __launch_bounds__(kBlock)
mi8_convert_kernel(const float* __restrict__ w, int K, int N, const unsigned* partials, int n_partials, float* d_quant_mult, int8_t* __restrict__ bt,
                   int words, int vec, int* status) {
  // (no pdl_launch_dependents(): a conversion is not part of a chain)
  __shared__ unsigned tile[32][33];   // [n][k / 4]
  __shared__ unsigned red[kBlock / 32];
  const int n0 = blockIdx.x * 32, k0 = (gridDim.y - 1 - blockIdx.y) * 128;   // (the rows that the search reads last are still in L2)
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int n = 4 * (lane & 7), q = 4 * warp + (lane >> 3);   // `vec`: four columns, four rows from 4 q on
  float4 v[4];
  if(vec) {
#pragma unroll
    for(int i = 0; i < 4; ++i)
      v[i] = k0 + 4 * q + i < K && n0 + n < N ? __ldcg(reinterpret_cast<const float4*>(w + static_cast<size_t>(k0 + 4 * q + i) * N + n0 + n))
                                              : make_float4(0.f, 0.f, 0.f, 0.f);
  } else {
    const int col = n0 + lane;
#pragma unroll
    for(int i = 0; i < 4; ++i) {
      const int k = k0 + 4 * (warp + 8 * i);
      const float* src = w + static_cast<size_t>(k) * N + col;
      v[i].x = (k < K && col < N) ? __ldcg(src) : 0.0f;
      v[i].y = (k + 1 < K && col < N) ? __ldcg(src + N) : 0.0f;
      v[i].z = (k + 2 < K && col < N) ? __ldcg(src + 2 * static_cast<size_t>(N)) : 0.0f;
      v[i].w = (k + 3 < K && col < N) ? __ldcg(src + 3 * static_cast<size_t>(N)) : 0.0f;
    }
  }
  pdl_wait();
  const float qm = parts_multiplier(partials, n_partials, red, d_quant_mult, status);
  if(vec) {
    tile[n][q] = pack4(make_float4(v[0].x, v[1].x, v[2].x, v[3].x), qm);
    tile[n + 1][q] = pack4(make_float4(v[0].y, v[1].y, v[2].y, v[3].y), qm);
    tile[n + 2][q] = pack4(make_float4(v[0].z, v[1].z, v[2].z, v[3].z), qm);
    tile[n + 3][q] = pack4(make_float4(v[0].w, v[1].w, v[2].w, v[3].w), qm);
  } else {
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

namespace {
// The maxima of x's parts into the workspace; how many there are (what reads them fetches x in front of its own wait: kernels in this file alone).
int launch_parts(const float* x, size_t n, unsigned* partials, cudaStream_t stream) {
  const int threads = n <= (5u << 18) ? 256 : n <= (15u << 18) ? 512 : 1024;   // (why: at the kernel)
  const size_t want = (n / 4 + threads) / threads, cap = static_cast<size_t>(std::min(sm_count(), kWsMaxAbsmaxBlocks));
  const int grid = static_cast<int>(std::min(want, cap));
  launch_kernel(threads == 256 ? mi8_absmax_kernel_parts<256> : threads == 512 ? mi8_absmax_kernel_parts<512> : mi8_absmax_kernel_parts<1024>, dim3(grid),
                dim3(threads), 0, stream, x, n, partials);
  count_launch();
  return grid;
}

template <int kHeld>
void launch_held(const float* x, size_t n, const unsigned* partials, int n_partials, float* d_quant_mult, int8_t* q, int* status, int early,
                 cudaStream_t stream) {
  const int grid = static_cast<int>((n / 4 + kHeld * kBlock - 1) / (kHeld * kBlock));
  launch_kernel(mi8_quantize_kernel_held<kHeld>, dim3(grid), dim3(kBlock), 0, stream, x, n, partials, n_partials, d_quant_mult, q, status, early);
  count_launch();
}

// Whether the device can hold a cluster of kWideCtas CTAs (more than eight are not portable).
bool wide_cluster_fits() {
  static std::atomic<int> known[64];   // 0 = not asked yet, 1 = yes, -1 = no
  int dev = 0;
  cudaGetDevice(&dev);
  if(dev < 0 || dev >= 64)
    return false;
  int k = known[dev].load(std::memory_order_acquire);
  if(k == 0) {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = kWideCtas;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.gridDim = dim3(kWideCtas);
    cfg.blockDim = dim3(1024);
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int n = 0;
    const bool yes = cudaFuncSetAttribute(mi8_prepare_cluster_kernel<kWideCtas>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
                     cudaOccupancyMaxActiveClusters(&n, mi8_prepare_cluster_kernel<kWideCtas>, &cfg) == cudaSuccess && n > 0;
    if(!yes)
      cudaGetLastError();
    known[dev].store(k = yes ? 1 : -1, std::memory_order_release);
  }
  return k > 0;
}
}  // namespace

int launch_prepare(const float* x, size_t n, float* d_quant_mult, int8_t* q, void* ws, size_t ws_bytes, cudaStream_t stream, Trigger trigger) {
  // Up to kOneCtaMaxN floats one CTA, up to kClusterMaxN a cluster, of kWideCtas from kWideMinN on (beyond, so few SMs read for longer than the other
  // launch costs).  Launches back to back, in us: one CTA 1.23 at 4096 floats, 1.51 at 8192; clusters of eight and sixteen 1.91 and 1.95 at 16384,
  // 2.01 and 2.01 at 32768, 2.42 and 2.22 at 66000, 3.04 and 2.49 at 131072, 4.13 (two chunks per thread) and 3.24 at 256000; two kernels 3.07 at 66000,
  // 3.11 at 131072, 3.31 at 256000, 3.45 at 270336.
  if(x == nullptr || n == 0)
    return MI8_ERR_BAD_ARG;
  if(ws == nullptr || ws_bytes < kWsHeaderBytes)   // (a cluster does not need it; the same arguments are refused for every size)
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
  const int early = trigger != Trigger::kDone ? 1 : 0;   // (larger tensors: the second kernel starts behind the first one's wait, and so may the next at its start)
  if(n < 4) {   // (no whole vector)
    const int rc = launch_max_absolute(x, n, nullptr, d_quant_mult, ws, ws_bytes, stream);
    return rc != MI8_OK ? rc : launch_quantize(x, n, d_quant_mult, q, stream);
  }
  const bool wide = n > kWideMinN && n % 16 == 0 && wide_cluster_fits();
  if(n % 16 != 0 || n > (wide ? kClusterMaxN : kNarrowMaxN)) {
    unsigned* partials = reinterpret_cast<unsigned*>(static_cast<uint8_t*>(ws) + kWsOffAbsmaxPartials);
    const int parts = launch_parts(x, n, partials, stream);
    const size_t per_vector = static_cast<size_t>(3 * sm_count()) * kBlock * 4;
    const size_t held = (n + per_vector - 1) / per_vector;
    (held <= 1 ? launch_held<1> : held <= 2 ? launch_held<2> : held <= 3 ? launch_held<3> : held <= 4 ? launch_held<4> : held <= 6 ? launch_held<6> : launch_held<8>)(
        x, n, partials, parts, d_quant_mult, q, status, early, stream);
    return check_launch();
  }
  const int n16 = static_cast<int>(n / 16);
  if(n <= kOneCtaMaxN)
    launch_kernel(mi8_prepare_cluster_kernel<1>, dim3(1), dim3((n16 + 31) / 32 * 32), 0, stream, x, n16, d_quant_mult, q, status, trigger);
  else if(wide)
    launch_kernel(mi8_prepare_cluster_kernel<kWideCtas>, dim3(kWideCtas), dim3(((n16 + kWideCtas - 1) / kWideCtas + 31) / 32 * 32), 0, stream, x, n16,
                  d_quant_mult, q, status, trigger);
  else
    launch_kernel(mi8_prepare_cluster_kernel<kPrepareCtas>, dim3(kPrepareCtas), dim3(((n16 + kPrepareCtas - 1) / kPrepareCtas + 31) / 32 * 32), 0, stream,
                  x, n16, d_quant_mult, q, status, trigger);
  count_launch();
  return check_launch();
}

int launch_convert(const float* w, int K, int N, float* d_quant_mult, int8_t* bt, void* ws, size_t ws_bytes, cudaStream_t stream) {
  if(w == nullptr || bt == nullptr || d_quant_mult == nullptr || K <= 0 || N <= 0)
    return MI8_ERR_BAD_ARG;
  if(ws == nullptr || ws_bytes < kWsHeaderBytes)
    return MI8_ERR_WORKSPACE;
  if(reinterpret_cast<uintptr_t>(w) & 15u)
    return MI8_ERR_MISALIGNED;
  if((K + 31) / 32 > 65535)
    return MI8_ERR_UNSUPPORTED;
  int* status = device_status_ptr();
  if(status == nullptr)
    return MI8_ERR_LAUNCH;
  unsigned* partials = reinterpret_cast<unsigned*>(static_cast<uint8_t*>(ws) + kWsOffAbsmaxPartials);
  const int parts = launch_parts(w, static_cast<size_t>(K) * N, partials, stream);
  const int words = K % 4 == 0 && (reinterpret_cast<uintptr_t>(bt) & 3u) == 0 ? 1 : 0;
  const int vec = N % 4 == 0 ? 1 : 0;
  launch_kernel(mi8_convert_kernel, dim3((N + 31) / 32, (K + 127) / 128), dim3(kBlock), 0, stream, w, K, N, partials, parts, d_quant_mult, bt, words, vec,
                status);
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

// Decode-step glue kernels around the int8 affines: embedding + position, residual add + LayerNorm,
// quantisation from a pre-reduced abs-max, single-query attention over a key/value history,
// history bookkeeping for the per-step re-projection of self-attention keys/values, and the
// log-softmax + top-k of the output layer.  All fp32, all HBM/latency-bound streaming kernels.
//
// Abs-max fusion: every producer of a tensor that is quantised next (embedding, LayerNorm, attention,
// the ReLU GEMM) reduces max|x| on the fly into a 4-byte slot (unsigned bit pattern, atomicMax), so
// the quantisation needs one launch instead of two.  Slots are zeroed once per step by the driver.
#include <cfloat>

#include "mi8_internal.h"
#include "mi8_math.cuh"
#include "mi8_ptx.cuh"

namespace mi8 {
namespace {

constexpr int kRowThreads = 256;
constexpr int kMaxVec = 4;  // float4 per thread: rows of up to 4096 floats
constexpr int kMaxHistLayers = 16;
constexpr int kMaxHistBeams = 6;   // hypotheses of a sentence that attention_hist_kernel serves together; from kHistBeams on for so many sentences only:
constexpr int kHistBeams = 4, kMaxHistSentences = 32;

__device__ __forceinline__ unsigned abs_bits(float v) { return __float_as_uint(v) & 0x7fffffffu; }

__device__ __forceinline__ unsigned block_max_u(unsigned v, unsigned* red) {
  v = __reduce_max_sync(0xffffffffu, v);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  __syncthreads();
  if(lane == 0)
    red[warp] = v;
  __syncthreads();
  unsigned t = 0u;
#pragma unroll
  for(int w = 0; w < kRowThreads / 32; ++w)
    t = max(t, red[w]);
  return t;
}

__device__ __forceinline__ unsigned max4u(unsigned m, const float4& v) {
  return max(max(max(m, abs_bits(v.x)), max(abs_bits(v.y), abs_bits(v.z))), abs_bits(v.w));
}

// out[r,:] = wemb[words[r],:] * scale + pos[(pos_mod ? r % pos_mod : 0),:]
// (words == nullptr: zero embedding, the start symbol; pos_mod = source width for the encoder, 0 for a decoder step)
__device__ __forceinline__ void embed_row(int r, const float* __restrict__ wemb, const int* __restrict__ words, const float* __restrict__ pos,
                                          int pos_mod, float scale, int dim, float* __restrict__ out, float* __restrict__ rowmax,
                                          unsigned* absmax_slot, unsigned* absmax_slot2, unsigned* red) {
  const float4* src = words ? reinterpret_cast<const float4*>(wemb + static_cast<size_t>(words[r]) * dim) : nullptr;
  const float4* p4 = reinterpret_cast<const float4*>(pos + static_cast<size_t>(pos_mod ? r % pos_mod : 0) * dim);
  float4* dst = reinterpret_cast<float4*>(out + static_cast<size_t>(r) * dim);
  unsigned m = 0u;
  for(int i = threadIdx.x; i < dim / 4; i += kRowThreads) {
    float4 e = src ? __ldg(src + i) : make_float4(0.f, 0.f, 0.f, 0.f);
    const float4 p = __ldg(p4 + i);
    float4 o;
    o.x = __fadd_rn(__fmul_rn(e.x, scale), p.x);
    o.y = __fadd_rn(__fmul_rn(e.y, scale), p.y);
    o.z = __fadd_rn(__fmul_rn(e.z, scale), p.z);
    o.w = __fadd_rn(__fmul_rn(e.w, scale), p.w);
    dst[i] = o;
    m = max4u(m, o);
  }
  m = block_max_u(m, red);
  if(threadIdx.x == 0) {
    if(rowmax)
      rowmax[r] = __uint_as_float(m);
    if(absmax_slot)
      atomicMax(absmax_slot, m);
    if(absmax_slot2)
      atomicMax(absmax_slot2, m);
  }
}

__global__ void __launch_bounds__(kRowThreads)
embed_kernel(const float* __restrict__ wemb, const int* __restrict__ words, const float* __restrict__ pos, int pos_mod, float scale,
             int dim, float* __restrict__ out, float* __restrict__ rowmax, unsigned* absmax_slot) {
  const TraceHandles th = trace_open_all();
  unsigned long long* const tb = th.first;
  pdl_wait_and_launch();
  trace_stamp_start(th, kTrEmbed);
  __shared__ unsigned red[kRowThreads / 32];
  embed_row(blockIdx.x, wemb, words, pos, pos_mod, scale, dim, out, rowmax, absmax_slot, nullptr, red);
  trace_stamp(tb, kTrEmbed, 2);
  trace_stamp(th.last, kTrEmbed, 3);
}

// The beginning of a decoder step: brings the step's control words (hypothesis rows, previous words, path scores, batch rows)
// from pinned host memory to the device and zeroes the abs-max slots and arrival counters.  One block, one round trip over
// PCIe, in place of a copy and a memset between the host's decision and the first kernel.  With finish_step and
// embed_ancestors_kernel below, which take three more commands out of a step: student, one sentence 4.95 -> 4.78 ms;
// student, 16 x beam 4 6.80 -> 6.55 ms; transformer-base, 16 x beam 4 19.27 -> 19.08 ms; transformer-big level.
__global__ void __launch_bounds__(1024)
step_begin_kernel(const int* host_ctrl, int* __restrict__ ctrl, int n_ctrl, unsigned* __restrict__ slots, int n_slots) {
  const TraceHandles th = trace_open_all();
  pdl_wait_and_launch();
  trace_stamp_start(th, kTrStepBegin);
  for(int i = threadIdx.x; i < n_slots; i += blockDim.x)
    slots[i] = 0u;
  const int4* src = reinterpret_cast<const int4*>(host_ctrl);   // (both arrays are 16-byte aligned and padded to whole vectors)
  for(int i = threadIdx.x; i < (n_ctrl + 3) / 4; i += blockDim.x)
    reinterpret_cast<int4*>(ctrl)[i] = __ldcv(src + i);
#ifndef MI8_NO_TRACE
  __syncthreads();   // (all stores are issued, so all words have arrived: the stamp counts their way over PCIe)
#endif
  trace_stamp(th.first, kTrStepBegin, 2);
}

// out = LayerNorm(a + resid) * gamma + beta, one block of 256 threads per row; biased variance
// (gamma * (x - mean) / sqrt(var + eps) + beta, src/tensors/cpu/tensor_operators.cpp:1087-1124).
// Arithmetic order (all operations rounded to nearest, restated identically by the CPU checker):
//   thread t owns the float4 chunks c = t + 256*j;  y = a + resid;
//   s_t = sum_j ((y0 + y1) + (y2 + y3));  mean = block256_sum(s) / dim;
//   q_t = sum_j fma(d0,d0, fma(d1,d1, fma(d2,d2, d3*d3))), d = y - mean;  var = block256_sum(q) / dim;
//   out = ((y - mean) / sqrt(var + eps)) * gamma + beta.
// More floats than kEarlyFloats: the next kernel may begin at once instead of behind the wait, beside a kernel that works for longer than its set-up.  Medians of 4 to 6
// passes by turns, at once / behind the wait, ms: transformer-big (1024 floats a row), 512 rows 38.9 / 39.3, 440 35.4 / 35.7, 400 36.2 / 36.6, 380 35.3 / 35.7, 336 33.5 /
// 33.2; transformer-base (512), 480 rows 28.4 / 27.7, 400 28.1 / 27.7, 360 33.3 / 32.8, 512 level.
constexpr unsigned kEarlyFloats = 368 * 1024;
__global__ void __launch_bounds__(kRowThreads)
add_layernorm_kernel(const float* __restrict__ a, const float* __restrict__ resid, const float* __restrict__ gamma,
                     const float* __restrict__ beta, float eps, int dim, float* __restrict__ out, float* __restrict__ rowmax,
                     unsigned* absmax_slot, unsigned* absmax_slot2) {
  const TraceHandles th = trace_open_all();
  unsigned long long* const tb = th.first;
  if(gridDim.x * static_cast<unsigned>(dim) > kEarlyFloats) {
    pdl_launch_dependents();
    pdl_wait();
  } else {
    pdl_wait_and_launch();
  }
  trace_stamp_start(th, kTrAddLn);
  __shared__ float redf[kRowThreads / 32];
  __shared__ unsigned redu[kRowThreads / 32];
  const int r = blockIdx.x;
  const float4* a4 = reinterpret_cast<const float4*>(a + static_cast<size_t>(r) * dim);
  const float4* r4 = resid ? reinterpret_cast<const float4*>(resid + static_cast<size_t>(r) * dim) : nullptr;
  float4 v[kMaxVec];
  float s = 0.f;
#pragma unroll
  for(int j = 0; j < kMaxVec; ++j) {
    const int i = threadIdx.x + j * kRowThreads;
    if(i < dim / 4) {
      float4 x = a4[i];
      if(r4) {
        const float4 y = r4[i];
        x.x = __fadd_rn(x.x, y.x); x.y = __fadd_rn(x.y, y.y); x.z = __fadd_rn(x.z, y.z); x.w = __fadd_rn(x.w, y.w);
      }
      v[j] = x;
      s = __fadd_rn(s, __fadd_rn(__fadd_rn(x.x, x.y), __fadd_rn(x.z, x.w)));
    }
  }
  const float mean = __fdiv_rn(block256_sum_det(s, redf), static_cast<float>(dim));
  float q = 0.f;
#pragma unroll
  for(int j = 0; j < kMaxVec; ++j) {
    const int i = threadIdx.x + j * kRowThreads;
    if(i < dim / 4) {
      const float dx = __fadd_rn(v[j].x, -mean), dy = __fadd_rn(v[j].y, -mean), dz = __fadd_rn(v[j].z, -mean), dw = __fadd_rn(v[j].w, -mean);
      q = __fadd_rn(q, __fmaf_rn(dx, dx, __fmaf_rn(dy, dy, __fmaf_rn(dz, dz, __fmul_rn(dw, dw)))));
    }
  }
  const float var = __fdiv_rn(block256_sum_det(q, redf), static_cast<float>(dim));
  const float denom = __fsqrt_rn(__fadd_rn(var, eps));
  const float4* g4 = reinterpret_cast<const float4*>(gamma);
  const float4* b4 = reinterpret_cast<const float4*>(beta);
  float4* o4 = reinterpret_cast<float4*>(out + static_cast<size_t>(r) * dim);
  unsigned m = 0u;
#pragma unroll
  for(int j = 0; j < kMaxVec; ++j) {
    const int i = threadIdx.x + j * kRowThreads;
    if(i < dim / 4) {
      const float4 g = __ldg(g4 + i), b = __ldg(b4 + i);
      float4 o;
      o.x = __fadd_rn(__fmul_rn(__fdiv_rn(__fadd_rn(v[j].x, -mean), denom), g.x), b.x);
      o.y = __fadd_rn(__fmul_rn(__fdiv_rn(__fadd_rn(v[j].y, -mean), denom), g.y), b.y);
      o.z = __fadd_rn(__fmul_rn(__fdiv_rn(__fadd_rn(v[j].z, -mean), denom), g.z), b.z);
      o.w = __fadd_rn(__fmul_rn(__fdiv_rn(__fadd_rn(v[j].w, -mean), denom), g.w), b.w);
      o4[i] = o;
      m = max4u(m, o);
    }
  }
  m = block_max_u(m, redu);
  if(threadIdx.x == 0) {
    if(rowmax)
      rowmax[r] = __uint_as_float(m);
    if(absmax_slot)
      atomicMax(absmax_slot, m);
    if(absmax_slot2)
      atomicMax(absmax_slot2, m);
  }
  trace_stamp(tb, kTrAddLn, 2);
  trace_stamp(th.last, kTrAddLn, 3);
}

__device__ __forceinline__ int quantize_one(float v, float qm) {
  int r = __float2int_rn(__fmul_rn(v, qm));
  return max(-127, min(127, r));
}
__device__ __forceinline__ unsigned pack4(const float4& v, float qm) {
  return (static_cast<unsigned>(quantize_one(v.x, qm)) & 0xffu) | ((static_cast<unsigned>(quantize_one(v.y, qm)) & 0xffu) << 8) |
         ((static_cast<unsigned>(quantize_one(v.z, qm)) & 0xffu) << 16) | ((static_cast<unsigned>(quantize_one(v.w, qm)) & 0xffu) << 24);
}
__device__ __forceinline__ float quant_mult_from_bits(unsigned bits) {
  return bits == 0u ? 1.0f : __fdiv_rn(127.0f, __uint_as_float(bits));
}

// Block `block` of `blocks` quantises its share of n floats (a multiple of four) at x into q: four 16-byte loads in flight per thread, the lanes of a warp
// side by side in each.  (A thread that took 64 consecutive bytes spread every load of its warp over 2 KB.)  The distance of a thread's vectors is a constant:
// from blockDim launches of up to 500000 floats were slower than with 64 consecutive bytes (16384 floats 1.52 us then, 1.63 with blockDim, 1.46 so; 524288
// 2.07, 2.11, 1.82; 4 M 3.87, 3.52, 2.97).
constexpr int kQuantizeThreads = 256;
__device__ __forceinline__ void quantize_range(const float* __restrict__ x, int8_t* __restrict__ q, size_t n, float qm, unsigned block, unsigned blocks) {
  const size_t n4 = n / 4;
  const float4* x4 = reinterpret_cast<const float4*>(x);
  unsigned* q4 = reinterpret_cast<unsigned*>(q);
  for(size_t base = static_cast<size_t>(block) * (4 * kQuantizeThreads) + threadIdx.x; base < n4; base += static_cast<size_t>(blocks) * (4 * kQuantizeThreads)) {
    float4 v[4];
#pragma unroll
    for(int e = 0; e < 4; ++e)
      if(base + e * kQuantizeThreads < n4)
        v[e] = __ldg(x4 + base + e * kQuantizeThreads);
#pragma unroll
    for(int e = 0; e < 4; ++e)
      if(base + e * kQuantizeThreads < n4)
        q4[base + e * kQuantizeThreads] = pack4(v[e], qm);
  }
}

// Quantise with the multiplier derived from an abs-max slot that a producer kernel already reduced.
// Optional row gather: source row of output row i is src_rows[i] (rows of `row_len` floats).
__global__ void __launch_bounds__(256)
quantize_slot_kernel(const float* __restrict__ x, size_t n, const unsigned* __restrict__ absmax_slot, int8_t* __restrict__ q,
                     float* __restrict__ d_quant_mult, int* status) {
  pdl_launch_dependents();   // (early: the GEMM behind it has a longer set-up than this kernel work)
  const TraceHandles th = trace_open_all();
  unsigned long long* const tb = th.first;
  pdl_wait();
  trace_stamp_start(th, kTrQuantSlot);
  const unsigned bits = *absmax_slot;
  const float qm = quant_mult_from_bits(bits);
  if(blockIdx.x == 0 && threadIdx.x == 0) {
    *d_quant_mult = qm;
    if(bits >= 0x7f800000u)
      atomicMax(status, static_cast<int>(kDevNonFinite));
  }
  quantize_range(x, q, n, qm, blockIdx.x, gridDim.x);
  if(blockIdx.x == 0 && threadIdx.x < (n & 3))
    q[n / 4 * 4 + threadIdx.x] = static_cast<int8_t>(quantize_one(x[n / 4 * 4 + threadIdx.x], qm));
  trace_stamp(tb, kTrQuantSlot, 2);
  trace_stamp(th.last, kTrQuantSlot, 3);
}

// add_layernorm_kernel and quantize_slot_kernel in one launch for few rows: one cluster of kCtas CTAs holds all rows (one per thread
// group), so the abs-max of the whole tensor is known after a cluster barrier and the rows are quantised from registers.  At a few
// dozen rows both kernels are launch and round trip (1.8 + 2.1 us and 0.9 + 2.1 us of work and hand-over in a step of the
// student).  A thread owns one float4 of a row (up to 1024 floats), a row's group is dim / 4 threads rounded up to whole warps, sums in
// the order of add_layernorm_kernel (the warps that kernel has beyond the row's end add +0).  With cell_old set, the first operand is the
// SSRU cell's output instead of `a`: the new state is computed (and stored) on the way, as ssru_cell_kernel does.
// Student, one sentence 4.80 -> 4.34 ms, 16 sentences 6.10 -> 5.64, 16 x beam 4 6.58 -> 6.29; transformer-base, one sentence 13.2 -> 12.6 ms.
struct SsruArgs {
  const float* cell_old = nullptr;   // [rows of the previous step, dim]
  const int* hyp = nullptr;          // row of cell_old per row (null: the same)
  const float* xw = nullptr;
  const float* f = nullptr;
  float* cell_new = nullptr;
};

template <int kCtas>
__global__ void __cluster_dims__(kCtas, 1, 1) __launch_bounds__(1024)
add_layernorm_quant_kernel(const float* __restrict__ a, const SsruArgs cell, const float* __restrict__ resid, const float* __restrict__ gamma,
                           const float* __restrict__ beta, float eps, int rows, int dim, int group_warps, float* __restrict__ out,
                           int8_t* __restrict__ q, float* __restrict__ d_quant_mult, int* status) {
  const TraceHandles th = trace_open_all();
  unsigned long long* const tb = th.first;
  __shared__ float red[32];
  __shared__ unsigned redu[32];
  __shared__ unsigned cta_max[kCtas];
  if(kCtas > 1)
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");   // (this CTA runs: the others may write to cta_max)
  pdl_wait_and_launch();
  trace_stamp_start(th, kTrAddLnQuant);
  const int rank = kCtas > 1 ? static_cast<int>(blockIdx.x) : 0;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = static_cast<int>(blockDim.x) >> 5;
  const int groups = warps / group_warps, group = warp / group_warps;
  const int chunk = (warp - group * group_warps) * 32 + lane;
  const int r = rank * groups + group;
  const bool live = chunk < dim / 4 && r < rows;
  const size_t o = static_cast<size_t>(live ? r : 0) * (dim / 4) + chunk;
  float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
  if(live) {
    if(cell.cell_old != nullptr) {
      const float4 c = reinterpret_cast<const float4*>(cell.cell_old)[static_cast<size_t>(cell.hyp ? cell.hyp[r] : r) * (dim / 4) + chunk];
      const float4 w = reinterpret_cast<const float4*>(cell.xw)[o], f = reinterpret_cast<const float4*>(cell.f)[o];
      float4 cn;
      cn.x = ssru_cell(c.x, w.x, f.x, &x.x);
      cn.y = ssru_cell(c.y, w.y, f.y, &x.y);
      cn.z = ssru_cell(c.z, w.z, f.z, &x.z);
      cn.w = ssru_cell(c.w, w.w, f.w, &x.w);
      reinterpret_cast<float4*>(cell.cell_new)[o] = cn;
    } else {
      x = reinterpret_cast<const float4*>(a)[o];
    }
    const float4 y = reinterpret_cast<const float4*>(resid)[o];
    x.x = __fadd_rn(x.x, y.x); x.y = __fadd_rn(x.y, y.y); x.z = __fadd_rn(x.z, y.z); x.w = __fadd_rn(x.w, y.w);
  }
  // the row's sum over its group: butterflies, then the warps' totals in ascending order
  auto row_sum = [&](float t) {
    t = warp_sum_det(t);
    __syncthreads();
    if(lane == 0)
      red[warp] = t;
    __syncthreads();
    t = 0.f;
    for(int w = 0; w < group_warps; ++w)
      t = __fadd_rn(t, red[group * group_warps + w]);
    return t;
  };
  const float mean = __fdiv_rn(row_sum(live ? __fadd_rn(0.f, __fadd_rn(__fadd_rn(x.x, x.y), __fadd_rn(x.z, x.w))) : 0.f), static_cast<float>(dim));
  float t = 0.f;
  if(live) {
    x.x = __fadd_rn(x.x, -mean); x.y = __fadd_rn(x.y, -mean); x.z = __fadd_rn(x.z, -mean); x.w = __fadd_rn(x.w, -mean);
    t = __fadd_rn(0.f, __fmaf_rn(x.x, x.x, __fmaf_rn(x.y, x.y, __fmaf_rn(x.z, x.z, __fmul_rn(x.w, x.w)))));
  }
  const float var = __fdiv_rn(row_sum(t), static_cast<float>(dim));
  const float denom = __fsqrt_rn(__fadd_rn(var, eps));
  unsigned m = 0u;
  if(live) {
    const float4 g = __ldg(reinterpret_cast<const float4*>(gamma) + chunk), b = __ldg(reinterpret_cast<const float4*>(beta) + chunk);
    x.x = __fadd_rn(__fmul_rn(__fdiv_rn(x.x, denom), g.x), b.x);
    x.y = __fadd_rn(__fmul_rn(__fdiv_rn(x.y, denom), g.y), b.y);
    x.z = __fadd_rn(__fmul_rn(__fdiv_rn(x.z, denom), g.z), b.z);
    x.w = __fadd_rn(__fmul_rn(__fdiv_rn(x.w, denom), g.w), b.w);
    reinterpret_cast<float4*>(out)[o] = x;
    m = max4u(0u, x);
  }
  m = __reduce_max_sync(0xffffffffu, m);
  if(lane == 0)
    redu[warp] = m;
  __syncthreads();
  m = __reduce_max_sync(0xffffffffu, lane < warps ? redu[lane] : 0u);
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
  const float qm = quant_mult_from_bits(m);
  if(rank == 0 && threadIdx.x == 0) {
    *d_quant_mult = qm;
    if(m >= 0x7f800000u)
      atomicMax(status, static_cast<int>(kDevNonFinite));
  }
  if(live)
    reinterpret_cast<unsigned*>(q)[o] = pack4(x, qm);
  trace_stamp(tb, kTrAddLnQuant, 2);
  trace_stamp(th.last, kTrAddLnQuant, 3);
}

// Two quantisations in one launch, for the start of a decoder self-attention block: blocks [0, blocks_x)
// quantise the layer input x with its own multiplier (the query projection's operand), the others the
// self-attention history with the multiplier of the whole live history (the key/value projections' operand):
// only the newest slab (`rows_new` live rows, the last of the slabs) when the history's abs-max
// still has the bits the stored keys/values were computed with (*prev_bits), everything otherwise.  (One slab row per block and iteration, a quarter of the
// threads at work at 1024 floats, made a whole history of 20 steps x 512 rows 22 us.  With whole blocks at work
// and quantize_range: transformer-base, 64 x beam 4, 34.5 -> 33.0 ms, transformer-big, 128 x 4, 41.25 -> 40.25; with two blocks per SM instead of four 33.1 and 41.5.)
__global__ void __launch_bounds__(256)
quantize_dual_kernel(const float* __restrict__ x, size_t n, const unsigned* __restrict__ slot_x, int8_t* __restrict__ q,
                     float* __restrict__ qm_x, int* status, int blocks_x, const float* __restrict__ slabs, int slab_rows, int steps,
                     int rows_new, int dim, const unsigned* __restrict__ slot_h, const unsigned* __restrict__ prev_bits,
                     int8_t* __restrict__ hq, float* __restrict__ qm_h) {
  const TraceHandles th = trace_open_all();
  unsigned long long* const tb = th.first;
  pdl_wait_and_launch();
  trace_stamp_start(th, kTrQuantDual);
  if(static_cast<int>(blockIdx.x) < blocks_x) {
    const unsigned bits = *slot_x;
    const float qm = quant_mult_from_bits(bits);
    if(blockIdx.x == 0 && threadIdx.x == 0) {
      *qm_x = qm;
      if(bits >= 0x7f800000u)
        atomicMax(status, static_cast<int>(kDevNonFinite));
    }
    quantize_range(x, q, n, qm, blockIdx.x, blocks_x);
  } else {
    const int hb = static_cast<int>(blockIdx.x) - blocks_x, nhb = static_cast<int>(gridDim.x) - blocks_x;
    const unsigned bits = *slot_h;
    const float qm = quant_mult_from_bits(bits);
    if(hb == 0 && threadIdx.x == 0)
      *qm_h = qm;
    const int total = (steps - 1) * slab_rows + rows_new;
    const int first = (*prev_bits == bits) ? (steps - 1) * slab_rows : 0;   // unchanged abs-max: only the newest slab
    quantize_range(slabs + static_cast<size_t>(first) * dim, hq + static_cast<size_t>(first) * dim, static_cast<size_t>(total - first) * dim, qm, hb, nhb);
  }
  trace_stamp(tb, kTrQuantDual, 2);
  trace_stamp(th.last, kTrQuantDual, 3);
}

// ---- self-attention history ------------------------------------------------------------------
// The decoder re-projects keys/values from the whole history of layer inputs every step, quantised
// with ONE multiplier over that history (src/models/transformer.h:401-417).  The history is kept as
// per-step slabs slab[t'][row][dim] in the row order of step t', plus an ancestor table
// anc[t'][r] = row of slab t' that current hypothesis r descends from, so a beam reorder only
// rewrites the small table.  rowmax[t'][row] holds max|x| of each slab row.

// anc_new[t'][r] = anc_old[t'][hyp[r]] (t' < t), anc_new[t][r] = r.
// With hist.layers > 0 the kernel also starts every layer's history abs-max of this step: for each layer l the
// maximum of rowmax_l[t'][anc_new[t'][r]] over the EARLIER slabs t' < t is reduced into hist.slot[l]; the producer
// of the layer's newest slab adds that slab's maximum to the same slot, which then holds what
// history_absmax_kernel computes in a launch of its own.
struct HistMaxArgs {
  int layers;
  const float* rowmax[kMaxHistLayers];
  unsigned* slot[kMaxHistLayers];
};
__device__ __forceinline__ void ancestors_slice(int block, const int* __restrict__ anc_old, int* __restrict__ anc_new, const int* __restrict__ hyp,
                                                int t, int rows, int stride, const HistMaxArgs& hist) {
  const int i = block * static_cast<int>(blockDim.x) + threadIdx.x;
  const bool in = i < (t + 1) * rows;
  int tp = 0, src = 0;
  if(in) {
    tp = i / rows;
    const int r = i - tp * rows;
    src = tp == t ? r : anc_old[tp * stride + hyp[r]];
    anc_new[tp * stride + r] = src;
  }
  for(int l = 0; l < hist.layers; ++l) {
    unsigned m = (in && tp < t) ? abs_bits(hist.rowmax[l][tp * stride + src]) : 0u;
    m = __reduce_max_sync(0xffffffffu, m);
    if((threadIdx.x & 31) == 0 && m != 0u)
      atomicMax(hist.slot[l], m);
  }
}

// The distinct slab rows that the hypotheses of sentence b descend from, position by position (hypotheses of one sentence share most of
// their history): list[i] = slab row, and which[j][p] = its place for hypothesis j at position p; ascending with the position.
// Both lie at the sentence's share b * beams * (t + 1) of their arrays, count[b] = length.  Read by attention_hist_kernel.
__device__ __forceinline__ void history_list(int b, const int* __restrict__ anc_old, const int* __restrict__ hyp, int t, int rows, int stride,
                                             const HistLists& out, unsigned* red) {
  const int beams = rows / out.batch, len = t + 1;
  int* list = out.list + static_cast<size_t>(b) * beams * len;
  int* which = out.which + static_cast<size_t>(b) * beams * len;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int base = 0;   // places taken by earlier positions
  for(int p0 = 0; p0 < len; p0 += kRowThreads) {
    const int p = p0 + threadIdx.x;
    int a[kMaxHistBeams], at[kMaxHistBeams];   // (unrolled: in registers)
    int n = 0;
#pragma unroll
    for(int j = 0; j < kMaxHistBeams; ++j) {
      a[j] = -1;
      at[j] = 0;
      if(p < len && j < beams) {
        const int r = j * out.batch + b;
        a[j] = p == t ? r : anc_old[p * stride + hyp[r]];
        at[j] = n;
        bool seen = false;
#pragma unroll
        for(int i = 0; i < j; ++i)
          if(!seen && a[i] == a[j]) {
            seen = true;
            at[j] = at[i];
          }
        n += seen ? 0 : 1;
      }
    }
    // places before this position: inclusive scan over the block
    int sum = n;
#pragma unroll
    for(int o = 1; o < 32; o <<= 1) {
      const int up = __shfl_up_sync(0xffffffffu, sum, o);
      sum += lane >= o ? up : 0;
    }
    __syncthreads();
    if(lane == 31)
      red[warp] = static_cast<unsigned>(sum);
    __syncthreads();
    int before = base + sum - n;
    for(int w = 0; w < kRowThreads / 32; ++w) {
      before += w < warp ? static_cast<int>(red[w]) : 0;
      base += static_cast<int>(red[w]);
    }
#pragma unroll
    for(int j = 0; j < kMaxHistBeams; ++j)
      if(p < len && j < beams) {
        list[before + at[j]] = p * stride + a[j];   // (equal rows write the same value)
        which[j * len + p] = before + at[j];
      }
  }
  if(threadIdx.x == 0)
    out.count[b] = base;
}

// The independent jobs at the start of a self-attention decoder's step in one launch: blocks [0, rows) embed the previous
// words (layer 0's newest slab), the next `lists.batch` list the sentences' distinct history rows, the others update the ancestor table and start
// the layers' history abs-max.
__global__ void __launch_bounds__(kRowThreads)
embed_ancestors_kernel(const float* __restrict__ wemb, const int* __restrict__ words, const float* __restrict__ pos, float scale, int dim,
                       float* __restrict__ out, float* __restrict__ rowmax, unsigned* absmax_slot, unsigned* absmax_slot2,
                       const int* __restrict__ anc_old, int* __restrict__ anc_new, const int* __restrict__ hyp, int t, int rows, int stride,
                       const HistMaxArgs hist, const HistLists lists) {
  const TraceHandles th = trace_open_all();
  unsigned long long* const tb = th.first;
  pdl_wait_and_launch();
  trace_stamp_start(th, kTrEmbed);
  __shared__ unsigned red[kRowThreads / 32];
  if(static_cast<int>(blockIdx.x) < rows)
    embed_row(blockIdx.x, wemb, words, pos, 0, scale, dim, out, rowmax, absmax_slot, absmax_slot2, red);
  else if(static_cast<int>(blockIdx.x) < rows + lists.batch)
    history_list(static_cast<int>(blockIdx.x) - rows, anc_old, hyp, t, rows, stride, lists, red);
  else
    ancestors_slice(static_cast<int>(blockIdx.x) - rows - lists.batch, anc_old, anc_new, hyp, t, rows, stride, hist);
  trace_stamp(tb, kTrEmbed, 2);
  trace_stamp(th.last, kTrEmbed, 3);
}

// The butterfly of the G threads of a head, for U positions at once: at the level that pairs lanes j and j ^ o the two
// lanes split the positions still held between them - each sends the partial sums of the half it gives up and adds
// what it receives to the half it keeps - so a level costs half as many shuffles and additions as the one before,
// instead of one of each per position.  Every sum is "own + partner's" of the same two operands as in the plain
// butterfly, hence the same bits.  Once a lane holds a single position the remaining levels are the plain butterfly.
// Returns the first position lane j holds afterwards (its sum in d[0], with U > G the next U / G - 1 behind it).
template <int G, int U>
__device__ __forceinline__ int head_butterfly(float (&d)[U], int j) {
  int pos = 0;
#pragma unroll
  for(int lvl = 0; ((G / 2) >> lvl) > 0; ++lvl) {
    const int o = (G / 2) >> lvl;
    const int c = (U >> lvl) > 1 ? (U >> lvl) : 1;   // positions a lane holds before this level
    if(c > 1) {
      const bool upper = (j & o) != 0;
#pragma unroll
      for(int i = 0; i < c / 2; ++i) {
        const float send = upper ? d[i] : d[i + c / 2];
        const float keep = upper ? d[i + c / 2] : d[i];
        d[i] = __fadd_rn(keep, __shfl_xor_sync(0xffffffffu, send, o));
      }
      pos += upper ? c / 2 : 0;
    } else {
      d[0] = __fadd_rn(d[0], __shfl_xor_sync(0xffffffffu, d[0], o));
    }
  }
  return pos;
}

// ---- single-query attention --------------------------------------------------------------------
// One block per query row; thread i owns elements 4i..4i+3 of the model dimension, i.e. a quarter-row
// slice of head i / G with G = DH/4 threads per head.  For every key position the block reads the whole
// key row (all heads) with one 16-byte load per thread - fully coalesced whatever the layout of the
// history - and the G threads of a head combine their partial dot products with a butterfly.
// Key/value row of position p for query row r is  kv_base(r) + p * kv_stride:
//   mode 0, decoder self-attention over the time-major history:  base = r,              stride = rows
//   mode 1, cross-attention over the context [batch, len, dim]:   base = (r % batch)*len, stride = 1, log mask row r % batch
//   mode 2, encoder self-attention, rows ordered [batch, len]:    base = (r / len)*len,   stride = 1, log mask row r / len
// softmax(q.k / sqrt(dh) + mask) . v in fp32 (src/models/transformer.h:240-277).
// Arithmetic order per (row, head), restated identically by the CPU checker:
//   thread j of the head: d_j = fma(q3,k3, fma(q2,k2, fma(q1,k1, q0*k0))) over its four elements
//   s_p = butterfly over the G threads (d_j + d_{j^o}, o = G/2 .. 1);  s_p = s_p * scale;  s_p = s_p + mask_p
//   mx = max_p s_p;  e_p = det_expf(s_p - mx)
//   thread j accumulates e_p for p = j, j+G, ... ascending; sum = butterfly over the G threads
//   w_p = e_p / sum;  out_i = fma-chain over p ascending of w_p * v_{p,i}, starting from 0.
template <int DH, int U>
__global__ void __launch_bounds__(256)
attention1_kernel(const float* __restrict__ q, const float* __restrict__ k, const float* __restrict__ v,
                  const float* __restrict__ log_mask, int heads, int len, int rows, int batch, int mode, float scale,
                  float* __restrict__ out, unsigned* absmax_slot, const int* __restrict__ anc, int anc_stride, int kv_rows) {
  const TraceHandles th = trace_open_all();
  unsigned long long* const tb = th.first;
  pdl_wait_and_launch();
  trace_stamp_start(th, kTrAttention1);
  extern __shared__ float sc_smem[];  // [heads][len] scores, then probabilities
  constexpr int G = DH / 4;
  const int r = blockIdx.x;
  // blockIdx.y selects the group of heads this block serves (blockDim.x / G heads, all of them when gridDim.y == 1);
  // `tid` is the thread's position in the row (quarter-row slice tid of the model dimension)
  const int hb = gridDim.y == 1 ? heads : static_cast<int>(blockDim.x) / G;
  const int tid = blockIdx.y * hb * G + threadIdx.x;
  const int dim = heads * DH;
  const bool active = tid < dim / 4;
  const int head = threadIdx.x / G, j = threadIdx.x % G;   // head inside the block's group
  const int group = mode == 1 ? r % batch : (mode == 2 ? r / len : 0);
  const size_t base = mode == 0 ? static_cast<size_t>(r) : static_cast<size_t>(group) * len;
  const size_t stride = (mode == 0 ? static_cast<size_t>(rows) : 1) * dim;
  const float* mask = (mode != 0 && log_mask) ? log_mask + static_cast<size_t>(group) * len : nullptr;
  const float4 qv = active ? __ldg(reinterpret_cast<const float4*>(q + static_cast<size_t>(r) * dim) + tid) : make_float4(0.f, 0.f, 0.f, 0.f);
  float* srow = sc_smem + (active ? head : 0) * len;
  // mode 0 with an ancestor table: keys/values are stored per step in that step's row order, and the row
  // of position p that query row r descends from is anc[p][r]
  const bool indirect = mode == 0 && anc != nullptr;
  int* anc_s = reinterpret_cast<int*>(sc_smem + hb * len);   // [len] ancestor rows of this query row
  if(indirect) {
    for(int p = threadIdx.x; p < len; p += blockDim.x)
      anc_s[p] = anc[static_cast<size_t>(p) * anc_stride + r];
    __syncthreads();
  }
  auto row_offset = [&](int p) -> size_t {
    if(indirect)
      return (static_cast<size_t>(p) * kv_rows + anc_s[p]) * dim + 4 * tid;
    return base * dim + 4 * tid + p * stride;
  };

  // scores: U key rows in flight per thread (the loads do not depend on one another; the arithmetic per
  // position is the same whatever U is)
  for(int p0 = 0; p0 < len; p0 += U) {
    float4 kk[U];
#pragma unroll
    for(int u = 0; u < U; ++u)
      kk[u] = (active && p0 + u < len) ? __ldg(reinterpret_cast<const float4*>(k + row_offset(p0 + u))) : make_float4(0.f, 0.f, 0.f, 0.f);
    float d[U];
#pragma unroll
    for(int u = 0; u < U; ++u) {
      d[u] = __fmul_rn(qv.x, kk[u].x);
      d[u] = __fmaf_rn(qv.y, kk[u].y, d[u]);
      d[u] = __fmaf_rn(qv.z, kk[u].z, d[u]);
      d[u] = __fmaf_rn(qv.w, kk[u].w, d[u]);
    }
    const int pos = head_butterfly<G, U>(d, j);
    // lanes that differ only in the bits of the plain levels hold the same position: the one with those bits clear writes
    // (with more positions than lanes a lane ends up holding U / G neighbouring positions)
    constexpr int kPlainMask = (U >= G) ? 0 : (G / U) - 1;
    constexpr int kHeld = U > G ? U / G : 1;
    if(active && (j & kPlainMask) == 0) {
#pragma unroll
      for(int i = 0; i < kHeld; ++i) {
        if(p0 + pos + i < len) {
          float sc = __fmul_rn(d[i], scale);
          if(mask)
            sc = __fadd_rn(sc, mask[p0 + pos + i]);
          srow[p0 + pos + i] = sc;
        }
      }
    }
  }
  __syncthreads();
  // softmax over the positions of this thread's head (the G threads of a head work together)
  float mx = -FLT_MAX;
  if(active)
    for(int p = j; p < len; p += G)
      mx = fmaxf(mx, srow[p]);
#pragma unroll
  for(int o = G / 2; o > 0; o >>= 1)
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  float part = 0.f;
  if(active)
    for(int p = j; p < len; p += G) {
      const float e = det_expf(__fadd_rn(srow[p], -mx));
      srow[p] = e;
      part = __fadd_rn(part, e);
    }
#pragma unroll
  for(int o = G / 2; o > 0; o >>= 1)
    part = __fadd_rn(part, __shfl_xor_sync(0xffffffffu, part, o));
  if(active)
    for(int p = j; p < len; p += G)
      srow[p] = __fdiv_rn(srow[p], part);
  __syncthreads();
  // weighted sum of the value rows, strictly in position order, loads U rows ahead
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
  for(int p0 = 0; p0 < len; p0 += U) {
    float4 vv[U];
#pragma unroll
    for(int u = 0; u < U; ++u)
      vv[u] = (active && p0 + u < len) ? __ldg(reinterpret_cast<const float4*>(v + row_offset(p0 + u))) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for(int u = 0; u < U; ++u) {
      if(p0 + u < len) {
        const float w = srow[p0 + u];
        acc.x = __fmaf_rn(w, vv[u].x, acc.x);
        acc.y = __fmaf_rn(w, vv[u].y, acc.y);
        acc.z = __fmaf_rn(w, vv[u].z, acc.z);
        acc.w = __fmaf_rn(w, vv[u].w, acc.w);
      }
    }
  }
  unsigned m_abs = 0u;
  if(active) {
    reinterpret_cast<float4*>(out + static_cast<size_t>(r) * dim)[tid] = acc;
    m_abs = max4u(0u, acc);
  }
  if(absmax_slot) {
    m_abs = __reduce_max_sync(0xffffffffu, m_abs);
    if((threadIdx.x & 31) == 0 && m_abs != 0u)
      atomicMax(absmax_slot, m_abs);
  }
  trace_stamp(tb, kTrAttention1, 2);
  trace_stamp(th.last, kTrAttention1, 3);
}

// Cross-attention (mode 1) for all hypotheses of a sentence together.  attention1_kernel reads a sentence's keys and values once
// per hypothesis (through L2) and waits for eight rows at a time.  Here a block serves 32 consecutive four-element slices
// (32 / G heads) of one sentence, a warp per hypothesis: every key and value row is copied once into a ring of
// kCrossStages x kCrossRows rows of shared memory, up to 32 rows ahead of their use and the first value rows during the softmax, and
// read from there by all warps.  Arithmetic and order per (row, head): those of attention1_kernel.
// A warp per hypothesis rather than one warp for all of them (each row read from shared memory once, four times the
// registers): the small batches need the warps - 64 sentences x beam 4 x 512 are 256 warps that way, 11.8 us inside a step.
// Bound by the chain of instructions of a warp and, where the keys and values of all layers exceed L2, by their read.
// Inside a decoder step, attention1_kernel -> here: transformer-base 64 x beam 4 x 38 positions 11.7 -> 8.5 us, transformer-big 128 x beam 4
// 15.1 -> 11 us; whole mini-batches: transformer-base, 64 x beam 4 40.7 -> 38.4 ms, big 46.4 -> 45.7 ms, four searches of big 219.5 -> 216.5 ms.
constexpr int kCrossStages = 3;
constexpr int kCrossRows = 16;     // rows per stage of the ring
constexpr int kCrossU = 8;         // positions whose scores a warp sums at once
constexpr int kCrossMaxBeams = 8;  // hypotheses per block

__device__ __forceinline__ void prefetch_l2(const void* p, int bytes) {   // 16-byte aligned, a multiple of 16 bytes
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(bytes) : "memory");
}
__device__ __forceinline__ void copy16_async(void* smem, const void* gmem) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(smem)), "l"(gmem) : "memory");
}
__device__ __forceinline__ void copy4_async(void* smem, const void* gmem) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(smem)), "l"(gmem) : "memory");
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void copy_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

template <int DH>
__global__ void __launch_bounds__(kCrossMaxBeams * 32)
attention_cross_kernel(const float* __restrict__ q, const float* __restrict__ k, const float* __restrict__ v,
                       const float* __restrict__ log_mask, int heads, int len, int rows, int batch, float scale, float* __restrict__ out,
                       unsigned* absmax_slot) {
  const TraceHandles th = trace_open_all();
  unsigned long long* const tb = th.first;
  constexpr int G = DH / 4, U = kCrossU, SR = kCrossRows;
  constexpr int kWarpHeads = 32 / G;
  static_assert(U <= G, "a lane holds one position after the butterfly");
  extern __shared__ float4 cross_smem[];   // [stages][SR][32] rows, then per warp and head [len4] scores
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
  const int j = lane % G;
  const int dim = heads * DH;
  const int slice = blockIdx.y * 32 + lane;   // this lane's four elements of the model dimension
  const bool active = slice < dim / 4;        // (whole heads are active or not)
  const int b = blockIdx.x;
  const int r = (blockIdx.z * warps + warp) * batch + b;
  const bool live = active && r < rows;
  const int len4 = (len + 3) & ~3;
  float* scores = reinterpret_cast<float*>(cross_smem + kCrossStages * SR * 32);
  float* sc = scores + (warp * kWarpHeads + lane / G) * len4;
  const size_t kv0 = static_cast<size_t>(b) * len * dim + 4 * slice;
  const int tiles = (len + SR - 1) / SR;
  // rows SR i .. SR i + SR - 1 of the keys (i < tiles), then of the values; the warps share the rows out
  auto fetch = [&](int i) {
    if(active && i < 2 * tiles) {
      const int p0 = (i < tiles ? i : i - tiles) * SR;
      const float* src = (i < tiles ? k : v) + kv0 + static_cast<size_t>(p0 + warp) * dim;
      float4* dst = cross_smem + (i % kCrossStages) * (SR * 32) + lane;
      const int n = min(SR, len - p0);
      for(int u = warp; u < n; u += warps, src += static_cast<size_t>(warps) * dim)
        copy16_async(dst + u * 32, src);
    }
    copy_commit();
  };
  // stage i is complete and the slot of stage i - 1 free again
  auto advance = [&](int i) {
    copy_wait<kCrossStages - 2>();
    __syncthreads();
    fetch(i + kCrossStages - 1);
    return cross_smem + (i % kCrossStages) * (SR * 32) + lane;
  };
  // The keys and values were projected long before the preceding kernel: their way from HBM to L2 starts while that one runs.
  // (A prefetch reads nothing into the program, so it may come before the wait even where they are still being written.)
  {
    const int bytes = min(512, (dim - static_cast<int>(blockIdx.y) * 128) * 4);
    for(int i = threadIdx.x; i < 2 * len; i += blockDim.x)
      prefetch_l2((i < len ? k : v) + (static_cast<size_t>(b) * len + (i < len ? i : i - len)) * dim + blockIdx.y * 128, bytes);
  }
  pdl_wait_and_launch();
  trace_stamp_start(th, kTrAttentionCross);
#pragma unroll
  for(int i = 0; i < kCrossStages - 1; ++i)
    fetch(i);
  const float4 qv = live ? __ldg(reinterpret_cast<const float4*>(q + static_cast<size_t>(r) * dim) + slice) : make_float4(0.f, 0.f, 0.f, 0.f);
  const float* mask = log_mask ? log_mask + static_cast<size_t>(b) * len : nullptr;
  constexpr int kPlainMask = (U >= G) ? 0 : (G / U) - 1;   // lanes that differ only in these bits hold the same position
  for(int i = 0; i < tiles; ++i) {
    const float4* src = advance(i);
#pragma unroll
    for(int h = 0; h < SR; h += U) {
      if(i * SR + h < len) {
        float d[U];
#pragma unroll
        for(int u = 0; u < U; ++u) {   // (rows past the end: whatever the ring holds; their sums are not written)
          const float4 kk = src[(h + u) * 32];
          d[u] = __fmul_rn(qv.x, kk.x);
          d[u] = __fmaf_rn(qv.y, kk.y, d[u]);
          d[u] = __fmaf_rn(qv.z, kk.z, d[u]);
          d[u] = __fmaf_rn(qv.w, kk.w, d[u]);
        }
        const int p = i * SR + h + head_butterfly<G, U>(d, j);
        if(active && (j & kPlainMask) == 0 && p < len) {
          float s = __fmul_rn(d[0], scale);
          if(mask)
            s = __fadd_rn(s, __ldg(mask + p));
          sc[p] = s;
        }
      }
    }
  }
  __syncwarp();
  float mx = -FLT_MAX, part = 0.f;
  if(active)
    for(int p = j; p < len; p += G)
      mx = fmaxf(mx, sc[p]);
#pragma unroll
  for(int o = G / 2; o > 0; o >>= 1)
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  if(active)
    for(int p = j; p < len; p += G) {
      const float e = det_expf(__fadd_rn(sc[p], -mx));
      sc[p] = e;
      part = __fadd_rn(part, e);
    }
#pragma unroll
  for(int o = G / 2; o > 0; o >>= 1)
    part = __fadd_rn(part, __shfl_xor_sync(0xffffffffu, part, o));
  if(active)
    for(int p = j; p < len; p += G)
      sc[p] = __fdiv_rn(sc[p], part);
  __syncwarp();
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
  for(int i = 0; i < tiles; ++i) {
    const float4* src = advance(tiles + i);
    const int n = active ? min(SR, len - i * SR) : 0;
    const float* w = sc + i * SR;
    int u = 0;
    for(; u + 4 <= n; u += 4) {
      const float4 w4 = *reinterpret_cast<const float4*>(w + u);
      const float wu[4] = {w4.x, w4.y, w4.z, w4.w};
#pragma unroll
      for(int e = 0; e < 4; ++e) {
        const float4 vv = src[(u + e) * 32];
        acc.x = __fmaf_rn(wu[e], vv.x, acc.x);
        acc.y = __fmaf_rn(wu[e], vv.y, acc.y);
        acc.z = __fmaf_rn(wu[e], vv.z, acc.z);
        acc.w = __fmaf_rn(wu[e], vv.w, acc.w);
      }
    }
    for(; u < n; ++u) {
      const float4 vv = src[u * 32];
      acc.x = __fmaf_rn(w[u], vv.x, acc.x);
      acc.y = __fmaf_rn(w[u], vv.y, acc.y);
      acc.z = __fmaf_rn(w[u], vv.z, acc.z);
      acc.w = __fmaf_rn(w[u], vv.w, acc.w);
    }
  }
  unsigned m_abs = 0u;
  if(live) {
    reinterpret_cast<float4*>(out + static_cast<size_t>(r) * dim)[slice] = acc;
    m_abs = max4u(0u, acc);
  }
  if(absmax_slot) {   // one atomic per block: all go to one address
    m_abs = __reduce_max_sync(0xffffffffu, m_abs);
    unsigned* red = reinterpret_cast<unsigned*>(scores);   // (used up)
    __syncthreads();
    if(lane == 0)
      red[warp] = m_abs;
    __syncthreads();
    if(warp == 0) {
      m_abs = __reduce_max_sync(0xffffffffu, lane < warps ? red[lane] : 0u);
      if(lane == 0 && m_abs != 0u)
        atomicMax(absmax_slot, m_abs);
    }
  }
  trace_stamp(tb, kTrAttentionCross, 2);
  trace_stamp(th.last, kTrAttentionCross, 3);
}

// Decoder self-attention for all hypotheses of a sentence together, as attention_cross_kernel does it: a warp per hypothesis, 32
// consecutive four-element slices per block, rows through the ring.  The rows are the sentence's distinct history rows (history_list), in
// the order of their positions; a warp takes from every stage of the ring the positions whose row lies in it.  attention1_kernel reads
// every ancestor row once per hypothesis, which L2 bounds: 512 rows x 24 positions x 8 KB are 100 MB a launch.
// Two to six hypotheses (one shares nothing; attention_hist_supported).  Whole mini-batches: transformer-base, 64 x beam 4 36.8 -> 35.1 ms; what
// transformer-big gains at 128 x beam 4, alone and four searches at once, is within the spread of runs.
template <int DH>
__global__ void __launch_bounds__(kMaxHistBeams * 32)
attention_hist_kernel(const float* __restrict__ q, const float* __restrict__ k, const float* __restrict__ v, int heads, int len, int batch, float scale,
                      float* __restrict__ out, unsigned* absmax_slot, const HistLists lists) {
  const TraceHandles th = trace_open_all();
  unsigned long long* const tb = th.first;
  constexpr int G = DH / 4, U = kCrossU, SR = kCrossRows;
  constexpr int kWarpHeads = 32 / G;
  extern __shared__ float4 hist_smem[];   // [stages][SR][32] rows, per warp and head [len4] scores, [beams * len] list, [beams][len] places
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, beams = blockDim.x >> 5;
  const int j = lane % G;
  const int dim = heads * DH;
  const int slice = blockIdx.y * 32 + lane;
  const bool active = slice < dim / 4;
  const int b = blockIdx.x, r = warp * batch + b;
  const int len4 = (len + 3) & ~3;
  float* scores = reinterpret_cast<float*>(hist_smem + kCrossStages * SR * 32);
  float* sc = scores + (warp * kWarpHeads + lane / G) * len4;
  int* list = reinterpret_cast<int*>(scores + beams * kWarpHeads * len4);
  int* which = list + beams * len + warp * len;
  pdl_wait_and_launch();
  trace_stamp_start(th, kTrAttentionHist);
  const float4 qv = active ? __ldg(reinterpret_cast<const float4*>(q + static_cast<size_t>(r) * dim) + slice) : make_float4(0.f, 0.f, 0.f, 0.f);
  const int n_rows = lists.count[b];
  {
    const size_t share = static_cast<size_t>(b) * beams * len;
    for(int i = threadIdx.x; i < beams * len; i += blockDim.x) {
      list[i] = lists.list[share + i];   // (places past n_rows are not used)
      list[beams * len + i] = lists.which[share + i];
    }
  }
  __syncthreads();
  const int tiles = (n_rows + SR - 1) / SR;
  auto fetch = [&](int i) {
    if(active && i < 2 * tiles) {
      const int i0 = (i < tiles ? i : i - tiles) * SR;
      const float* src = (i < tiles ? k : v) + 4 * slice;
      float4* dst = hist_smem + (i % kCrossStages) * (SR * 32) + lane;
      const int n = min(SR, n_rows - i0);
      for(int u = warp; u < n; u += beams)
        copy16_async(dst + u * 32, src + static_cast<size_t>(list[i0 + u]) * dim);
    }
    copy_commit();
  };
  auto advance = [&](int i) {
    copy_wait<kCrossStages - 2>();
    __syncthreads();
    fetch(i + kCrossStages - 1);
    return hist_smem + (i % kCrossStages) * (SR * 32) + lane;
  };
#pragma unroll
  for(int i = 0; i < kCrossStages - 1; ++i)
    fetch(i);
  constexpr int kPlainMask = (U >= G) ? 0 : (G / U) - 1;
  // positions from p on whose rows lie in stage i (at most SR: every position has a row of its own)
  auto in_stage = [&](int p, int i) { return __popc(__ballot_sync(0xffffffffu, p + lane < len && which[min(p + lane, len - 1)] < (i + 1) * SR)); };
  int p = 0;
  for(int i = 0; i < tiles; ++i) {
    const float4* src = advance(i) - static_cast<ptrdiff_t>(i) * SR * 32;
    const int n = in_stage(p, i);
#pragma unroll 1
    for(int h = 0; h < n; h += U) {
      float d[U];
#pragma unroll
      for(int u = 0; u < U; ++u) {
        const float4 kk = src[which[p + min(h + u, n - 1)] * 32];
        d[u] = __fmul_rn(qv.x, kk.x);
        d[u] = __fmaf_rn(qv.y, kk.y, d[u]);
        d[u] = __fmaf_rn(qv.z, kk.z, d[u]);
        d[u] = __fmaf_rn(qv.w, kk.w, d[u]);
      }
      const int pos = h + head_butterfly<G, U>(d, j);
      if(active && (j & kPlainMask) == 0 && pos < n)
        sc[p + pos] = __fmul_rn(d[0], scale);
    }
    p += n;
  }
  __syncwarp();
  float mx = -FLT_MAX, part = 0.f;
  if(active)
    for(int e = j; e < len; e += G)
      mx = fmaxf(mx, sc[e]);
#pragma unroll
  for(int o = G / 2; o > 0; o >>= 1)
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  if(active)
    for(int e = j; e < len; e += G) {
      const float x = det_expf(__fadd_rn(sc[e], -mx));
      sc[e] = x;
      part = __fadd_rn(part, x);
    }
#pragma unroll
  for(int o = G / 2; o > 0; o >>= 1)
    part = __fadd_rn(part, __shfl_xor_sync(0xffffffffu, part, o));
  if(active)
    for(int e = j; e < len; e += G)
      sc[e] = __fdiv_rn(sc[e], part);
  __syncwarp();
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
  p = 0;
  for(int i = 0; i < tiles; ++i) {
    const float4* src = advance(tiles + i) - static_cast<ptrdiff_t>(i) * SR * 32;
    const int n = in_stage(p, i);
    if(active) {
#pragma unroll 4
      for(int e = p; e < p + n; ++e) {
        const float w = sc[e];
        const float4 vv = src[which[e] * 32];
        acc.x = __fmaf_rn(w, vv.x, acc.x);
        acc.y = __fmaf_rn(w, vv.y, acc.y);
        acc.z = __fmaf_rn(w, vv.z, acc.z);
        acc.w = __fmaf_rn(w, vv.w, acc.w);
      }
    }
    p += n;
  }
  unsigned m_abs = 0u;
  if(active) {
    reinterpret_cast<float4*>(out + static_cast<size_t>(r) * dim)[slice] = acc;
    m_abs = max4u(0u, acc);
  }
  if(absmax_slot) {   // one atomic per block: all go to one address
    m_abs = __reduce_max_sync(0xffffffffu, m_abs);
    unsigned* red = reinterpret_cast<unsigned*>(scores);   // (used up)
    __syncthreads();
    if(lane == 0)
      red[warp] = m_abs;
    __syncthreads();
    if(warp == 0) {
      m_abs = __reduce_max_sync(0xffffffffu, lane < beams ? red[lane] : 0u);
      if(lane == 0 && m_abs != 0u)
        atomicMax(absmax_slot, m_abs);
    }
  }
  trace_stamp(tb, kTrAttentionHist, 2);
  trace_stamp(th.last, kTrAttentionHist, 3);
}

// Encoder self-attention (mode 2): block (b, h, i) has 32 query positions of one (sentence, head), a lane each, and its keys and values in shared memory.
// attention1_kernel re-reads every key/value row once per query; here they cross L2 -> SM once per 32 queries.  The eight warps share the key positions out
// (position p is warp p % 8's: its scores, exponentials and the interleaved partial sums they belong to) and then the elements of the output.
// The arithmetic per (row, head) is that of attention1_kernel restated for one lane: the G = DH/4 four-element partial dot products are combined in the
// butterfly's order (pairs G/2 apart first), the softmax sum as G interleaved partial sums combined the same way,
// the output as a fused-multiply-add chain over the positions in ascending order.
// Bound by one warp's chain of instructions where blocks are few, by shared-memory reads (a broadcast of four floats feeds four multiply-adds) where they are many.
// With a thread per query position, one or two warps of a block at work on all key positions, before: a layer of transformer-big, 128 sentences of 31 words,
// 95 -> 43 us (47 with registers for two blocks per SM instead of three), of transformer-base, 64 of 38 words, 42 -> 27, of the student, one sentence 9 -> 3.7,
// 16 sentences 14 -> 4.6; student, 16 sentences, a mini-batch 3.14 -> 3.035 ms, one sentence 2.22 -> 2.135.
// Longer sentences, 16 heads of 64: 16 sentences of 64 words 42 -> 21, 100 words 53 -> 49, 128 words 113 -> 68, 200 words 319 -> 261; 64 of 64 words 123 -> 67, 100
// words 221 -> 190.  Beyond 200 words (64 floats a head; 264 of 32), which attention1_kernel had: 250 words, one sentence 89 -> 25, 16 511 -> 355; 290 words 104 -> 56
// and 679 -> 514.  Of 142 sizes from 1 x 16 to 128 x 64 and 16 x 330 none is slower.
template <int G>
__device__ __forceinline__ float butterfly_order_sum(float (&a)[G]) {
#pragma unroll
  for(int o = G / 2; o > 0; o >>= 1) {
#pragma unroll
    for(int j = 0; j < o; ++j)
      a[j] = __fadd_rn(a[j], a[j + o]);
  }
  return a[0];
}

constexpr int kEncWarps = 8, kEncRows = 32;
constexpr size_t attention_enc_smem(int dim_head, size_t len) {   // keys, values, scores, mask; queries; partial sums; maxima
  return sizeof(float) * (len * (2 * dim_head + kEncRows + 1) + kEncRows * (dim_head + 4) + kEncRows * (dim_head / 4) + kEncRows * kEncWarps + 4);
}

template <int DH>
__global__ void __launch_bounds__(kEncWarps * 32, DH == 64 ? 3 : 2)
attention_enc_kernel(const float* __restrict__ q, const float* __restrict__ k, const float* __restrict__ v,
                     const float* __restrict__ log_mask, int heads, int len, float scale, float* __restrict__ out,
                     unsigned* absmax_slot) {
  const TraceHandles th = trace_open_all();
  unsigned long long* const tb = th.first;
  pdl_wait_and_launch();
  trace_stamp_start(th, kTrAttentionEnc);
  extern __shared__ float4 enc_smem[];
  constexpr int G = DH / 4, W = kEncWarps, kQPitch = DH + 4, kOwn = DH / W;   // (a row of queries 4 floats longer: eight lanes' reads on different banks)
  static_assert(G % W == 0 && kOwn % 4 == 0, "");
  const int b = blockIdx.x, h = blockIdx.y, q0 = blockIdx.z * kEncRows;
  const int dim = heads * DH, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float* ks = reinterpret_cast<float*>(enc_smem);   // [len][DH]
  float* vs = ks + static_cast<size_t>(len) * DH;   // [len][DH]
  float* qs = vs + static_cast<size_t>(len) * DH;   // [32][DH + 4]
  float* parts = qs + kEncRows * kQPitch;           // [G][32]
  float* maxima = parts + G * kEncRows;             // [W][32]
  float* sc = maxima + W * kEncRows;                // [len][32] scores / probabilities
  float* ms = sc + static_cast<size_t>(len) * kEncRows;   // [len]
  const size_t row0 = static_cast<size_t>(b) * len;
  for(int i = threadIdx.x; i < len * G; i += W * 32) {
    const size_t off = (row0 + i / G) * dim + h * DH + 4 * (i % G);
    reinterpret_cast<float4*>(ks)[i] = __ldg(reinterpret_cast<const float4*>(k + off));
    reinterpret_cast<float4*>(vs)[i] = __ldg(reinterpret_cast<const float4*>(v + off));
  }
  for(int i = threadIdx.x; i < kEncRows * G; i += W * 32)   // (beyond the end the last query once more)
    *reinterpret_cast<float4*>(qs + (i / G) * kQPitch + 4 * (i % G)) =
        __ldg(reinterpret_cast<const float4*>(q + (row0 + min(q0 + i / G, len - 1)) * dim + h * DH + 4 * (i % G)));
  for(int i = threadIdx.x; i < len; i += W * 32)
    ms[i] = log_mask ? __ldg(log_mask + row0 + i) : 0.f;
  __syncthreads();
  float qv[DH];
#pragma unroll
  for(int c = 0; c < G; ++c) {
    const float4 t = *reinterpret_cast<const float4*>(qs + lane * kQPitch + 4 * c);
    qv[4 * c] = t.x; qv[4 * c + 1] = t.y; qv[4 * c + 2] = t.z; qv[4 * c + 3] = t.w;
  }
  float mx = -FLT_MAX;
  for(int p = warp; p < len; p += W) {
    const float4* kr = reinterpret_cast<const float4*>(ks + p * DH);
    float a[G];
#pragma unroll
    for(int j = 0; j < G; ++j) {
      const float4 t = kr[j];
      a[j] = __fmul_rn(qv[4 * j], t.x);
      a[j] = __fmaf_rn(qv[4 * j + 1], t.y, a[j]);
      a[j] = __fmaf_rn(qv[4 * j + 2], t.z, a[j]);
      a[j] = __fmaf_rn(qv[4 * j + 3], t.w, a[j]);
    }
    float sv = __fmul_rn(butterfly_order_sum<G>(a), scale);
    if(log_mask)
      sv = __fadd_rn(sv, ms[p]);
    sc[p * kEncRows + lane] = sv;
    mx = fmaxf(mx, sv);
  }
  maxima[warp * kEncRows + lane] = mx;
  __syncthreads();
#pragma unroll
  for(int w = 0; w < W; ++w)
    mx = fmaxf(mx, maxima[w * kEncRows + lane]);
#pragma unroll
  for(int j = 0; j < G; j += W) {   // partial sum j + warp: positions j + warp, j + warp + G, ...
    float part = 0.f;
    for(int p = j + warp; p < len; p += G) {
      const float e = det_expf(__fadd_rn(sc[p * kEncRows + lane], -mx));
      sc[p * kEncRows + lane] = e;
      part = __fadd_rn(part, e);
    }
    parts[(j + warp) * kEncRows + lane] = part;
  }
  __syncthreads();
  {
    float a[G];
#pragma unroll
    for(int j = 0; j < G; ++j)
      a[j] = parts[j * kEncRows + lane];
    const float total = butterfly_order_sum<G>(a);
    for(int p = warp; p < len; p += W)
      sc[p * kEncRows + lane] = __fdiv_rn(sc[p * kEncRows + lane], total);
  }
  __syncthreads();
  float acc[kOwn];
#pragma unroll
  for(int e = 0; e < kOwn; ++e)
    acc[e] = 0.f;
#pragma unroll 4
  for(int p = 0; p < len; ++p) {
    const float w = sc[p * kEncRows + lane];
    const float4* vr = reinterpret_cast<const float4*>(vs + p * DH + warp * kOwn);
#pragma unroll
    for(int c = 0; c < kOwn / 4; ++c) {
      const float4 t = vr[c];
      acc[4 * c] = __fmaf_rn(w, t.x, acc[4 * c]);
      acc[4 * c + 1] = __fmaf_rn(w, t.y, acc[4 * c + 1]);
      acc[4 * c + 2] = __fmaf_rn(w, t.z, acc[4 * c + 2]);
      acc[4 * c + 3] = __fmaf_rn(w, t.w, acc[4 * c + 3]);
    }
  }
  unsigned m_abs = 0u;
  if(q0 + lane < len) {
    float4* o4 = reinterpret_cast<float4*>(out + (row0 + q0 + lane) * dim + h * DH + warp * kOwn);
#pragma unroll
    for(int c = 0; c < kOwn / 4; ++c) {
      const float4 t = make_float4(acc[4 * c], acc[4 * c + 1], acc[4 * c + 2], acc[4 * c + 3]);
      o4[c] = t;
      m_abs = max4u(m_abs, t);
    }
  }
  if(absmax_slot) {   // one atomic per block: all go to one address
    m_abs = __reduce_max_sync(0xffffffffu, m_abs);
    unsigned* red = reinterpret_cast<unsigned*>(maxima);   // (used up)
    if(lane == 0)
      red[warp] = m_abs;
    __syncthreads();
    if(warp == 0) {
      m_abs = __reduce_max_sync(0xffffffffu, lane < W ? red[lane] : 0u);
      if(lane == 0 && m_abs != 0u)
        atomicMax(absmax_slot, m_abs);
    }
  }
  trace_stamp(tb, kTrAttentionEnc, 2);
  trace_stamp(th.last, kTrAttentionEnc, 3);
}

// ---- output layer: log-softmax + per-row top-k --------------------------------------------------
// Tree merge of the 256 per-thread sorted candidate lists in shared memory; the result is in list 0.
template <int K>
__device__ __forceinline__ void topk_block_merge(float* s_v, int* s_i) {
  for(int active = 128; active >= 1; active >>= 1) {
    if(threadIdx.x < active) {
      TopK a;
#pragma unroll
      for(int j = 0; j < K; ++j) {
        a.v[j] = s_v[threadIdx.x * K + j];
        a.i[j] = s_i[threadIdx.x * K + j];
      }
#pragma unroll
      for(int j = 0; j < K; ++j)
        topk_insert<K>(a, s_v[(threadIdx.x + active) * K + j], s_i[(threadIdx.x + active) * K + j]);
#pragma unroll
      for(int j = 0; j < K; ++j) {
        s_v[threadIdx.x * K + j] = a.v[j];
        s_i[threadIdx.x * K + j] = a.i[j];
      }
    }
    __syncthreads();
  }
}

// The end of a step, run by whichever block of the output layer's last kernel finishes a sentence's last row (an arrival counter per
// sentence, zeroed at the start of the step): the beam x k row candidates of sentence b (rows beam-major: row = j * batch + b)
// become its k best, sorted; on ties the smaller flattened key (beam, word) first.  A candidate's place is the number of valid
// candidates before it; places that stay empty get score -inf, beam 0, word 0.  Block 0 also remembers, per layer, the history
// abs-max the stored keys/values now belong to (prev_bits[l] = slots[first + l * stride]; stats: pairs unchanged, all pairs).
// In place of two launches, each of a launch's hand-over (6 us together in a transformer-base step).
// It also leaves the next step's control words where that step is launched already (StepEnd::next_ctrl).
// The sentence's candidates lie in c_v / c_i: beam * k <= kStepEndCandidates (both launchers refuse more; mi8d_step then merges the
// n-best lists with nbest_merge_kernel, which has no such limit).
__device__ __forceinline__ void finish_step(const StepEnd& e, int r, int k, int vocab, const float* cand_score, const int* cand_word, float* c_v,
                                            int* c_i, int* s_last) {
  if(blockIdx.x == 0 && static_cast<int>(threadIdx.x) < e.layers) {
    const unsigned now = e.slots[e.first + threadIdx.x * e.stride];
    if(e.prev_bits[threadIdx.x] == now)
      atomicAdd(e.stats, 1u);
    atomicAdd(e.stats + 1, 1u);
    e.prev_bits[threadIdx.x] = now;
  }
  if(e.arrivals == nullptr)
    return;
  const int b = r % e.batch;
  __syncthreads();   // the row's candidates are written
  if(e.beam > 1) {   // (a sentence's only row is its last)
    if(threadIdx.x == 0) {
      __threadfence();
      *s_last = atomicAdd(e.arrivals + b, 1u) == static_cast<unsigned>(e.beam - 1) ? 1 : 0;
      __threadfence();
    }
    __syncthreads();
    if(!*s_last)
      return;
  }
  if(threadIdx.x >= 32)
    return;
  const auto store_entry = [&](int place, float score, int from, int word, int key) {
    if(e.tagged != nullptr) {
      volatile unsigned long long* at = e.tagged + 2 * (b * k + place);
      at[0] = static_cast<unsigned long long>(e.tag) << 32 | __float_as_uint(score);
      at[1] = static_cast<unsigned long long>(e.tag) << 32 | static_cast<unsigned>(key);
    } else {
      e.out_score[b * k + place] = score;
      e.out_beam[b * k + place] = from;
      e.out_word[b * k + place] = word;
    }
  };
  const int n = e.beam * k;
  int valid = 0;
  for(int c0 = 0; c0 < n; c0 += 32) {
    const int c = c0 + threadIdx.x;
    bool ok = false;
    if(c < n) {
      const int row = (c / k) * e.batch + b;
      const float v = __ldcg(cand_score + row * k + c % k);
      // not -inf: a dummy hypothesis; not a filler, neither of a row with fewer than k entries nor of one without a number (its
      // log-sum-exp is one, and would lift the filler's score)
      const int word = __ldcg(cand_word + row * k + c % k);
      ok = v > -FLT_MAX && static_cast<unsigned>(word) < static_cast<unsigned>(vocab);
      c_v[c] = ok ? v : -FLT_MAX;
      c_i[c] = ok ? (c / k) * vocab + word : 0x7fffffff;
    }
    valid += __popc(__ballot_sync(0xffffffffu, ok));
  }
  __syncwarp();
  for(int c = threadIdx.x; c < n; c += 32) {
    const float v = c_v[c];
    const int key = c_i[c];
    if(v > -FLT_MAX) {
      int place = 0;
      for(int o = 0; o < n; ++o)
        place += (c_v[o] > -FLT_MAX && better(c_v[o], c_i[o], v, key)) ? 1 : 0;
      if(place < k) {
        const int from = key / vocab, word = key % vocab;
        store_entry(place, v, from, word, key);
        if(e.next_ctrl != nullptr && place < e.hyps[b]) {
          int* next = e.next_ctrl + place * e.batch + b;
          next[0] = from * e.batch + b;
          next[k * e.batch] = word;
          next[2 * k * e.batch] = __float_as_int(v);
          if(word == e.eos)
            *e.next_stop = 1u;
        }
      }
    }
  }
  for(int c = valid + threadIdx.x; c < k; c += 32) {
    store_entry(c, -INFINITY, 0, 0, 0);
  }
  if(e.next_ctrl != nullptr) {
    const int alive = e.hyps[b];
    for(int c = alive + threadIdx.x; c < k; c += 32) {   // (no hypothesis: end of sentence and score -inf)
      int* next = e.next_ctrl + c * e.batch + b;
      next[0] = 0;
      next[k * e.batch] = e.eos;
      next[2 * k * e.batch] = __float_as_int(-INFINITY);
    }
    if(threadIdx.x == 0) {
      e.next_ctrl[3 * k * e.batch + b] = b;
      if(valid < alive)
        *e.next_stop = 1u;
    }
  }
}

// mx + log(sum of the nb terms, added in ascending order).
__device__ __forceinline__ float lse_of_terms(const float* terms, int nb, float mx) {
  float total = 0.f;
#pragma unroll 16
  for(int b = 0; b < nb; ++b)   // (unrolled: the loads run ahead of the chain of additions)
    total = __fadd_rn(total, terms[b]);
  return __fadd_rn(mx, det_logf(total));
}

// Combines the per-block pairs (m_b, s_b) of one row, held in shared memory, into the row's log-sum-exp:
// M = max_b m_b;  S = sum over b ascending of s_b * exp(m_b - M), product and sum rounded separately;
// lse = M + log(S).  bm/bs: nb entries each; red: 33 floats.  Every thread returns the same value.
__device__ __forceinline__ float lse_from_blocks(const float* bm, float* bs, int nb, float* red) {
  float mx = -FLT_MAX;
  for(int b = threadIdx.x; b < nb; b += blockDim.x)
    mx = fmaxf(mx, bm[b]);
  for(int o = 16; o > 0; o >>= 1)
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  __syncthreads();
  if((threadIdx.x & 31) == 0)
    red[threadIdx.x >> 5] = mx;
  __syncthreads();
  mx = red[0];
  for(int w = 1; w < static_cast<int>(blockDim.x >> 5); ++w)
    mx = fmaxf(mx, red[w]);
  for(int b = threadIdx.x; b < nb; b += blockDim.x)
    bs[b] = __fmul_rn(bs[b], det_expf(__fadd_rn(bm[b], -mx)));
  __syncthreads();
  if(threadIdx.x == 0)
    red[32] = lse_of_terms(bs, nb, mx);
  __syncthreads();
  return red[32];
}

constexpr size_t kLseBlockBytes = 32 * 1024;   // the blocks' maxima and sums of the widest row that is taken
__host__ __device__ constexpr size_t lse_staged_floats(int threads, bool from_blocks) { return from_blocks ? 0 : static_cast<size_t>(threads) * 32; }

__device__ __forceinline__ float warp_max(float v) {   // (no NaN)
  float m;
  asm volatile("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(m) : "f"(v));
  return m;
}

// One block per row: cand_score[r][j] = (j-th largest logit - logsumexp(row)) + prev_score[r], cand_word[r][j].
// The log-sum-exp is defined over blocks of 128 consecutive entries (the unit the output GEMM's write-back
// owns): per block its maximum m_b and s_b = sum of det_expf(x - m_b) with the entries added one after the
// other in ascending order; the blocks are combined as lse_from_blocks does it.
//
// Bound by instruction issue (about 20 per logit, most of them the exponential), so the work per logit is kept small:
//   * Four neighbouring lanes share a block of 128 entries, 32 consecutive ones each, held in registers from the one
//     read of the row on.  The ordered sum runs through the four lanes in turn: in round q every lane extends the running
//     sum by its own entries and the result of lane q is the one that counts.
//   * A warp copies the 1024 entries of its next eight blocks to shared memory as whole lines (16 bytes a lane, or a word each where the
//     rows are not 16-byte aligned) while it works on the last ones.  A lane reads its 32 entries from there in units of 16 bytes,
//     unit u of lane l stored at u ^ (l & 7), without bank conflicts in either direction.
//     Against lanes that read their own 128 bytes from L2: 512 rows of 32000 back to back 30.4 us to 29.6, 768 rows 49.2 to 43.2; 512
//     rows of 32001, whose words came one by one, 78.8 us to 36.1.
//   * No candidate lists while scanning.  The k best entries lie in the k blocks with the best (maximum, then smaller
//     index): each of those blocks has an entry that precedes every entry of any other block.  So the k blocks are picked
//     from the block maxima, their entries that reach the k-th maximum are collected, and an entry's place in the
//     output is the number of collected entries before it.
// 512 rows of 32000 logits with a list of k per thread and a block of 128 per lane: 55.6 us back to back and 42.6 us inside a
// decoder step (logits in L2); 34.0 and 24.7 us as described, 26.9 back to back with the block sizes below.
// kThreads: 1024 (one pass over 32000 logits, one block per SM) while every row has an SM to itself, 512 (two blocks per SM) up to two
// rows per SM, 256 (four) beyond, registers held to 64 so that they fit: 256 rows 29.1 us with 256 threads, 18.0 with 512.
// After the scan no warp waits for the block's maximum (each takes it from the warps' maxima), one warp picks the blocks with two warp
// reductions a pick while another walks the chain of additions.  Back to back, against the maximum by two block-wide waits and picks by
// shuffles: rows of 32000: one 14.0 us to 10.8, 148 14.8 to 11.7, 296 20.7 to 17.6, 512 29.7 to 26.6, 768 43.2 to 37.0.  (That warp
// collecting the picked blocks' entries as well, while the sum runs, instead of all warps behind it: 512 rows 31.1 us.)
// kFromBlocks: the blocks' maxima and sums were left by the output layer's write-back (few rows); no scan.
template <int kThreads, bool kFromBlocks = false>
__global__ void __launch_bounds__(kThreads, 1024 / kThreads)
lse_topk_kernel(const float* __restrict__ logits, int vocab, int k, const float* __restrict__ prev_scores, float* cand_score, int* cand_word,
                const StepEnd end, const float* __restrict__ block_max, const float* __restrict__ block_sum) {
  const TraceHandles th = trace_open_all();
  unsigned long long* const tb = th.first;
  pdl_wait_and_launch();
  if(end.stop != nullptr && *end.stop != 0u)
    return;
  trace_stamp_start(th, kTrLseTopk);
  extern __shared__ __align__(16) float lse_smem[];   // [kThreads / 32][1024] staged entries (none from blocks), [nb] block maxima, [nb] block sums
  static_assert(kStepEndCandidates <= kMaxK * 128, "finish_step reuses these arrays");
  __shared__ float c_v[kMaxK * 128];      // collected candidates
  __shared__ int c_i[kMaxK * 128];
  __shared__ float red[33];
  __shared__ int pick[kMaxK];
  __shared__ int n_cand;
  __shared__ int s_last;
  __shared__ float s_floor;
  const int r = blockIdx.x;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const float* row = logits + static_cast<size_t>(r) * vocab;
  const int nb = (vocab + 127) / 128;
  float most = -FLT_MAX;   // of the blocks' maxima that this lane has seen
  float* bm = lse_smem + lse_staged_floats(kThreads, kFromBlocks);
  float* bs = bm + nb;
  const bool vec = (vocab & 3) == 0 && (reinterpret_cast<uintptr_t>(logits) & 15u) == 0;
  if(threadIdx.x == 0)
    n_cand = 0;
  if(kFromBlocks) {
    for(int b = threadIdx.x; b < nb; b += kThreads) {
      bm[b] = __ldg(block_max + static_cast<size_t>(r) * nb + b);
      most = fmaxf(most, bm[b]);
      bs[b] = __ldg(block_sum + static_cast<size_t>(r) * nb + b);
    }
  }
  float* const staged = lse_smem + warp * 1024;
  auto stage = [&](int b0) {
    const int left = vocab - b0 * 128;
    const float* src = row + static_cast<size_t>(b0) * 128;
    if(left > 0 && vec) {
#pragma unroll
      for(int j = 0; j < 8; ++j) {
        const int owner = 4 * j + (lane >> 3);   // the lane whose entries these are
        float* dst = staged + owner * 32 + (((lane & 7) ^ (owner & 7)) << 2);
        const int e = 128 * j + 4 * lane;
        if(e < left)
          copy16_async(dst, src + e);
        else
          *reinterpret_cast<float4*>(dst) = make_float4(-FLT_MAX, -FLT_MAX, -FLT_MAX, -FLT_MAX);
      }
    } else if(left > 0) {
#pragma unroll 8
      for(int owner = 0; owner < 32; ++owner) {
        float* dst = staged + owner * 32 + (((lane >> 2) ^ (owner & 7)) << 2) + (lane & 3);
        const int e = 32 * owner + lane;
        if(e < left)
          copy4_async(dst, src + e);
        else
          *dst = -FLT_MAX;
      }
    }
    copy_commit();
  };
  if(!kFromBlocks)
    stage(warp * 8);
  for(int b0 = warp * 8; !kFromBlocks && b0 < nb; b0 += kThreads / 4) {
    const int b = b0 + (lane >> 2);
    const int lo = b * 128 + (lane & 3) * 32;
    const int cnt = b < nb ? max(0, min(32, vocab - lo)) : 0;   // this lane's entries that exist
    float x[32];
    copy_wait<0>();
    __syncwarp();
#pragma unroll
    for(int j = 0; j < 8; ++j) {
      const float4 q = *reinterpret_cast<const float4*>(staged + lane * 32 + ((j ^ (lane & 7)) << 2));
      x[4 * j] = q.x; x[4 * j + 1] = q.y; x[4 * j + 2] = q.z; x[4 * j + 3] = q.w;
    }
    __syncwarp();
    stage(b0 + kThreads / 4);
    float m = -FLT_MAX;
#pragma unroll
    for(int j = 0; j < 32; ++j)
      m = fmaxf(m, x[j]);
    m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 1));
    m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 2));
    most = fmaxf(most, m);
    if(cnt == 32) {
#pragma unroll
      for(int j = 0; j < 32; ++j)
        x[j] = det_expf_nonpos(__fadd_rn(x[j], -m));
    } else {
#pragma unroll
      for(int j = 0; j < 32; ++j)   // adding 0 for entries that do not exist leaves the sum as it is
        x[j] = j < cnt ? det_expf_nonpos(__fadd_rn(x[j], -m)) : 0.f;
    }
    float sum = 0.f;
#pragma unroll
    for(int q = 0; q < 4; ++q) {
      float t = sum;
#pragma unroll
      for(int j = 0; j < 32; ++j)
        t = __fadd_rn(t, x[j]);
      sum = __shfl_sync(0xffffffffu, t, (lane & 28) | q);
    }
    if((lane & 3) == 0 && b < nb) {
      bm[b] = m;
      bs[b] = sum;
    }
  }
  most = warp_max(most);
  if(lane == 0)
    red[warp] = most;
  __syncthreads();
  if(warp != 1) {
    // Every warp but one: the blocks' terms of the sum; warp 0 then adds them up.
    const float mx = warp_max(lane < kThreads / 32 ? red[lane] : -FLT_MAX);
    for(int b = warp == 0 ? lane : threadIdx.x - 32; b < nb; b += kThreads - 32)
      bs[b] = __fmul_rn(bs[b], det_expf(__fadd_rn(bm[b], -mx)));
    if(warp == 0) {
      asm volatile("bar.sync 1, %0;" ::"n"(kThreads - 32) : "memory");
      if(lane == 0)
        red[32] = lse_of_terms(bs, nb, mx);
    } else {
      asm volatile("bar.arrive 1, %0;" ::"n"(kThreads - 32) : "memory");
    }
  } else {
    // Warp 1 meanwhile: the k blocks with the best maxima, k rounds, each picks the best block that follows the last pick; a lane keeps
    // the best of its own blocks.
    float v, last_v = FLT_MAX;
    int i, last_i = -1;
    auto next_own = [&]() {
      v = -FLT_MAX;
      i = 0x7fffffff;
      for(int b = lane; b < nb; b += 32) {
        const float bv = bm[b];
        if((last_i < 0 || better(last_v, last_i, bv, b)) && better(bv, b, v, i)) {
          v = bv;
          i = b;
        }
      }
    };
    next_own();
    for(int j = 0; j < k; ++j) {
      last_v = warp_max(v);
      last_i = __reduce_min_sync(0xffffffffu, v == last_v ? i : 0x7fffffff);
      if(lane == 0)
        pick[j] = last_i;   // 0x7fffffff: there are fewer than k blocks
      if(i == last_i && i != 0x7fffffff)
        next_own();
    }
    if(lane == 0)
      s_floor = last_v;
  }
  __syncthreads();
  const float lse = red[32];
  const float floor_v = s_floor;
  // Without k maxima above the lowest finite value the argument above does not hold (a block without a single number shares that
  // maximum): then the k best are searched for one by one.
  const bool by_pick = floor_v > -FLT_MAX || nb <= k;
  if(by_pick) {
    for(int c = threadIdx.x; c < k * 128; c += kThreads) {
      const int b = pick[c >> 7];
      if(b < nb) {
        const int i = b * 128 + (c & 127);
        if(i < vocab) {
          const float v = __ldg(row + i);
          if(v >= floor_v) {
            const int at = atomicAdd(&n_cand, 1);
            c_v[at] = v;
            c_i[at] = i;
          }
        }
      }
    }
  }
  __syncthreads();
  const float ps = prev_scores ? prev_scores[r] : 0.f;
  if(by_pick) {
    const int n = n_cand;
    for(int c = threadIdx.x; c < n; c += kThreads) {
      const float v = c_v[c];
      const int i = c_i[c];
      int place = 0;
      for(int o = 0; o < n; ++o)
        place += better(c_v[o], c_i[o], v, i) ? 1 : 0;
      if(place < k) {
        cand_score[r * k + place] = __fadd_rn(__fadd_rn(v, -lse), ps);
        cand_word[r * k + place] = i;
      }
    }
    for(int c = n + threadIdx.x; c < k; c += kThreads) {
      cand_score[r * k + c] = __fadd_rn(__fadd_rn(-FLT_MAX, -lse), ps);
      cand_word[r * k + c] = 0x7fffffff;
    }
  } else if(warp == 0) {
    float last_v = 0.f;
    int last_i = 0;
    for(int j = 0; j < k; ++j) {
      float v = -FLT_MAX;
      int i = 0x7fffffff;
      for(int e = lane; e < vocab; e += 32) {
        const float ev = __ldg(row + e);
        if((j == 0 || better(last_v, last_i, ev, e)) && better(ev, e, v, i)) {
          v = ev;
          i = e;
        }
      }
#pragma unroll
      for(int o = 16; o > 0; o >>= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, v, o);
        const int oi = __shfl_xor_sync(0xffffffffu, i, o);
        if(better(ov, oi, v, i)) {
          v = ov;
          i = oi;
        }
      }
      last_v = v;
      last_i = i;
      if(lane == 0) {
        cand_score[r * k + j] = __fadd_rn(__fadd_rn(v, -lse), ps);
        cand_word[r * k + j] = i;
      }
    }
  }
  __syncthreads();   // (c_v and c_i are reused)
  finish_step(end, r, k, vocab, cand_score, cand_word, c_v, c_i, &s_last);
  trace_stamp(tb, kTrLseTopk, 2);
  trace_stamp(th.last, kTrLseTopk, 3);
}

// Second half of the fused output layer: the GEMM's write-back left, per (row, block of 128 vocabulary entries),
// the block maximum, the block's sum of exponentials and its KT best entries; one block per row combines them
// into the row's log-sum-exp (lse_from_blocks) and its k best entries overall, exactly what lse_topk_kernel
// computes from materialised logits.
template <int KT>
__global__ void __launch_bounds__(256)
lse_merge_kernel(const float* __restrict__ blk_max, const float* __restrict__ blk_sum, const float* __restrict__ blk_topv,
                 const int* __restrict__ blk_topi, int nb, int k, const float* __restrict__ prev_scores, float* cand_score, int* cand_word, int vocab,
                 const StepEnd end) {
  const TraceHandles th = trace_open_all();
  unsigned long long* const tb = th.first;
  pdl_wait_and_launch();
  trace_stamp_start(th, kTrLseMerge);
  static_assert(kStepEndCandidates <= 256 * KT, "finish_step reuses these arrays");
  extern __shared__ float lse_blocks[];
  __shared__ float s_v[256 * KT];
  __shared__ int s_i[256 * KT];
  __shared__ float red[33];
  __shared__ int s_last;
  const int r = blockIdx.x;
  float* bm = lse_blocks;
  float* bs = lse_blocks + nb;
  TopK t;
#pragma unroll
  for(int j = 0; j < KT; ++j) {
    t.v[j] = -FLT_MAX;
    t.i[j] = 0x7fffffff;
  }
  for(int b = threadIdx.x; b < nb; b += 256) {
    const size_t slot = static_cast<size_t>(r) * nb + b;
    bm[b] = blk_max[slot];
    bs[b] = blk_sum[slot];
#pragma unroll
    for(int j = 0; j < KT; ++j)
      topk_insert<KT>(t, blk_topv[slot * KT + j], blk_topi[slot * KT + j]);
  }
#pragma unroll
  for(int j = 0; j < KT; ++j) {
    s_v[threadIdx.x * KT + j] = t.v[j];
    s_i[threadIdx.x * KT + j] = t.i[j];
  }
  __syncthreads();
  const float lse = lse_from_blocks(bm, bs, nb, red);
  topk_block_merge<KT>(s_v, s_i);
  if(threadIdx.x < k) {
    const float ps = prev_scores ? prev_scores[r] : 0.f;
    cand_score[r * k + threadIdx.x] = __fadd_rn(__fadd_rn(s_v[threadIdx.x], -lse), ps);
    cand_word[r * k + threadIdx.x] = s_i[threadIdx.x];
  }
  __syncthreads();   // (s_v and s_i are reused)
  finish_step(end, r, k, vocab, cand_score, cand_word, s_v, s_i, &s_last);
  trace_stamp(tb, kTrLseMerge, 2);
  trace_stamp(th.last, kTrLseMerge, 3);
}

// Per sentence b: merge the beam x K row candidates (rows beam-major: row = j * batch + b) into the
// K best, sorted; key order on ties = (beam j, rank) ascending, i.e. smaller flattened key first.
// out_score[b][n], out_beam[b][n], out_word[b][n].
template <int K>
__global__ void nbest_merge_kernel(const float* __restrict__ cand_score, const int* __restrict__ cand_word, int beam, int batch,
                                   int vocab, float* __restrict__ out_score, int* __restrict__ out_beam, int* __restrict__ out_word) {
  const TraceHandles th = trace_open_all();
  unsigned long long* const tb = th.first;
  pdl_wait_and_launch();
  trace_stamp_start(th, kTrNbest);
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if(b >= batch) {
    trace_stamp(tb, kTrNbest, 2);
    trace_stamp(th.last, kTrNbest, 3);
    return;
  }
  TopK t;
#pragma unroll
  for(int j = 0; j < K; ++j) {
    t.v[j] = -FLT_MAX;
    t.i[j] = 0x7fffffff;
  }
  for(int j = 0; j < beam; ++j) {
    const int row = j * batch + b;
    for(int c = 0; c < K; ++c) {
      const float s = cand_score[row * K + c];
      const int word = cand_word[row * K + c];
      if(static_cast<unsigned>(word) >= static_cast<unsigned>(vocab))   // (a filler)
        continue;
      const int key = j * vocab + word;  // the reference's flattened (beam, word) key
      // -inf candidates (dummy hypotheses) must stay behind every real one but keep a defined order
      topk_insert<K>(t, s == -INFINITY ? -FLT_MAX : s, key);
    }
  }
#pragma unroll
  for(int n = 0; n < K; ++n) {
    const bool valid = t.i[n] != 0x7fffffff && t.v[n] > -FLT_MAX;
    out_score[b * K + n] = valid ? t.v[n] : -INFINITY;
    out_beam[b * K + n] = valid ? t.i[n] / vocab : 0;
    out_word[b * K + n] = valid ? t.i[n] % vocab : 0;
  }
  trace_stamp(tb, kTrNbest, 2);
  trace_stamp(th.last, kTrNbest, 3);
}

// rows gather: out[i,:] = in[idx[i],:]  (16-byte copies when the row length allows it)
__global__ void gather_rows_kernel(const float* __restrict__ in, const int* __restrict__ idx, int dim, float* __restrict__ out) {
  const TraceHandles th = trace_open_all();
  unsigned long long* const tb = th.first;
  pdl_wait_and_launch();
  trace_stamp_start(th, kTrGather);
  const int r = blockIdx.x;
  const float* src = in + static_cast<size_t>(idx[r]) * dim;
  float* dst = out + static_cast<size_t>(r) * dim;
  if((dim & 3) == 0) {
    const float4* s4 = reinterpret_cast<const float4*>(src);
    float4* d4 = reinterpret_cast<float4*>(dst);
    for(int i = threadIdx.x; i < dim / 4; i += blockDim.x)
      d4[i] = __ldg(s4 + i);
  } else {
    for(int i = threadIdx.x; i < dim; i += blockDim.x)
      dst[i] = __ldg(src + i);
  }
  trace_stamp(tb, kTrGather, 2);
  trace_stamp(th.last, kTrGather, 3);
}

// SSRU cell (src/rnn/cells.h:1052-1066): c' = c[hyp] * sigmoid(f) + x * (1 - sigmoid(f)); h = relu(c').
// Writes the new cell state and y = LayerNorm(h + resid) * gamma + beta is done by add_layernorm on h.
__global__ void ssru_cell_kernel(const float* __restrict__ cell_old, const int* __restrict__ hyp, const float* __restrict__ xw,
                                 const float* __restrict__ f, int dim, float* __restrict__ cell_new, float* __restrict__ h_out) {
  const TraceHandles th = trace_open_all();
  unsigned long long* const tb = th.first;
  pdl_wait_and_launch();
  trace_stamp_start(th, kTrSsru);
  const int r = blockIdx.x;
  const float* c = cell_old + static_cast<size_t>(hyp ? hyp[r] : r) * dim;
  for(int i = threadIdx.x; i < dim; i += blockDim.x) {
    const size_t o = static_cast<size_t>(r) * dim + i;
    cell_new[o] = ssru_cell(c[i], xw[o], f[o], h_out + o);
  }
  trace_stamp(tb, kTrSsru, 2);
  trace_stamp(th.last, kTrSsru, 3);
}

int g_attention_block_heads = 8;   // heads one block of attention1_kernel serves (0 = all heads of the row)
int g_attention_unroll = 8;   // key/value rows a thread of attention1_kernel keeps in flight (8 or 16; 16 costs a block per SM and measured 7 % slower)

}  // namespace

MI8_DEFINE_TRACE_SETTER(trace_set_glue)
void set_attention_unroll(int u) { g_attention_unroll = u; }
void set_attention_block_heads(int h) { g_attention_block_heads = h; }

// ------------------------------------------------------------------------------------------------ launchers
int launch_embed(const float* wemb, const int* words, const float* pos, int pos_mod, float scale, int rows, int dim, float* out,
                 float* rowmax, unsigned* slot, cudaStream_t s) {
  if(rows <= 0 || dim <= 0 || dim % 4 != 0 || dim > kRowThreads * 4 * kMaxVec || out == nullptr || pos == nullptr)
    return MI8_ERR_BAD_ARG;
  launch_kernel(embed_kernel, dim3(rows), dim3(kRowThreads), 0, s, wemb, words, pos, pos_mod, scale, dim, out, rowmax, slot);
  count_launch();
  return check_launch();
}

int launch_step_begin(const int* host_ctrl, int* ctrl, int n_ctrl, unsigned* slots, int n_slots, cudaStream_t s) {
  launch_kernel(step_begin_kernel, dim3(1), dim3(1024), 0, s, host_ctrl, ctrl, n_ctrl, slots, n_slots);
  count_launch();
  return check_launch();
}

int launch_add_layernorm(const float* a, const float* resid, const float* gamma, const float* beta, float eps, int rows, int dim,
                         float* out, float* rowmax, unsigned* slot, cudaStream_t s, unsigned* slot2) {
  if(rows <= 0 || dim <= 0 || dim % 4 != 0 || dim > kRowThreads * 4 * kMaxVec || a == nullptr || out == nullptr)
    return MI8_ERR_BAD_ARG;
  launch_kernel(add_layernorm_kernel, dim3(rows), dim3(kRowThreads), 0, s, a, resid, gamma, beta, eps, dim, out, rowmax, slot, slot2);
  count_launch();
  return check_launch();
}

// One row per thread group and eight CTAs: 32 rows of 1024 floats, 64 of 512, 128 of 256.  More rows per group in turn were slower than the two
// launches (256 rows of 512, four each: 8.2 us against 1.8 + 2.2 + 1.6 of both kernels and the hand-over between them).
constexpr int kLnQuantCtas = 8;
bool add_layernorm_quant_supported(int rows, int dim) {
  return dim % 16 == 0 && dim <= 1024 && rows > 0 && rows <= kLnQuantCtas * (32 / ((dim / 4 + 31) / 32));
}

int launch_add_layernorm_quant(const float* a, const float* resid, const float* gamma, const float* beta, float eps, int rows, int dim, float* out,
                               int8_t* q, float* d_qm, cudaStream_t s, const float* cell_old, const int* hyp, const float* xw, const float* f,
                               float* cell_new) {
  if(!add_layernorm_quant_supported(rows, dim))
    return MI8_ERR_UNSUPPORTED;
  int* status = device_status_ptr();
  if(status == nullptr)
    return MI8_ERR_LAUNCH;
  SsruArgs cell;
  cell.cell_old = cell_old;
  cell.hyp = hyp;
  cell.xw = xw;
  cell.f = f;
  cell.cell_new = cell_new;
  const int group_warps = (dim / 4 + 31) / 32;
  if(rows <= 2)   // no other CTA to wait for
    launch_kernel(add_layernorm_quant_kernel<1>, dim3(1), dim3(32 * group_warps * rows), 0, s, a, cell, resid, gamma, beta, eps, rows, dim, group_warps,
                  out, q, d_qm, status);
  else
    launch_kernel(add_layernorm_quant_kernel<kLnQuantCtas>, dim3(kLnQuantCtas), dim3(32 * group_warps * ((rows + kLnQuantCtas - 1) / kLnQuantCtas)), 0, s,
                  a, cell, resid, gamma, beta, eps, rows, dim, group_warps, out, q, d_qm, status);
  count_launch();
  return check_launch();
}

int launch_quantize_slot(const float* x, size_t n, const unsigned* slot, int8_t* q, float* d_qm, cudaStream_t s) {
  if(x == nullptr || q == nullptr || slot == nullptr || d_qm == nullptr || n == 0)
    return MI8_ERR_BAD_ARG;
  if((reinterpret_cast<uintptr_t>(x) & 15u) || (reinterpret_cast<uintptr_t>(q) & 15u))
    return MI8_ERR_MISALIGNED;
  int* status = device_status_ptr();
  if(status == nullptr)
    return MI8_ERR_LAUNCH;
  size_t blocks = (n / 16 + 255) / 256;
  const size_t cap = static_cast<size_t>(sm_count()) * 8;
  blocks = blocks < 1 ? 1 : (blocks > cap ? cap : blocks);
  launch_kernel(quantize_slot_kernel, dim3(static_cast<int>(blocks)), dim3(256), 0, s, x, n, slot, q, d_qm, status);
  count_launch();
  return check_launch();
}

int launch_embed_ancestors(const float* wemb, const int* words, const float* pos, float scale, int dim, float* out, float* rowmax, unsigned* slot,
                           unsigned* slot2, const int* anc_old, int* anc_new, const int* hyp, int t, int rows, int stride, cudaStream_t s,
                           int hist_layers, const float* const* hist_rowmax, unsigned* const* hist_slot, const HistLists& lists) {
  if(lists.batch > 0 && (rows % lists.batch != 0 || rows / lists.batch > kMaxHistBeams || lists.list == nullptr || lists.which == nullptr ||
                         lists.count == nullptr))
    return MI8_ERR_BAD_ARG;
  if(rows <= 0 || dim <= 0 || dim % 4 != 0 || dim > kRowThreads * 4 * kMaxVec || out == nullptr || pos == nullptr)
    return MI8_ERR_BAD_ARG;
  if(hist_layers < 0 || hist_layers > kMaxHistLayers)
    return MI8_ERR_UNSUPPORTED;
  HistMaxArgs hist;
  hist.layers = hist_layers;
  for(int l = 0; l < kMaxHistLayers; ++l) {
    hist.rowmax[l] = l < hist_layers ? hist_rowmax[l] : nullptr;
    hist.slot[l] = l < hist_layers ? hist_slot[l] : nullptr;
  }
  const int n = (t + 1) * rows;
  launch_kernel(embed_ancestors_kernel, dim3(rows + lists.batch + (n + kRowThreads - 1) / kRowThreads), dim3(kRowThreads), 0, s, wemb, words, pos, scale, dim,
                out, rowmax, slot, slot2, anc_old, anc_new, hyp, t, rows, stride, hist, lists);
  count_launch();
  return check_launch();
}

int launch_quantize_dual(const float* x, size_t n, const unsigned* slot_x, int8_t* q, float* qm_x, const float* slabs, int slab_rows,
                         int steps, int rows_new, int dim, const unsigned* slot_h, const unsigned* prev_bits, int8_t* hq, float* qm_h,
                         cudaStream_t s) {
  if(x == nullptr || q == nullptr || slot_x == nullptr || qm_x == nullptr || slabs == nullptr || slot_h == nullptr || prev_bits == nullptr ||
     hq == nullptr || qm_h == nullptr || n == 0 || steps <= 0 || rows_new <= 0 || rows_new > slab_rows)
    return MI8_ERR_BAD_ARG;
  if(dim % 16 != 0 || n % 16 != 0 || (reinterpret_cast<uintptr_t>(x) & 15u) || (reinterpret_cast<uintptr_t>(q) & 15u))
    return MI8_ERR_MISALIGNED;
  int* status = device_status_ptr();
  if(status == nullptr)
    return MI8_ERR_LAUNCH;
  size_t bx = (n / 16 + 255) / 256;
  const size_t cap = static_cast<size_t>(sm_count()) * 4;
  bx = bx < 1 ? 1 : (bx > cap ? cap : bx);
  // history part: blocks for all slabs, up to what is resident at once (with an unchanged abs-max those of the newest slab work)
  const size_t hist = (static_cast<size_t>(steps) * rows_new * dim + 4095) / 4096, hcap = static_cast<size_t>(sm_count()) * 4;
  const int bh = static_cast<int>(hist < hcap ? hist : hcap);
  launch_kernel(quantize_dual_kernel, dim3(static_cast<unsigned>(bx) + bh), dim3(256), 0, s, x, n, slot_x, q, qm_x, status,
                static_cast<int>(bx), slabs, slab_rows, steps, rows_new, dim, slot_h, prev_bits, hq, qm_h);
  count_launch();
  return check_launch();
}

int launch_attention1(const float* q, const float* k, const float* v, const float* log_mask, int rows, int heads, int dim_head,
                      int len, int batch, int mode, float* out, unsigned* slot, cudaStream_t s, const int* anc, int anc_stride,
                      int kv_rows) {
  if(rows <= 0 || heads <= 0 || len <= 0)
    return MI8_ERR_BAD_ARG;
  if(mode < 0 || mode > 2)
    return MI8_ERR_BAD_ARG;
  const float scale = 1.0f / sqrtf(static_cast<float>(dim_head));
  const int dim = heads * dim_head;
  if(dim > 1024)
    return MI8_ERR_UNSUPPORTED;
  if(mode == 2 && batch > 0 && rows == batch * len && anc == nullptr && (dim_head == 64 || dim_head == 32)) {
    // encoder: keys/values of a (sentence, head) staged in shared memory
    const size_t esmem = attention_enc_smem(dim_head, len);
    if(esmem <= 200 * 1024) {
      static bool attr_set[64][2] = {};
      int dev = 0;
      cudaGetDevice(&dev);
      const int which = dim_head == 64 ? 0 : 1;
      if(dev >= 0 && dev < 64 && !attr_set[dev][which]) {
        cudaError_t e = which == 0 ? cudaFuncSetAttribute(attention_enc_kernel<64>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024)
                                   : cudaFuncSetAttribute(attention_enc_kernel<32>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
        if(e != cudaSuccess) {
          set_last_cuda_error(e);
          return MI8_ERR_LAUNCH;
        }
        attr_set[dev][which] = true;
      }
      const dim3 egrid(batch, heads, (len + kEncRows - 1) / kEncRows);
      if(which == 0)
        launch_kernel(attention_enc_kernel<64>, egrid, dim3(kEncWarps * 32), esmem, s, q, k, v, log_mask, heads, len, scale, out, slot);
      else
        launch_kernel(attention_enc_kernel<32>, egrid, dim3(kEncWarps * 32), esmem, s, q, k, v, log_mask, heads, len, scale, out, slot);
      count_launch();
      return check_launch();
    }
  }
  if(mode == 1 && batch > 0 && (dim_head == 64 || dim_head == 32)) {
    // the hypotheses of a sentence together; sentences so long that the scores leave no room for the ring within 48 KB go one
    // row at a time below
    const int beams = (rows + batch - 1) / batch;
    const int groups = (beams + kCrossMaxBeams - 1) / kCrossMaxBeams, warps = (beams + groups - 1) / groups;
    const int warp_heads = 128 / dim_head;
    const size_t xsmem = kCrossStages * kCrossRows * 32 * sizeof(float4) + static_cast<size_t>(warps) * warp_heads * ((len + 3) & ~3) * sizeof(float);
    if(xsmem <= 48 * 1024 && groups <= 65535) {
      const dim3 xgrid(batch, (heads + warp_heads - 1) / warp_heads, groups);
      if(dim_head == 64)
        launch_kernel(attention_cross_kernel<64>, xgrid, dim3(warps * 32), xsmem, s, q, k, v, log_mask, heads, len, rows, batch, scale, out, slot);
      else
        launch_kernel(attention_cross_kernel<32>, xgrid, dim3(warps * 32), xsmem, s, q, k, v, log_mask, heads, len, rows, batch, scale, out, slot);
      count_launch();
      return check_launch();
    }
  }
  // A block serves `hb` heads of one query row.  Splitting a row over several smaller blocks changes nothing in the
  // arithmetic (heads are independent) and lets the SMs share the rows out evenly: 512 rows of 256 threads are 3.46
  // blocks per SM - some SMs get four, the others three - while halves or quarters of rows balance to within a few per cent.
  const int G = dim_head / 4;
  int hb = heads;
  if(g_attention_block_heads > 0 && heads % g_attention_block_heads == 0 && (g_attention_block_heads * G) % 32 == 0)
    hb = g_attention_block_heads;
  const int threads = ((hb * G + 31) / 32) * 32;
  const dim3 agrid(rows, heads / hb);
  const size_t smem = (static_cast<size_t>(hb) + 1) * len * sizeof(float);
  if(smem > 48 * 1024)
    return MI8_ERR_UNSUPPORTED;
  const bool wide = g_attention_unroll >= 16;
  if(dim_head == 64 && wide)
    launch_kernel(attention1_kernel<64, 16>, agrid, dim3(threads), smem, s, q, k, v, log_mask, heads, len, rows, batch, mode, scale, out, slot, anc, anc_stride, kv_rows);
  else if(dim_head == 64)
    launch_kernel(attention1_kernel<64, 8>, agrid, dim3(threads), smem, s, q, k, v, log_mask, heads, len, rows, batch, mode, scale, out, slot, anc, anc_stride, kv_rows);
  else if(dim_head == 32 && wide)
    launch_kernel(attention1_kernel<32, 16>, agrid, dim3(threads), smem, s, q, k, v, log_mask, heads, len, rows, batch, mode, scale, out, slot, anc, anc_stride, kv_rows);
  else if(dim_head == 32)
    launch_kernel(attention1_kernel<32, 8>, agrid, dim3(threads), smem, s, q, k, v, log_mask, heads, len, rows, batch, mode, scale, out, slot, anc, anc_stride, kv_rows);
  else
    return MI8_ERR_UNSUPPORTED;
  count_launch();
  return check_launch();
}

namespace {
size_t attention_hist_smem(int beams, int dim_head, int len) {
  return kCrossStages * kCrossRows * 32 * sizeof(float4) +
         sizeof(float) * (static_cast<size_t>(beams) * (128 / dim_head) * ((len + 3) & ~3) + 2 * static_cast<size_t>(beams) * len);
}
}  // namespace
// Two to four hypotheses, five and six up to 32 sentences: a wider beam's hypotheses share less, and its warps wait for one another at every stage.
// Whole mini-batches, this kernel against attention1_kernel, in turn: transformer-base, beam 4, 4 to 64 sentences x 8 to 36 words 0 to -2 %; beam 6
// 4 x 36 -2.0 %, 16 x 36 -2.8 %, 32 x 30 -2.2 %, 48 x 30 -1.8 %, 64 x 24 +1.2 %; beam 7 8 x 30 +1.2 %, 16 x 30 -2.6 %; beam 8 4 x 30 +2.0 %,
// 8 x 30 +1.2 %, 64 x 8 +1.7 %; transformer-big, beam 5 64 x 30 +1.0 %; beam 6 16 x 36 -3.0 %, 32 x 30 -2.6 %, 48 x 30 +1.3 %, 64 x 24 +2.0 %; beam 8
// 8 x 30 +1.9 %, 32 x 24 +2.2 %.
bool attention_hist_supported(int beams, int sentences, int dim_head, int len) {
  return beams >= 2 && (beams <= kHistBeams || (beams <= kMaxHistBeams && sentences <= kMaxHistSentences)) && (dim_head == 64 || dim_head == 32) &&
         attention_hist_smem(beams, dim_head, len) <= 48 * 1024;
}
int launch_attention_hist(const float* q, const float* k, const float* v, int rows, int heads, int dim_head, int len, float* out, unsigned* slot,
                          cudaStream_t s, const HistLists& lists) {
  const int beams = lists.batch > 0 ? rows / lists.batch : 0;
  if(rows <= 0 || heads <= 0 || len <= 0 || beams * lists.batch != rows || !attention_hist_supported(beams, lists.batch, dim_head, len))
    return MI8_ERR_UNSUPPORTED;
  const float scale = 1.0f / sqrtf(static_cast<float>(dim_head));
  const int warp_heads = 128 / dim_head;
  const dim3 grid(lists.batch, (heads + warp_heads - 1) / warp_heads);
  const size_t smem = attention_hist_smem(beams, dim_head, len);
  if(dim_head == 64)
    launch_kernel(attention_hist_kernel<64>, grid, dim3(beams * 32), smem, s, q, k, v, heads, len, lists.batch, scale, out, slot, lists);
  else
    launch_kernel(attention_hist_kernel<32>, grid, dim3(beams * 32), smem, s, q, k, v, heads, len, lists.batch, scale, out, slot, lists);
  count_launch();
  return check_launch();
}

int launch_lse_topk(const float* logits, int rows, int vocab, int k, const float* prev_scores, float* cand_score, int* cand_word,
                    cudaStream_t s, const StepEnd& end, const float* block_max, const float* block_sum) {
  if(rows <= 0 || vocab <= 0 || k < 1 || k > kMaxK)
    return MI8_ERR_BAD_ARG;
  if(end.arrivals != nullptr && !step_end_fits(end.beam, k))
    return MI8_ERR_UNSUPPORTED;
  const size_t smem = 2 * static_cast<size_t>((vocab + 127) / 128) * sizeof(float);
  if(smem > kLseBlockBytes)
    return MI8_ERR_UNSUPPORTED;
  auto launch = [&](auto kernel, int which, int threads) -> int {
    static bool attr_set[64][4] = {};
    const size_t staged = lse_staged_floats(threads, which == 3) * sizeof(float);
    int dev = 0;
    cudaGetDevice(&dev);
    if(staged > 0 && (dev < 0 || dev >= 64 || !attr_set[dev][which])) {
      cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(staged + kLseBlockBytes));
      if(e != cudaSuccess) {
        set_last_cuda_error(e);
        return MI8_ERR_LAUNCH;
      }
      if(dev >= 0 && dev < 64)
        attr_set[dev][which] = true;
    }
    launch_kernel(kernel, dim3(rows), dim3(threads), staged + smem, s, logits, vocab, k, prev_scores, cand_score, cand_word, end, block_max, block_sum);
    count_launch();
    return check_launch();
  };
  if(block_max != nullptr)
    return launch(lse_topk_kernel<256, true>, 3, 256);
  if(rows <= sm_count())
    return launch(lse_topk_kernel<1024>, 2, 1024);
  if(rows <= 2 * sm_count())
    return launch(lse_topk_kernel<512>, 1, 512);
  return launch(lse_topk_kernel<256>, 0, 256);
}

int launch_lse_merge(const float* blk_max, const float* blk_sum, const float* blk_topv, const int* blk_topi, int rows, int vocab,
                     int k_top, int k, const float* prev_scores, float* cand_score, int* cand_word, cudaStream_t s, const StepEnd& end) {
  if(rows <= 0 || vocab <= 0 || k < 1 || k > k_top || (k_top != 4 && k_top != 8))
    return MI8_ERR_BAD_ARG;
  if(end.arrivals != nullptr && !step_end_fits(end.beam, k))
    return MI8_ERR_UNSUPPORTED;
  const int nb = (vocab + 127) / 128;
  const size_t smem = 2 * static_cast<size_t>(nb) * sizeof(float);
  if(smem > 32 * 1024)
    return MI8_ERR_UNSUPPORTED;
  if(k_top == 4)
    launch_kernel(lse_merge_kernel<4>, dim3(rows), dim3(256), smem, s, blk_max, blk_sum, blk_topv, blk_topi, nb, k, prev_scores, cand_score,
                  cand_word, vocab, end);
  else
    launch_kernel(lse_merge_kernel<8>, dim3(rows), dim3(256), smem, s, blk_max, blk_sum, blk_topv, blk_topi, nb, k, prev_scores, cand_score,
                  cand_word, vocab, end);
  count_launch();
  return check_launch();
}

int launch_nbest_merge(const float* cand_score, const int* cand_word, int beam, int batch, int vocab, int k, float* out_score,
                       int* out_beam, int* out_word, cudaStream_t s) {
  if(k < 1 || k > kMaxK || beam < 1 || batch < 1)
    return MI8_ERR_BAD_ARG;
  const int blocks = (batch + 127) / 128;
  switch(k) {
    case 1: launch_kernel(nbest_merge_kernel<1>, dim3(blocks), dim3(128), 0, s, cand_score, cand_word, beam, batch, vocab, out_score, out_beam, out_word); break;
    case 2: launch_kernel(nbest_merge_kernel<2>, dim3(blocks), dim3(128), 0, s, cand_score, cand_word, beam, batch, vocab, out_score, out_beam, out_word); break;
    case 3: launch_kernel(nbest_merge_kernel<3>, dim3(blocks), dim3(128), 0, s, cand_score, cand_word, beam, batch, vocab, out_score, out_beam, out_word); break;
    case 4: launch_kernel(nbest_merge_kernel<4>, dim3(blocks), dim3(128), 0, s, cand_score, cand_word, beam, batch, vocab, out_score, out_beam, out_word); break;
    case 5: launch_kernel(nbest_merge_kernel<5>, dim3(blocks), dim3(128), 0, s, cand_score, cand_word, beam, batch, vocab, out_score, out_beam, out_word); break;
    case 6: launch_kernel(nbest_merge_kernel<6>, dim3(blocks), dim3(128), 0, s, cand_score, cand_word, beam, batch, vocab, out_score, out_beam, out_word); break;
    case 7: launch_kernel(nbest_merge_kernel<7>, dim3(blocks), dim3(128), 0, s, cand_score, cand_word, beam, batch, vocab, out_score, out_beam, out_word); break;
    default: launch_kernel(nbest_merge_kernel<8>, dim3(blocks), dim3(128), 0, s, cand_score, cand_word, beam, batch, vocab, out_score, out_beam, out_word); break;
  }
  count_launch();
  return check_launch();
}

int launch_gather_rows(const float* in, const int* idx, int rows, int dim, float* out, cudaStream_t s) {
  if(rows <= 0 || dim <= 0)
    return MI8_ERR_BAD_ARG;
  launch_kernel(gather_rows_kernel, dim3(rows), dim3(128), 0, s, in, idx, dim, out);
  count_launch();
  return check_launch();
}

int launch_ssru_cell(const float* cell_old, const int* hyp, const float* xw, const float* f, int rows, int dim, float* cell_new,
                     float* h_out, cudaStream_t s) {
  launch_kernel(ssru_cell_kernel, dim3(rows), dim3(256), 0, s, cell_old, hyp, xw, f, dim, cell_new, h_out);
  count_launch();
  return check_launch();
}

}  // namespace mi8

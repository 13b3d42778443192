// The layers of an SSRU decoder step for few rows in one launch: embedding, and per layer the recurrent cell, cross-attention and the
// feed-forward block with their LayerNorms and quantisations (DecoderTransformer::step, src/models/transformer.h:713-896, with
// rnn::SSRU, src/rnn/cells.h:1052-1066, in the place of the self-attention).
//
// What bounds the step there is its chain, not its work: 24 launches of one to three microseconds of work each and two of hand-over, for
// one megabyte of weights a layer.  So ONE cluster of 16 CTAs runs the whole chain.  A CTA owns 1/16 of every weight matrix's columns; what
// the next affine needs of all of them - the rows' results, or their quantised values - is stored into the shared memory of every CTA
// (distributed shared memory) and a hardware cluster barrier takes the place of a launch boundary: six per layer.  LayerNorm and
// quantisation of the few rows are then done by every CTA for itself, which costs less than another exchange, and the abs-max of the whole
// tensor is at hand without one.
//   * Weights.  A CTA's share of all matrices is a stream of units of 16 weight rows x 128 bytes of K (one TMA box, 128-byte
//     swizzle).  Unit u belongs to warp u % 16; a warp keeps its next units in flight in shared memory, across phases and layers (weights do
//     not depend on anything), from the start of the launch on.  With few rows the student's whole decoder fits.
//   * Products.  mma.sync m16n8k32 with the weights as the 16-row operand: tcgen05 needs 128 weight rows per instruction, a CTA has 16 to 96
//     here.  A lane reads 16 consecutive bytes of K and feeds them to two MMAs; operand A and B take the same K for the same lane, so the
//     order inside a 128-byte block does not matter.  Chunks 2t + i (lane t of a quad) keep the eight lanes of a load phase on
//     different banks under the swizzle.  Integer sums are exact in any order: units add into shared memory with atomics.
//   * Floats.  Every operation and its order are those of the kernels of mi8_glue.cu, so the bits are too.
// Student decoder (two layers), whole mini-batches: one sentence 4.22 -> 2.82 ms, 16 sentences 5.55 -> 3.94 ms (the launch takes 35 and 45 us
// of a step where the separate ones took 88 and 95).  Eight CTAs instead of 16: 1 % slower.  Not bound by the weights (64 KB a layer and
// CTA, a microsecond) but by the latencies of its phases: about 1000 cycles per exchange, 1000 to 1500 per LayerNorm, 700 per quantisation.
#include <cfloat>

#include "mi8_internal.h"
#include "mi8_math.cuh"
#include "mi8_ptx.cuh"

namespace mi8 {
namespace {

constexpr int kWarps = 16;
constexpr int kThreads = kWarps * 32;
constexpr int kUnitRows = 16;
constexpr int kUnitBytes = kUnitRows * 128;
constexpr int kMaxRing = 8;        // units a warp keeps in flight
constexpr int kPhases = 5;         // affines per layer: W|Wf, Wq, Wo, W1, W2
constexpr int kMaxDynSmem = 225 * 1024;

enum Phase { kCell = 0, kQuery, kOut, kFfn1, kFfn2 };

__device__ __forceinline__ unsigned abs_bits(float v) { return __float_as_uint(v) & 0x7fffffffu; }
__device__ __forceinline__ unsigned max4u(unsigned m, const float4& v) {
  return max(max(max(m, abs_bits(v.x)), max(abs_bits(v.y), abs_bits(v.z))), abs_bits(v.w));
}
__device__ __forceinline__ unsigned pack4(const float4& v, float qm) {
  const int a = max(-127, min(127, __float2int_rn(__fmul_rn(v.x, qm))));
  const int b = max(-127, min(127, __float2int_rn(__fmul_rn(v.y, qm))));
  const int c = max(-127, min(127, __float2int_rn(__fmul_rn(v.z, qm))));
  const int d = max(-127, min(127, __float2int_rn(__fmul_rn(v.w, qm))));
  return (static_cast<unsigned>(a) & 0xffu) | ((static_cast<unsigned>(b) & 0xffu) << 8) | ((static_cast<unsigned>(c) & 0xffu) << 16) |
         ((static_cast<unsigned>(d) & 0xffu) << 24);
}
__device__ __forceinline__ float mult_of(unsigned bits) { return bits == 0u ? 1.0f : __fdiv_rn(127.0f, __uint_as_float(bits)); }
__device__ __forceinline__ float unquant_of(float qa, float qb) { return __fdiv_rn(1.0f, __fmul_rn(qa, qb)); }
__device__ __forceinline__ float4 dequant(const int4& a, float unquant) {
  return make_float4(__fmul_rn(__int2float_rn(a.x), unquant), __fmul_rn(__int2float_rn(a.y), unquant), __fmul_rn(__int2float_rn(a.z), unquant),
                     __fmul_rn(__int2float_rn(a.w), unquant));
}
__device__ __forceinline__ float4 add4(const float4& a, const float4& b) {
  return make_float4(__fadd_rn(a.x, b.x), __fadd_rn(a.y, b.y), __fadd_rn(a.z, b.z), __fadd_rn(a.w, b.w));
}
__device__ __forceinline__ void mma_16x8x32(int (&c)[4], unsigned a0, unsigned a1, unsigned a2, unsigned a3, unsigned b0, unsigned b1) {
  asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
               : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void st_cluster_f4(uint32_t addr, const float4& v) {
  asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w) : "memory");
}
__device__ __forceinline__ void st_cluster_u4(uint32_t addr, const uint4& v) {
  asm volatile("st.shared::cluster.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}
// byte offset of byte `b` (0..127) of K block kb of row r in an operand of `rows` rows
__device__ __forceinline__ int operand_offset(int kb, int rows, int r, int b) {
  return (kb * rows + r) * 128 + ((((b >> 4) ^ r) & 7) << 4) + (b & 15);
}

__device__ __forceinline__ void cluster_barrier() {
  __syncwarp();
  cluster_sync_all();
}

// i / n for i * n < 65536, with inv = 65536 / n + 1 (rounded down)
__device__ __forceinline__ int div_small(int i, int inv) { return (i * inv) >> 16; }

__device__ __forceinline__ void copy_async16(void* smem, const void* gmem) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(smem)), "l"(gmem) : "memory");
}
__device__ __forceinline__ void copy_async4(void* smem, const void* gmem) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(smem)), "l"(gmem) : "memory");
}
__device__ __forceinline__ void copy_async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// The split of a layer over the CTAs, known at compile time but for the feed-forward dimension f = 16 kCtas n.
template <int kDim, int kDh, int kCtas>
struct Split {
  static constexpr int kHeads = kDim / kDh;
  static constexpr int kNd = kDim / kCtas;                               // own columns of the model dimension
  static constexpr int kShare = kCtas > kHeads ? kCtas / kHeads : 1;     // CTAs that share a head: each takes every kShare-th row
  static constexpr int kOwnHeads = kHeads > kCtas ? kHeads / kCtas : 1;
  static constexpr int kNq = kOwnHeads * kDh;                            // own columns of the query projection
  static constexpr int kKb = kDim / 128;
  static_assert(kNd % kUnitRows == 0 && kDim % 128 == 0 && (kHeads % kCtas == 0 || kCtas % kHeads == 0), "");
  __host__ __device__ static constexpr int m_tiles(int phase, int f) {
    return (phase == kCell ? 2 * kNd : phase == kQuery ? kNq : phase == kFfn1 ? f / kCtas : kNd) / kUnitRows;
  }
  __host__ __device__ static constexpr int k_blocks(int phase, int f) { return phase == kFfn2 ? f / 128 : kKb; }
  static int units(int f) {   // of a layer
    int n = 0;
    for(int ph = 0; ph < kPhases; ++ph)
      n += m_tiles(ph, f) * k_blocks(ph, f);
    return n;
  }
  // widest accumulator row, floats of a CTA's biases and multipliers and of all LayerNorms per layer, scores (or a head's output) of a warp
  __host__ __device__ static constexpr int acc_cols(int f) { return f / kCtas > 2 * kNd ? (f / kCtas > kNq ? f / kCtas : kNq) : (2 * kNd > kNq ? 2 * kNd : kNq); }
  __host__ __device__ static constexpr int params(int f) { return 3 * kNd + kNq + f / kCtas + 8; }
  static constexpr int kNorms = 6 * kDim;
  __host__ __device__ static constexpr int scores(int src) { return ((src + 3) & ~3) > kDh ? ((src + 3) & ~3) : kDh; }
  static size_t smem(int rows, int f, int layers, int src, int ring) {
    const int Rp = (rows + 7) & ~7;
    return 1024 + static_cast<size_t>(kWarps) * ring * kUnitBytes + static_cast<size_t>(kDim + f) * Rp + 2 * sizeof(float) * rows * kDim +
           sizeof(int) * Rp * (acc_cols(f) + 4) + sizeof(float) * (rows * kNd * (1 + layers) + layers * (params(f) + kNorms) + kWarps * scores(src));
  }
};

// kRw: rows a warp normalises (row = warp + 16 i).
template <int kDim, int kDh, int kCtas, int kRw>
__global__ void __launch_bounds__(kThreads, 1) decoder_rows_kernel(const __grid_constant__ DecoderRowsParams p) {
  using T = Split<kDim, kDh, kCtas>;
  constexpr int kNd = T::kNd, kNq = T::kNq, kNv = T::kKb;   // (a row is kNv float4 per lane of a warp)
  extern __shared__ uint8_t smem_raw[];
  __shared__ uint64_t full[kWarps][kMaxRing];
  __shared__ unsigned redu[kWarps];
  __shared__ unsigned cta_max[kCtas];
  __shared__ int abort_word;
  volatile int* abort_flag = &abort_word;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = static_cast<int>(cluster_ctarank());
  const int R = p.rows, Rp = (p.rows + 7) & ~7, f = p.ffn, nf = p.ffn / kCtas, S = p.src, ring_n = p.ring;
  const int head0 = rank / T::kShare * T::kOwnHeads;

  uint8_t* ring = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);   // (swizzled boxes start on 1024 bytes; the same in every CTA)
  int8_t* Q = reinterpret_cast<int8_t*>(ring + kWarps * ring_n * kUnitBytes);    // [d / 128][Rp][128] the current operand
  int8_t* H = Q + kDim * Rp;                                                    // [f / 128][Rp][128] the feed-forward's hidden operand
  float* Y = reinterpret_cast<float*>(H + f * Rp);                              // [2][R][d] rows on their way, two in turn
  int* acc = reinterpret_cast<int*>(Y + 2 * R * kDim);                          // [Rp][columns + 4]
  float* xs = reinterpret_cast<float*>(acc + Rp * (T::acc_cols(f) + 4));        // [R][kNd] residual, own columns
  float* cell = xs + R * kNd;                                                   // [layers][R][kNd] previous SSRU state, own columns
  float* prm = cell + p.layers * R * kNd;                                       // [layers][params] own columns' biases, the weights' multipliers
  float* norms = prm + p.layers * T::params(f);                                 // [layers][6][d] LayerNorm scales and biases
  float* sc = norms + p.layers * T::kNorms + warp * T::scores(S);               // this warp's scores, then the head's output

  const TraceHandles th = trace_open_all();

  // ---- what does not depend on the kernel in front
  // ---- the weight stream: lane k knows the warp's k-th unit
  const CUtensorMap* my_map = nullptr;
  int my_row = 0, my_unit = -1;   // first weight row; phase | m tile << 8 | K block << 16, phase counted over the layers
  {
    int u = warp + lane * kWarps;
#pragma unroll 1
    for(int l = 0; l < p.layers && my_unit < 0; ++l) {
#pragma unroll
      for(int ph = 0; ph < kPhases; ++ph) {
        const int mts = T::m_tiles(ph, f), n = mts * T::k_blocks(ph, f);
        if(my_unit < 0) {
          if(u < n) {
            const int kb = ph == kFfn1 ? div_small(u, p.inv_mt_ffn1) : u / mts, mt = u - kb * mts;
            my_unit = (l * kPhases + ph) | (mt << 8) | (kb << 16);
            my_map = &p.map[l][ph];
            my_row = mt * kUnitRows;
            if(ph == kCell)
              my_row += rank * kNd + (my_row < kNd ? 0 : kDim - kNd);
            else
              my_row += ph == kQuery ? head0 * kDh : ph == kFfn1 ? rank * nf : rank * kNd;
          }
          u -= n;
        }
      }
    }
  }
  auto request = [&](int slot) {   // by the lane that knows the unit (test hook: a withheld unit never arrives)
    if(lane == p.withhold_item)
      return;
    mbar_arrive_expect_tx(&full[warp][slot], kUnitBytes);
    tma_load_2d(ring + (warp * ring_n + slot) * kUnitBytes, my_map, (my_unit >> 16) * 128, my_row, &full[warp][slot]);
  };
  if(lane < ring_n)
    mbar_init(&full[warp][lane], 1);
  fence_mbar_init();
  fence_proxy_async_smem();
  if(lane < ring_n && my_unit >= 0)
    request(lane);
  __syncwarp();
  const int total = __popc(__ballot_sync(0xffffffffu, my_unit >= 0));
  int used = 0, requested = min(ring_n, total), slot = 0;
  uint32_t parity = 0;
  bool ok = true;

  // The LayerNorms, this CTA's columns of the biases and the weights' multipliers, from where they were registered: a caller may rewrite
  // them between steps.  Like the weights above they are read in front of the wait: only mi8d_search's steps, which have its own kernels in front of them, are
  // launched over the end of those; a step that a caller asks for starts when all in front of it has completed (launch_decoder_rows).
#pragma unroll 1
  for(int l = 0; l < p.layers; ++l) {
    const DecoderRowsVectors& v = p.vec[l];
    float* own = prm + l * T::params(f);
    constexpr int kLn = kDim / 4, kOwn = kNd / 4;   // 16-byte chunks
#pragma unroll 1
    for(int i = threadIdx.x; i < 6 * kLn + 3 * kOwn + (kNq + nf) / 4; i += kThreads) {
      const int c = i - 6 * kLn, q = c - 3 * kOwn;
      if(c < 0)
        copy_async16(norms + l * T::kNorms + 4 * i, v.ln[i / kLn] + 4 * (i % kLn));
      else if(q < 0)
        copy_async16(own + 4 * c, v.own[c / kOwn] + rank * kNd + 4 * (c % kOwn));
      else
        copy_async16(own + 4 * c, q < kNq / 4 ? v.b_q + head0 * kDh + 4 * q : v.b_1 + rank * nf + 4 * q - kNq);
    }
    if(threadIdx.x < kRowsMultipliers)
      copy_async4(own + 3 * kNd + kNq + nf + threadIdx.x, v.qb[threadIdx.x]);
  }
  float4 pv[kNv];
#pragma unroll
  for(int v = 0; v < kNv; ++v)
    pv[v] = __ldg(reinterpret_cast<const float4*>(p.pos) + 32 * v + lane);

#pragma unroll 1
  for(int i = threadIdx.x; i < Rp * (T::acc_cols(f) + 4) / 4; i += kThreads)
    reinterpret_cast<int4*>(acc)[i] = make_int4(0, 0, 0, 0);
  if(threadIdx.x == 0)
    abort_word = 0;
  pdl_wait_and_launch();
  trace_stamp_start(th, kTrDecoderRows);
  // ---- embedding * sqrt(d) + position, and the cells' previous state.  The control words come with the launch's parameters, which are
  // there at once (reads of pinned memory by every CTA went over PCIe lane by lane: 16 rows 250 us), or from the device, where the step in front left
  // them (StepEnd::next_ctrl): launched before the host has seen that step's words, this one has its weights under way when they come.
  const bool with_words = p.n_ctrl > 0;
  int word[kRw];
  const unsigned stopped = p.stop != nullptr ? *p.stop : 0u;   // (looked at once the loads beside it are under way)
#pragma unroll
  for(int i = 0; i < kRw; ++i) {
    const int r = min(warp + i * kWarps, R - 1);
    word[i] = with_words ? p.ctrl_words[R + r] : (p.words ? p.words[r] : -1);
  }
  const int own_row = min(static_cast<int>(threadIdx.x) / (kNd / 4), R - 1);
  const int own_src = with_words ? p.ctrl_words[own_row] : (p.hyp ? p.hyp[own_row] : own_row);
  const bool brings = rank == kCtas - 1 && static_cast<int>(threadIdx.x) < p.n_lists;
  const unsigned long long entry = brings ? p.lists[threadIdx.x] : 0ull;
  auto bring = [&]() {   // the lists of the step in front, to the host
    if(brings)
      const_cast<volatile unsigned long long*>(p.host_lists)[threadIdx.x] = entry;
  };
  if(stopped != 0u) {   // (the same word for every CTA) a hypothesis has ended: the host launches this step anew
    int no_abort = 0;
    for(int i = 0; i < requested; ++i)
      mbar_wait_bounded(&full[warp][i], 0u, &no_abort, p.spin_limit);
    copy_async_wait();
    bring();
    return;
  }
  float4 x[kRw][kNv];
#pragma unroll
  for(int i = 0; i < kRw; ++i) {
    const int r = warp + i * kWarps;
    if(r < R) {
      const float4* src = reinterpret_cast<const float4*>(p.wemb + static_cast<size_t>(max(word[i], 0)) * kDim) + lane;
#pragma unroll
      for(int v = 0; v < kNv; ++v)
        x[i][v] = word[i] >= 0 ? __ldg(src + 32 * v) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
  }
#pragma unroll 1
  for(int l = 0; l < p.layers; ++l)
#pragma unroll 1
    for(int i = threadIdx.x; i < R * (kNd / 4); i += kThreads) {
      const int r = i / (kNd / 4), c = 4 * (i % (kNd / 4));
      const int src = i < kThreads ? own_src : with_words ? p.ctrl_words[r] : (p.hyp ? p.hyp[r] : r);
      copy_async16(cell + (l * R + r) * kNd + c, p.cell_old + l * p.layer_stride + static_cast<size_t>(src) * kDim + rank * kNd + c);
    }
  bring();
  __syncthreads();
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");   // (this CTA runs: the others may store into it)

  // this CTA's columns of one affine: acc[r][column] += operand rows x weight rows; ends with a block barrier
  auto affine = [&](int phase, int cols, const int8_t* operand) {
    const int stride = cols + 4;
    const int g = lane >> 2, t = lane & 3;
    while(used < total) {
      const int unit = __shfl_sync(0xffffffffu, my_unit, used);
      if((unit & 0xff) != phase)
        break;
      const int mt = (unit >> 8) & 0xff, kb = unit >> 16;
      if(ok)
        ok = __all_sync(0xffffffffu, mbar_wait_bounded(&full[warp][slot], parity, abort_flag,
                                                     p.withhold_item == kWithholdWarp && warp == 3 ? 0u : p.spin_limit));   // (test hook: one warp gives up at once)
      if(!ok) {
        if(lane == 0) {
          *abort_flag = 1;
          atomicMax(p.status, static_cast<int>(kDevTimeoutMma));
        }
        break;
      }
      const uint8_t* w = ring + (warp * ring_n + slot) * kUnitBytes + g * 128;
      const uint8_t* a = reinterpret_cast<const uint8_t*>(operand) + kb * Rp * 128 + g * 128;
      uint4 lo[2], hi[2];
#pragma unroll
      for(int h = 0; h < 2; ++h) {
        const int chunk = ((2 * t + h) ^ g) << 4;
        lo[h] = *reinterpret_cast<const uint4*>(w + chunk);
        hi[h] = *reinterpret_cast<const uint4*>(w + 1024 + chunk);
      }
#pragma unroll 1
      for(int nt = 0; nt < Rp / 8; ++nt) {
        int c[4] = {0, 0, 0, 0};
#pragma unroll
        for(int h = 0; h < 2; ++h) {
          const uint4 b = *reinterpret_cast<const uint4*>(a + nt * 1024 + (((2 * t + h) ^ g) << 4));
          mma_16x8x32(c, lo[h].x, hi[h].x, lo[h].y, hi[h].y, b.x, b.y);
          mma_16x8x32(c, lo[h].z, hi[h].z, lo[h].w, hi[h].w, b.z, b.w);
        }
        int* dst = acc + (nt * 8 + 2 * t) * stride + mt * kUnitRows + g;
        atomicAdd(dst, c[0]);
        atomicAdd(dst + stride, c[1]);
        atomicAdd(dst + 8, c[2]);
        atomicAdd(dst + stride + 8, c[3]);
      }
      __syncwarp();   // (every lane has read the unit: its place is free)
      if(requested < total) {
        if(lane == requested)
          request(slot);
        ++requested;
      }
      ++used;
      if(++slot == ring_n) {
        slot = 0;
        parity ^= 1u;
      }
    }
    __syncthreads();
  };
  auto clear_acc = [&](int cols) {   // (read by everyone before the last barrier, added to after the next)
#pragma unroll 1
    for(int i = threadIdx.x; i < Rp * (cols + 4) / 4; i += kThreads)
      reinterpret_cast<int4*>(acc)[i] = make_int4(0, 0, 0, 0);
  };

  if(rank == 0) {   // for the kernels behind this one
    for(int i = threadIdx.x; i < p.n_ctrl; i += kThreads)
      p.ctrl[i] = p.ctrl_words[i];
    if(threadIdx.x == 0 && p.next_stop != nullptr)
      *p.next_stop = 0u;
    for(int i = threadIdx.x; i < p.n_slots; i += kThreads)
      p.slots[i] = 0u;
  }
#pragma unroll
  for(int i = 0; i < kRw; ++i)
#pragma unroll
    for(int v = 0; v < kNv; ++v) {
      x[i][v].x = __fadd_rn(__fmul_rn(x[i][v].x, p.emb_scale), pv[v].x);
      x[i][v].y = __fadd_rn(__fmul_rn(x[i][v].y, p.emb_scale), pv[v].y);
      x[i][v].z = __fadd_rn(__fmul_rn(x[i][v].z, p.emb_scale), pv[v].z);
      x[i][v].w = __fadd_rn(__fmul_rn(x[i][v].w, p.emb_scale), pv[v].w);
    }
  // x: rows of this warp -> their abs-max over all rows -> quantised into Q; ends with a block barrier
  auto quantise = [&]() -> float {
    unsigned m = 0u;
#pragma unroll
    for(int i = 0; i < kRw; ++i)
      if(warp + i * kWarps < R) {
#pragma unroll
        for(int v = 0; v < kNv; ++v)
          m = max4u(m, x[i][v]);
      }
    m = __reduce_max_sync(0xffffffffu, m);
    if(lane == 0)
      redu[warp] = m;
    __syncthreads();
    m = __reduce_max_sync(0xffffffffu, redu[lane & (kWarps - 1)]);
    const float qm = mult_of(m);
    if(m >= 0x7f800000u && rank == 0 && threadIdx.x == 0)
      atomicMax(p.status, static_cast<int>(kDevNonFinite));
#pragma unroll
    for(int i = 0; i < kRw; ++i) {
      const int r = warp + i * kWarps;
      if(r < R) {
#pragma unroll
        for(int v = 0; v < kNv; ++v)
          *reinterpret_cast<unsigned*>(Q + operand_offset(v, Rp, r, 4 * lane)) = pack4(x[i][v], qm);
      }
    }
    __syncthreads();
    return qm;
  };
  // keeps this CTA's columns of x as the next residual
  auto keep_residual = [&]() {
#pragma unroll
    for(int i = 0; i < kRw; ++i) {
      const int r = warp + i * kWarps;
      if(r < R) {
#pragma unroll
        for(int v = 0; v < kNv; ++v) {
          const int c = 4 * (32 * v + lane) - rank * kNd;
          if(c >= 0 && c < kNd)
            *reinterpret_cast<float4*>(xs + r * kNd + c) = x[i][v];
        }
      }
    }
  };
  auto load_rows = [&](const float* y) {
#pragma unroll
    for(int i = 0; i < kRw; ++i) {
      const int r = warp + i * kWarps;
      if(r < R) {
#pragma unroll
        for(int v = 0; v < kNv; ++v)
          x[i][v] = reinterpret_cast<const float4*>(y + r * kDim)[32 * v + lane];
      }
    }
  };
  // LayerNorm of x in place (kDim is a power of two: the product with 1 / kDim is the quotient), sums in the order of add_layernorm_kernel
  // (its 256 threads' warps are the v here)
  auto layernorm = [&](const float* gamma) {   // (the biases lie behind the scales)
    float4 gm[kNv], bt[kNv];
#pragma unroll
    for(int v = 0; v < kNv; ++v) {
      gm[v] = reinterpret_cast<const float4*>(gamma)[32 * v + lane];
      bt[v] = reinterpret_cast<const float4*>(gamma + kDim)[32 * v + lane];
    }
#pragma unroll
    for(int i = 0; i < kRw; ++i) {
      if(warp + i * kWarps < R) {
        float s[kNv];
#pragma unroll
        for(int v = 0; v < kNv; ++v)
          s[v] = __fadd_rn(0.f, __fadd_rn(__fadd_rn(x[i][v].x, x[i][v].y), __fadd_rn(x[i][v].z, x[i][v].w)));
#pragma unroll
        for(int o = 16; o > 0; o >>= 1)
#pragma unroll
          for(int v = 0; v < kNv; ++v)
            s[v] = __fadd_rn(s[v], __shfl_xor_sync(0xffffffffu, s[v], o));
        float t = 0.f;
#pragma unroll
        for(int v = 0; v < kNv; ++v)
          t = __fadd_rn(t, s[v]);
        const float mean = __fmul_rn(t, 1.0f / kDim);
#pragma unroll
        for(int v = 0; v < kNv; ++v) {
          x[i][v].x = __fadd_rn(x[i][v].x, -mean);
          x[i][v].y = __fadd_rn(x[i][v].y, -mean);
          x[i][v].z = __fadd_rn(x[i][v].z, -mean);
          x[i][v].w = __fadd_rn(x[i][v].w, -mean);
          s[v] = __fadd_rn(0.f, __fmaf_rn(x[i][v].x, x[i][v].x, __fmaf_rn(x[i][v].y, x[i][v].y, __fmaf_rn(x[i][v].z, x[i][v].z, __fmul_rn(x[i][v].w, x[i][v].w)))));
        }
#pragma unroll
        for(int o = 16; o > 0; o >>= 1)
#pragma unroll
          for(int v = 0; v < kNv; ++v)
            s[v] = __fadd_rn(s[v], __shfl_xor_sync(0xffffffffu, s[v], o));
        t = 0.f;
#pragma unroll
        for(int v = 0; v < kNv; ++v)
          t = __fadd_rn(t, s[v]);
        const float denom = __fsqrt_rn(__fadd_rn(__fmul_rn(t, 1.0f / kDim), 1e-6f));
#pragma unroll
        for(int v = 0; v < kNv; ++v) {
          x[i][v].x = __fadd_rn(__fmul_rn(__fdiv_rn(x[i][v].x, denom), gm[v].x), bt[v].x);
          x[i][v].y = __fadd_rn(__fmul_rn(__fdiv_rn(x[i][v].y, denom), gm[v].y), bt[v].y);
          x[i][v].z = __fadd_rn(__fmul_rn(__fdiv_rn(x[i][v].z, denom), gm[v].z), bt[v].z);
          x[i][v].w = __fadd_rn(__fmul_rn(__fdiv_rn(x[i][v].w, denom), gm[v].w), bt[v].w);
        }
      }
    }
  };
  // value(r, c) of this CTA's columns c .. c + 3 into the rows of every CTA (each thread computes what it stores: cheaper than one more
  // block barrier between computing once and storing kCtas times)
  auto spread = [&](float* y, auto&& value) {
#pragma unroll 1
    for(int i = threadIdx.x; i < R * kCtas * (kNd / 4); i += kThreads) {
      const int c = 4 * (i % (kNd / 4)), dest = i / (kNd / 4) % kCtas, r = i / (kNd / 4 * kCtas);
      st_cluster_f4(mapa_shared(smem_u32(y + r * kDim + rank * kNd + c), dest), value(r, c, dest == rank));
    }
  };

  keep_residual();
  copy_async_wait();
  float qa = quantise();
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");   // every CTA of the cluster runs

  float* y = Y;   // where the next rows go, the two places in turn (rows stored two exchanges ago have been read by every CTA)
  auto next_y = [&]() { y = y == Y ? Y + R * kDim : Y; };
#pragma unroll 1
  for(int l = 0; l < p.layers; ++l) {
    const float* norm = norms + l * T::kNorms;
    const float *b_wf = prm + l * T::params(f), *b_o = b_wf + kNd, *b_2 = b_o + kNd, *b_q = b_2 + kNd, *b_1 = b_q + kNq, *qb = b_1 + nf;
    // ---- SSRU cell
    affine(l * kPhases + kCell, 2 * kNd, Q);
    {
      const float uw = unquant_of(qa, qb[0]), uf = unquant_of(qa, qb[1]);
      spread(y, [&](int r, int c, bool own) {
        const int* a = acc + r * (2 * kNd + 4) + c;
        const float4 xw = dequant(*reinterpret_cast<const int4*>(a), uw);
        const float4 fg = add4(dequant(*reinterpret_cast<const int4*>(a + kNd), uf), *reinterpret_cast<const float4*>(b_wf + c));
        const float4 c0 = *reinterpret_cast<const float4*>(cell + (l * R + r) * kNd + c);
        float4 h, cn;
        cn.x = ssru_cell(c0.x, xw.x, fg.x, &h.x);
        cn.y = ssru_cell(c0.y, xw.y, fg.y, &h.y);
        cn.z = ssru_cell(c0.z, xw.z, fg.z, &h.z);
        cn.w = ssru_cell(c0.w, xw.w, fg.w, &h.w);
        if(own)
          *reinterpret_cast<float4*>(p.cell_new + l * p.layer_stride + static_cast<size_t>(r) * kDim + rank * kNd + c) = cn;
        return add4(h, *reinterpret_cast<const float4*>(xs + r * kNd + c));
      });
    }
    cluster_barrier();
    clear_acc(2 * kNd);
    load_rows(y);
    next_y();
    layernorm(norm);

    // ---- cross-attention, arithmetic and order of attention1_kernel: warp w has one (row, head).  Its first keys and all it needs of
    // the mask are on their way while the query is computed.
    constexpr int G = kDh / 4, kGroups = 32 / G, kU = 4;   // lanes of a head's dot product, positions at once, times kU in flight
    const int own_rows = (R - rank % T::kShare + T::kShare - 1) / T::kShare;
    const bool has_unit = warp < own_rows * T::kOwnHeads;
    const int hl = T::kOwnHeads > 1 ? div_small(warp, p.inv_rows) : 0;
    const int r = has_unit ? rank % T::kShare + (warp - hl * own_rows) * T::kShare : 0, head = head0 + (has_unit ? hl : 0);
    const int b = r - div_small(r, p.inv_batch) * p.batch;
    const int j = lane % G, grp = lane / G;
    const float* kp = p.cross_k + l * p.layer_stride + static_cast<size_t>(b) * S * kDim + head * kDh + 4 * j;
    const float* vp = p.cross_v + l * p.layer_stride + static_cast<size_t>(b) * S * kDim + head * kDh + (kDh / 32) * lane;
    const float* mask = p.log_mask + static_cast<size_t>(b) * S;
    float4 kk[kU];
    float mk[kU];
    auto load_k = [&](int p0) {   // (past the end: the last position again, not written)
#pragma unroll
      for(int e = 0; e < kU; ++e) {
        const int pos = min(p0 + e * kGroups + grp, S - 1);
        kk[e] = __ldg(reinterpret_cast<const float4*>(kp + static_cast<size_t>(pos) * kDim));
        mk[e] = __ldg(mask + pos);
      }
    };
    if(has_unit)
      load_k(0);
    keep_residual();
    qa = quantise();
    affine(l * kPhases + kQuery, kNq, Q);
    if(has_unit) {
      const float4 qv = add4(dequant(*reinterpret_cast<const int4*>(acc + r * (kNq + 4) + hl * kDh + 4 * j), unquant_of(qa, qb[2])),
                             *reinterpret_cast<const float4*>(b_q + hl * kDh + 4 * j));
      constexpr int kAhead = kDh == 32 ? 16 : 8;   // (what 128 registers hold)
      float2 vv[kAhead];
      auto load_v = [&](int pos) -> float2 {
        const float* src = vp + static_cast<size_t>(min(pos, S - 1)) * kDim;
        return kDh == 64 ? __ldg(reinterpret_cast<const float2*>(src)) : make_float2(__ldg(src), 0.f);
      };
#pragma unroll 1
      for(int p0 = 0; p0 < S; p0 += kU * kGroups) {
        if(p0 > 0)
          load_k(p0);
        float dt[kU];
#pragma unroll
        for(int e = 0; e < kU; ++e) {
          dt[e] = __fmul_rn(qv.x, kk[e].x);
          dt[e] = __fmaf_rn(qv.y, kk[e].y, dt[e]);
          dt[e] = __fmaf_rn(qv.z, kk[e].z, dt[e]);
          dt[e] = __fmaf_rn(qv.w, kk[e].w, dt[e]);
        }
#pragma unroll
        for(int o = G / 2; o > 0; o >>= 1)
#pragma unroll
          for(int e = 0; e < kU; ++e)
            dt[e] = __fadd_rn(dt[e], __shfl_xor_sync(0xffffffffu, dt[e], o));
        if(p0 == 0) {
#pragma unroll
          for(int e = 0; e < kAhead; ++e)   // the first value rows: on their way during the softmax
            vv[e] = load_v(e);
        }
        if(j == 0) {
#pragma unroll
          for(int e = 0; e < kU; ++e) {
            const int pos = p0 + e * kGroups + grp;
            if(pos < S)
              sc[pos] = __fadd_rn(__fmul_rn(dt[e], p.att_scale), mk[e]);
          }
        }
      }
      __syncwarp();
      float mx = -FLT_MAX;
#pragma unroll 1
      for(int pos = lane; pos < S; pos += 32)
        mx = fmaxf(mx, sc[pos]);
#pragma unroll
      for(int o = 16; o > 0; o >>= 1)
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
#pragma unroll 1
      for(int pos = lane; pos < S; pos += 32)
        sc[pos] = det_expf(__fadd_rn(sc[pos], -mx));
      __syncwarp();
      float part = 0.f;
      for(int pos = j; pos < S; pos += G)
        part = __fadd_rn(part, sc[pos]);
#pragma unroll
      for(int o = G / 2; o > 0; o >>= 1)
        part = __fadd_rn(part, __shfl_xor_sync(0xffffffffu, part, o));
      __syncwarp();
#pragma unroll 1
      for(int pos = lane; pos < S; pos += 32)
        sc[pos] = __fdiv_rn(sc[pos], part);
      __syncwarp();
      float2 out = make_float2(0.f, 0.f);
#pragma unroll 1
      for(int p0 = 0; p0 < S; p0 += kAhead) {
        if(p0 > 0) {
#pragma unroll
          for(int e = 0; e < kAhead; ++e)
            vv[e] = load_v(p0 + e);
        }
#pragma unroll
        for(int e = 0; e < kAhead; ++e) {
          if(p0 + e < S) {
            const float w = sc[p0 + e];
            out.x = __fmaf_rn(w, vv[e].x, out.x);
            out.y = __fmaf_rn(w, vv[e].y, out.y);
          }
        }
      }
      __syncwarp();   // (the weights are used up)
      if(kDh == 64)
        *reinterpret_cast<float2*>(sc + 2 * lane) = out;
      else
        sc[lane] = out.x;
      __syncwarp();
#pragma unroll
      for(int i = lane; i < G * kCtas; i += 32)
        st_cluster_f4(mapa_shared(smem_u32(y + r * kDim + head * kDh + 4 * (i % G)), i / G), *reinterpret_cast<const float4*>(sc + 4 * (i % G)));
    }
    cluster_barrier();
    clear_acc(kNq);
    load_rows(y);
    next_y();
    qa = quantise();

    // ---- its output projection, residual, LayerNorm
    auto residual_affine = [&](int ph, const int8_t* operand, float qb_w, const float* bias, const float* scales) {
      affine(l * kPhases + ph, kNd, operand);
      const float uo = unquant_of(qa, qb_w);
      spread(y, [&](int row, int c, bool) {
        const float4 o = add4(dequant(*reinterpret_cast<const int4*>(acc + row * (kNd + 4) + c), uo), *reinterpret_cast<const float4*>(bias + c));
        return add4(o, *reinterpret_cast<const float4*>(xs + row * kNd + c));
      });
      cluster_barrier();
      clear_acc(kNd);
      load_rows(y);
      next_y();
      layernorm(scales);
      keep_residual();
      qa = quantise();
    };
    residual_affine(kOut, Q, qb[3], b_o, norm + 2 * kDim);

    // ---- feed-forward: the hidden rows stay with the CTA that owns the columns until their abs-max is known to all
    affine(l * kPhases + kFfn1, nf, Q);
    {
      const float u1 = unquant_of(qa, qb[4]);
      const int tasks = R * (nf / 4);
      float4 hv[2];
      int at[2];
      unsigned m = 0u;
#pragma unroll
      for(int k = 0; k < 2; ++k) {
        const int i = threadIdx.x + k * kThreads;
        if(i < tasks) {
          const int row = div_small(i, p.inv_nf4), c = 4 * (i - row * (nf / 4));
          float4 h = add4(dequant(*reinterpret_cast<const int4*>(acc + row * (nf + 4) + c), u1), *reinterpret_cast<const float4*>(b_1 + c));
          h.x = h.x > 0.f ? h.x : 0.f;
          h.y = h.y > 0.f ? h.y : 0.f;
          h.z = h.z > 0.f ? h.z : 0.f;
          h.w = h.w > 0.f ? h.w : 0.f;
          hv[k] = h;
          m = max4u(m, h);
          const int col = rank * nf + (c & ~15);
          at[k] = operand_offset(col >> 7, Rp, row, col & 127);
        }
      }
      m = __reduce_max_sync(0xffffffffu, m);
      if(lane == 0)
        redu[warp] = m;
      __syncthreads();
      if(warp == 0) {
        m = __reduce_max_sync(0xffffffffu, redu[lane & (kWarps - 1)]);
        if(lane < kCtas)
          st_cluster_u32(mapa_shared(smem_u32(&cta_max[rank]), lane), m);
      }
      cluster_barrier();
      clear_acc(nf);
      m = __reduce_max_sync(0xffffffffu, cta_max[lane % kCtas]);
      qa = mult_of(m);
      if(m >= 0x7f800000u && rank == 0 && threadIdx.x == 0)
        atomicMax(p.status, static_cast<int>(kDevNonFinite));
      // four neighbouring lanes hold 16 consecutive columns (nf is a multiple of 16): each stores the chunk into a quarter of the CTAs
#pragma unroll
      for(int k = 0; k < 2; ++k) {
        const int i = threadIdx.x + k * kThreads;
        if((i & ~31) < tasks) {
          const unsigned own = i < tasks ? pack4(hv[k], qa) : 0u;
          uint4 chunk;
          chunk.x = __shfl_sync(0xffffffffu, own, 0, 4);
          chunk.y = __shfl_sync(0xffffffffu, own, 1, 4);
          chunk.z = __shfl_sync(0xffffffffu, own, 2, 4);
          chunk.w = __shfl_sync(0xffffffffu, own, 3, 4);
          if(i < tasks) {
#pragma unroll
            for(int c = 0; c < kCtas; c += 4)
              st_cluster_u4(mapa_shared(smem_u32(H + at[k]), c + (lane & 3)), chunk);
          }
        }
      }
    }
    cluster_barrier();
    residual_affine(kFfn2, H, qb[5], b_2, norm + 4 * kDim);
  }
  if(!ok)   // (a wait ran out: no copy may land after the CTA has gone)
    for(int no_abort = 0; used < requested; ++used)
      mbar_wait_bounded(&full[warp][used % ring_n], (used / ring_n) & 1, &no_abort, p.spin_limit);
  // ---- the output layer's operand
#pragma unroll
  for(int i = 0; i < kRw; ++i) {
    const int row = warp + i * kWarps;
    if(row < R && row % kCtas == rank) {
#pragma unroll
      for(int v = 0; v < kNv; ++v)
        *reinterpret_cast<unsigned*>(p.out_q + static_cast<size_t>(row) * kDim + 128 * v + 4 * lane) = pack4(x[i][v], qa);
    }
  }
  if(rank == 0 && threadIdx.x == 0)
    *p.out_qm = qa;
  trace_stamp(th.first, kTrDecoderRows, 2);
  trace_stamp(th.last, kTrDecoderRows, 3);
}

template <int kDim, int kDh, int kCtas, int kRw>
struct RowsKernel {
  using T = Split<kDim, kDh, kCtas>;
  static constexpr auto kernel = decoder_rows_kernel<kDim, kDh, kCtas, kRw>;
  // whether the device can hold the cluster
  static bool available() {
    static int known[64] = {};   // 0 = not asked yet, 1 = yes, -1 = no
    int dev = 0;
    cudaGetDevice(&dev);
    if(dev < 0 || dev >= 64)
      return false;
    if(known[dev] == 0) {
      cudaLaunchConfig_t cfg = {};
      cudaLaunchAttribute attr[1];
      attr[0].id = cudaLaunchAttributeClusterDimension;
      attr[0].val.clusterDim.x = kCtas;
      attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
      cfg.gridDim = dim3(kCtas);
      cfg.blockDim = dim3(kThreads);
      cfg.dynamicSmemBytes = kMaxDynSmem;
      cfg.attrs = attr;
      cfg.numAttrs = 1;
      int n = 0;
      const bool yes = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxDynSmem) == cudaSuccess &&
                       (kCtas <= 8 || cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess) &&
                       cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) == cudaSuccess && n > 0;
      if(!yes)
        cudaGetLastError();
      known[dev] = yes ? 1 : -1;
    }
    return known[dev] > 0;
  }
  static bool supported(int rows, int f, int layers, int src) {
    return rows * kDim <= kRw * kWarps * kDim && rows * T::kHeads <= kWarps * kCtas && f % (kUnitRows * kCtas) == 0 && f % 128 == 0 &&
           rows * (f / kCtas / 4) <= 2 * kThreads && rows * (f / kCtas / 4) * (f / kCtas / 4) < 65536 && layers * T::units(f) <= 32 * kWarps &&
           T::smem(rows, f, layers, src, 1) <= static_cast<size_t>(kMaxDynSmem) && available();
  }
  static int launch(DecoderRowsParams& p, cudaStream_t stream, bool params_settled) {
    // as many units in flight per warp as fit, up to all of a warp's
    const int most = (p.layers * T::units(p.ffn) + kWarps - 1) / kWarps;
    p.ring = 1;
    while(p.ring < kMaxRing && p.ring < most && T::smem(p.rows, p.ffn, p.layers, p.src, p.ring + 1) <= static_cast<size_t>(kMaxDynSmem))
      ++p.ring;
    p.inv_mt_ffn1 = 65536 / T::m_tiles(kFfn1, p.ffn) + 1;
    p.inv_nf4 = 65536 / (p.ffn / kCtas / 4) + 1;
    p.inv_batch = 65536 / p.batch + 1;
    p.inv_rows = 65536 / p.rows + 1;   // (read where a CTA has several heads: all rows are its own then)
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = kCtas;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.gridDim = dim3(kCtas);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = T::smem(p.rows, p.ffn, p.layers, p.src, p.ring);
    cfg.stream = stream;
    cfg.attrs = attr;
    const bool timed = kernel_times_on();
    cfg.numAttrs = pdl_enabled() && params_settled && !timed ? 2 : 1;
    if(timed)
      kernel_times_before(reinterpret_cast<const void*>(kernel), stream);
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, static_cast<const DecoderRowsParams&>(p));
    if(timed)
      kernel_times_after(stream);
    if(e != cudaSuccess) {
      set_last_cuda_error(e);
      return MI8_ERR_LAUNCH;
    }
    count_launch();
    return check_launch();
  }
};
using Rows256 = RowsKernel<256, 32, 16, 2>;   // up to 32 rows
using Rows512 = RowsKernel<512, 64, 16, 1>;   // up to 16 rows

}  // namespace

MI8_DEFINE_TRACE_SETTER(trace_set_rows)

// The sizes that a kernel exists for; the conditions are what the split over the CTAs and the shared memory need.
bool decoder_rows_supported(int rows, int d, int f, int heads, int layers, int src) {
  if(rows < 1 || rows > kDecoderRowsMax || src < 1 || layers < 1 || layers > kDecoderRowsLayers || f < 1)
    return false;
  if(d == 256 && heads == 8)
    return Rows256::supported(rows, f, layers, src);
  if(d == 512 && heads == 8)
    return Rows512::supported(rows, f, layers, src);
  return false;
}

int launch_decoder_rows(DecoderRowsParams& p, int d, int heads, cudaStream_t stream, bool params_settled) {
  if(!decoder_rows_supported(p.rows, d, p.ffn, heads, p.layers, p.src))
    return MI8_ERR_UNSUPPORTED;
  test_wait_limits(&p.withhold_item, &p.spin_limit);
  p.status = device_status_ptr();
  if(p.status == nullptr)
    return MI8_ERR_LAUNCH;
  return d == 256 ? Rows256::launch(p, stream, params_settled) : Rows512::launch(p, stream, params_settled);
}

}  // namespace mi8

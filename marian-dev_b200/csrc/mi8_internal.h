// Internal declarations shared by the translation units of libmarian_i8.so.
#pragma once
#include <cstddef>
#include <cstdint>
#include <cuda.h>
#include <cuda_runtime.h>

#include "../../include/marian_i8.h"
#include "../../include/marian_i8_measure.h"

namespace mi8 {

// ------------------------------------------------------------------ workspace layout (bytes)
// [0, 256)            abs-max block counter (first 4 bytes) and reserved words
// [256, 16640)        split-K arrival counters, one uint32 per output tile
// [16640, 20736)      abs-max per-block partial maxima (1024 x uint32)
// [20736, ...)        split-K accumulation buffers, int32 [tile][column][128 rows]
// Everything except the abs-max partials must be zero between calls; kernels restore that.
constexpr size_t kWsOffAbsmaxCounter = 0;
constexpr size_t kWsOffTileCounters = 256;
constexpr int kWsMaxTileCounters = 4096;
constexpr size_t kWsOffAbsmaxPartials = kWsOffTileCounters + sizeof(uint32_t) * kWsMaxTileCounters;
constexpr int kWsMaxAbsmaxBlocks = 1024;
constexpr size_t kWsOffPartials = kWsOffAbsmaxPartials + sizeof(uint32_t) * kWsMaxAbsmaxBlocks;
constexpr size_t kWsHeaderBytes = kWsOffPartials;

// ------------------------------------------------------------------ per-thread error / launch bookkeeping
void set_last_cuda_error(cudaError_t e);
void count_launch();

// Device status word of the current device (address of a __device__ int, resolved once per device).
int* device_status_ptr();
int sm_count();

// Checks cudaGetLastError() after a launch; returns MI8_OK or MI8_ERR_LAUNCH.
int check_launch();

// ------------------------------------------------------------------ GEMM plan
struct GemmPlan {
  int tile_m;        // activation rows per tile (MMA N): 16, 32, 64, 128 or 256
  int pair;          // 1: CTA-pair kernel (256 weight rows x 256 activation rows per cluster of two CTAs)
  int duo;           // 1: two CTAs of a cluster share a 64-row tile's inner dimension (splits == 2, no workspace)
  int stages;        // shared-memory pipeline depth
  int splits;        // split-K factor
  int n_tiles;       // tiles of 128 weight rows
  int m_tiles;       // tiles of tile_m activation rows
  int kb_total;      // 128-byte K blocks
  int kb_per_split;
  int grid;
  int smem_bytes;
  size_t partial_bytes;   // behind the workspace's header: what a call brings, of which a product that is not split uses nothing
};
int make_gemm_plan(int M, int N, int K, int force_tile_m, int force_splits, GemmPlan* plan, bool allow_duo = false);

// mi8_peak.cu: TOPS of a loop of this library's int8 MMAs alone (k_blocks 128-byte K blocks per SM).
int measure_int8_mma_peak(int k_blocks, float* tops_out, cudaStream_t stream);

int profile_begin(int max_records);
int profile_end(mi8_gemm_record* out, int capacity, int* count);

// quantisation kernels (mi8_quant.cu)
int launch_max_absolute(const float* x, size_t n, float* d_absmax, float* d_quant_mult, void* ws, size_t ws_bytes,
                        cudaStream_t stream);
int launch_quantize(const float* x, size_t n, const float* d_quant_mult, int8_t* q, cudaStream_t stream);
// When the last kernel of launch_prepare lets the next one start: when it is done, behind its own wait (what is in front has completed then), or at its start.
enum class Trigger { kDone, kBehindWait, kAtStart };
// both in turn (d_quant_mult = 127 / max|x|, q = x quantised with it); one launch for small tensors
int launch_prepare(const float* x, size_t n, float* d_quant_mult, int8_t* q, void* ws, size_t ws_bytes, cudaStream_t stream, Trigger trigger);
// W [K, N] -> Bt [N, K] and its multiplier
int launch_convert(const float* w, int K, int N, float* d_quant_mult, int8_t* bt, void* ws, size_t ws_bytes, cudaStream_t stream);
int launch_transpose_f32(const float* in, int batch, int rows, int cols, float* out, cudaStream_t stream);

// GEMM (mi8_gemm.cu)
// absmax_out (optional): 4-byte slot that receives max|C| (unsigned bit pattern, atomicMax) for the
// quantisation of C as the next affine's input.
// weights_settled: whatever may still be at work in front of the launch on its stream does not write the weight, so that the first of it is fetched in front of the
// kernel's wait.  Where the caller of the library orders the launches nobody knows that (a kernel that quantises a weight lets the next one start before it is done).
int launch_gemm(const int8_t* aq, const int8_t* bt, int M, int N, int K, const float* d_qa, const float* d_qb, float scale,
                const float* bias, int relu, void* c, int out_dtype, int32_t* acc_out, void* ws, size_t ws_bytes,
                cudaStream_t stream, int force_tile_m, int force_splits, unsigned* absmax_out = nullptr,
                const unsigned* skip_a = nullptr, const unsigned* skip_b = nullptr, int skip_rows_below = 0, bool weights_settled = false);

// The general form: one activation against up to three weight matrices of the same shape stored one behind the
// other (N = nseg * rows of one of them), each with its own multiplier, bias and output matrix [M, N / nseg].
constexpr int kBlockRows = 32;
struct GemmCall {
  const int8_t* aq = nullptr;
  const int8_t* bt = nullptr;
  int M = 0, N = 0, K = 0;
  const float* d_qa = nullptr;
  float scale = 1.0f;
  int relu = 0;
  int out_dtype = MI8_F32;
  int32_t* acc_out = nullptr;
  int nseg = 1;
  const float* seg_qb[3] = {nullptr, nullptr, nullptr};
  const float* seg_bias[3] = {nullptr, nullptr, nullptr};
  void* seg_c[3] = {nullptr, nullptr, nullptr};
  void* ws = nullptr;
  size_t ws_bytes = 0;
  cudaStream_t stream = nullptr;
  int force_tile_m = 0, force_splits = 0;
  unsigned* absmax_out = nullptr;
  const unsigned* skip_a = nullptr;
  const unsigned* skip_b = nullptr;
  int skip_rows_below = 0;
  // with the three above: the segments from the second on also take the skip_rows_below rows in front of their own (of the operand's buffer and of their results,
  // which continue there), unless the two words are equal.  Needs force_tile_m of 16 to 128.
  bool rows_below = false;
  // optional, up to kBlockRows rows of one fp32 result: per (row, block of 128 columns) the maximum and the sum of exponentials [M][ceil(N / 128)]
  float* block_max = nullptr;
  float* block_sum = nullptr;
  int a_rows_cap = 0;   // rows the activation buffer holds (extent of its tensor map); 0 = M
  int a_row0 = 0;       // the M rows start at this row of the buffer `aq` points to (needs a_rows_cap >= a_row0 + M)
  // per segment, where it differs: the first of its M activation rows (-1: a_row0) and their multiplier (null: d_qa)
  int seg_row0[3] = {-1, -1, -1};
  const float* seg_qa[3] = {nullptr, nullptr, nullptr};
  bool weights_settled = false;
};
int launch_gemm_call(const GemmCall& g);

// Test hook behind mi8_test_wait_fault (marian_i8_measure.h).
void test_wait_fault(int withhold_item, unsigned spin_limit);

// The GEMM that quantises its activation itself: `a_f32` [M,K] fp32 and `a_slot`, the 4-byte slot its
// producer reduced max|A| into.  MI8_ERR_UNSUPPORTED when the shape does not give every CTA exactly one
// tile (quant_a_tile() == 0): the caller then quantises with a kernel of its own and calls launch_gemm.
int quant_a_tile(int M, int N);
int launch_gemm_quant_a(const float* a_f32, const unsigned* a_slot, float* qa_out, const int8_t* bt, int M, int N, int K,
                        const float* d_qb, float scale, const float* bias, int relu, void* c, int out_dtype, int32_t* acc_out,
                        cudaStream_t stream, unsigned* absmax_out = nullptr, int8_t* aq_out = nullptr, bool weights_settled = false);
// ... and without a slot, where every CTA finds the maximum itself (aq_out: the quantised activation, M * K bytes).
bool quant_a_own_max(int M, int N, int K);

// The cluster GEMM for decode shapes: quantises the fp32 activation `a_f32` [M, K] itself with the multiplier of the abs-max
// slot `a_slot` (its CTAs share the quantised tile through distributed shared memory, so the fp32 values are read once
// per cluster), and with `ln` set writes LayerNorm(C + ln_resid) * ln_gamma + ln_beta (the arithmetic of
// add_layernorm_kernel, bit for bit) instead of C, with the row maxima and abs-max slots that kernel produces.
// gemm_cq_supported() says whether a shape can take this route (K a multiple of 128 up to 4096, N a multiple of 128;
// with `ln`: N <= 1024).
struct CqCall {
  const float* a_f32 = nullptr;
  const unsigned* a_slot = nullptr;
  float* qa_out = nullptr;
  const int8_t* bt = nullptr;
  const float* d_qb = nullptr;
  int M = 0, N = 0, K = 0;
  float scale = 1.0f;
  const float* bias = nullptr;
  int relu = 0;
  float* c = nullptr;
  unsigned* absmax_out = nullptr;
  int ln = 0;
  const float* ln_resid = nullptr;
  const float* ln_gamma = nullptr;
  const float* ln_beta = nullptr;
  float ln_eps = 0.0f;
  float* ln_out = nullptr;
  float* ln_rowmax = nullptr;
  unsigned* ln_slot = nullptr;
  unsigned* ln_slot2 = nullptr;
  cudaStream_t stream = nullptr;
  int force_tile_m = 0;     // 0 = chosen from M and N
  int force_cluster = 0;    // 0 = the largest of 8, 4, 2, 1 that divides N / 128 (ln: N / 128)
  bool weights_settled = false;
};
bool gemm_cq_supported(int M, int N, int K, bool ln);
int launch_gemm_cq(const CqCall& g);

// packed8avx512 scheme (mi8_packed8.cu, mi8_gemm.cu): weight item back to Bt[N,K]; per-row uint8 quantisation of
// the activation; uint8 x int8 GEMM whose write-back applies the zero points, the scales and the bias.  `segs`: several matrices of N / n columns
// each in the place of the one that the arguments name; block_max / block_sum: as in GemmCall.
constexpr int kMaxSegments = 3;
struct P8Segments {
  int n = 0;
  const int8_t* bt[kMaxSegments];
  const float* scale_b[kMaxSegments];
  const int32_t *zp_b[kMaxSegments], *off_b[kMaxSegments];
  const float* bias[kMaxSegments];
  float* c[kMaxSegments];
};
int launch_p8_prepare_b(const float* w, int K, int N, int8_t* packed, cudaStream_t stream);
int launch_p8_unpack_bt(const int8_t* packed, int K, int N, int8_t* bt, cudaStream_t stream);
int launch_p8_quantize_rows(const float* a, int M, int K, uint8_t* aq, float* scale_a, int32_t* zp_a, int32_t* sum_a, cudaStream_t stream, bool early = true);
int launch_gemm_p8(const uint8_t* aq, const float* scale_a, const int32_t* zp_a, const int32_t* sum_a, const int8_t* bt,
                   const float* scale_b, const int32_t* zp_b, const int32_t* off_b, int M, int N, int K, const float* bias, int relu,
                   float* c, int32_t* acc_out, void* ws, size_t ws_bytes, cudaStream_t stream, int force_tile_m, int force_splits,
                   const P8Segments* segs = nullptr, float* block_max = nullptr, float* block_sum = nullptr);

constexpr int kDecoderRowsMax = 32;   // rows of a step that launch_decoder_rows takes
// What the last kernel of a decoder step does besides the rows' candidates: the n-best lists of the sentences (arrivals != nullptr; one
// zeroed counter per sentence; the outputs may be pinned host memory) and the record of the history abs-max per layer (layers > 0).
struct StepEnd {
  int beam = 0, batch = 0;
  unsigned* arrivals = nullptr;
  float* out_score = nullptr;
  int* out_beam = nullptr;
  int* out_word = nullptr;
  int layers = 0, first = 0, stride = 0;
  const unsigned* slots = nullptr;
  unsigned* prev_bits = nullptr;
  unsigned* stats = nullptr;
  // A step whose successor is launched before the host has seen its n-best lists (mi8d_search, few rows): the control words of the successor, which are
  // those of the lists as long as no hypothesis ends - otherwise `next_stop` is set, and the successor does nothing.  hyps: hypotheses of each sentence that
  // are alive, of k.  stop: this step itself is such a successor.  tagged ([batch * k][2], in the place of the three lists): an entry's score and its
  // beam * vocab + word, each below `tag`, so that the host sees when a word is new.  With a successor they stay on the device and its first kernel brings
  // them to the host (DecoderRowsParams::lists): stores to the host held the end of this kernel, and with it the successor, up (student, one sentence: 9.0 us
  // with a fence and a flag behind them, 7.8 with tagged words alone, 6.9 so).
  int* next_ctrl = nullptr;   // hypothesis rows, previous words, path scores [k * batch] each, batch rows [batch]
  unsigned* next_stop = nullptr;
  const unsigned* stop = nullptr;
  unsigned long long* tagged = nullptr;
  unsigned tag = 0;
  int eos = 0;
  unsigned char hyps[kDecoderRowsMax] = {};
};
// Candidates of one sentence (beam x k) that the row kernels' shared memory holds; wider beams end with launch_nbest_merge.
constexpr int kStepEndCandidates = 1024;
constexpr bool step_end_fits(int beam, int k) { return beam <= kStepEndCandidates / k; }

// Output layer: GEMM whose write-back reduces every (row, block of 128 vocabulary entries) to its maximum, its sum
// of exponentials and its k_top (4 or 8) best entries (blk_* arrays: [rows][ceil(vocab/128)] (x k_top)); then
// launch_lse_merge turns those into the per-row candidates launch_lse_topk would have produced from the logits.
int launch_gemm_logits(const int8_t* aq, const float* d_qa, const int8_t* wq, const float* d_qw, int rows, int vocab, int K,
                       const float* bias, float scale, int k_top, float* blk_max, float* blk_sum, float* blk_topv, int* blk_topi,
                       float* logits_out, cudaStream_t stream);
int launch_lse_merge(const float* blk_max, const float* blk_sum, const float* blk_topv, const int* blk_topi, int rows, int vocab,
                     int k_top, int k, const float* prev_scores, float* cand_score, int* cand_word, cudaStream_t s, const StepEnd& end = StepEnd());

// decode-step glue (mi8_glue.cu)
int launch_embed(const float* wemb, const int* words, const float* pos, int pos_mod, float scale, int rows, int dim, float* out,
                 float* rowmax, unsigned* slot, cudaStream_t s);
// host_ctrl: pinned host memory; ctrl and host_ctrl 16-byte aligned, room for whole 16-byte vectors
int launch_step_begin(const int* host_ctrl, int* ctrl, int n_ctrl, unsigned* slots, int n_slots, cudaStream_t s);
// slot2 (optional): a second 4-byte slot that receives the same maximum (the self-attention history's abs-max)
int launch_add_layernorm(const float* a, const float* resid, const float* gamma, const float* beta, float eps, int rows, int dim,
                         float* out, float* rowmax, unsigned* slot, cudaStream_t s, unsigned* slot2 = nullptr);
// the same for few rows with the quantisation of the result (q, d_qm) in the same launch; cell_old != nullptr: the SSRU cell's output
// in the place of `a` (see launch_ssru_cell)
bool add_layernorm_quant_supported(int rows, int dim);
int launch_add_layernorm_quant(const float* a, const float* resid, const float* gamma, const float* beta, float eps, int rows, int dim, float* out,
                               int8_t* q, float* d_qm, cudaStream_t s, const float* cell_old = nullptr, const int* hyp = nullptr,
                               const float* xw = nullptr, const float* f = nullptr, float* cell_new = nullptr);
int launch_quantize_slot(const float* x, size_t n, const unsigned* slot, int8_t* q, float* d_qm, cudaStream_t s);
// Per sentence the distinct slab rows its hypotheses descend from (mi8_glue.cu, history_list); batch == 0: none.
struct HistLists {
  int batch = 0;
  int *list = nullptr, *which = nullptr, *count = nullptr;
};
// the embedding of a step (slot2: the history's abs-max of layer 0) and the ancestor table (and, optionally, the history lists); hist_layers > 0: also reduces, per layer, the
// maximum of rowmax over the earlier slabs' ancestor rows into hist_slot[l]
int launch_embed_ancestors(const float* wemb, const int* words, const float* pos, float scale, int dim, float* out, float* rowmax, unsigned* slot,
                           unsigned* slot2, const int* anc_old, int* anc_new, const int* hyp, int t, int rows, int stride, cudaStream_t s,
                           int hist_layers, const float* const* hist_rowmax, unsigned* const* hist_slot, const HistLists& lists = HistLists());
// decoder self-attention (mode 0 with an ancestor table) for all hypotheses of a sentence together, from the lists of this step
bool attention_hist_supported(int beams, int sentences, int dim_head, int len);
int launch_attention_hist(const float* q, const float* k, const float* v, int rows, int heads, int dim_head, int len, float* out, unsigned* slot,
                          cudaStream_t s, const HistLists& lists);
// layer input x and the self-attention history quantised by one launch (see quantize_dual_kernel)
int launch_quantize_dual(const float* x, size_t n, const unsigned* slot_x, int8_t* q, float* qm_x, const float* slabs, int slab_rows,
                         int steps, int rows_new, int dim, const unsigned* slot_h, const unsigned* prev_bits, int8_t* hq, float* qm_h,
                         cudaStream_t s);
void set_attention_unroll(int u);
void set_attention_block_heads(int h);
// in-situ timeline: each translation unit with kernels installs the buffer in its own copy of the pointer
int trace_set_glue(unsigned long long* buf);
int trace_set_gemm(unsigned long long* buf);
int trace_set_quant(unsigned long long* buf);
int launch_attention1(const float* q, const float* k, const float* v, const float* log_mask, int rows, int heads, int dim_head,
                      int len, int batch, int mode, float* out, unsigned* slot, cudaStream_t s, const int* anc = nullptr,
                      int anc_stride = 0, int kv_rows = 0);
// block_max / block_sum (optional, both): what GemmCall's write-back left of the rows' blocks, in the place of a scan of the logits
int launch_lse_topk(const float* logits, int rows, int vocab, int k, const float* prev_scores, float* cand_score, int* cand_word,
                    cudaStream_t s, const StepEnd& end = StepEnd(), const float* block_max = nullptr, const float* block_sum = nullptr);
int launch_nbest_merge(const float* cand_score, const int* cand_word, int beam, int batch, int vocab, int k, float* out_score,
                       int* out_beam, int* out_word, cudaStream_t s);
int launch_gather_rows(const float* in, const int* idx, int rows, int dim, float* out, cudaStream_t s);
int launch_ssru_cell(const float* cell_old, const int* hyp, const float* xw, const float* f, int rows, int dim, float* cell_new,
                     float* h_out, cudaStream_t s);

// The layers of an SSRU decoder's step for few rows in one launch (mi8_rows.cu).
constexpr int kDecoderRowsLayers = 4, kRowsMultipliers = 6;
// A layer's parameters apart from the matrices, read from here by every launch; 16-byte aligned but for the multipliers.
struct DecoderRowsVectors {
  const float* qb[kRowsMultipliers];   // multipliers of W, Wf, Wq, Wo, W1, W2
  const float* own[3];                 // biases of d columns that a CTA takes its share of: Wf's, Wo's, W2's
  const float *b_q, *b_1;
  const float* ln[6];                  // scale and bias behind the cell, the cross-attention, the feed-forward block
};
struct DecoderRowsParams {
  int rows = 0, ffn = 0, layers = 0, src = 0, batch = 0;
  float emb_scale = 0.f, att_scale = 0.f;
  const float *wemb = nullptr, *pos = nullptr, *log_mask = nullptr;
  // layer 0's; layer l's lie l * layer_stride floats behind
  const float *cross_k = nullptr, *cross_v = nullptr, *cell_old = nullptr;
  float* cell_new = nullptr;
  size_t layer_stride = 0;
  const int *words = nullptr, *hyp = nullptr;   // null: the first step
  int* ctrl = nullptr;
  int n_ctrl = 0, n_slots = 0;
  unsigned* slots = nullptr;    // zeroed
  const unsigned* stop = nullptr;   // optional: the launch does nothing where this word is set (StepEnd)
  unsigned* next_stop = nullptr;    // optional: zeroed
  const unsigned long long* lists = nullptr;   // optional: what the step in front left for the host (StepEnd::tagged), and where it goes
  unsigned long long* host_lists = nullptr;
  int n_lists = 0;
  int8_t* out_q = nullptr;      // [rows, d] the last LayerNorm's result, quantised, and its multiplier
  float* out_qm = nullptr;
  int* status = nullptr;
  int withhold_item = -1;       // (test hook, as in the GEMMs; `status`, these two and the next line are set by the launcher)
  uint32_t spin_limit = 0;
  int ring = 0, inv_mt_ffn1 = 0, inv_nf4 = 0, inv_batch = 0, inv_rows = 0;
  // n_ctrl > 0: the control words (hypothesis rows, previous words, path scores, batch rows), used from here and brought to `ctrl`
  int ctrl_words[4 * kDecoderRowsMax];
  DecoderRowsVectors vec[kDecoderRowsLayers];
  // per layer W above Wf, Wq, Wo, W1, W2: boxes of 16 rows x 128 bytes (rows_weight_map)
  CUtensorMap map[kDecoderRowsLayers][5];
};
static_assert(sizeof(DecoderRowsParams) <= 4096, "kernel parameters");
// What mi8_test_wait_fault asked for: the item whose loads are left out (-1: none; kWithholdWarp) and the bound of every wait.
constexpr int kWithholdWarp = MI8_TEST_ONE_WARP;
void test_wait_limits(int* withhold_item, uint32_t* spin_limit);
int rows_weight_map(CUtensorMap* map, const int8_t* bt, int N, int K);
bool decoder_rows_supported(int rows, int d, int f, int heads, int layers, int src);
// `params_settled`: what lies in front on the stream, as far as it has not completed when the launch is due, writes none of the registered parameters, which the kernel
// reads in front of its wait.  Otherwise the launch is not overlapped.
int launch_decoder_rows(DecoderRowsParams& p, int d, int heads, cudaStream_t stream, bool params_settled);
int trace_set_rows(unsigned long long* buf);

// Whether kernels are launched with programmatic dependent launch (mi8_set_pdl; on by default).
bool pdl_enabled();
void set_pdl(bool on);

// Per-kernel device times (mi8_kernel_times_begin / _end): when on, every launch made through launch_kernel by
// the calling thread is bracketed by CUDA events on its stream and attributed to the kernel function.
bool kernel_times_on();
void kernel_times_before(const void* func, cudaStream_t stream);
void kernel_times_after(cudaStream_t stream);

// Launches `kernel` with or without the programmatic-stream-serialization attribute.
template <typename... KArgs, typename... Args>
inline cudaError_t launch_kernel(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, Args&&... args) {
  if(kernel_times_on()) {
    kernel_times_before(reinterpret_cast<const void*>(kernel), stream);
    cudaLaunchConfig_t tcfg = {};
    tcfg.gridDim = grid;
    tcfg.blockDim = block;
    tcfg.dynamicSmemBytes = smem;
    tcfg.stream = stream;
    const cudaError_t te = cudaLaunchKernelEx(&tcfg, kernel, static_cast<KArgs>(args)...);   // no launch overlap while timing
    kernel_times_after(stream);
    return te;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl_enabled() ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
}

inline cudaStream_t as_stream(void* s) { return s ? reinterpret_cast<cudaStream_t>(s) : cudaStreamPerThread; }

}  // namespace mi8

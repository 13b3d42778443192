// Host-side driver of one decoder time step (declared in include/marian_i8_decode.h): sequences the
// int8 affines and the glue kernels on one stream, with all buffers carved out of a caller-owned
// arena.  Restates DecoderTransformer::step (src/models/transformer.h:713-896): per layer
// self-attention over the re-projected history (or the SSRU cell), cross-attention over cached
// encoder keys/values, the ReLU feed-forward block, each followed by residual add + LayerNorm
// ("transformer-postprocess: dan"), then the tied output layer, log-softmax and n-best selection.
// mi8d_search adds the beam-search bookkeeping around the step (BeamSearch::search,
// src/translator/beam_search.cpp:249-538), so a mini-batch is translated by one call.
#include <thread>
#include <algorithm>
#include <atomic>
#include <chrono>
#include <cmath>
#include <cstring>
#include <string>
#include <unordered_map>
#include <vector>

#include "../../include/marian_i8_decode.h"
#include "mi8_internal.h"
#include "mi8_tagged.h"

namespace mi8 {
namespace {

struct Weight {
  const int8_t* bt = nullptr;
  int K = 0, N = 0;
  const float* qm() const { return reinterpret_cast<const float*>(bt + static_cast<size_t>(K) * N); }
};

// One affine as the step loop uses it: everything resolved to pointers once (no name lookups per step).
struct Aff {
  const int8_t* bt = nullptr;
  const float* qm = nullptr;       // intgemm8: the weight's multiplier
  const float* bias = nullptr;
  int K = 0, N = 0;
  // packed8avx512: per-column scale, zero point and column offset instead of one multiplier
  bool p8 = false;
  const float* scale_b = nullptr;
  const int32_t* zp_b = nullptr;
  const int32_t* off_b = nullptr;
};
struct P8Weight {
  const int8_t* bt = nullptr;
  const float* scale_b = nullptr;
  const int32_t* zp_b = nullptr;
  const int32_t* off_b = nullptr;
  int K = 0, N = 0;
};
// Several weights of the same shape multiplied with the same activation in one launch (Wk|Wv, Wq|Wk|Wv,
// the SSRU's W|Wf): their int8 matrices copied one behind the other into the arena.  packed8avx512 matrices stay where they were registered.
struct Fused {
  int8_t* bt = nullptr;   // intgemm8: [nseg * n, K] in the arena
  int nseg = 0, n = 0, K = 0;
  const float* qm[3] = {nullptr, nullptr, nullptr};
  const float* bias[3] = {nullptr, nullptr, nullptr};
  P8Segments p8;          // packed8avx512; the outputs are the caller's
  bool ready = false;
};
struct Norm {
  const float* g = nullptr;
  const float* b = nullptr;
};
struct EncLayerW {
  Aff q, k, v, o, w1, w2;
  Fused qkv;
  Norm ln_att, ln_ffn;
};
struct DecLayerW {
  Aff self_q, self_k, self_v, self_o, rnn_w, rnn_wf, ctx_q, ctx_k, ctx_v, ctx_o, w1, w2;
  Fused self_qkv, rnn, ctx_kv;
  Norm ln_self, ln_ctx, ln_ffn;
};

size_t align_up(size_t v, size_t a = 256) { return (v + a - 1) / a * a; }

struct Arena {
  uint8_t* base = nullptr;
  size_t size = 0, used = 0;
  template <typename T>
  T* take(size_t count) {
    size_t bytes = align_up(count * sizeof(T));
    T* p = base ? reinterpret_cast<T*>(base + used) : nullptr;
    used += bytes;
    return p;
  }
};

struct LayerBufs {
  float* slab = nullptr;     // [max_steps][slab_rows][d]  layer inputs (self-attention decoders), row order of each step
  float* rowmax = nullptr;   // [max_steps][slab_rows]     max|x| per slab row
  float* kslab = nullptr;    // [max_steps][slab_rows][d]  projected keys / values of the slabs, valid for the
  float* vslab = nullptr;    //                            history abs-max remembered in prev_bits
  int8_t* hq = nullptr;      // [max_steps][slab_rows][d]  quantised slabs, then [max_rows][d] the newest slab with the multiplier of
                             // its own (the query projection's operand), then both multipliers (history's, own)
  float* cross_k = nullptr;  // [max_batch * max_src, d]
  float* cross_v = nullptr;
  float* cell[2] = {nullptr, nullptr};  // SSRU state, double-buffered [max_rows, d]
};

// Slots of the per-step abs-max array: slot 0 belongs to the embedding (input of layer 0), then eight per layer.
enum LayerSlot { kSlotSelfLn = 0, kSlotHistory, kSlotSelfAtt, kSlotCtxAtt, kSlotCtxLn, kSlotRelu, kSlotOut, kSlotsPerLayer = 8 };

}  // namespace
}  // namespace mi8

using namespace mi8;

struct mi8d_decoder {
  mi8d_config cfg;
  Arena arena;
  void* ws = nullptr;
  size_t ws_bytes = 0;
  std::unordered_map<std::string, Weight> weights;
  std::unordered_map<std::string, P8Weight> p8_weights;   // packed8avx512 model: every affine's weight is registered here instead
  bool p8 = false;
  std::unordered_map<std::string, const float*> params;
  const float* positions = nullptr;
  // resolved model (rebuilt by resolve() after a parameter was registered)
  bool dirty = true;
  bool can_fuse = false;              // dim_emb is a multiple of 128: a weight tile never straddles two fused matrices
  std::vector<EncLayerW> enc_w;
  std::vector<DecLayerW> dec_w;
  const float* wemb = nullptr;
  const float* out_bias = nullptr;
  Aff out_w;
  std::vector<int8_t*> fused_enc, fused_self, fused_ctx;   // arena storage of the fused matrices
  DecoderRowsParams rows;             // for launch_decoder_rows: what does not change from step to step is filled in by resolve()
  bool rows_ready = false;

  std::vector<LayerBufs> layers;
  float* x_in = nullptr;                 // layer-0 input when there are no slabs (SSRU) and the final layer output
  float* x_final = nullptr;
  float *x1 = nullptr, *x2 = nullptr;    // after self / cross blocks
  float *qbuf = nullptr, *abuf = nullptr, *obuf = nullptr, *hbuf = nullptr, *fbuf = nullptr;
  int8_t *aq = nullptr, *cq = nullptr;
  HistLists lists;                 // of the running step; `batch` is set where they are used
  unsigned* prev_bits = nullptr;   // per layer: history abs-max (bit pattern) the stored keys/values were computed with
  unsigned* reuse_stats = nullptr; // [0] (layer, step) pairs that reused stored keys/values, [1] all pairs
  int slab_rows = 0;               // rows reserved per history slab for the current mini-batch
  float* logits = nullptr;
  float* cand_score = nullptr;
  int* cand_word = nullptr;
  float* enc_x[2] = {nullptr, nullptr};
  float *enc_q = nullptr, *enc_k = nullptr, *enc_v = nullptr, *enc_h = nullptr;
  int8_t* enc_aq = nullptr;
  float* context[2] = {nullptr, nullptr};
  float* log_mask[2] = {nullptr, nullptr};
  int* anc[2] = {nullptr, nullptr};
  // beam-search bookkeeping (mi8d_search): per-step control words and n-best lists, device side and pinned host side
  int* s_ctrl[2] = {nullptr, nullptr};   // [3 * max_rows + max_batch]: hypothesis rows, previous words, path scores (as bits), batch rows; steps in turn
  int* h_ctrl = nullptr;            // pinned; read by the step's first kernel
  int* h_out = nullptr;             // pinned, [2][3][max_batch * 8]: scores (as bits), beams, words, written by the step's last kernel; steps in turn
  unsigned long long* h_tagged = nullptr;   // pinned, [2][kDecoderRowsMax * 2]: StepEnd::tagged; steps in turn
  unsigned* stops = nullptr;        // [2] StepEnd::next_stop
  unsigned long long* s_tagged = nullptr;   // [2][kDecoderRowsMax * 2] the same on the device, on its way through the step behind
  unsigned tag = 0;
  float *blk_max = nullptr, *blk_sum = nullptr, *blk_topv = nullptr;   // per (row, 128-word block) partials of the output layer
  int* blk_topi = nullptr;
  bool keep_logits = false;
  const int* step_ctrl = nullptr;   // set by mi8d_search around a step: pinned control words to bring to s_ctrl first, and how many
  int n_step_ctrl = 0;
  unsigned* slots = nullptr;
  int n_slots = 0;
  // packed8avx512: scale, zero point and sum of every row of the activation quantised last
  float* p8_scale_a = nullptr;
  int32_t *p8_zp_a = nullptr, *p8_sum_a = nullptr;
  // Re-projecting the keys/values of the EARLIER history slabs (needed only when the history's abs-max changed) does
  // not depend on the query projection: it runs on an internal stream, forked from and joined to the caller's
  // stream with events, beside the query projection and the newest slab's keys/values.
  cudaStream_t side = nullptr;
  cudaEvent_t ev_fork = nullptr, ev_join = nullptr;
  cudaEvent_t ev_step = nullptr;   // blocking-sync event: the host thread sleeps instead of spinning while a step runs (opt_blocking_wait)
  int opt_blocking_wait = 0;
  bool overlap = false;
  // tuning switches (mi8d_set_option)
  int opt_fuse = 1, opt_quant_in_gemm = 0, opt_fused_out_rows = 0, opt_side_stream = 1, opt_shared_history = 1, opt_one_launch_rows = kDecoderRowsMax, opt_step_ahead = 1;
  int opt_gemm_tile = 0;
  int opt_cluster = 0, opt_fused_ln = 1, opt_cluster_max_rows = 1024, opt_cluster_size = 0, opt_cluster_max_k = 2048;
  // host-side timing of mi8d_search
  double t_issue = 0, t_wait = 0, t_host = 0, n_steps = 0;

  int t = 0, batch = 0, src = 0, ctx_cur = 0, anc_cur = 0, cell_cur = 0;
  bool cross_valid = false;

  // lays the arena out; with a null base it only measures
  void layout() {
    const mi8d_config& c = cfg;
    const size_t d = c.dim_emb, f = c.dim_ffn, R = c.max_rows, T = c.max_steps, B = c.max_batch, S = c.max_src;
    arena.used = 0;
    layers.assign(c.dec_depth, LayerBufs());
    for(auto& L : layers) {
      if(!c.ssru) {
        L.slab = arena.take<float>(T * R * d);
        L.rowmax = arena.take<float>(T * R);
        L.kslab = arena.take<float>(T * R * d);
        L.vslab = arena.take<float>(T * R * d);
        L.hq = arena.take<int8_t>((T + 1) * R * d + 256);
      } else {
        L.cell[0] = arena.take<float>(R * d);
        L.cell[1] = arena.take<float>(R * d);
      }
      L.cross_k = arena.take<float>(B * S * d);
      L.cross_v = arena.take<float>(B * S * d);
    }
    x_in = arena.take<float>(R * d);
    x_final = arena.take<float>(R * d);
    x1 = arena.take<float>(R * d);
    x2 = arena.take<float>(R * d);
    qbuf = arena.take<float>(R * d);
    abuf = arena.take<float>(R * d);
    obuf = arena.take<float>(R * d);
    fbuf = arena.take<float>(R * d);
    hbuf = arena.take<float>(R * f);
    aq = arena.take<int8_t>(R * (f > d ? f : d) + 256);
    if(!c.ssru) {
      anc[0] = arena.take<int>(T * R);
      anc[1] = arena.take<int>(T * R);
      lists.list = arena.take<int>(T * R);
      lists.which = arena.take<int>(T * R);
      lists.count = arena.take<int>(B);
      prev_bits = arena.take<unsigned>(c.dec_depth);
      reuse_stats = arena.take<unsigned>(2);
    }
    cq = arena.take<int8_t>(B * S * d + 256);
    logits = arena.take<float>(R * static_cast<size_t>(c.vocab));
    const size_t nb = (static_cast<size_t>(c.vocab) + 127) / 128;
    blk_max = arena.take<float>(R * nb);
    blk_sum = arena.take<float>(R * nb);
    blk_topv = arena.take<float>(R * nb * 8);
    blk_topi = arena.take<int>(R * nb * 8);
    for(int*& ctrl : s_ctrl)
      ctrl = arena.take<int>(3 * R + B);   // (the arena rounds every array up to 256 bytes)
    stops = arena.take<unsigned>(2);
    s_tagged = arena.take<unsigned long long>(4 * kDecoderRowsMax);
    cand_score = arena.take<float>(R * 8);
    cand_word = arena.take<int>(R * 8);
    for(int i = 0; i < 2; ++i) {
      context[i] = arena.take<float>(B * S * d);
      log_mask[i] = arena.take<float>(B * S);
    }
    if(c.enc_depth > 0) {
      const size_t M = B * S;
      for(int i = 0; i < 2; ++i)
        enc_x[i] = arena.take<float>(M * d);
      enc_q = arena.take<float>(M * d);
      enc_k = arena.take<float>(M * d);
      enc_v = arena.take<float>(M * d);
      enc_h = arena.take<float>(M * f);
      enc_aq = arena.take<int8_t>(M * (f > d ? f : d) + 256);
    }
    n_slots = kSlotsPerLayer * c.dec_depth + 8 + 4 * c.enc_depth + c.max_batch;
    slots = arena.take<unsigned>(n_slots);
    const size_t max_act_rows = R > B * S ? R : B * S;
    p8_scale_a = arena.take<float>(max_act_rows);
    p8_zp_a = arena.take<int32_t>(max_act_rows);
    p8_sum_a = arena.take<int32_t>(max_act_rows);
    // storage of the fused weight matrices (copies of the registered int8 matrices, made once by resolve())
    can_fuse = d % 128 == 0;
    fused_enc.assign(c.enc_depth, nullptr);
    fused_self.assign(c.dec_depth, nullptr);
    fused_ctx.assign(c.dec_depth, nullptr);
    if(can_fuse) {
      for(auto& p : fused_enc)
        p = arena.take<int8_t>(3 * d * d);
      for(auto& p : fused_self)
        p = arena.take<int8_t>((c.ssru ? 2 : 3) * d * d);
      for(auto& p : fused_ctx)
        p = arena.take<int8_t>(2 * d * d);
    }
  }

  unsigned* layer_slot(int l, int which) const { return slots + 1 + kSlotsPerLayer * l + which; }
  unsigned* arrivals() const { return slots + n_slots - cfg.max_batch; }   // per sentence: rows whose candidates are ready
  unsigned* input_slot(int l) const { return l == 0 ? slots : layer_slot(l - 1, kSlotOut); }
  unsigned* enc_slot(int l, int which) const { return slots + 1 + kSlotsPerLayer * cfg.dec_depth + 4 * l + which; }

  const Weight* W(const std::string& name) const {
    auto it = weights.find(name);
    return it == weights.end() ? nullptr : &it->second;
  }
  const float* P(const std::string& name) const {
    auto it = params.find(name);
    return it == params.end() ? nullptr : it->second;
  }
  bool aff(Aff& a, const std::string& wname, const std::string& bname) const {
    a = Aff();
    if(p8) {
      auto it = p8_weights.find(wname);
      if(it == p8_weights.end())
        return false;
      a.p8 = true;
      a.bt = it->second.bt;
      a.scale_b = it->second.scale_b;
      a.zp_b = it->second.zp_b;
      a.off_b = it->second.off_b;
      a.K = it->second.K;
      a.N = it->second.N;
    } else {
      const Weight* w = W(wname);
      if(w == nullptr)
        return false;
      a.bt = w->bt;
      a.qm = w->qm();
      a.K = w->K;
      a.N = w->N;
    }
    a.bias = nullptr;
    if(!bname.empty()) {
      a.bias = P(bname);
      if(a.bias == nullptr)
        return false;
    }
    return true;
  }
  bool norm(Norm& n, const std::string& prefix) const {
    n.g = P(prefix + "_ln_scale");
    n.b = P(prefix + "_ln_bias");
    return n.g != nullptr && n.b != nullptr;
  }
  // puts `parts` together; intgemm8: copies the matrices one behind the other into `store` (stream-ordered on s)
  bool fuse(Fused& f, int8_t* store, std::initializer_list<const Aff*> parts, cudaStream_t s) {
    f = Fused();
    if(store == nullptr)
      return true;   // not fusable for this model: the step falls back to one launch per matrix
    int i = 0;
    for(const Aff* a : parts) {
      if(i == 0) {
        f.n = a->N;
        f.K = a->K;
      } else if(a->N != f.n || a->K != f.K) {
        return true;
      }
      if(p8) {
        f.p8.bt[i] = a->bt;
        f.p8.scale_b[i] = a->scale_b;
        f.p8.zp_b[i] = a->zp_b;
        f.p8.off_b[i] = a->off_b;
        f.p8.bias[i] = a->bias;
      } else if(cudaMemcpyAsync(store + static_cast<size_t>(i) * f.n * f.K, a->bt, static_cast<size_t>(f.n) * f.K, cudaMemcpyDeviceToDevice, s) !=
                cudaSuccess) {
        return false;
      }
      f.qm[i] = a->qm;
      f.bias[i] = a->bias;
      ++i;
    }
    f.bt = store;
    f.nseg = f.p8.n = i;
    f.ready = f.n % 128 == 0;
    return true;
  }

  // What launch_decoder_rows needs of the layers, where all of them have it (an SSRU decoder whose W and Wf lie one behind the other).
  void resolve_rows() {
    const mi8d_config& c = cfg;
    rows_ready = false;
    if(!c.ssru || p8 || c.dec_depth > kDecoderRowsLayers)
      return;
    const int dm = c.dim_emb, f = c.dim_ffn;
    for(int l = 0; l < c.dec_depth; ++l) {
      const DecLayerW& w = dec_w[l];
      auto shape = [](const Aff& a, int K, int N) { return a.K == K && a.N == N && a.bias != nullptr; };
      if(!w.rnn.ready || w.rnn.n != dm || w.rnn.K != dm || w.rnn.bias[0] != nullptr || w.rnn.bias[1] == nullptr || !shape(w.ctx_q, dm, dm) ||
         !shape(w.ctx_o, dm, dm) || !shape(w.w1, dm, f) || !shape(w.w2, f, dm))
        return;
      CUtensorMap* m = rows.map[l];
      if(rows_weight_map(m, w.rnn.bt, 2 * dm, dm) != MI8_OK || rows_weight_map(m + 1, w.ctx_q.bt, dm, dm) != MI8_OK ||
         rows_weight_map(m + 2, w.ctx_o.bt, dm, dm) != MI8_OK || rows_weight_map(m + 3, w.w1.bt, f, dm) != MI8_OK ||
         rows_weight_map(m + 4, w.w2.bt, dm, f) != MI8_OK)
        return;
      DecoderRowsVectors& v = rows.vec[l];
      v = DecoderRowsVectors{{w.rnn.qm[0], w.rnn.qm[1], w.ctx_q.qm, w.ctx_o.qm, w.w1.qm, w.w2.qm}, {w.rnn.bias[1], w.ctx_o.bias, w.w2.bias},
                             w.ctx_q.bias, w.w1.bias, {w.ln_self.g, w.ln_self.b, w.ln_ctx.g, w.ln_ctx.b, w.ln_ffn.g, w.ln_ffn.b}};
      const float* copied[] = {v.own[0], v.own[1], v.own[2], v.b_q, v.b_1, v.ln[0], v.ln[1], v.ln[2], v.ln[3], v.ln[4], v.ln[5]};
      for(const float* x : copied)   // (the launch copies them 16 bytes at a time; the general route reads biases word by word)
        if(reinterpret_cast<uintptr_t>(x) & 15u)
          return;
    }
    rows_ready = true;
  }

  // Looks every parameter up once and builds the fused matrices.  MI8_ERR_BAD_ARG names a missing parameter.
  int resolve(cudaStream_t s) {
    const mi8d_config& c = cfg;
    enc_w.assign(c.enc_depth, EncLayerW());
    dec_w.assign(c.dec_depth, DecLayerW());
    bool ok = true, copies = true;
    for(int l = 0; l < c.enc_depth; ++l) {
      EncLayerW& e = enc_w[l];
      const std::string pre = "encoder_l" + std::to_string(l + 1) + "_self", ffn = "encoder_l" + std::to_string(l + 1) + "_ffn";
      ok = ok && aff(e.q, pre + "_Wq", pre + "_bq") && aff(e.k, pre + "_Wk", pre + "_bk") && aff(e.v, pre + "_Wv", pre + "_bv") &&
           aff(e.o, pre + "_Wo", pre + "_bo") && aff(e.w1, ffn + "_W1", ffn + "_b1") && aff(e.w2, ffn + "_W2", ffn + "_b2") &&
           norm(e.ln_att, pre + "_Wo") && norm(e.ln_ffn, ffn + "_ffn");
      if(ok)
        copies = copies && fuse(e.qkv, fused_enc[l], {&e.q, &e.k, &e.v}, s);
    }
    for(int l = 0; l < c.dec_depth && ok; ++l) {
      DecLayerW& w = dec_w[l];
      const std::string li = "decoder_l" + std::to_string(l + 1);
      if(c.ssru) {
        const std::string pre = li + "_rnn";
        ok = ok && aff(w.rnn_w, pre + "_W", "") && aff(w.rnn_wf, pre + "_Wf", pre + "_bf") && norm(w.ln_self, pre + "_ffn");
        if(ok)
          copies = copies && fuse(w.rnn, fused_self[l], {&w.rnn_w, &w.rnn_wf}, s);
      } else {
        const std::string pre = li + "_self";
        ok = ok && aff(w.self_q, pre + "_Wq", pre + "_bq") && aff(w.self_k, pre + "_Wk", pre + "_bk") &&
             aff(w.self_v, pre + "_Wv", pre + "_bv") && aff(w.self_o, pre + "_Wo", pre + "_bo") && norm(w.ln_self, pre + "_Wo");
        if(ok)
          copies = copies && fuse(w.self_qkv, fused_self[l], {&w.self_q, &w.self_k, &w.self_v}, s);
      }
      const std::string pre = li + "_context", ffn = li + "_ffn";
      ok = ok && aff(w.ctx_q, pre + "_Wq", pre + "_bq") && aff(w.ctx_k, pre + "_Wk", pre + "_bk") && aff(w.ctx_v, pre + "_Wv", pre + "_bv") &&
           aff(w.ctx_o, pre + "_Wo", pre + "_bo") && norm(w.ln_ctx, pre + "_Wo") && aff(w.w1, ffn + "_W1", ffn + "_b1") &&
           aff(w.w2, ffn + "_W2", ffn + "_b2") && norm(w.ln_ffn, ffn + "_ffn");
      if(ok)
        copies = copies && fuse(w.ctx_kv, fused_ctx[l], {&w.ctx_k, &w.ctx_v}, s);
    }
    if(ok)
      resolve_rows();
    wemb = P("Wemb");
    ok = ok && wemb != nullptr && aff(out_w, p8 ? "Wemb_packed8" : "Wemb_intgemm8", "decoder_ff_logit_out_b");
    out_bias = out_w.bias;
    if(!ok)
      return MI8_ERR_BAD_ARG;
    if(!copies) {
      set_last_cuda_error(cudaGetLastError());
      return MI8_ERR_LAUNCH;
    }
    dirty = false;
    return MI8_OK;
  }
};

namespace {

#define MI8D_CUDA(expr)               \
  do {                                \
    cudaError_t ce_ = (expr);         \
    if(ce_ != cudaSuccess) {          \
      set_last_cuda_error(ce_);       \
      return MI8_ERR_LAUNCH;          \
    }                                 \
  } while(0)

#define MI8D_TRY(expr)      \
  do {                      \
    int rc_ = (expr);       \
    if(rc_ != MI8_OK)       \
      return rc_;           \
  } while(0)

// MI8D_OPT_GEMM_TILE_ROWS: the widest tile up to the option's value that M still fills more than half of (512 = the
// CTA-pair kernel, for more than 256 rows); 0 = leave the choice to the plan.
int wide_tile(const mi8d_decoder* d, int M) {
  int t = d->opt_gemm_tile;
  if(t <= 0 || M <= 16 || M > 1024)   // (encoder-sized products already fill the GPU: the plan's two-CTA kernel is the fastest there)
    return 0;
  if(t == 512 && M <= 256)
    t = 256;
  while(t > 32 && M <= t / 2)
    t >>= 1;
  return t;
}

// The driver's products may fetch their weights in front of their wait: an encoder begins with a copy, a step with a kernel that lets the next one start behind its own
// wait (a step in one launch sees to itself, launch_decoder_rows), so that all a caller has put in front has completed, and the driver's kernels write no weight.
constexpr bool kOwnChain = true;

// Few rows: 16-row tiles for up to 64 of them, where that is one wave of CTAs (the plan takes the smallest tile that holds all rows), and inner dimensions of up
// to 2048 unsplit (the plan splits 2048).  A tile's operands, MMAs and write-back are then the shortest, and the split path's fence, atomics and counter cost more
// than eight K blocks.  Whole mini-batches, the plan / 16-row tiles / those and no splits: transformer-base, 4 x beam 4 13.5 / 13.5 / 13.25 ms, 10 x 4 15.0 /
// 14.5 / 14.4, 16 x 4 15.5 / 14.95 / 14.75; transformer-big, 10 x 4 17.25 / 16.75 / 16.75, 16 x 4 17.2 / 16.9 / 16.9; student, 40 sentences 4.95 / 4.8 / 4.8.
// (32-row tiles: 10 x 4 14.55 and 16.95.  No splits of 4096: transformer-big, 4 x 4 15.3 -> 15.8.)
constexpr int kNarrowRows = 64, kUnsplitK = 2048;
int narrow_tile(int M, int N) {
  return M > 16 && M <= kNarrowRows && static_cast<long long>((N + 127) / 128) * ((M + 15) / 16) <= sm_count() ? 16 : 0;
}
int few_rows_splits(int M, int K) { return M <= kNarrowRows && K <= kUnsplitK ? 1 : 0; }

// The tile of the launch that projects a step's newest history slab and, when the history's abs-max changed, the earlier slabs as well (GemmCall::rows_below), or 0
// for a launch of their own beside it (`below`: floats of the earlier slabs).  Together as long as the earlier slabs are short: the launch has one tile width, which
// the newest slab wants narrow and they want wide, and a launch of their own runs beside the newest slab's.  They are what a beam's reordering changes often and what
// one hypothesis per sentence rarely does, so that its tiles are those of the newest slab.  Whole mini-batches, apart / together up to 2 M / 4 M / any number of
// floats, ms: transformer-base, 4 x beam 4 (40 words) 25.5 / 23.8 / 23.8 / 23.9, 20 x 4 28.0 / 27.5 / 27.5 / 27.9, 64 x 4 30.4 / 30.4 / 30.4 / 31.3, 30 x 6 25.8 /
// 25.6 / 26.1 / 26.9, 64 x 1 29.2 / 27.6 / 27.6 / 27.7; transformer-big, 16 x 4 16.95 / 16.6 / 16.5 / 16.7, 60 x 4 21.9 / 21.75 / 21.6 / 21.4, 128 x 4 39.1 /
// 39.05 / 38.9 / 39.35, 20 x 1 16.1 / 15.1 / 15.1 / 15.2, 60 x 1 32.6 / 31.65 / 31.1 / 31.0.  Tiles of 16 / 32 / 64 / 128 rows: base, 4 x 4 13.3 / 12.9 / 12.9 / -,
// 20 x 4 15.8 / 15.7 / 15.6 / 15.4, 64 x 1 14.6 / 15.2 / 15.3 / -.  Not on a GPU that several searches share: the launch has a CTA on every SM.
int below_tile(int rows, int beam, size_t below) {
  if(rows > 512 || below > (beam == 1 ? size_t{4} << 20 : size_t{2} << 20))
    return 0;
  if(beam == 1)
    return rows <= 64 ? 16 : rows <= 128 ? 32 : 64;
  return rows <= 64 ? 64 : 128;
}

// aq (already quantised, multiplier behind the data) x weight -> c
int gemm(mi8d_decoder* d, const int8_t* a, int M, const Aff& w, bool relu, float* c, cudaStream_t s, unsigned* absmax_out = nullptr,
         int force_splits = 0, int force_tile_m = 0) {
  const float* qa = reinterpret_cast<const float*>(a + static_cast<size_t>(M) * w.K);
  if(force_tile_m == 0 && w.N <= 8192 && wide_tile(d, M) != 0) {
    // several searches share the GPU: wider tiles on fewer SMs fetch every weight tile fewer times (throughput over latency)
    force_tile_m = wide_tile(d, M);
    force_splits = 1;
  }
  if(force_tile_m == 0)
    force_tile_m = narrow_tile(M, w.N);
  if(force_splits == 0 && w.N <= 8192)
    force_splits = few_rows_splits(M, w.K);
  return launch_gemm(a, w.bt, M, w.N, w.K, qa, w.qm, 1.0f, w.bias, relu ? 1 : 0, c, MI8_F32, nullptr, d->ws, d->ws_bytes, s, force_tile_m,
                     force_splits, absmax_out, nullptr, nullptr, 0, kOwnChain);
}

// M rows of `a` against the matrices [first, last) of a fused group, one launch; outputs and the activation's details are the caller's
GemmCall fused_call(mi8d_decoder* d, const int8_t* a, const Fused& f, int M, int first, int last, int a_rows_cap, cudaStream_t s) {
  GemmCall g;
  g.aq = a;
  g.bt = f.bt + static_cast<size_t>(first) * f.n * f.K;
  g.M = M;
  g.N = (last - first) * f.n;
  g.K = f.K;
  g.nseg = last - first;
  for(int i = first; i < last; ++i) {
    g.seg_qb[i - first] = f.qm[i];
    g.seg_bias[i - first] = f.bias[i];
  }
  g.ws = d->ws;
  g.ws_bytes = d->ws_bytes;
  g.stream = s;
  g.a_rows_cap = a_rows_cap;
  g.weights_settled = kOwnChain;
  g.force_tile_m = narrow_tile(M, g.N);
  g.force_splits = few_rows_splits(M, f.K);
  return g;
}

// the same activation against all matrices of a fused group; outs[i] receives [M, f.n].  (packed8avx512, a launch per matrix before: transformer-base,
// 16 sentences x beam 4 19.4 -> 17.2 ms a mini-batch, transformer-big, 8 x 4 20.6 -> 18.4, student, 4 x 4 5.7 -> 5.2.)
int gemm_fused(mi8d_decoder* d, const int8_t* a, const float* qa, int M, const Fused& f, float* const* outs, cudaStream_t s) {
  if(d->p8) {
    P8Segments segs = f.p8;
    std::copy(outs, outs + f.nseg, segs.c);
    return launch_gemm_p8(reinterpret_cast<const uint8_t*>(a), d->p8_scale_a, d->p8_zp_a, d->p8_sum_a, nullptr, nullptr, nullptr, nullptr, M,
                          f.nseg * f.n, f.K, nullptr, 0, nullptr, nullptr, d->ws, d->ws_bytes, s, narrow_tile(M, f.nseg * f.n), few_rows_splits(M, f.K), &segs);
  }
  GemmCall g = fused_call(d, a, f, M, 0, f.nseg, 0, s);
  g.d_qa = qa;
  for(int i = 0; i < f.nseg; ++i)
    g.seg_c[i] = outs[i];
  return launch_gemm_call(g);
}

// The activation quantisation of either scheme into `q`: intgemm8 - Int8::PrepareA with the multiplier 127 / max|x| from the
// slot the producer reduced (stored behind the data); packed8avx512 - uint8 per row with its own scale, zero point and sum
// (src/tensors/cpu/mjdgemm/mjdgemm_avx512.cpp:195-276), kept in the decoder's per-row arrays until the next quantisation.
int quantize_act(mi8d_decoder* d, const float* x, int M, int K, const unsigned* slot, int8_t* q, cudaStream_t s) {
  if(d->p8)
    return launch_p8_quantize_rows(x, M, K, reinterpret_cast<uint8_t*>(q), d->p8_scale_a, d->p8_zp_a, d->p8_sum_a, s, false);
  return launch_quantize_slot(x, static_cast<size_t>(M) * K, slot, q, reinterpret_cast<float*>(q + static_cast<size_t>(M) * K), s);
}

// ... and the product of that quantised activation with one weight
int gemm_act(mi8d_decoder* d, const int8_t* q, int M, const Aff& w, bool relu, float* c, cudaStream_t s, unsigned* absmax_out = nullptr,
             int force_splits = 0) {
  if(w.p8)
    return launch_gemm_p8(reinterpret_cast<const uint8_t*>(q), d->p8_scale_a, d->p8_zp_a, d->p8_sum_a, w.bt, w.scale_b, w.zp_b, w.off_b, M, w.N,
                          w.K, w.bias, relu ? 1 : 0, c, nullptr, d->ws, d->ws_bytes, s, narrow_tile(M, w.N),
                          force_splits != 0 || w.N > 8192 ? force_splits : few_rows_splits(M, w.K));
  return gemm(d, q, M, w, relu, c, s, absmax_out, force_splits);
}

// Int8::PrepareA of x (multiplier from the slot its producer reduced) followed by the affine: either the
// quantisation kernel and the GEMM, or - with the option set and a shape that gives every CTA one tile - the GEMM
// that quantises its operand while loading it.
// `ready`: d->aq already holds the quantised x (see ln_quantises).
int quant_gemm(mi8d_decoder* d, const float* x, int M, const unsigned* slot, const Aff& w, bool relu, float* c, cudaStream_t s,
               unsigned* absmax_out = nullptr, bool ready = false) {
  if(ready)
    return gemm_act(d, d->aq, M, w, relu, c, s, absmax_out);
  float* qa = reinterpret_cast<float*>(d->aq + static_cast<size_t>(M) * w.K);
  if(!w.p8 && d->opt_cluster && M <= d->opt_cluster_max_rows && w.K <= d->opt_cluster_max_k && gemm_cq_supported(M, w.N, w.K, false)) {
    // the cluster GEMM: the CTAs of neighbouring weight tiles quantise the activation tile together (one launch, no int8 copy)
    CqCall g;
    g.a_f32 = x;
    g.a_slot = slot;
    g.bt = w.bt;
    g.d_qb = w.qm;
    g.M = M;
    g.N = w.N;
    g.K = w.K;
    g.bias = w.bias;
    g.relu = relu ? 1 : 0;
    g.c = c;
    g.absmax_out = absmax_out;
    g.weights_settled = kOwnChain;
    g.force_cluster = d->opt_cluster_size;
    g.stream = s;
    return launch_gemm_cq(g);
  }
  if(!w.p8 && d->opt_quant_in_gemm && w.K <= 1024 && quant_a_tile(M, w.N) != 0)
    return launch_gemm_quant_a(x, slot, qa, w.bt, M, w.N, w.K, w.qm, 1.0f, w.bias, relu ? 1 : 0, c, MI8_F32, nullptr, s, absmax_out, nullptr, kOwnChain);
  MI8D_TRY(quantize_act(d, x, M, w.K, slot, d->aq, s));
  return gemm_act(d, d->aq, M, w, relu, c, s, absmax_out);
}

int add_ln(mi8d_decoder* d, const float* a, const float* resid, const Norm& n, int rows, float* out, float* rowmax, unsigned* slot,
           cudaStream_t s, unsigned* slot2 = nullptr) {
  return launch_add_layernorm(a, resid, n.g, n.b, 1e-6f, rows, d->cfg.dim_emb, out, rowmax, slot, s, slot2);
}

// Whether a LayerNorm of `rows` rows whose result only feeds affines of its own multiplier also quantises it (into d->aq / enc_aq).
bool ln_quantises(const mi8d_decoder* d, int rows) {
  return !d->p8 && !d->opt_cluster && !d->opt_quant_in_gemm && add_layernorm_quant_supported(rows, d->cfg.dim_emb);
}
// Whether launch_decoder_rows runs the layers of a step of `rows` rows.
bool decoder_rows_apply(const mi8d_decoder* d, int rows) {
  const mi8d_config& c = d->cfg;
  return rows <= d->opt_one_launch_rows && d->rows_ready && d->opt_fuse && !d->opt_cluster && !d->opt_quant_in_gemm &&
         decoder_rows_supported(rows, c.dim_emb, c.dim_ffn, c.heads, c.dec_depth, d->src);
}
int add_ln_quant(mi8d_decoder* d, const float* a, const float* resid, const Norm& n, int rows, float* out, int8_t* q, cudaStream_t s) {
  return launch_add_layernorm_quant(a, resid, n.g, n.b, 1e-6f, rows, d->cfg.dim_emb, out, q,
                                    reinterpret_cast<float*>(q + static_cast<size_t>(rows) * d->cfg.dim_emb), s);
}

// out = LayerNorm(affine(x) + resid): the "dan" post-processing of a sub-layer's last affine (src/models/transformer.h:189-214).
// One launch when the row fits a cluster (the cluster GEMM's LayerNorm write-back), else affine (into `tmp`) and LayerNorm.
// `quant_next` (ln_quantises): the result is also quantised into d->aq for the next affine, and the slots and row maxima are left alone.
int quant_gemm_ln(mi8d_decoder* d, const float* x, int M, const unsigned* slot, const Aff& w, const float* resid, const Norm& n, float* tmp,
                  float* out, float* rowmax, unsigned* out_slot, cudaStream_t s, unsigned* out_slot2 = nullptr, bool quant_next = false) {
  if(!w.p8 && d->opt_cluster && d->opt_fused_ln && M <= d->opt_cluster_max_rows && w.K <= d->opt_cluster_max_k && w.N == d->cfg.dim_emb &&
     gemm_cq_supported(M, w.N, w.K, true)) {
    CqCall g;
    g.a_f32 = x;
    g.a_slot = slot;
    g.bt = w.bt;
    g.d_qb = w.qm;
    g.M = M;
    g.N = w.N;
    g.K = w.K;
    g.bias = w.bias;
    g.ln = 1;
    g.ln_resid = resid;
    g.ln_gamma = n.g;
    g.ln_beta = n.b;
    g.ln_eps = 1e-6f;
    g.ln_out = out;
    g.ln_rowmax = rowmax;
    g.ln_slot = out_slot;
    g.ln_slot2 = out_slot2;
    g.weights_settled = kOwnChain;
    g.stream = s;
    return launch_gemm_cq(g);
  }
  MI8D_TRY(quant_gemm(d, x, M, slot, w, false, tmp, s));
  if(quant_next)
    return add_ln_quant(d, tmp, resid, n, M, out, d->aq, s);
  return add_ln(d, tmp, resid, n, M, out, rowmax, out_slot, s, out_slot2);
}

}  // namespace

extern "C" {

size_t mi8d_arena_bytes(const mi8d_config* cfg) {
  if(cfg == nullptr)
    return 0;
  mi8d_decoder tmp;
  tmp.cfg = *cfg;
  tmp.layout();
  return tmp.arena.used + 4096;
}

int mi8d_create(const mi8d_config* cfg, void* arena, size_t arena_bytes, void* workspace, size_t workspace_bytes,
                mi8d_decoder** out) {
  if(cfg == nullptr || arena == nullptr || out == nullptr || workspace == nullptr)
    return MI8_ERR_BAD_ARG;
  if(cfg->enc_depth < 0 || cfg->dim_emb % 16 != 0 || cfg->dim_ffn % 16 != 0 || cfg->heads <= 0 || cfg->dim_emb % cfg->heads != 0 || cfg->dec_depth <= 0 ||
     cfg->max_rows <= 0 || cfg->max_steps <= 0 || cfg->max_batch <= 0 || cfg->max_src <= 0 || cfg->vocab <= 0)
    return MI8_ERR_BAD_ARG;
  if(cfg->dec_depth > 16)
    return MI8_ERR_UNSUPPORTED;
  const int dh = cfg->dim_emb / cfg->heads;
  if(dh != 64 && dh != 32)
    return MI8_ERR_UNSUPPORTED;
  if(reinterpret_cast<uintptr_t>(arena) & 255u)
    return MI8_ERR_MISALIGNED;
  if(arena_bytes < mi8d_arena_bytes(cfg) || workspace_bytes < mi8_workspace_bytes(0, 0, 0))
    return MI8_ERR_WORKSPACE;
  mi8d_decoder* d = new mi8d_decoder();
  d->cfg = *cfg;
  d->arena.base = static_cast<uint8_t*>(arena);
  d->arena.size = arena_bytes;
  d->layout();
  d->ws = workspace;
  d->ws_bytes = workspace_bytes;
  if(d->reuse_stats != nullptr)
    cudaMemset(d->reuse_stats, 0, 2 * sizeof(unsigned));
  {
    // pinned host staging for the beam search's per-step upload and download
    const size_t nc = 3 * static_cast<size_t>(cfg->max_rows) + cfg->max_batch + 3, no = 2 * 3 * static_cast<size_t>(cfg->max_batch) * 8;
    if(cudaHostAlloc(reinterpret_cast<void**>(&d->h_ctrl), nc * sizeof(int), cudaHostAllocDefault) != cudaSuccess ||
       cudaHostAlloc(reinterpret_cast<void**>(&d->h_out), no * sizeof(int) + 4 * kDecoderRowsMax * sizeof(unsigned long long), cudaHostAllocDefault) != cudaSuccess) {
      cudaGetLastError();
      if(d->h_ctrl)
        cudaFreeHost(d->h_ctrl);
      d->h_ctrl = d->h_out = nullptr;   // mi8d_search then reports MI8_ERR_WORKSPACE; stepping by hand still works
    } else {
      d->h_tagged = reinterpret_cast<unsigned long long*>(d->h_out + no);   // (an even number of words behind)
      std::fill(d->h_tagged, d->h_tagged + 4 * kDecoderRowsMax, 0ull);
    }
  }
  if(!cfg->ssru) {
    bool ok = cudaStreamCreateWithFlags(&d->side, cudaStreamNonBlocking) == cudaSuccess;
    for(cudaEvent_t* e : {&d->ev_fork, &d->ev_join})
      ok = ok && cudaEventCreateWithFlags(e, cudaEventDisableTiming) == cudaSuccess;
    d->overlap = ok;   // without them the step simply runs on the caller's stream alone
    if(!ok)
      cudaGetLastError();
  }
  if(cudaEventCreateWithFlags(&d->ev_step, cudaEventDisableTiming | cudaEventBlockingSync) != cudaSuccess) {
    d->ev_step = nullptr;
    cudaGetLastError();
  }
  *out = d;
  return MI8_OK;
}

void mi8d_destroy(mi8d_decoder* d) {
  if(d == nullptr)
    return;
  if(d->ev_step != nullptr)
    cudaEventDestroy(d->ev_step);
  if(d->side != nullptr) {
    cudaStreamSynchronize(d->side);
    cudaStreamDestroy(d->side);
  }
  for(cudaEvent_t e : {d->ev_fork, d->ev_join})
    if(e != nullptr)
      cudaEventDestroy(e);
  if(d->h_ctrl)
    cudaFreeHost(d->h_ctrl);
  if(d->h_out)
    cudaFreeHost(d->h_out);
  delete d;
}

int mi8d_set_weight(mi8d_decoder* d, const char* name, const int8_t* bt, int K, int N) {
  if(d == nullptr || name == nullptr || bt == nullptr || K <= 0 || N <= 0)
    return MI8_ERR_BAD_ARG;
  if(K % 16 != 0 || (reinterpret_cast<uintptr_t>(bt) & 15u))
    return MI8_ERR_MISALIGNED;
  Weight w;
  w.bt = bt;
  w.K = K;
  w.N = N;
  d->weights[name] = w;
  d->dirty = true;
  return MI8_OK;
}

int mi8d_set_packed8_weight(mi8d_decoder* d, const char* name, const int8_t* bt, const float* scale_b, const int32_t* zp_b, const int32_t* off_b,
                            int K, int N) {
  if(d == nullptr || name == nullptr || bt == nullptr || scale_b == nullptr || zp_b == nullptr || off_b == nullptr || K <= 0 || N <= 0)
    return MI8_ERR_BAD_ARG;
  if(K % 16 != 0 || (reinterpret_cast<uintptr_t>(bt) & 15u))
    return MI8_ERR_MISALIGNED;
  P8Weight w;
  w.bt = bt;
  w.scale_b = scale_b;
  w.zp_b = zp_b;
  w.off_b = off_b;
  w.K = K;
  w.N = N;
  d->p8_weights[name] = w;
  d->p8 = true;
  d->dirty = true;
  return MI8_OK;
}

int mi8d_set_param(mi8d_decoder* d, const char* name, const float* p) {
  if(d == nullptr || name == nullptr || p == nullptr)
    return MI8_ERR_BAD_ARG;
  d->params[name] = p;
  d->dirty = true;
  return MI8_OK;
}

int mi8d_set_positions(mi8d_decoder* d, const float* table) {
  if(d == nullptr || table == nullptr)
    return MI8_ERR_BAD_ARG;
  d->positions = table;
  return MI8_OK;
}

int mi8d_set_option(mi8d_decoder* d, int option, int value) {
  if(d == nullptr && option != MI8D_OPT_ATTENTION_UNROLL && option != MI8D_OPT_ATTENTION_BLOCK_HEADS)
    return MI8_ERR_BAD_ARG;   // (the process-wide switches need no decoder)
  switch(option) {
    case MI8D_OPT_FUSE_WEIGHTS: d->opt_fuse = value != 0; break;
    case MI8D_OPT_QUANT_IN_GEMM: d->opt_quant_in_gemm = value != 0; break;
    case MI8D_OPT_FUSED_OUTPUT_MAX_ROWS: d->opt_fused_out_rows = value; break;
    case MI8D_OPT_SIDE_STREAM: d->opt_side_stream = value != 0; break;
    case MI8D_OPT_SHARED_HISTORY: d->opt_shared_history = value != 0; break;
    case MI8D_OPT_ONE_LAUNCH_ROWS: d->opt_one_launch_rows = value; break;
    case MI8D_OPT_STEP_AHEAD: d->opt_step_ahead = value != 0; break;
    case MI8D_OPT_CLUSTER_AFFINE: d->opt_cluster = value != 0; break;
    case MI8D_OPT_FUSED_LAYERNORM: d->opt_fused_ln = value != 0; break;
    case MI8D_OPT_CLUSTER_MAX_ROWS: d->opt_cluster_max_rows = value; break;
    case MI8D_OPT_CLUSTER_SIZE:
      if(value != 0 && value != 1 && value != 2 && value != 4 && value != 8)
        return MI8_ERR_BAD_ARG;
      d->opt_cluster_size = value;
      break;
    case MI8D_OPT_CLUSTER_MAX_K: d->opt_cluster_max_k = value; break;
    case MI8D_OPT_BLOCKING_WAIT:
      if(value < 0 || value > 2)
        return MI8_ERR_BAD_ARG;
      d->opt_blocking_wait = value;
      break;
    case MI8D_OPT_GEMM_TILE_ROWS:
      if(value != 0 && value != 32 && value != 64 && value != 128 && value != 256 && value != 512)
        return MI8_ERR_BAD_ARG;
      d->opt_gemm_tile = value;
      break;
    case MI8D_OPT_ATTENTION_UNROLL:
      if(value != 8 && value != 16)
        return MI8_ERR_BAD_ARG;
      set_attention_unroll(value);
      break;
    case MI8D_OPT_ATTENTION_BLOCK_HEADS: set_attention_block_heads(value); break;
    default: return MI8_ERR_BAD_ARG;
  }
  return MI8_OK;
}

int mi8d_search_stats(mi8d_decoder* d, double out[4], int reset) {
  if(d == nullptr || out == nullptr)
    return MI8_ERR_BAD_ARG;
  out[0] = d->t_issue;
  out[1] = d->t_wait;
  out[2] = d->t_host;
  out[3] = d->n_steps;
  if(reset)
    d->t_issue = d->t_wait = d->t_host = d->n_steps = 0;
  return MI8_OK;
}

const float* mi8d_last_logits(const mi8d_decoder* d) { return d ? d->logits : nullptr; }

int mi8d_keep_logits(mi8d_decoder* d, int keep) {
  if(d == nullptr)
    return MI8_ERR_BAD_ARG;
  d->keep_logits = keep != 0;
  return MI8_OK;
}

size_t mi8g_output_scratch_bytes(int rows, int vocab) {
  if(rows <= 0 || vocab <= 0)
    return 0;
  return static_cast<size_t>(rows) * ((static_cast<size_t>(vocab) + 127) / 128) * 18 * sizeof(float);
}

int mi8g_output_topk(const int8_t* aq, const float* d_qa, const int8_t* wq, const float* d_qw, int rows, int vocab, int K,
                     const float* bias, int k, const float* prev_scores, void* scratch, size_t scratch_bytes, float* logits_out,
                     float* cand_score, int* cand_word, void* stream) {
  if(rows <= 0 || vocab <= 0 || k < 1 || k > 8 || scratch == nullptr || cand_score == nullptr || cand_word == nullptr)
    return MI8_ERR_BAD_ARG;
  if(scratch_bytes < mi8g_output_scratch_bytes(rows, vocab))
    return MI8_ERR_WORKSPACE;
  const size_t cells = static_cast<size_t>(rows) * ((static_cast<size_t>(vocab) + 127) / 128);
  float* blk_max = static_cast<float*>(scratch);
  float* blk_sum = blk_max + cells;
  float* blk_topv = blk_sum + cells;
  int* blk_topi = reinterpret_cast<int*>(blk_topv + cells * 8);
  const int k_top = k <= 4 ? 4 : 8;
  int rc = launch_gemm_logits(aq, d_qa, wq, d_qw, rows, vocab, K, bias, 1.0f, k_top, blk_max, blk_sum, blk_topv, blk_topi, logits_out,
                              as_stream(stream));
  if(rc != MI8_OK)
    return rc;
  return launch_lse_merge(blk_max, blk_sum, blk_topv, blk_topi, rows, vocab, k_top, k, prev_scores, cand_score, cand_word, as_stream(stream));
}

int mi8d_history_reuse(mi8d_decoder* d, unsigned out[2], int reset) {
  if(d == nullptr || out == nullptr)
    return MI8_ERR_BAD_ARG;
  out[0] = out[1] = 0;
  if(d->reuse_stats == nullptr)
    return MI8_OK;
  cudaError_t e = cudaDeviceSynchronize();
  if(e == cudaSuccess)
    e = cudaMemcpy(out, d->reuse_stats, 2 * sizeof(unsigned), cudaMemcpyDeviceToHost);
  if(e == cudaSuccess && reset)
    e = cudaMemset(d->reuse_stats, 0, 2 * sizeof(unsigned));
  if(e != cudaSuccess) {
    set_last_cuda_error(e);
    return MI8_ERR_LAUNCH;
  }
  return MI8_OK;
}

int mi8g_embed(const float* wemb, const int* words, const float* pos, int pos_mod, float scale, int rows, int dim, float* out,
               float* rowmax, unsigned* absmax_slot, void* stream) {
  return launch_embed(wemb, words, pos, pos_mod, scale, rows, dim, out, rowmax, absmax_slot, as_stream(stream));
}
int mi8g_add_layernorm(const float* a, const float* resid, const float* gamma, const float* beta, float eps, int rows, int dim,
                       float* out, float* rowmax, unsigned* absmax_slot, void* stream) {
  if(gamma == nullptr || beta == nullptr)
    return MI8_ERR_BAD_ARG;
  return launch_add_layernorm(a, resid, gamma, beta, eps, rows, dim, out, rowmax, absmax_slot, as_stream(stream));
}
int mi8g_affine_slot(const float* a, const unsigned* absmax_slot, const int8_t* bt, const float* d_qb, int M, int N, int K,
                     float scale, const float* bias, int relu, float* c, unsigned* absmax_out, int tile_rows, int cluster,
                     void* stream) {
  CqCall g;
  g.a_f32 = a;
  g.a_slot = absmax_slot;
  g.bt = bt;
  g.d_qb = d_qb;
  g.M = M;
  g.N = N;
  g.K = K;
  g.scale = scale;
  g.bias = bias;
  g.relu = relu;
  g.c = c;
  g.absmax_out = absmax_out;
  g.force_tile_m = tile_rows;
  g.force_cluster = cluster;
  g.stream = as_stream(stream);
  return launch_gemm_cq(g);
}
int mi8g_affine_slot_add_layernorm(const float* a, const unsigned* absmax_slot, const int8_t* bt, const float* d_qb, int M,
                                   int N, int K, float scale, const float* bias, const float* resid, const float* gamma,
                                   const float* beta, float eps, float* out, float* rowmax, unsigned* out_slot,
                                   unsigned* out_slot2, void* stream) {
  CqCall g;
  g.a_f32 = a;
  g.a_slot = absmax_slot;
  g.bt = bt;
  g.d_qb = d_qb;
  g.M = M;
  g.N = N;
  g.K = K;
  g.scale = scale;
  g.bias = bias;
  g.ln = 1;
  g.ln_resid = resid;
  g.ln_gamma = gamma;
  g.ln_beta = beta;
  g.ln_eps = eps;
  g.ln_out = out;
  g.ln_rowmax = rowmax;
  g.ln_slot = out_slot;
  g.ln_slot2 = out_slot2;
  g.stream = as_stream(stream);
  return launch_gemm_cq(g);
}
int mi8g_quantize_slot(const float* x, size_t n, const unsigned* absmax_slot, int8_t* q, float* d_quant_mult, void* stream) {
  return launch_quantize_slot(x, n, absmax_slot, q, d_quant_mult, as_stream(stream));
}
int mi8g_attention1(const float* q, const float* k, const float* v, const float* log_mask, int rows, int heads, int dim_head,
                    int len, int batch, int mode, float* out, unsigned* absmax_slot, void* stream) {
  if(q == nullptr || k == nullptr || v == nullptr || out == nullptr)
    return MI8_ERR_BAD_ARG;
  return launch_attention1(q, k, v, log_mask, rows, heads, dim_head, len, batch, mode, out, absmax_slot, as_stream(stream));
}
int mi8g_lse_topk(const float* logits, int rows, int vocab, int k, const float* prev_scores, float* cand_score, int* cand_word,
                  void* stream) {
  if(logits == nullptr || cand_score == nullptr || cand_word == nullptr)
    return MI8_ERR_BAD_ARG;
  return launch_lse_topk(logits, rows, vocab, k, prev_scores, cand_score, cand_word, as_stream(stream));
}
int mi8g_nbest_merge(const float* cand_score, const int* cand_word, int beam, int batch, int vocab, int k, float* out_score,
                     int* out_beam, int* out_word, void* stream) {
  if(cand_score == nullptr || cand_word == nullptr || out_score == nullptr || out_beam == nullptr || out_word == nullptr)
    return MI8_ERR_BAD_ARG;
  return launch_nbest_merge(cand_score, cand_word, beam, batch, vocab, k, out_score, out_beam, out_word, as_stream(stream));
}
int mi8g_lse_topk_nbest(const float* logits, int beam, int batch, int vocab, int k, const float* prev_scores, float* cand_score,
                        int* cand_word, unsigned* arrivals, float* out_score, int* out_beam, int* out_word, void* stream) {
  if(logits == nullptr || cand_score == nullptr || cand_word == nullptr || arrivals == nullptr || out_score == nullptr || out_beam == nullptr ||
     out_word == nullptr || beam < 1 || batch < 1 || beam > INT32_MAX / batch)
    return MI8_ERR_BAD_ARG;
  StepEnd end;
  end.beam = beam;
  end.batch = batch;
  end.arrivals = arrivals;
  end.out_score = out_score;
  end.out_beam = out_beam;
  end.out_word = out_word;
  return launch_lse_topk(logits, beam * batch, vocab, k, prev_scores, cand_score, cand_word, as_stream(stream), end);
}

int mi8d_start(mi8d_decoder* d, const float* context, const float* log_mask, int batch, int src, void* stream) {
  if(d == nullptr || context == nullptr || log_mask == nullptr || batch <= 0 || src <= 0)
    return MI8_ERR_BAD_ARG;
  if(batch > d->cfg.max_batch || src > d->cfg.max_src)
    return MI8_ERR_UNSUPPORTED;
  cudaStream_t s = as_stream(stream);
  const size_t dm = d->cfg.dim_emb;
  cudaError_t e = cudaMemcpyAsync(d->context[0], context, sizeof(float) * batch * src * dm, cudaMemcpyDeviceToDevice, s);
  if(e == cudaSuccess)
    e = cudaMemcpyAsync(d->log_mask[0], log_mask, sizeof(float) * batch * src, cudaMemcpyDeviceToDevice, s);
  if(e == cudaSuccess && d->cfg.ssru)
    for(auto& L : d->layers)
      if(e == cudaSuccess)
        e = cudaMemsetAsync(L.cell[0], 0, sizeof(float) * static_cast<size_t>(batch) * dm, s);
  if(e != cudaSuccess) {
    set_last_cuda_error(e);
    return MI8_ERR_LAUNCH;
  }
  d->t = 0;
  d->batch = batch;
  d->src = src;
  d->ctx_cur = 0;
  d->anc_cur = 0;
  d->cell_cur = 0;
  d->cross_valid = false;
  d->slab_rows = (d->cfg.max_rows / d->cfg.max_batch) * batch;
  return MI8_OK;
}

int mi8d_encode(mi8d_decoder* d, const int* ids, const float* log_mask, int batch, int src, void* stream) {
  if(d == nullptr || ids == nullptr || log_mask == nullptr || batch <= 0 || src <= 0)
    return MI8_ERR_BAD_ARG;
  const mi8d_config& c = d->cfg;
  if(c.enc_depth <= 0 || batch > c.max_batch || src > c.max_src || src > c.max_steps)
    return MI8_ERR_UNSUPPORTED;
  if(d->positions == nullptr)
    return MI8_ERR_BAD_ARG;
  cudaStream_t s = as_stream(stream);
  if(d->dirty)
    MI8D_TRY(d->resolve(s));
  const int dm = c.dim_emb, M = batch * src;
  const size_t n_d = static_cast<size_t>(M) * dm;
  cudaError_t e = cudaMemsetAsync(d->slots, 0, sizeof(unsigned) * d->n_slots, s);
  if(e == cudaSuccess)
    e = cudaMemcpyAsync(d->log_mask[0], log_mask, sizeof(float) * batch * src, cudaMemcpyDeviceToDevice, s);
  if(e != cudaSuccess) {
    set_last_cuda_error(e);
    return MI8_ERR_LAUNCH;
  }
  float* aq_tail = reinterpret_cast<float*>(d->enc_aq + n_d);
  // embeddings * sqrt(d) + positions 0..src-1 (src/models/transformer.h:93,110-114)
  float* x = d->enc_x[0];
  unsigned* x_slot = d->slots;
  const bool lq = ln_quantises(d, M);
  MI8D_TRY(launch_embed(d->wemb, ids, d->positions, src, sqrtf(static_cast<float>(dm)), M, dm, x, nullptr, x_slot, s));
  for(int l = 0; l < c.enc_depth; ++l) {
    const EncLayerW& w = d->enc_w[l];
    unsigned *sa = d->enc_slot(l, 0), *s1 = d->enc_slot(l, 1), *s3 = d->enc_slot(l, 2);
    // q, keys and values are the same tensor: one quantisation serves the three projections, and with fused
    // weights one launch computes all three
    if(l == 0 || !lq)
      MI8D_TRY(quantize_act(d, x, M, dm, x_slot, d->enc_aq, s));
    if(d->opt_fuse && w.qkv.ready) {
      float* outs[3] = {d->enc_q, d->enc_k, d->enc_v};
      MI8D_TRY(gemm_fused(d, d->enc_aq, aq_tail, M, w.qkv, outs, s));
    } else {
      MI8D_TRY(gemm_act(d, d->enc_aq, M, w.q, false, d->enc_q, s));
      MI8D_TRY(gemm_act(d, d->enc_aq, M, w.k, false, d->enc_k, s));
      MI8D_TRY(gemm_act(d, d->enc_aq, M, w.v, false, d->enc_v, s));
    }
    float* a = d->enc_x[1];   // attention output, then reused as x1
    MI8D_TRY(launch_attention1(d->enc_q, d->enc_k, d->enc_v, d->log_mask[0], M, c.heads, dm / c.heads, src, batch, 2, a, sa, s));
    MI8D_TRY(quantize_act(d, a, M, dm, sa, d->enc_aq, s));
    MI8D_TRY(gemm_act(d, d->enc_aq, M, w.o, false, d->enc_q, s));
    if(lq) {                                                                                  // x1 = LN(Wo(a) + x)
      MI8D_TRY(add_ln_quant(d, d->enc_q, x, w.ln_att, M, a, d->enc_aq, s));
    } else {
      MI8D_TRY(add_ln(d, d->enc_q, x, w.ln_att, M, a, nullptr, s1, s));
      MI8D_TRY(quantize_act(d, a, M, dm, s1, d->enc_aq, s));
    }
    MI8D_TRY(gemm_act(d, d->enc_aq, M, w.w1, true, d->enc_h, s, s3));                        // ReLU (and max|h|) in the write-back
    MI8D_TRY(quantize_act(d, d->enc_h, M, c.dim_ffn, s3, d->enc_aq, s));
    MI8D_TRY(gemm_act(d, d->enc_aq, M, w.w2, false, d->enc_q, s));
    const bool last = l + 1 == c.enc_depth;
    float* nx = last ? d->context[0] : x;                                                     // the last layer writes the context
    x_slot = d->enc_slot(l, 3);
    if(lq && !last)
      MI8D_TRY(add_ln_quant(d, d->enc_q, a, w.ln_ffn, M, nx, d->enc_aq, s));
    else
      MI8D_TRY(add_ln(d, d->enc_q, a, w.ln_ffn, M, nx, nullptr, x_slot, s));
    x = nx;
  }
  if(c.ssru) {
    for(auto& L : d->layers) {
      e = cudaMemsetAsync(L.cell[0], 0, sizeof(float) * static_cast<size_t>(batch) * dm, s);
      if(e != cudaSuccess) {
        set_last_cuda_error(e);
        return MI8_ERR_LAUNCH;
      }
    }
  }
  d->t = 0;
  d->batch = batch;
  d->src = src;
  d->ctx_cur = 0;
  d->anc_cur = 0;
  d->cell_cur = 0;
  d->cross_valid = false;
  d->slab_rows = (c.max_rows / c.max_batch) * batch;
  return MI8_OK;
}

}  // extern "C"

namespace {

// How a step of mi8d_search is tied to the one behind it (StepEnd has the words' meaning): `end` carries them to the step's last kernel.
struct StepLink {
  bool in_search = false;   // (what lies in front of the step is the search's own)
  const unsigned* stop = nullptr;
  unsigned* next_stop = nullptr;
  int* next_ctrl = nullptr;
  unsigned long long *tagged = nullptr, *host_lists = nullptr;   // where the last kernel leaves the lists; where the first brings those of the step in front
  const unsigned long long* lists = nullptr;
  int n_lists = 0;
  unsigned tag = 0;
  int eos = 0;
  unsigned char hyps[kDecoderRowsMax] = {};
};

int run_step(mi8d_decoder* d, const int* hyp_idx, const int* prev_words, const int* batch_idx, const float* prev_scores, int beam, int batch, int n_best,
             float* out_score, int* out_beam, int* out_word, void* stream, const StepLink& link) {
  if(d == nullptr || beam <= 0 || batch <= 0 || n_best <= 0 || n_best > 8 || out_score == nullptr || out_beam == nullptr ||
     out_word == nullptr)
    return MI8_ERR_BAD_ARG;
  const mi8d_config& c = d->cfg;
  const int t = d->t;
  const int R = beam * batch;
  if(R > c.max_rows || t >= c.max_steps || batch > d->batch || (!c.ssru && R > d->slab_rows))
    return MI8_ERR_UNSUPPORTED;
  if(t > 0 && (hyp_idx == nullptr || prev_words == nullptr))
    return MI8_ERR_BAD_ARG;
  if(t == 0 && beam != 1)
    return MI8_ERR_BAD_ARG;
  if(d->positions == nullptr)
    return MI8_ERR_BAD_ARG;
  cudaStream_t s = as_stream(stream);
  if(d->dirty)
    MI8D_TRY(d->resolve(s));
  const int dm = c.dim_emb, S = d->src;
  const int SR = d->slab_rows;
  const size_t slab_stride = static_cast<size_t>(SR) * dm;
  const size_t n_d = static_cast<size_t>(R) * dm;

  // Few rows of an SSRU decoder: all layers in one launch, which also brings the control words to the device unless the batch
  // changed (the gather below reads them).
  const bool rows_path = decoder_rows_apply(d, R);
  const bool begin_apart = !rows_path || batch != d->batch;
  if(begin_apart)
    MI8D_TRY(launch_step_begin(d->step_ctrl, d->s_ctrl[t & 1], d->n_step_ctrl, d->slots, d->n_slots, s));

  // sentences that finished leave the batch: compact the encoder context, recompute cross K/V
  if(batch != d->batch) {
    if(batch_idx == nullptr)
      return MI8_ERR_BAD_ARG;
    const int nxt = d->ctx_cur ^ 1;
    MI8D_TRY(launch_gather_rows(d->context[d->ctx_cur], batch_idx, batch, S * dm, d->context[nxt], s));
    MI8D_TRY(launch_gather_rows(d->log_mask[d->ctx_cur], batch_idx, batch, S, d->log_mask[nxt], s));
    d->ctx_cur = nxt;
    d->batch = batch;
    d->cross_valid = false;
  }
  const float* ctx = d->context[d->ctx_cur];
  const float* lmask = d->log_mask[d->ctx_cur];
  if(!d->cross_valid) {
    // one quantisation of the context serves the key and value projections of every layer
    const size_t n = static_cast<size_t>(batch) * S * dm;
    float* cq_tail = reinterpret_cast<float*>(d->cq + n);
    if(d->p8) {
      MI8D_TRY(quantize_act(d, ctx, batch * S, dm, nullptr, d->cq, s));
    } else {
      MI8D_TRY(launch_prepare(ctx, n, cq_tail, d->cq, d->ws, d->ws_bytes, s, Trigger::kBehindWait));
    }
    for(int l = 0; l < c.dec_depth; ++l) {
      const DecLayerW& w = d->dec_w[l];
      if(d->opt_fuse && w.ctx_kv.ready) {
        float* outs[2] = {d->layers[l].cross_k, d->layers[l].cross_v};
        MI8D_TRY(gemm_fused(d, d->cq, cq_tail, batch * S, w.ctx_kv, outs, s));
      } else {
        MI8D_TRY(gemm_act(d, d->cq, batch * S, w.ctx_k, false, d->layers[l].cross_k, s));
        MI8D_TRY(gemm_act(d, d->cq, batch * S, w.ctx_v, false, d->layers[l].cross_v, s));
      }
    }
    d->cross_valid = true;
  }

  // layer-0 input: scaled embedding of the previous word (zero at the first step) + position t.  For self-attention also, in the same
  // launch, the ancestor table of this step and every layer's history abs-max over the earlier slabs; the producer of a
  // layer's newest slab (this embedding / the previous layer's last LayerNorm) adds that slab's maximum.
  const int anc_new = d->anc_cur ^ 1;
  HistLists lists = d->lists;
  lists.batch = 0;
  // single-query attention over the stored keys/values of steps 0 .. t
  auto self_attention = [&](const LayerBufs& L, unsigned* sa) {
    if(lists.batch > 0)
      return launch_attention_hist(d->qbuf, L.kslab, L.vslab, R, c.heads, dm / c.heads, t + 1, d->abuf, sa, s, lists);
    return launch_attention1(d->qbuf, L.kslab, L.vslab, nullptr, R, c.heads, dm / c.heads, t + 1, batch, 0, d->abuf, sa, s, d->anc[anc_new], SR, SR);
  };
  float* x = c.ssru ? d->x_in : d->layers[0].slab + static_cast<size_t>(t) * slab_stride;
  const int* words = t == 0 ? nullptr : prev_words;
  const float* pos = d->positions + static_cast<size_t>(t) * dm;
  const float emb_scale = sqrtf(static_cast<float>(dm));
  const int cell_new = d->cell_cur ^ 1;
  float* aq_tail = reinterpret_cast<float*>(d->aq + n_d);
  if(rows_path) {
    DecoderRowsParams& p = d->rows;
    p.rows = R;
    p.ffn = c.dim_ffn;
    p.layers = c.dec_depth;
    p.src = S;
    p.batch = batch;
    p.emb_scale = emb_scale;
    p.att_scale = 1.0f / sqrtf(static_cast<float>(dm / c.heads));
    p.wemb = d->wemb;
    p.pos = pos;
    p.log_mask = lmask;
    p.words = words;
    p.hyp = t == 0 ? nullptr : hyp_idx;
    p.ctrl = d->s_ctrl[t & 1];
    p.stop = link.stop;
    p.next_stop = link.next_stop;
    p.lists = link.lists;
    p.host_lists = link.host_lists;
    p.n_lists = link.n_lists;
    p.n_ctrl = begin_apart ? 0 : d->n_step_ctrl;
    std::copy(d->step_ctrl, d->step_ctrl + p.n_ctrl, p.ctrl_words);   // (3 R + batch words, batch <= R <= kDecoderRowsMax)
    p.slots = d->slots;
    p.n_slots = begin_apart ? 0 : d->n_slots;
    p.out_q = d->aq;
    p.out_qm = aq_tail;
    const LayerBufs &first = d->layers[0], &next = d->layers[c.dec_depth > 1 ? 1 : 0];   // (every layer's buffers are laid out alike)
    p.cross_k = first.cross_k;
    p.cross_v = first.cross_v;
    p.cell_old = first.cell[d->cell_cur];
    p.cell_new = first.cell[cell_new];
    p.layer_stride = static_cast<size_t>(next.cross_k - first.cross_k);
    MI8D_TRY(launch_decoder_rows(p, dm, c.heads, s, link.in_search));
  } else if(c.ssru) {
    MI8D_TRY(launch_embed(d->wemb, words, pos, 0, emb_scale, R, dm, x, nullptr, d->input_slot(0), s));
  } else {
    const float* rowmax[16];
    unsigned* hslot[16];
    for(int l = 0; l < c.dec_depth; ++l) {
      rowmax[l] = d->layers[l].rowmax;
      hslot[l] = d->layer_slot(l, kSlotHistory);
    }
    lists.batch = d->opt_shared_history && attention_hist_supported(beam, batch, dm / c.heads, t + 1) ? batch : 0;
    MI8D_TRY(launch_embed_ancestors(d->wemb, words, pos, emb_scale, dm, x, d->layers[0].rowmax + static_cast<size_t>(t) * SR, d->input_slot(0),
                                    d->layer_slot(0, kSlotHistory), d->anc[d->anc_cur], d->anc[anc_new], hyp_idx, t, R, SR, s,
                                    d->p8 ? 0 : c.dec_depth, rowmax, hslot, lists));
  }

  const bool lq = rows_path || ln_quantises(d, R);
  for(int l = 0; l < c.dec_depth && !rows_path; ++l) {
    LayerBufs& L = d->layers[l];
    const DecLayerW& w = d->dec_w[l];
    unsigned* x_slot = d->input_slot(l);
    unsigned* s1 = d->layer_slot(l, kSlotSelfLn);
    if(c.ssru) {
      if(l == 0 || !lq)
        MI8D_TRY(quantize_act(d, x, R, dm, x_slot, d->aq, s));
      if(d->opt_fuse && w.rnn.ready) {
        float* outs[2] = {d->qbuf, d->fbuf};
        MI8D_TRY(gemm_fused(d, d->aq, aq_tail, R, w.rnn, outs, s));            // dot(input, W) and affine(input, Wf, bf)
      } else {
        MI8D_TRY(gemm_act(d, d->aq, R, w.rnn_w, false, d->qbuf, s));
        MI8D_TRY(gemm_act(d, d->aq, R, w.rnn_wf, false, d->fbuf, s));
      }
      if(lq) {
        MI8D_TRY(launch_add_layernorm_quant(nullptr, x, w.ln_self.g, w.ln_self.b, 1e-6f, R, dm, d->x1, d->aq, aq_tail, s, L.cell[d->cell_cur],
                                            t == 0 ? nullptr : hyp_idx, d->qbuf, d->fbuf, L.cell[cell_new]));
      } else {
        MI8D_TRY(launch_ssru_cell(L.cell[d->cell_cur], t == 0 ? nullptr : hyp_idx, d->qbuf, d->fbuf, R, dm, L.cell[cell_new], d->abuf, s));
        MI8D_TRY(add_ln(d, d->abuf, x, w.ln_self, R, d->x1, nullptr, s1, s));
      }
    } else if(d->p8) {
      // packed8avx512 quantises every ROW of an activation on its own, so the keys/values of earlier steps never change:
      // the newest slab is projected and stored, the rest is a plain key/value cache (what the reference recomputes from the
      // concatenated history, src/models/transformer.h:401-417, comes out identical row by row)
      unsigned* sa = d->layer_slot(l, kSlotSelfAtt);
      MI8D_TRY(quantize_act(d, x, R, dm, nullptr, d->aq, s));
      float* outs[3] = {d->qbuf, L.kslab + static_cast<size_t>(t) * slab_stride, L.vslab + static_cast<size_t>(t) * slab_stride};
      if(d->opt_fuse && w.self_qkv.ready) {
        MI8D_TRY(gemm_fused(d, d->aq, nullptr, R, w.self_qkv, outs, s));
      } else {
        MI8D_TRY(gemm_act(d, d->aq, R, w.self_q, false, outs[0], s));
        MI8D_TRY(gemm_act(d, d->aq, R, w.self_k, false, outs[1], s));
        MI8D_TRY(gemm_act(d, d->aq, R, w.self_v, false, outs[2], s));
      }
      MI8D_TRY(self_attention(L, sa));
      MI8D_TRY(quant_gemm_ln(d, d->abuf, R, sa, w.self_o, x, w.ln_self, d->obuf, d->x1, nullptr, s1, s, nullptr, lq));
    } else {
      unsigned* sh = d->layer_slot(l, kSlotHistory);
      unsigned* sa = d->layer_slot(l, kSlotSelfAtt);
      // Keys and values are projections of the WHOLE history of layer inputs, quantised with one multiplier over the
      // live part of that history.  The projections of earlier steps are kept per slab and stay valid as long as that
      // multiplier's abs-max does not change (compared bit for bit on the device): then only the newest slab is
      // quantised and projected, otherwise everything is.  One launch quantises the layer input twice - with its own
      // multiplier for the query projection and, as the newest history slab, with the history's.
      const int steps = t + 1;
      const int cap_rows = c.max_steps * c.max_rows;   // slabs of hq; the operand of the query projection lies behind them
      int8_t* xq = L.hq + static_cast<size_t>(cap_rows) * dm;
      float* hq_tail = reinterpret_cast<float*>(xq + static_cast<size_t>(c.max_rows) * dm);
      float* xq_tail = hq_tail + 1;
      MI8D_TRY(launch_quantize_dual(x, n_d, x_slot, xq, xq_tail, L.slab, SR, steps, R, dm, sh, d->prev_bits + l, L.hq, hq_tail, s));
      const bool fused = d->opt_fuse && w.self_qkv.ready;
      float* kv_new[2] = {L.kslab + static_cast<size_t>(t) * slab_stride, L.vslab + static_cast<size_t>(t) * slab_stride};
      // Query, key and value projections of the newest slab are one launch (the query's segment takes its rows and multiplier from
      // another place of hq).  The earlier slabs' keys and values, recomputed only when the abs-max changed, are in it as well (below_tile), or run
      // beside it on the internal stream, or in front of it.
      // (As three launches, the query's on its own stream beside the others with tiles for half of the SMs each: 38.4, 19.1 and 45.7 ms.)
      const int below = fused && t > 0 && d->opt_gemm_tile == 0 && d->opt_side_stream ? below_tile(R, beam, static_cast<size_t>(t) * SR * dm) : 0;
      const bool side = d->overlap && d->opt_side_stream && t > 0 && below == 0;
      cudaStream_t so = side ? d->side : s;
      if(side) {
        MI8D_CUDA(cudaEventRecord(d->ev_fork, s));
        MI8D_CUDA(cudaStreamWaitEvent(so, d->ev_fork, 0));
      }
      if(t > 0 && below == 0) {
        // all tiles skipped when the stored results still hold; no split-K: the two streams must not share the workspace's counters
        if(fused) {
          GemmCall g = fused_call(d, L.hq, w.self_qkv, t * SR, 1, 3, cap_rows + c.max_rows, so);
          g.d_qa = hq_tail;
          g.seg_c[0] = L.kslab;
          g.seg_c[1] = L.vslab;
          g.force_splits = 1;
          g.skip_a = d->prev_bits + l;
          g.skip_b = sh;
          g.skip_rows_below = t * SR;
          MI8D_TRY(launch_gemm_call(g));
        } else {
          MI8D_TRY(launch_gemm(L.hq, w.self_k.bt, t * SR, w.self_k.N, w.self_k.K, hq_tail, w.self_k.qm, 1.0f, w.self_k.bias, 0, L.kslab, MI8_F32,
                               nullptr, d->ws, d->ws_bytes, so, 0, 1, nullptr, d->prev_bits + l, sh, t * SR));
          MI8D_TRY(launch_gemm(L.hq, w.self_v.bt, t * SR, w.self_v.N, w.self_v.K, hq_tail, w.self_v.qm, 1.0f, w.self_v.bias, 0, L.vslab, MI8_F32,
                               nullptr, d->ws, d->ws_bytes, so, 0, 1, nullptr, d->prev_bits + l, sh, t * SR));
        }
      }
      if(side)
        MI8D_CUDA(cudaEventRecord(d->ev_join, so));
      if(fused) {
        GemmCall g = fused_call(d, L.hq, w.self_qkv, R, 0, 3, cap_rows + c.max_rows, s);
        g.d_qa = hq_tail;
        g.a_row0 = t * SR;
        g.seg_row0[0] = cap_rows;
        g.seg_qa[0] = xq_tail;
        g.seg_c[0] = d->qbuf;
        g.seg_c[1] = kv_new[0];
        g.seg_c[2] = kv_new[1];
        if(below != 0) {
          g.rows_below = true;
          g.force_tile_m = below;
          g.force_splits = 1;
          g.skip_a = d->prev_bits + l;
          g.skip_b = sh;
          g.skip_rows_below = t * SR;
        } else if(wide_tile(d, R) != 0) {
          g.force_tile_m = wide_tile(d, R);
          g.force_splits = 1;
        }
        MI8D_TRY(launch_gemm_call(g));
      } else {
        const int8_t* a_new = L.hq + static_cast<size_t>(t) * slab_stride;
        MI8D_TRY(launch_gemm(xq, w.self_q.bt, R, w.self_q.N, w.self_q.K, xq_tail, w.self_q.qm, 1.0f, w.self_q.bias, 0, d->qbuf, MI8_F32,
                             nullptr, d->ws, d->ws_bytes, s, 0, 1, nullptr, nullptr, nullptr, 0, kOwnChain));
        MI8D_TRY(launch_gemm(a_new, w.self_k.bt, R, w.self_k.N, w.self_k.K, hq_tail, w.self_k.qm, 1.0f, w.self_k.bias, 0, kv_new[0], MI8_F32,
                             nullptr, d->ws, d->ws_bytes, s, 0, 1, nullptr, nullptr, nullptr, 0, kOwnChain));
        MI8D_TRY(launch_gemm(a_new, w.self_v.bt, R, w.self_v.N, w.self_v.K, hq_tail, w.self_v.qm, 1.0f, w.self_v.bias, 0, kv_new[1], MI8_F32,
                             nullptr, d->ws, d->ws_bytes, s, 0, 1, nullptr, nullptr, nullptr, 0, kOwnChain));
      }
      if(side)
        MI8D_CUDA(cudaStreamWaitEvent(s, d->ev_join, 0));
      MI8D_TRY(self_attention(L, sa));
      MI8D_TRY(quant_gemm_ln(d, d->abuf, R, sa, w.self_o, x, w.ln_self, d->obuf, d->x1, nullptr, s1, s, nullptr, lq));
    }
    {
      unsigned* sa = d->layer_slot(l, kSlotCtxAtt);
      unsigned* s2 = d->layer_slot(l, kSlotCtxLn);
      MI8D_TRY(quant_gemm(d, d->x1, R, s1, w.ctx_q, false, d->qbuf, s, nullptr, lq));
      MI8D_TRY(launch_attention1(d->qbuf, L.cross_k, L.cross_v, lmask, R, c.heads, dm / c.heads, S, batch, 1, d->abuf, sa, s));
      MI8D_TRY(quant_gemm_ln(d, d->abuf, R, sa, w.ctx_o, d->x1, w.ln_ctx, d->obuf, d->x2, nullptr, s2, s, nullptr, lq));

      unsigned* s3 = d->layer_slot(l, kSlotRelu);
      MI8D_TRY(quant_gemm(d, d->x2, R, s2, w.w1, true, d->hbuf, s, s3, lq));   // ReLU and max|h| fused in the write-back

      // the block's output is the next layer's input: write it straight into that layer's history slab, and its
      // maximum into that layer's history abs-max as well
      const bool last = l + 1 == c.dec_depth;
      float* nx = last ? d->x_final : (c.ssru ? d->x_in : d->layers[l + 1].slab + static_cast<size_t>(t) * slab_stride);
      float* nx_rowmax = (last || c.ssru) ? nullptr : d->layers[l + 1].rowmax + static_cast<size_t>(t) * SR;
      unsigned* nx_hist = (last || c.ssru) ? nullptr : d->layer_slot(l + 1, kSlotHistory);
      MI8D_TRY(quant_gemm_ln(d, d->hbuf, R, s3, w.w2, d->x2, w.ln_ffn, d->obuf, nx, nx_rowmax, d->layer_slot(l, kSlotOut), s, nx_hist,
                             lq && (last || c.ssru)));
      x = nx;
    }
  }

  // tied output layer, then log-softmax + n-best per sentence over beam x vocabulary
  unsigned* x_slot = d->input_slot(c.dec_depth);
  if(!lq)
    MI8D_TRY(quantize_act(d, x, R, dm, x_slot, d->aq, s));
  // Beyond kBlockRows rows the plain GEMM followed by the scanning log-softmax / top-k kernel is the faster route since that kernel
  // scans without candidate lists (beam 6, 2 sentences of transformer-base: 16.2 ms a mini-batch with the reducing write-back, 15.2 ms
  // without; student, 16 sentences x beam 4: 7.3 and 7.0; 64 x 4 and 128 x 4 rows: level).  opt_fused_out_rows > 0 brings the other back.
  const bool fused_output = !d->p8 && !d->keep_logits && R <= d->opt_fused_out_rows && n_best >= 2;
  const bool merge_apart = !step_end_fits(beam, n_best);
  StepEnd end;
  end.beam = beam;
  end.batch = batch;
  end.arrivals = merge_apart ? nullptr : d->arrivals();
  end.out_score = out_score;
  end.out_beam = out_beam;
  end.out_word = out_word;
  end.stop = link.stop;
  end.next_stop = link.next_stop;
  end.next_ctrl = link.next_ctrl;
  end.tagged = link.tagged;
  end.tag = link.tag;
  end.eos = link.eos;
  std::copy(link.hyps, link.hyps + kDecoderRowsMax, end.hyps);
  if(!c.ssru && !d->p8) {   // remember which abs-max the stored keys/values of every layer now belong to
    end.layers = c.dec_depth;
    end.first = 1 + kSlotHistory;
    end.stride = kSlotsPerLayer;
    end.slots = d->slots;
    end.prev_bits = d->prev_bits;
    end.stats = d->reuse_stats;
  }
  if(!fused_output && R <= kBlockRows) {
    // few rows: the write-back reduces the blocks of the log-softmax as well
    if(d->p8) {
      const Aff& w = d->out_w;
      MI8D_TRY(launch_gemm_p8(reinterpret_cast<const uint8_t*>(d->aq), d->p8_scale_a, d->p8_zp_a, d->p8_sum_a, w.bt, w.scale_b, w.zp_b, w.off_b, R, w.N,
                              w.K, w.bias, 0, d->logits, nullptr, d->ws, d->ws_bytes, s, 0, 0, nullptr, d->blk_max, d->blk_sum));
    } else {
      GemmCall g;
      g.aq = d->aq;
      g.bt = d->out_w.bt;
      g.M = R;
      g.N = d->out_w.N;
      g.K = d->out_w.K;
      g.d_qa = aq_tail;
      g.seg_qb[0] = d->out_w.qm;
      g.seg_bias[0] = d->out_bias;
      g.seg_c[0] = d->logits;
      g.weights_settled = kOwnChain;
      g.stream = s;
      g.block_max = d->blk_max;
      g.block_sum = d->blk_sum;
      MI8D_TRY(launch_gemm_call(g));
    }
    MI8D_TRY(launch_lse_topk(d->logits, R, c.vocab, n_best, prev_scores, d->cand_score, d->cand_word, s, end, d->blk_max, d->blk_sum));
  } else if(!fused_output) {
    MI8D_TRY(gemm_act(d, d->aq, R, d->out_w, false, d->logits, s));
    MI8D_TRY(launch_lse_topk(d->logits, R, c.vocab, n_best, prev_scores, d->cand_score, d->cand_word, s, end));
  } else {
    // the GEMM's write-back reduces every 128-word block of a row; the logits never reach memory
    const int k_top = n_best <= 4 ? 4 : 8;
    MI8D_TRY(launch_gemm_logits(d->aq, aq_tail, d->out_w.bt, d->out_w.qm, R, c.vocab, dm, d->out_bias, 1.0f, k_top, d->blk_max, d->blk_sum,
                                d->blk_topv, d->blk_topi, nullptr, s));
    MI8D_TRY(launch_lse_merge(d->blk_max, d->blk_sum, d->blk_topv, d->blk_topi, R, c.vocab, k_top, n_best, prev_scores, d->cand_score,
                              d->cand_word, s, end));
  }
  if(merge_apart)
    MI8D_TRY(launch_nbest_merge(d->cand_score, d->cand_word, beam, batch, c.vocab, n_best, out_score, out_beam, out_word, s));
  d->anc_cur = anc_new;
  d->cell_cur = cell_new;
  d->t = t + 1;
  return MI8_OK;
}

}  // namespace

extern "C" {

int mi8d_step(mi8d_decoder* d, const int* hyp_idx, const int* prev_words, const int* batch_idx, const float* prev_scores, int beam,
              int batch, int n_best, float* out_score, int* out_beam, int* out_word, void* stream) {
  return run_step(d, hyp_idx, prev_words, batch_idx, prev_scores, beam, batch, n_best, out_score, out_beam, out_word, stream, StepLink());
}

// Beam search over one mini-batch: the bookkeeping of BeamSearch::search (src/translator/beam_search.cpp:249-538)
// around mi8d_encode / mi8d_step.  Per step: every sentence still in the batch contributes its surviving
// hypotheses (beam-major rows, dummy slots with EOS and score -inf), the n-best lists come back, each sentence keeps
// as many candidates as it had hypotheses (toHyps, :24-210), hypotheses that ended in EOS are scored
// ((pathScore - wordPenalty * length) / length^normalize, src/translator/history.h:22-35) and leave the beam, a
// sentence whose beam is empty leaves the batch (purgeBeams, :224-245), and everything stops at
// length >= max_length_factor * width (:521-531).  The best finished hypothesis of every sentence is traced back
// through the per-step parent links.  One wait per step (the n-best download).
// Where a step's layers are one launch (few rows of an SSRU decoder), step t + 1 is launched before the host has seen step t's lists, with the control
// words that step t's last kernel leaves on the device (StepEnd): the GPU no longer waits for the host's turn, 12 of 58 us of a step of one sentence.
// Those words hold while no hypothesis ends; otherwise the three launches do nothing or only fill scratch, and the host launches step t + 1 anew.  The output GEMM of
// a step so stopped still runs, 4 to 5 us in front of the new one, where the host's turn had stood.  Student with a bias on the end of the sentence, step by step /
// ahead, ms: 16 sentences that end after 8.5 words on average (at most 41) 3.09 / 2.63, 32 after 3.5 3.21 / 2.79, 8 x beam 4 after 29 3.03 / 2.72, 2 x 4 after 21 2.42 /
// 2.15; none ends 3.55 / 3.04 (16), 2.65 / 2.19 (one); a search that ends with its first words 0.65 / 0.65 to 0.73 (16).
int mi8d_search(mi8d_decoder* d, const int* ids, const float* log_mask, int batch, int width, const mi8d_search_config* sc,
                int* out_tokens, int max_out, int* out_len, float* out_score, unsigned long long* h2d_bytes, unsigned long long* d2h_bytes,
                void* stream) {
  if(d == nullptr || ids == nullptr || log_mask == nullptr || sc == nullptr || out_tokens == nullptr || out_len == nullptr || batch <= 0 ||
     width <= 0 || max_out <= 0 || sc->beam <= 0 || sc->beam > 8)
    return MI8_ERR_BAD_ARG;
  if(d->h_ctrl == nullptr || d->h_out == nullptr)
    return MI8_ERR_WORKSPACE;
  const mi8d_config& c = d->cfg;
  const int beam = sc->beam, eos = sc->eos_id, B0 = batch;
  if(beam * batch > c.max_rows || batch > c.max_batch)
    return MI8_ERR_UNSUPPORTED;
  cudaStream_t s = as_stream(stream);
  int rc = mi8d_encode(d, ids, log_mask, batch, width, stream);
  if(rc != MI8_OK)
    return rc;

  struct Final { double norm; int t, pos; };
  struct StepRecord { std::vector<int> words, prev, unpurged; };   // [B0 * beam] each
  std::vector<int> W(B0, beam), step_map(B0), new_n(B0), new_W(B0);
  std::vector<int> words(B0 * beam, 0), prev_state(B0 * beam, 0), new_words(B0 * beam), new_prev(B0 * beam);
  std::vector<float> scores(B0 * beam, 0.f), new_scores(B0 * beam);
  std::vector<std::vector<Final>> finals(B0);
  std::vector<StepRecord> history;
  std::vector<int> active;
  for(int o = 0; o < B0; ++o)
    step_map[o] = o;
  int prev_dim = B0;
  unsigned long long up_bytes = 0, down_bytes = 0;

  using clk = std::chrono::steady_clock;
  auto secs = [](clk::time_point a, clk::time_point b) { return std::chrono::duration<double>(b - a).count(); };
  const auto last_step = [&](int t) { return static_cast<double>(t + 1) >= static_cast<double>(sc->max_length_factor) * width; };
  const bool may_run_ahead = d->opt_step_ahead && d->opt_blocking_wait != 1 && d->opt_fused_out_rows == 0 && !d->keep_logits;
  // Step t + 1 may be launched before step t's lists are seen: both take the cluster launch, with nothing between them but the control words.
  const auto ahead_of = [&](int t, int nb, int max_beam) {
    return may_run_ahead && !last_step(t) && t + 1 < c.max_steps && max_beam * nb <= kBlockRows && decoder_rows_apply(d, max_beam * nb) &&
           (t > 0 || decoder_rows_apply(d, nb));
  };
  // What step t needs to know of its neighbours, while `active` and W are those of step t
  const auto link_of = [&](int t, int nb, int max_beam, bool launched_ahead) {
    StepLink link;
    link.in_search = true;
    const int own = (t & 1) * 2 * kDecoderRowsMax, front = 2 * kDecoderRowsMax - own;
    const bool ahead = ahead_of(t, nb, max_beam);
    if(launched_ahead) {
      link.stop = d->stops + (t & 1);
      link.lists = d->s_tagged + front;
      link.host_lists = d->h_tagged + front;
      link.n_lists = 2 * nb * max_beam;
    }
    if(launched_ahead || ahead) {
      link.tagged = (ahead ? d->s_tagged : d->h_tagged) + own;
      d->tag = d->tag == 0xffffffffu ? 1u : d->tag + 1u;
      link.tag = d->tag;
    }
    if(ahead) {
      link.next_stop = d->stops + ((t + 1) & 1);
      link.next_ctrl = d->s_ctrl[(t + 1) & 1];
      link.eos = eos;
      for(int a = 0; a < nb; ++a)
        link.hyps[a] = static_cast<unsigned char>(W[active[a]]);
    }
    return link;
  };
  // Launches step t: hypotheses from the control words in s_ctrl[t & 1] (t > 0); the lists go to the step's half of h_out
  const auto launch = [&](int t, int nb, int max_beam, const StepLink& link) {
    const int tensor_beam = t == 0 ? 1 : max_beam, R = tensor_beam * nb, cells = nb * max_beam;
    int *ctrl = d->s_ctrl[t & 1], *out = d->h_out + (t & 1) * 3 * c.max_batch * 8;
    return run_step(d, t > 0 ? ctrl : nullptr, t > 0 ? ctrl + R : nullptr, t > 0 ? ctrl + 3 * R : nullptr,
                    t > 0 ? reinterpret_cast<const float*>(ctrl + 2 * R) : nullptr, tensor_beam, nb, max_beam, reinterpret_cast<float*>(out), out + cells,
                    out + 2 * cells, stream, link);
  };
  // An error behind a launch: what is in flight still writes to pinned memory and to the caller's arena
  const auto settled = [&](int code) {
    cudaStreamSynchronize(s);
    if(d->side != nullptr)
      cudaStreamSynchronize(d->side);
    cudaGetLastError();
    return code;
  };
  StepLink link, next_link;   // of the running step, and of the one launched ahead of it
  bool launched = false;      // the running step was launched ahead, and stands
  bool loose_end = false;     // the stream may still be at work
  clk::time_point mark = clk::now();
  for(int t = 0;; ++t) {
    int max_beam = 0;
    active.clear();
    for(int o = 0; o < B0; ++o) {
      max_beam = W[o] > max_beam ? W[o] : max_beam;
      if(W[o] > 0)
        active.push_back(o);
    }
    if(max_beam == 0)
      break;
    const int nb = static_cast<int>(active.size());
    const int n_best = max_beam;
    const int tensor_beam = t == 0 ? 1 : max_beam;
    const int R = tensor_beam * nb;
    if(t > 0 && !launched) {
      int* hc = d->h_ctrl;
      for(int j = 0; j < max_beam; ++j) {
        for(int a = 0; a < nb; ++a) {
          const int o = active[a];
          const bool valid = j < W[o];
          const int idx = j * nb + a;
          hc[idx] = valid ? prev_state[o * beam + j] * prev_dim + step_map[o] : 0;
          hc[R + idx] = valid ? words[o * beam + j] : eos;                       // dummy slots carry EOS
          const float sv = valid ? scores[o * beam + j] : -INFINITY;
          memcpy(&hc[2 * R + idx], &sv, sizeof(float));
        }
      }
      for(int a = 0; a < nb; ++a)
        hc[3 * R + a] = step_map[active[a]];
      const size_t n_up = static_cast<size_t>(3 * R + nb) * sizeof(int);
      d->step_ctrl = hc;
      d->n_step_ctrl = 3 * R + nb;
      up_bytes += n_up;
    }
    const int cells = nb * n_best;
    const clk::time_point t_a = clk::now();
    if(launched) {
      link = next_link;
    } else {
      link = link_of(t, nb, max_beam, false);
      rc = launch(t, nb, max_beam, link);
      d->step_ctrl = nullptr;
      d->n_step_ctrl = 0;
      if(rc != MI8_OK)
        return settled(rc);
    }
    const int was_t = d->t, was_cell = d->cell_cur, was_anc = d->anc_cur;
    const bool ahead = link.next_ctrl != nullptr;
    if(ahead) {
      next_link = link_of(t + 1, nb, max_beam, true);
      rc = launch(t + 1, nb, max_beam, next_link);
      if(rc != MI8_OK)
        return settled(rc);
    }
    const clk::time_point t_b = clk::now();
    int* out = d->h_out + (t & 1) * 3 * c.max_batch * 8;
    if(link.tagged != nullptr) {
      const volatile unsigned long long* word = d->h_tagged + (t & 1) * 2 * kDecoderRowsMax;
      loose_end = true;
      const auto pause = [&]() {
        if(d->opt_blocking_wait == 2)
          std::this_thread::yield();
      };
      cudaError_t qe = cudaSuccess;
      const auto state = [&]() {
        qe = cudaStreamQuery(s);
        return qe == cudaSuccess ? StreamState::kIdle : qe == cudaErrorNotReady ? StreamState::kBusy : StreamState::kFailed;
      };
      const TaggedWait waited = wait_for_tagged(word, 2 * cells, link.tag, 4096, pause, state);
      if(waited == TaggedWait::kFailed)
        MI8D_CUDA(qe);
      if(waited == TaggedWait::kMissing)
        return MI8_ERR_DEVICE;
      for(int e = 0; e < cells; ++e) {
        const unsigned score = static_cast<unsigned>(word[2 * e]), key = static_cast<unsigned>(word[2 * e + 1]);
        memcpy(out + e, &score, sizeof(float));
        out[cells + e] = static_cast<int>(key / static_cast<unsigned>(c.vocab));
        out[2 * cells + e] = static_cast<int>(key % static_cast<unsigned>(c.vocab));
      }
    } else if(d->opt_blocking_wait == 2 && d->ev_step != nullptr) {
      // several searches (and ranks) share the host's cores: poll, and hand the core to another thread between polls - as
      // quick as spinning while cores are free, fair when there are more waiting threads than cores
      MI8D_CUDA(cudaEventRecord(d->ev_step, s));
      cudaError_t qe;
      while((qe = cudaEventQuery(d->ev_step)) == cudaErrorNotReady)
        std::this_thread::yield();
      MI8D_CUDA(qe);
      loose_end = false;
    } else if(d->opt_blocking_wait && d->ev_step != nullptr) {
      // sleep until the step's results have arrived (an interrupt wakes the thread: tens of microseconds later than polling)
      MI8D_CUDA(cudaEventRecord(d->ev_step, s));
      MI8D_CUDA(cudaEventSynchronize(d->ev_step));
      loose_end = false;
    } else {
      MI8D_CUDA(cudaStreamSynchronize(s));
      loose_end = false;
    }
    const clk::time_point t_c = clk::now();
    d->t_host += secs(mark, t_a);
    d->t_issue += secs(t_a, t_b);
    d->t_wait += secs(t_b, t_c);
    d->n_steps += 1;
    mark = t_c;
    down_bytes += static_cast<size_t>(cells) * (link.tagged != nullptr ? 2 * sizeof(unsigned long long) : 3 * sizeof(int));
    const float* nv = reinterpret_cast<const float*>(out);
    const int* nbm = out + cells;
    const int* nw = out + 2 * cells;

    // toHyps: every sentence keeps its current number of hypotheses, skipping invalid scores
    std::fill(new_n.begin(), new_n.end(), 0);
    std::fill(new_words.begin(), new_words.end(), 0);
    std::fill(new_prev.begin(), new_prev.end(), 0);
    std::fill(new_scores.begin(), new_scores.end(), 0.f);
    for(int a = 0; a < nb; ++a) {
      const int o = active[a];
      int cnt = 0;
      for(int cidx = 0; cidx < n_best && cnt < W[o]; ++cidx) {
        const float v = nv[a * n_best + cidx];
        if(!(v > -INFINITY))
          continue;
        new_words[o * beam + cnt] = nw[a * n_best + cidx];
        new_scores[o * beam + cnt] = v;
        new_prev[o * beam + cnt] = nbm[a * n_best + cidx];
        ++cnt;
      }
      new_n[o] = cnt;
    }
    // purgeBeams and History::add
    const int length = t + 1;
    const bool max_len_reached = last_step(t);
    bool one_ended = false;   // (or one without a successor: what finish_step takes as a reason to stop)
    StepRecord rec;
    rec.words = new_words;
    rec.prev = new_prev;
    rec.unpurged.assign(B0 * beam, 0);
    std::fill(new_W.begin(), new_W.end(), 0);
    for(int o = 0; o < B0; ++o) {
      int surv = 0;
      for(int j = 0; j < new_n[o]; ++j)
        if(new_words[o * beam + j] != eos)
          ++surv;
      new_W[o] = surv;
      one_ended = one_ended || surv != W[o];
      const bool last = surv == 0 || max_len_reached;
      int rank = 0;
      for(int j = 0; j < new_n[o]; ++j) {
        const bool is_eos = new_words[o * beam + j] == eos;
        if(is_eos || last) {
          const double norm = (static_cast<double>(new_scores[o * beam + j]) - static_cast<double>(sc->word_penalty) * length) /
                              std::pow(static_cast<double>(length), static_cast<double>(sc->normalize));
          finals[o].push_back(Final{norm, t, j});
        }
        if(!is_eos)
          rec.unpurged[o * beam + rank++] = j;
      }
    }
    history.push_back(std::move(rec));
    launched = ahead && !one_ended;
    if(ahead && one_ended) {   // the step launched ahead is launched anew: its words were not these
      d->t = was_t;
      d->cell_cur = was_cell;
      d->anc_cur = was_anc;
    }
    if(max_len_reached)
      break;
    const StepRecord& cur = history.back();
    std::fill(words.begin(), words.end(), 0);
    std::fill(scores.begin(), scores.end(), 0.f);
    std::fill(prev_state.begin(), prev_state.end(), 0);
    for(int o = 0; o < B0; ++o) {
      for(int r2 = 0; r2 < new_W[o]; ++r2) {
        const int j = cur.unpurged[o * beam + r2];
        words[o * beam + r2] = new_words[o * beam + j];
        scores[o * beam + r2] = new_scores[o * beam + j];
        prev_state[o * beam + r2] = new_prev[o * beam + j];
      }
    }
    W = new_W;
    std::fill(step_map.begin(), step_map.end(), -1);
    for(int a = 0; a < nb; ++a)
      step_map[active[a]] = a;
    prev_dim = nb;
  }

  if(loose_end)
    MI8D_CUDA(cudaStreamSynchronize(s));

  // best finished hypothesis per sentence (highest score; ties to the earlier step, then the earlier position), traced back
  for(int o = 0; o < B0; ++o) {
    out_len[o] = 0;
    if(out_score)
      out_score[o] = -INFINITY;
    if(finals[o].empty())
      continue;
    const Final* best = &finals[o][0];
    for(const Final& f : finals[o])
      if(f.norm > best->norm || (f.norm == best->norm && (f.t < best->t || (f.t == best->t && f.pos < best->pos))))
        best = &f;
    int t = best->t, pos = best->pos;
    const int len = t + 1;
    if(len > max_out)
      return MI8_ERR_WORKSPACE;
    for(;;) {
      out_tokens[static_cast<size_t>(o) * max_out + t] = history[t].words[o * beam + pos];
      if(t == 0)
        break;
      // the parent is addressed by its row in the previous step's purged beam: map it back to that step's unpurged list
      pos = history[t - 1].unpurged[o * beam + history[t].prev[o * beam + pos]];
      --t;
    }
    out_len[o] = len;
    if(out_score)
      out_score[o] = static_cast<float>(best->norm);
  }
  if(h2d_bytes)
    *h2d_bytes = up_bytes;
  if(d2h_bytes)
    *d2h_bytes = down_bytes;
  return MI8_OK;
}

}  // extern "C"

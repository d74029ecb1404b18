// dsk_hybrid_host.cuh — host side of the layer-list ("hybrid") model family inside libdsk: model description, tensor upload by
// name, the per-sequence state (recurrent states, convolution histories, latent ring caches) and the chunk step that
// dsk_forward / dsk_forward_chunk / dsk_decode_greedy drive.  Included at the end of dsk_engine.cu (it uses that file's error,
// allocation and sampling helpers); dsk_model::hy / dsk_state::hy point at the structures below.
//
// Tensor names (safetensors, [out, in] matrices):  embed, side.embed, final.norm, head (untied LM head), loop.step (layer loop),
// and per layer i ("l<i>."):
//   norm1 (and norm1b, norm2, norm2b in sandwich blocks)
//         | mix.in, mix.conv, mix.conv.b, mix.dt_bias, mix.A_log, mix.D, mix.norm, mix.o              (state-space mixer)
//         | mix.q, mix.dkv, mix.dkv.norm, mix.uk, mix.uv, mix.o                                        (latent attention)
//         | mix.q, mix.k, mix.q.norm, mix.k.norm, mix.talk, mix.o                                      (grouped-query attention)
//   mlp.router, mlp.correction, mlp.e<j>.gate|up|down                                                 (routed feed-forward)
//   mlp.up, mlp.up.b, mlp.down, mlp.down.b, mlp.act                                                   (dense feed-forward)
//   side.gate, side.proj, side.norm                                                                   (per-layer token input)
//   shift (token shift), norm1.b / norm2.b / final.norm.b (layer norms with a bias)
//         | mix.q, mix.f, mix.f.b, mix.lower, mix.v, mix.norm, mix.o                                   (gated linear recurrence)
//   mlp.router, mlp.router.b, mlp.e<j>.up|down                                                        (routed feed-forward, top-softmax router)
//   mix.q|k|v (+ .conv), mix.b, mix.a, mix.A_log, mix.dt_bias, mix.norm, mix.g, mix.o                 (gated delta rule)
//   mix.q|k|v|g, mix.norm, mix.o                                                                      (lightning attention)
//   mix.q|k|v|g, mix.i, mix.i.b, mix.f, mix.f.b, mix.norm, mix.o                                      (mLSTM matrix memory)
//   mlp.shared.gate|up|down|sg (shared expert), loop.in (product that opens a loop pass), mix.q|k|v.conv (attention behind convolutions)
// Two mixers side by side name theirs mix.left.* and mix.right.*.
// Grouped-query attention with its switches on adds mix.v, mix.q.b / k.b / v.b, mix.rel, mix.sink, mix.vmix; latent attention with a
// rotated key part (DSK_MIX_MLA) has mix.dq, dq.norm, uq, dkv, dkv.norm, uk, uv, sink, g, o; a gated dense feed-forward mlp.gate / up / down;
// DSK_BLOCK_POST layers norm1 / norm2, ls1 / ls2, canon1 / canon2, rg1 / rg2 (+ .b); the model "bigram" beside "embed".
// A parallel block computes, with h = norm1(x):  x += m (mixer(h) + ff(h));  a sandwich block  x += norm1b(mixer(norm1(x))),
// x += norm2b(ff(norm2(x))) (with layer scales: ls1 / ls2 times the norms' results);  a pre-norm block  x += m mixer(norm1(x)), x += m ff(norm2(x)).  Then, when the model has a per-layer token table,
// g = gelu_tanh(side.gate x) * side.embed[token][i*sd : (i+1)*sd],  y = side.proj g,  x += m * rmsnorm(y) * side.norm.
// A layer loop repeats a range of layers with the same weights; each repetition ("layer run") keeps a separate cache / state.
#pragma once

namespace hyb {
using namespace dsk;
using namespace dsk::hy;

struct HTensor {
  void* p = nullptr;       // model quant type (float | bf16)
  long long rows = 0, cols = 0;
  bool present = false;
};

struct HLayer {
  dsk_layer_spec sp;
  float *norm1 = nullptr, *norm1b = nullptr, *norm2 = nullptr, *norm2b = nullptr;
  // state-space mixer
  HTensor in, o;
  float *conv_w = nullptr, *conv_b = nullptr, *dt_bias = nullptr, *A_log = nullptr, *D = nullptr, *mnorm = nullptr;
  // latent attention
  HTensor q, dkv, ukT, uk, uv;      // ukT: [heads][kv_rank][dim], the transposed key up-projection (absorbed into the query);
                                    // uk: the same matrix as stored, for portions that up-project the keys instead
  float* dkv_norm = nullptr;
  int owner = -1;                   // layer whose latent cache this layer reads (itself unless kv_from)
  int ring = 0;                     // rows of this layer's own ring cache (owners only)
  // grouped-query attention (with q, o above): key projection, whole-projection norm weights, score mixing, rotation table
  HTensor kproj;
  float *q_norm = nullptr, *k_norm = nullptr, *talk = nullptr, *rot_freq = nullptr;
  float rot_mag = 1.f;
  // grouped-query attention with a value matrix: q, k and v rows (and the output gate's rows, when there is one) stacked into one
  // matrix (one product per step) with their biases; a layer that reads another layer's keys and values stacks [q | gate]
  HTensor qkv;
  float *qkv_b = nullptr, *rel = nullptr, *sink = nullptr;
  int* rel_bucket = nullptr;        // distance (0 .. att_rel_max) -> row of rel
  int rel_rows = 0;
  float vmix = 0.f;                 // value-mixing weight (mix.vmix), read once at upload
  char have_qkv[4] = {0, 0, 0, 0}, have_qkvb[3] = {0, 0, 0}, have_vmix = 0;   // have_qkv[3]: the output gate's rows behind q / k / v
  // latent attention with a rotated key part: the two down-projections stacked [q_rank | kv_rank + rot_dim], query up-projection, output gate
  HTensor in2, uq, gmat;
  float* dq_norm = nullptr;
  char have_in2[2] = {0, 0};
  // DSK_BLOCK_POST: input convolutions, residual gates; closing norm weights (norm weight x layer scale, folded when the model is finalised)
  HTensor rg1, rg2;
  float *rg1_b = nullptr, *rg2_b = nullptr, *canon1 = nullptr, *canon2 = nullptr, *ls1 = nullptr, *ls2 = nullptr, *close1 = nullptr, *close2 = nullptr;
  float norm1_s = 1.f, norm2_s = 1.f;   // single-number norm weights
  char have_n1 = 0, have_n2 = 0;
  // dense feed-forward (gate_d: the gate matrix of a gated one)
  HTensor up, down, gate_d;
  float *up_b = nullptr, *down_b = nullptr, *act = nullptr;
  float act_a = 0.f, act_b = 0.f;
  // routed feed-forward
  HTensor gate_s, up_s, down_s;     // expert stacks [E][ff][width], [E][ff][width], [E][width][ff]
  std::vector<char> have;           // 3 E flags
  float *router = nullptr, *correction = nullptr;   // with a shared expert the row of its weight (mlp.shared.sg) stands behind the router's
  HTensor gate_sh, up_sh, down_sh;  // shared expert
  char have_router[2] = {0, 0};
  // per-layer token input
  HTensor sgate, sproj;
  float* snorm = nullptr;
  // token shift weight; biases of the layer norms; bias of a top-softmax router
  float *shift = nullptr, *norm1_bias = nullptr, *norm2_bias = nullptr, *router_b = nullptr;
  // gated linear recurrence: [q | f | v] rows stacked into one matrix, the forget gate's bias at the f rows of a stacked bias
  // (zeros elsewhere), lower bounds, and the output norm's weight (one vector for all heads)
  HTensor lin_in;
  float *lin_bias = nullptr, *lower = nullptr, *lin_norm = nullptr;
  char have_lin[4] = {0, 0, 0, 0}, have_linb = 0;   // lightning attention: [q | k | v | g]
  float *decay = nullptr, *log_decay = nullptr;     // lightning attention: one number per head
  // gated delta rule: its projections ride in qkv (att_layout), convolution taps of the [q | k | v] channels in one array; A_log, dt_bias
  // and lin_norm as above.  Side by side with attention, o holds both output matrices column by column: [left | right]
  float* gdn_conv_w = nullptr;
  // attention behind short convolutions: taps of the q, k and v channels in conv_w, three blocks [taps][channels], have_conv as below.  mLSTM: lin_in [q | k | v | g | i | f],
  // padded to a multiple of 8 rows, lin_bias with the gates' biases, mnorm
  char have_gate[2] = {0, 0}, have_gateb[2] = {0, 0};
  char have_gdn[6] = {0, 0, 0, 0, 0, 0}, have_conv[3] = {0, 0, 0}, have_o[2] = {0, 0};
};

// one execution of a layer: layers inside the loop range run once per pass, each time with a state of their own
struct Run {
  int layer;
  int pass;        // >= 0: this run opens pass `pass` of the loop (loop.step[pass] is added to the residual stream first)
  int owner_run;   // latent attention: the run whose latent cache this run reads (itself unless kv_from)
};

struct Model {
  dsk_hybrid_config c;
  std::vector<HLayer> L;
  std::vector<Run> runs;
  HTensor embed, side_embed, head, bigram, loop_in;
  float *final_norm = nullptr, *final_norm_b = nullptr, *loop_step = nullptr;
  int vmix_first = -1;              // the first layer whose values later value-mixing layers blend in
  size_t wsize = 4;                 // bytes per matrix element
};

struct LayerState {
  float* ssm = nullptr;             // [heads][vdim][state]
  float* hist = nullptr;            // [conv - 1][channels]
  void* cache = nullptr;            // [ring][kv_rank] (owner layers); grouped-query attention: keys [ring][kv_heads * dim]
  void* vcache = nullptr;           // grouped-query attention: values [ring][kv_heads * vdim]
  float* canon = nullptr;           // DSK_BLOCK_POST: [2][taps - 1][width] rings of the two input convolutions
  float* shift = nullptr;           // token shift: the mixer input of the sequence's last token [width]
  float* lin = nullptr;             // gated linear recurrence: [heads][dim][vdim]; mLSTM: then n [heads][dim] and m [heads]
  // gated delta rule (and attention behind convolutions): state in lin, the convolutions' inputs in hist, a ring over positions of taps - 1 + kConvSpare rows
  size_t ssm_bytes = 0, hist_bytes = 0, cache_bytes = 0, vcache_bytes = 0, canon_bytes = 0, shift_bytes = 0, lin_bytes = 0;
};

struct State {
  std::vector<LayerState> L;
  int chunk = 0, width = 0;
  int next_pos = 0;
  int *d_tok = nullptr, *d_want = nullptr, *d_ctl = nullptr, *d_idx = nullptr, *d_perm = nullptr, *d_ntiles = nullptr;
  int4* d_tiles = nullptr;
  int max_tiles = 0;
  int head_rows = 0;                         // rows of the logits buffer: the LM head runs over the wanted rows in groups of this size
  float* part = nullptr;                     // partial softmax results of key-split attention (decode-sized chunks)
  // prefill attention as matrix products (blocks of kPrefillQ queries): up-projected keys / values, their per-head packing, scores
  float *kf = nullptr, *vf = nullptr, *sc = nullptr;
  int talk_q = 0;   // queries per block of layers that mix heads
  void *kb = nullptr, *vt = nullptr;
  int* d_rows = nullptr;
  int prefill_keys = 0;                      // keys a block of queries can see at most; 0: the matrix path is off
  float* y = nullptr;                        // a sublayer's output before its closing norm (sandwich and post blocks)
  float* emb = nullptr;                      // the step's embedding output (a layer loop that adds it again)
  float* xin = nullptr;                      // [chunk][2 width]: [stream | embedding output], what the product that opens a loop pass reads
  float *lgate = nullptr, *lden = nullptr;   // mLSTM: log gates and running maxima of the step, normalisers
  float* wsh = nullptr;                      // [chunk] weights of the shared expert
  // linear attention: prepared q, k and v rows, per-block records, outputs ahead of their norm
  float *lq = nullptr, *lk = nullptr, *lv = nullptr, *lrec = nullptr, *lout = nullptr;
  float* lseg = nullptr;                     // lin_mma: states between the segments of a step
  float* hs = nullptr;                       // the token-shifted mixer input of the step
  float* vfirst = nullptr;                   // [chunk][kv_heads * vdim] values of the step's tokens in the first value-mixing layer
  int* d_prev = nullptr;                     // the sequence's last token (bigram embedding)
  float *x = nullptr, *h = nullptr, *b0 = nullptr, *b1 = nullptr, *b2 = nullptr, *b3 = nullptr, *wgt = nullptr, *logits = nullptr;
  // pinned staging of a chunk's first position, token ids and wanted rows (behind dsk_state::h_ctrl, with h_err), two of them: [4] [chunk] [chunk], on the
  // device d_ctl, d_tok and d_want
  int* h_in[2] = {nullptr, nullptr};
  cudaEvent_t in_ev[2] = {nullptr, nullptr};   // its copy is through
  // attention of portions in one kernel (pattn): split keys and values of the visible positions, queries it takes at a time
  __nv_bfloat16 *k16 = nullptr, *v16 = nullptr;
  float* ppart = nullptr;                    // partial softmax results of shares of the keys: a CTA of 128 rows an SM (launches that fill the chip are not split)
  int pattn_q = 0;
  // bf16 products of portions: activations rounded for the product that follows, hidden rows of a feed-forward, and a host word that a wait
  // which gave up sets
  __nv_bfloat16 *a16 = nullptr, *hid16 = nullptr;
  // rows of the width that products read, rounded by the kernel that made them (h, hs or x: `mirror`, until something else writes it)
  __nv_bfloat16* h16 = nullptr;
  const float* mirror = nullptr;
  size_t a16_elems = 0, hid16_elems = 0;
  int* h_err = nullptr;
  // device memory of the state: one allocation, cut into the pieces that salloc was asked for (portion: one that only the attention of portions needs; seq: caches and carried
  // states of the sequence)
  struct Piece { void** at; size_t bytes; bool portion, seq; };
  std::vector<Piece> pieces;
  char *arena = nullptr, *seq = nullptr;     // seq: what a new sequence finds zeroed (Piece::seq), in one run
  size_t seq_bytes = 0;
  // side-by-side mixers run on two streams, forked and joined by events
  cudaStream_t side = nullptr;
  cudaEvent_t ev_fork = nullptr, ev_join = nullptr;
  cudaGraphExec_t step_graph = nullptr;      // captured greedy decode step (arg-max -> token -> one-token chunk)
  // DSK_HY_TIMELINE=1: CUDA events between the groups of launches of every step, summed per label and printed to stderr
  bool timeline = false;
  std::vector<cudaEvent_t> tl_events;
  std::vector<const char*> tl_labels;
  size_t tl_used = 0;
  long long launches = 0;
};

static constexpr int kPrefillQ = 256, kPrefillMin = 32;   // prefill attention: queries per block / smallest portion that takes the matrix path
// Buffers of the attention of portions: a state takes them up to this size (blocks of kPrefillQ queries of the fused kernel, the smallest there are: up to
// half as much again).  Heads x keys decide: 16 key heads of 64 + 64 entries take 25 KB a key.
static constexpr size_t kPortionBytes = (size_t)4 << 30;
static constexpr int kNarrowMin = 448;                           // rows from which a product of up to 96 columns runs on gemm_narrow
static constexpr int kAttnSplitMax = 64, kAttnSplitTokens = 4;   // decode-sized chunks split a window over up to 64 CTAs

static bool is_ssd(const dsk_layer_spec& s) { return s.mixer == DSK_MIX_SSD; }
static long long ssd_inner(const dsk_layer_spec& s) { return (long long)s.ssm_heads * s.ssm_vdim; }
static long long ssd_channels(const dsk_layer_spec& s) { return ssd_inner(s) + 2LL * s.ssm_groups * s.ssm_state; }
static long long ssd_proj(const dsk_layer_spec& s) { return ssd_inner(s) + ssd_channels(s) + s.ssm_heads; }

static bool has_gdn(const dsk_layer_spec& s) { return s.mixer == DSK_MIX_GDN || s.mixer2 == DSK_MIX_GDN; }
static long long gdn_qk(const dsk_layer_spec& s) { return has_gdn(s) ? (long long)s.gdn_kv_heads * s.gdn_dim : 0; }
static long long gdn_v(const dsk_layer_spec& s) { return has_gdn(s) ? (long long)s.gdn_heads * s.gdn_vdim : 0; }

// Columns of the stacked projection of attention with a value matrix and of the delta rule:  [q | k | v | gate], or, with a delta
// rule beside it (or alone),  [q | k | v | dq | dk | dv | dg | gate | db | da], padded with zero rows to a multiple of 8.
struct AttLayout {
  long long k = 0, v = 0, gate = 0, gate_rows = 0, dq = 0, dk = 0, dv = 0, dg = 0, db = 0, da = 0, total = 0;
};
static AttLayout att_layout(const dsk_layer_spec& s) {
  AttLayout a;
  long long n = 0;
  if (s.mixer == DSK_MIX_GQA) {
    a.k = (long long)s.att_heads * s.att_dim; a.v = a.k + (long long)s.att_kv_heads * s.att_dim; n = a.v + (long long)s.att_kv_heads * s.att_vdim;
    a.gate_rows = s.att_out_gate == DSK_GATE_ENTRY ? (long long)s.att_heads * s.att_vdim : s.att_out_gate == DSK_GATE_HEAD ? s.att_heads : 0;
  }
  if (has_gdn(s)) { a.dq = n; a.dk = a.dq + gdn_qk(s); a.dv = a.dk + gdn_qk(s); a.dg = a.dv + gdn_v(s); n = a.dg + gdn_v(s); }
  a.gate = n; n += a.gate_rows;
  if (has_gdn(s)) { a.db = n; a.da = n + s.gdn_heads; n = (a.da + s.gdn_heads + 7) / 8 * 8; }
  a.total = n;
  return a;
}

// rows of an mLSTM mixer's stacked projection: [q | k | v | g | i | f], padded with zero rows to a multiple of 8
struct MlstmLayout { long long k, v, g, i, f, total; };
static MlstmLayout mlstm_layout(const dsk_layer_spec& s) {
  const long long HN = (long long)s.lin_heads * s.lin_dim, HP = (long long)s.lin_heads * s.lin_vdim;
  MlstmLayout a{HN, 2 * HN, 2 * HN + HP, 2 * HN + 2 * HP, 2 * HN + 2 * HP + s.lin_heads, 0};
  a.total = (a.f + s.lin_heads + 7) / 8 * 8;
  return a;
}
static bool has_attn(const dsk_layer_spec& s) { return s.mixer == DSK_MIX_GQA || s.mixer == DSK_MIX_MLA || s.mixer == DSK_MIX_LATENT_SWA; }

// key heads per CTA of the decode-sized attention kernel: without score mixing as few as keep four query heads (half the warps) busy
static int gqa_key_heads(int H, int G, bool talk) {
  int GL = G;
  if (!talk)
    for (int d = G; d >= 1; d--) if (G % d == 0 && d * (H / G) >= 4) GL = d;
  return GL;
}

static int validate(const dsk_hybrid_config& c, const dsk_layer_spec* L) {
  if (c.dim <= 0 || c.vocab_size <= 0 || c.n_layers <= 0 || c.max_seq_len <= 0) return fail(-1, "hybrid model: bad dimensions");
  if (c.quant != DSK_F32 && c.quant != DSK_BF16) return fail(-1, "hybrid models run with quant fp32 or bf16");
  if (c.norm_groups <= 0 || c.dim % c.norm_groups != 0) return fail(-1, "norm groups %d do not divide width %d", c.norm_groups, c.dim);
  if (c.chunk < 1 || c.chunk > 4096) return fail(-1, "chunk %d out of range (1..4096)", c.chunk);
  if (c.side_dim < 0) return fail(-1, "negative side_dim");
  if (c.block != DSK_BLOCK_PARALLEL && c.block != DSK_BLOCK_SANDWICH && c.block != DSK_BLOCK_POST && c.block != DSK_BLOCK_PRE) return fail(-1, "unknown block kind %d", c.block);
  if (c.block == DSK_BLOCK_PRE && (c.norm_kind != DSK_NORM_RMS || c.norm_groups != 1 || c.token_shift || c.side_dim > 0))
    return fail(-1, "pre-norm blocks run with ungrouped RMS norms, without a token shift and without the per-layer token input");
  if (c.norm_one_plus && (c.norm_kind != DSK_NORM_RMS || c.norm_scalar)) return fail(-1, "norm weights stored around zero belong to RMS norms with a weight vector");
  if (c.loop_embed && c.block != DSK_BLOCK_PRE) return fail(-1, "a layer loop that adds the embedding again belongs to pre-norm blocks");
  if (!(c.logit_softcap >= 0.f)) return fail(-1, "negative logit cap");
  if (c.block == DSK_BLOCK_POST && (c.norm_groups != 1 || c.loop_times >= 1))
    return fail(-1, "post-norm blocks run with ungrouped norms and without a layer loop");
  if (c.block == DSK_BLOCK_POST && c.norm_kind == DSK_NORM_LAYER && c.norm_scalar) return fail(-1, "single-number norm weights belong to RMS norms");
  if (c.norm_bias && c.norm_kind != DSK_NORM_LAYER) return fail(-1, "norm biases belong to layer norms");
  if (c.norm_bias && c.block == DSK_BLOCK_SANDWICH) return fail(-1, "sandwich blocks run their layer norms without a bias");
  if (c.block != DSK_BLOCK_POST && (c.canon_taps || c.res_gate || c.norm_scalar))
    return fail(-1, "input convolutions, gated residuals and single-number norm weights belong to post-norm blocks");
  if (c.layer_scale && c.block != DSK_BLOCK_POST && c.block != DSK_BLOCK_SANDWICH) return fail(-1, "layer scales belong to post-norm and sandwich blocks");
  if (c.loop_in && (c.block != DSK_BLOCK_SANDWICH || c.loop_embed)) return fail(-1, "loop passes that open with a product belong to sandwich blocks");
  if (c.canon_taps < 0 || c.canon_taps > kCanonMaxTaps) return fail(-1, "input convolution of %d taps unsupported (at most %d)", c.canon_taps, kCanonMaxTaps);
  if (c.bigram_buckets < 0) return fail(-1, "negative bigram table size");
  if (c.norm_kind != DSK_NORM_RMS && c.norm_kind != DSK_NORM_LAYER) return fail(-1, "unknown norm kind %d", c.norm_kind);
  if (c.loop_times >= 1 && (c.loop_start < 0 || c.loop_stop > c.n_layers || c.loop_start > c.loop_stop))
    return fail(-1, "layer loop %d..%d outside the %d layers", c.loop_start, c.loop_stop, c.n_layers);
  for (int i = 0; i < c.n_layers; i++) {
    const dsk_layer_spec& s = L[i];
    if (s.mixer2 != 0 && !(s.mixer2 == DSK_MIX_GDN && s.mixer == DSK_MIX_GQA && s.att_value_proj && s.att_kv_from < 0 && !s.att_vmix))
      return fail(-1, "layer %d: two mixers side by side are attention with its own value matrix and the delta rule", i);
    if (has_gdn(s)) {
      if (s.gdn_heads <= 0 || s.gdn_kv_heads <= 0 || s.gdn_dim <= 0 || s.gdn_vdim <= 0 || s.gdn_conv < 1) return fail(-1, "layer %d: bad delta-rule sizes", i);
      if (s.gdn_heads % s.gdn_kv_heads != 0) return fail(-1, "layer %d: delta-rule heads %d not a multiple of its key heads %d", i, s.gdn_heads, s.gdn_kv_heads);
      if (s.gdn_dim > 256) return fail(-1, "layer %d: key size %d > 256 unsupported (the recurrence keeps the state in registers)", i, s.gdn_dim);
    }
    if (s.mixer == DSK_MIX_SSD) {
      if (s.ssm_heads <= 0 || s.ssm_vdim <= 0 || s.ssm_state <= 0 || s.ssm_groups <= 0 || s.ssm_conv < 1 || s.ssm_norm_groups <= 0)
        return fail(-1, "layer %d: bad state-space mixer sizes", i);
      if (s.ssm_heads % s.ssm_groups != 0) return fail(-1, "layer %d: heads %d not a multiple of groups %d", i, s.ssm_heads, s.ssm_groups);
      if ((s.ssm_heads * s.ssm_vdim) % s.ssm_norm_groups != 0) return fail(-1, "layer %d: norm_groups does not divide the inner width", i);
      if (s.ssm_state > 256) return fail(-1, "layer %d: state size %d > 256 unsupported (the scan keeps the state in registers)", i, s.ssm_state);
    } else if (s.mixer == DSK_MIX_LATENT_SWA) {
      if (s.att_heads <= 0 || s.att_dim <= 0 || s.att_vdim <= 0 || s.att_kv_rank <= 0 || s.att_window <= 0)
        return fail(-1, "layer %d: bad latent-attention sizes", i);
      if (s.att_kv_rank > 1024) return fail(-1, "layer %d: kv_rank %d > 1024 unsupported", i, s.att_kv_rank);
      if (s.att_kv_from >= 0) {
        const int j = s.att_kv_from;
        if (j >= i || L[j].mixer != DSK_MIX_LATENT_SWA || L[j].att_kv_from >= 0 || L[j].att_kv_rank != s.att_kv_rank)
          return fail(-1, "layer %d: kv_from %d must name an earlier latent-attention layer that projects its own latent of the same rank", i, j);
      }
    } else if (s.mixer == DSK_MIX_GQA) {
      if (s.att_heads <= 0 || s.att_kv_heads <= 0 || s.att_dim <= 0 || s.att_vdim <= 0 || s.att_window <= 0) return fail(-1, "layer %d: bad attention sizes", i);
      if (s.att_heads % s.att_kv_heads != 0) return fail(-1, "layer %d: heads %d not a multiple of kv_heads %d", i, s.att_heads, s.att_kv_heads);
      if (!s.att_value_proj && s.att_vdim != s.att_dim) return fail(-1, "layer %d: values come out of the key matrix, so vdim %d must equal dim %d", i, s.att_vdim, s.att_dim);
      if (s.att_bias && !s.att_value_proj) return fail(-1, "layer %d: projection biases need the stacked q / k / v projection (att_value_proj)", i);
      if (s.att_talk && (s.att_softcap > 0.f || s.att_rel_max > 0)) return fail(-1, "layer %d: head mixing together with a score cap or distance bias is undefined", i);
      if (s.att_keep_first < 0 || (s.att_keep_first > 0 && s.att_mask != DSK_MASK_WINDOW)) return fail(-1, "layer %d: kept first positions belong to a window mask", i);
      if (s.att_rel_max < 0 || s.att_softcap < 0.f) return fail(-1, "layer %d: negative score cap or distance limit", i);
      if (s.rot_dims < 0 || s.rot_dims > s.att_dim || s.rot_dims % 2 != 0) return fail(-1, "layer %d: rot dims %d must be even and at most dim %d", i, s.rot_dims, s.att_dim);
      if (s.rot_dims > 0 && !(s.rot_base > 0.f)) return fail(-1, "layer %d: bad rotation base", i);
      if ((s.rot_layout != DSK_ROT_PAIRS && s.rot_layout != DSK_ROT_HALF) || (s.rot_scale != DSK_ROTSCALE_YARN && s.rot_scale != DSK_ROTSCALE_BANDS) ||
          (s.att_qk_norm != DSK_QKNORM_WHOLE && s.att_qk_norm != DSK_QKNORM_HEAD && s.att_qk_norm != DSK_QKNORM_HEAD_WEIGHT))
        return fail(-1, "layer %d: unknown rotation layout, rotation scaling or query / key norm", i);
      if (s.rot_scale == DSK_ROTSCALE_BANDS && s.rot_factor > 0.f && (!(s.rot_fast > s.rot_slow) || s.rot_original <= 0))
        return fail(-1, "layer %d: wavelength-band rotation scaling needs high > low and a positive original length", i);
      if (s.att_out_gate < DSK_GATE_NONE || s.att_out_gate > DSK_GATE_HEAD) return fail(-1, "layer %d: unknown output gate %d", i, s.att_out_gate);
      if (s.att_out_gate && !s.att_value_proj) return fail(-1, "layer %d: the output gate's rows ride in the stacked q / k / v projection (att_value_proj)", i);
      if (s.att_kv_from >= 0) {
        const int j = s.att_kv_from;
        if (j >= i || L[j].mixer != DSK_MIX_GQA || L[j].att_kv_from >= 0)
          return fail(-1, "layer %d: kv_from %d must name an earlier attention layer that projects its own keys and values", i, j);
        const dsk_layer_spec& o = L[j];
        if (s.att_out_gate == DSK_GATE_HEAD) return fail(-1, "layer %d: a per-head output gate belongs to a layer with its own keys and values", i);
        if (o.att_kv_heads != s.att_kv_heads || o.att_dim != s.att_dim || o.att_vdim != s.att_vdim || o.att_keep_first != s.att_keep_first || !o.att_value_proj ||
            !s.att_value_proj || s.att_vmix || s.att_bias)
          return fail(-1, "layer %d: a layer that reads layer %d's keys and values needs its key heads, sizes and kept positions, a value matrix there, and no biases or value mixing of its own", i, j);
      }
      if (s.att_sink < DSK_SINK_NONE || s.att_sink > DSK_SINK_ONE) return fail(-1, "layer %d: unknown softmax sink %d", i, s.att_sink);
      if (s.att_conv < 0 || (s.att_conv > 0 && (!s.att_value_proj || s.att_qk_norm != DSK_QKNORM_HEAD_WEIGHT || s.att_kv_from >= 0 || s.att_vmix || s.mixer2)))
        return fail(-1, "layer %d: convolutions behind the projections need a value matrix, weighted per-head norms, and no shared caches, value mixing or second mixer", i);
      if (s.att_conv > 0 && s.att_dim > 1024) return fail(-1, "layer %d: head size %d > 1024 unsupported behind convolutions", i, s.att_dim);
      const int GL = gqa_key_heads(s.att_heads, s.att_kv_heads, s.att_talk != 0);
      if (gqa_attn_smem_floats(GL * (s.att_heads / s.att_kv_heads), GL, s.att_dim, s.att_vdim, s.att_talk != 0) * 4 > 200 * 1024)
        return fail(-1, "layer %d: %d heads x %d with %d key heads do not fit the attention kernel's shared memory", i, s.att_heads, s.att_dim, s.att_kv_heads);
    } else if (s.mixer == DSK_MIX_MLA) {
      if (s.att_heads <= 0 || s.att_dim <= 0 || s.att_rot_dim < 0 || s.att_vdim <= 0 || s.att_kv_rank <= 0 || s.att_q_rank <= 0 || s.att_window <= 0)
        return fail(-1, "layer %d: bad latent-attention sizes", i);
      if (s.att_kv_rank + s.att_rot_dim > 1024) return fail(-1, "layer %d: kv_rank + rot_dim %d > 1024 unsupported", i, s.att_kv_rank + s.att_rot_dim);
      if (s.rot_dims < 0 || s.rot_dims > s.att_rot_dim || s.rot_dims % 2 != 0) return fail(-1, "layer %d: rot dims %d must be even and at most rot_dim %d", i, s.rot_dims, s.att_rot_dim);
      if (s.rot_dims > 0 && !(s.rot_base > 0.f)) return fail(-1, "layer %d: bad rotation base", i);
      if (s.rot_layout != DSK_ROT_PAIRS && s.rot_layout != DSK_ROT_HALF) return fail(-1, "layer %d: unknown rotation layout", i);
      if (s.rot_factor > 0.f && (s.rot_scale != DSK_ROTSCALE_YARN || !(s.rot_base > 1.f) || s.rot_original <= 0 || !(s.rot_fast > 0.f) || !(s.rot_slow > 0.f)))
        return fail(-1, "layer %d: bad rotation scaling", i);
      if (s.att_sink < DSK_SINK_NONE || s.att_sink > DSK_SINK_ONE) return fail(-1, "layer %d: unknown softmax sink %d", i, s.att_sink);
    } else if (s.mixer == DSK_MIX_MLSTM) {
      if (s.lin_heads <= 0 || s.lin_dim <= 0 || s.lin_vdim <= 0 || !(s.lin_gate_cap > 0.f)) return fail(-1, "layer %d: bad matrix-memory sizes or gate cap", i);
      if (s.lin_dim > 256) return fail(-1, "layer %d: key size %d > 256 unsupported (the recurrence keeps the state in registers)", i, s.lin_dim);
    } else if (s.mixer == DSK_MIX_HGRN2) {
      if (s.lin_heads <= 0 || s.lin_dim <= 0 || s.lin_vdim <= 0) return fail(-1, "layer %d: bad linear-recurrence sizes", i);
      if (s.lin_dim > 256) return fail(-1, "layer %d: key size %d > 256 unsupported (the recurrence keeps the state in registers)", i, s.lin_dim);
    } else if (s.mixer == DSK_MIX_LIGHTNING) {
      if (s.lin_heads <= 0 || s.lin_dim <= 0 || s.lin_vdim <= 0 || !s.lin_decay) return fail(-1, "layer %d: bad lightning-attention sizes or no decays", i);
      if (s.lin_dim > 256) return fail(-1, "layer %d: key size %d > 256 unsupported (the recurrence keeps the state in registers)", i, s.lin_dim);
      for (int h = 0; h < s.lin_heads; h++) if (!(s.lin_decay[h] >= 0.f && s.lin_decay[h] <= 1.f)) return fail(-1, "layer %d: decay %g of head %d outside 0..1", i, (double)s.lin_decay[h], h);
    } else if (s.mixer != DSK_MIX_GDN) return fail(-1, "layer %d: unknown mixer %d", i, s.mixer);
    if (has_attn(s) && s.att_mask != DSK_MASK_WINDOW && s.att_mask != DSK_MASK_CHUNK) return fail(-1, "layer %d: unknown mask %d", i, s.att_mask);
    if (s.ff_kind == DSK_FF_DENSE) {
      if (s.ff_hidden <= 0) return fail(-1, "layer %d: bad feed-forward size", i);
      if (s.ff_act != DSK_ACT_XIELU && s.ff_act != DSK_ACT_GEGLU && s.ff_act != DSK_ACT_GLU_CLAMPED && s.ff_act != DSK_ACT_SWIGLU) return fail(-1, "layer %d: unknown activation %d", i, s.ff_act);
    } else if (s.ff_kind == DSK_FF_MOE) {
      if (s.ff_experts <= 0 || s.ff_top <= 0 || s.ff_top > s.ff_experts || s.ff_hidden <= 0) return fail(-1, "layer %d: bad routed feed-forward sizes", i);
      if (s.ff_experts > 4096) return fail(-1, "layer %d: more than 4096 experts unsupported", i);
      if (s.ff_router < DSK_ROUTER_SIGMOID || s.ff_router > DSK_ROUTER_SOFTMAX_GROUPS || s.ff_expert < DSK_EXPERT_GLU_CLAMPED || s.ff_expert > DSK_EXPERT_SWIGLU)
        return fail(-1, "layer %d: unknown router or expert kind", i);
      const int groups = std::max(1, s.ff_groups), keep = s.ff_groups > 0 ? s.ff_groups_keep : 1;
      if (s.ff_groups < 0 || s.ff_experts % groups != 0 || keep < 1 || keep > groups || s.ff_top > s.ff_experts / groups * keep)
        return fail(-1, "layer %d: %d expert groups, %d kept, do not fit %d experts of which %d are taken", i, s.ff_groups, s.ff_groups_keep, s.ff_experts, s.ff_top);
      if (groups > 1 && s.ff_router != DSK_ROUTER_SOFTMAX_GROUPS) return fail(-1, "layer %d: expert groups belong to the softmax router", i);
      if (s.ff_shared < 0 || (s.ff_shared > 0 && s.ff_expert == DSK_EXPERT_RELU2)) return fail(-1, "layer %d: a shared expert needs gated experts", i);
    } else if (s.ff_kind != DSK_FF_NONE) return fail(-1, "layer %d: unknown feed-forward kind %d", i, s.ff_kind);
  }
  return 0;
}

// attention of portions in one kernel: sizes and the layers that take it (no mixing of the heads' scores, a tile of keys that fits)
static constexpr int kPattnSmemMax = 220 * 1024, kPattn5SmemMax = 226 * 1024;
struct PattnSize { int parts, G, D, V, Dp, Vp, VN; };
static PattnSize pattn_size(const dsk_layer_spec& s, bool bf16) {
  PattnSize z;
  z.parts = s.mixer == DSK_MIX_LATENT_SWA && bf16 ? 1 : 3;
  z.G = s.mixer == DSK_MIX_GQA ? s.att_kv_heads : s.att_heads;
  z.D = s.att_dim + (s.mixer == DSK_MIX_MLA ? s.att_rot_dim : 0); z.V = s.att_vdim;
  z.VN = z.V <= 64 ? 8 : 16;
  z.Dp = (z.D + 15) / 16 * 16; z.Vp = (z.V + z.VN * 8 - 1) / (z.VN * 8) * (z.VN * 8);
  return z;
}
static bool takes_pattn(const dsk_layer_spec& s, bool bf16) {
  if (!has_attn(s) || (s.mixer == DSK_MIX_GQA && s.att_talk)) return false;
  const PattnSize z = pattn_size(s, bf16);
  return pattn_smem(z.parts, 2, z.Dp, z.VN, 4) <= (size_t)kPattnSmemMax;
}

static void set_kernel_attrs() {
  static bool done = false;
  if (done) return;
  const int big = 200 * 1024;
  cudaFuncSetAttribute(ssd_scan<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, big); cudaFuncSetAttribute(ssd_scan<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, big);
  cudaFuncSetAttribute(ssd_scan<3>, cudaFuncAttributeMaxDynamicSharedMemorySize, big); cudaFuncSetAttribute(ssd_scan<4>, cudaFuncAttributeMaxDynamicSharedMemorySize, big);
  cudaFuncSetAttribute(ssd_scan<6>, cudaFuncAttributeMaxDynamicSharedMemorySize, big); cudaFuncSetAttribute(ssd_scan<8>, cudaFuncAttributeMaxDynamicSharedMemorySize, big);
  cudaFuncSetAttribute(gemm_mma<HEPI_STORE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMmaSmem);
  cudaFuncSetAttribute(gemm_mma<HEPI_ADD>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMmaSmem);
  cudaFuncSetAttribute(gemm_mma<HEPI_GLU>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMmaSmem);
  cudaFuncSetAttribute(gemm_mma<HEPI_GELU_MUL>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMmaSmem);
  cudaFuncSetAttribute(gemm_mma<HEPI_XIELU>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMmaSmem);
  cudaFuncSetAttribute(gemm_mma<HEPI_GEGLU>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMmaSmem);
  cudaFuncSetAttribute(gemm_mma<HEPI_SIGMUL>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMmaSmem);
  cudaFuncSetAttribute(gemm_mma<HEPI_RELU2>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMmaSmem);
  cudaFuncSetAttribute(gemm_mma<HEPI_LINGATE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMmaSmem);
  cudaFuncSetAttribute(hgrn2_scan<1, 8>, cudaFuncAttributeMaxDynamicSharedMemorySize, big); cudaFuncSetAttribute(hgrn2_scan<2, 8>, cudaFuncAttributeMaxDynamicSharedMemorySize, big);
  cudaFuncSetAttribute(hgrn2_scan<3, 8>, cudaFuncAttributeMaxDynamicSharedMemorySize, big); cudaFuncSetAttribute(hgrn2_scan<4, 8>, cudaFuncAttributeMaxDynamicSharedMemorySize, big);
  cudaFuncSetAttribute(hgrn2_scan<6, 8>, cudaFuncAttributeMaxDynamicSharedMemorySize, big); cudaFuncSetAttribute(hgrn2_scan<8, 8>, cudaFuncAttributeMaxDynamicSharedMemorySize, big);
  cudaFuncSetAttribute(hgrn2_scan<1, 16>, cudaFuncAttributeMaxDynamicSharedMemorySize, big); cudaFuncSetAttribute(hgrn2_scan<2, 16>, cudaFuncAttributeMaxDynamicSharedMemorySize, big);
  cudaFuncSetAttribute(hgrn2_scan<3, 16>, cudaFuncAttributeMaxDynamicSharedMemorySize, big); cudaFuncSetAttribute(hgrn2_scan<4, 16>, cudaFuncAttributeMaxDynamicSharedMemorySize, big);
  cudaFuncSetAttribute(hgrn2_scan<1, 32>, cudaFuncAttributeMaxDynamicSharedMemorySize, big); cudaFuncSetAttribute(hgrn2_scan<2, 32>, cudaFuncAttributeMaxDynamicSharedMemorySize, big);
  cudaFuncSetAttribute(gemm_mma<HEPI_SILU_SIG>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMmaSmem);
  cudaFuncSetAttribute(gemm_mma<HEPI_SOFTCAP>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMmaSmem);
  cudaFuncSetAttribute(lin_mma<8>, cudaFuncAttributeMaxDynamicSharedMemorySize, LinMma<8>::SMEM); cudaFuncSetAttribute(lin_mma<16>, cudaFuncAttributeMaxDynamicSharedMemorySize, LinMma<16>::SMEM);
#define DSK_LSCAN_ATTR(A, B, C) \
  cudaFuncSetAttribute(lin_scan<true, A, B, C>, cudaFuncAttributeMaxDynamicSharedMemorySize, big); \
  cudaFuncSetAttribute(lin_scan<false, A, B, C>, cudaFuncAttributeMaxDynamicSharedMemorySize, big)
  DSK_LSCAN_ATTR(8, 1, 2); DSK_LSCAN_ATTR(16, 1, 2); DSK_LSCAN_ATTR(32, 1, 2); DSK_LSCAN_ATTR(8, 1, 4); DSK_LSCAN_ATTR(16, 1, 4); DSK_LSCAN_ATTR(32, 1, 4); DSK_LSCAN_ATTR(32, 2, 4);
#undef DSK_LSCAN_ATTR
  cudaFuncSetAttribute(gemm_mma<HEPI_SWIGLU>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMmaSmem);
#define DSK_PATTN_ATTR(A, B) cudaFuncSetAttribute(pattn<A, B, 4, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kPattnSmemMax); cudaFuncSetAttribute(pattn<A, B, 2, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kPattnSmemMax); \
  cudaFuncSetAttribute(pattn<A, B, 4, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kPattnSmemMax); cudaFuncSetAttribute(pattn<A, B, 2, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kPattnSmemMax)
  DSK_PATTN_ATTR(1, 8); DSK_PATTN_ATTR(1, 16); DSK_PATTN_ATTR(3, 8); DSK_PATTN_ATTR(3, 16);
#undef DSK_PATTN_ATTR
#define DSK_PATTN5_ATTR(A, B) cudaFuncSetAttribute(pattn5<A, B>, cudaFuncAttributeMaxDynamicSharedMemorySize, kPattn5SmemMax)
  DSK_PATTN5_ATTR(1, 1); DSK_PATTN5_ATTR(1, 2); DSK_PATTN5_ATTR(3, 1); DSK_PATTN5_ATTR(3, 2);
#undef DSK_PATTN5_ATTR
#define DSK_SPLIT_ATTR(E) cudaFuncSetAttribute(gemm_split<E, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, split_smem(kSplitStages)); \
  cudaFuncSetAttribute(gemm_split<E, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, split_smem(kSplitStages))
  DSK_SPLIT_ATTR(HEPI_STORE); DSK_SPLIT_ATTR(HEPI_ADD); DSK_SPLIT_ATTR(HEPI_GLU); DSK_SPLIT_ATTR(HEPI_XIELU); DSK_SPLIT_ATTR(HEPI_GEGLU); DSK_SPLIT_ATTR(HEPI_SIGMUL);
  DSK_SPLIT_ATTR(HEPI_RELU2); DSK_SPLIT_ATTR(HEPI_LINGATE); DSK_SPLIT_ATTR(HEPI_SILU_SIG); DSK_SPLIT_ATTR(HEPI_SOFTCAP); DSK_SPLIT_ATTR(HEPI_SWIGLU); DSK_SPLIT_ATTR(HEPI_GELU_MUL);
#undef DSK_SPLIT_ATTR
#define DSK_TC5_ATTR(E) cudaFuncSetAttribute(gemm_tc5<E>, cudaFuncAttributeMaxDynamicSharedMemorySize, kTcSmem)
  DSK_TC5_ATTR(HEPI_STORE); DSK_TC5_ATTR(HEPI_ADD); DSK_TC5_ATTR(HEPI_GLU); DSK_TC5_ATTR(HEPI_XIELU); DSK_TC5_ATTR(HEPI_GEGLU); DSK_TC5_ATTR(HEPI_SIGMUL);
  DSK_TC5_ATTR(HEPI_RELU2); DSK_TC5_ATTR(HEPI_LINGATE); DSK_TC5_ATTR(HEPI_SILU_SIG); DSK_TC5_ATTR(HEPI_SOFTCAP); DSK_TC5_ATTR(HEPI_SWIGLU); DSK_TC5_ATTR(HEPI_GELU_MUL);
#undef DSK_TC5_ATTR
#define DSK_DECODE_ATTR(KV, CV) cudaFuncSetAttribute(decode_attn<KV, CV, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, big); cudaFuncSetAttribute(decode_attn<KV, CV, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, big)
  DSK_DECODE_ATTR(true, 1); DSK_DECODE_ATTR(true, 2); DSK_DECODE_ATTR(true, 4); DSK_DECODE_ATTR(false, 1); DSK_DECODE_ATTR(false, 2); DSK_DECODE_ATTR(false, 4);
#undef DSK_DECODE_ATTR
  cudaFuncSetAttribute(ssd_gram, cudaFuncAttributeMaxDynamicSharedMemorySize, big);
  cudaFuncSetAttribute(gqa_attn, cudaFuncAttributeMaxDynamicSharedMemorySize, big);
  cudaFuncSetAttribute(mix_softmax<0>, cudaFuncAttributeMaxDynamicSharedMemorySize, big); cudaFuncSetAttribute(mix_softmax<16>, cudaFuncAttributeMaxDynamicSharedMemorySize, big);
  cudaFuncSetAttribute(mix_softmax<32>, cudaFuncAttributeMaxDynamicSharedMemorySize, big);
  done = true;
}

static dsk_model* model_create(const dsk_hybrid_config* cfg, const dsk_layer_spec* layers, int rank, int n_ranks) {
  if (need_device()) return nullptr;
  if (!cfg || !layers) { fail(-1, "bad arguments"); return nullptr; }
  if (n_ranks != 1 || rank != 0) { fail(-1, "hybrid models run on one GPU (n_ranks must be 1)"); return nullptr; }
  if (validate(*cfg, layers)) return nullptr;
  set_kernel_attrs();
  dsk_model* m = new dsk_model();
  Model* M = new Model();
  m->hy = M;
  M->c = *cfg;
  M->wsize = cfg->quant == DSK_BF16 ? 2 : 4;
  m->c = dsk_config{};
  m->c.dim = cfg->dim; m->c.vocab_size = cfg->vocab_size; m->c.n_layers = cfg->n_layers; m->c.max_seq_len = cfg->max_seq_len;
  m->c.quant = cfg->quant; m->c.norm_eps = cfg->norm_eps;
  M->L.resize(cfg->n_layers);
  for (int i = 0; i < cfg->n_layers; i++) {
    HLayer& L = M->L[i];
    L.sp = layers[i];
    if (L.sp.mixer == DSK_MIX_LIGHTNING) {   // the decays and their logarithms (taken in double, rounded once)
      const size_t n = (size_t)L.sp.lin_heads * 4;
      std::vector<float> lg(L.sp.lin_heads);
      for (int h = 0; h < L.sp.lin_heads; h++) lg[h] = L.sp.lin_decay[h] > 0.f ? (float)std::log((double)L.sp.lin_decay[h]) : -1e30f;
      if (dmalloc(m, (void**)&L.decay, n) || dmalloc(m, (void**)&L.log_decay, n) || cudaMemcpy(L.decay, L.sp.lin_decay, n, cudaMemcpyHostToDevice) != cudaSuccess ||
          cudaMemcpy(L.log_decay, lg.data(), n, cudaMemcpyHostToDevice) != cudaSuccess) {
        fail(-2, "decay table allocation failed"); dsk_model_destroy(m); return nullptr;
      }
    }
    L.sp.lin_decay = nullptr;   // the caller's array
    if ((L.sp.mixer == DSK_MIX_GQA || L.sp.mixer == DSK_MIX_MLA) && L.sp.att_sink == DSK_SINK_ONE) {   // e^0 joins the softmax denominators
      if (dmalloc(m, (void**)&L.sink, (size_t)L.sp.att_heads * 4) || cudaMemset(L.sink, 0, (size_t)L.sp.att_heads * 4) != cudaSuccess) {
        fail(-2, "sink allocation failed"); dsk_model_destroy(m); return nullptr;
      }
    }
    if (L.sp.ff_kind == DSK_FF_MOE) L.have.assign(3 * (size_t)L.sp.ff_experts, 0);
    if (L.sp.mixer == DSK_MIX_LATENT_SWA) L.owner = L.sp.att_kv_from >= 0 ? L.sp.att_kv_from : i;
    if (L.sp.mixer == DSK_MIX_GQA) L.owner = L.sp.att_kv_from >= 0 ? L.sp.att_kv_from : i;
    if (L.sp.mixer == DSK_MIX_MLA) L.owner = i;
    if (L.sp.mixer == DSK_MIX_GQA && L.sp.att_vmix) {
      if (M->vmix_first < 0) M->vmix_first = i;
      else if ((long long)L.sp.att_kv_heads * L.sp.att_vdim != (long long)M->L[M->vmix_first].sp.att_kv_heads * M->L[M->vmix_first].sp.att_vdim) {
        fail(-1, "layer %d: value mixing needs as many value entries per token as layer %d has", i, M->vmix_first); dsk_model_destroy(m); return nullptr;
      }
    }
  }
  // ring caches: the owner keeps the widest window (or chunk of the mask) among its readers plus one step, capped by the sequence limit
  for (int i = 0; i < cfg->n_layers; i++) {
    const HLayer& L = M->L[i];
    if (L.owner < 0) continue;
    HLayer& O = M->L[L.owner];
    const long long need = (long long)L.sp.att_window - 1 + cfg->chunk;
    O.ring = (int)std::max<long long>(O.ring, std::min<long long>(need, (long long)cfg->max_seq_len));
  }
  // the order of layer runs: layers before the loop, the loop's passes, the layers after it
  const bool looped = cfg->loop_times >= 1 && cfg->loop_stop > cfg->loop_start;   // one pass is a loop too: it has its pass vector
  const int ls = looped ? cfg->loop_start : 0, le = looped ? cfg->loop_stop : 0, lt = looped ? cfg->loop_times : 0;
  for (int i = 0; i < ls; i++) M->runs.push_back(Run{i, -1, -1});
  for (int t = 0; t < lt; t++)
    for (int i = ls; i < le; i++) M->runs.push_back(Run{i, i == ls ? t : -1, -1});
  for (int i = le; i < cfg->n_layers; i++) M->runs.push_back(Run{i, -1, -1});
  for (size_t r = 0; r < M->runs.size(); r++) {   // a reader of another layer's latent cache reads that layer's latest run
    const int o = M->L[M->runs[r].layer].owner;
    if (o < 0) continue;
    for (int q = (int)r; q >= 0; q--)
      if (M->runs[q].layer == o) { M->runs[r].owner_run = q; break; }
    if (M->runs[r].owner_run < 0) { fail(-1, "layer %d reads the latent cache of layer %d, which has not run before it", M->runs[r].layer, o); dsk_model_destroy(m); return nullptr; }
  }
  // rotation tables of the attention layers that rotate: frequency per pair, in double, rounded once to fp32
  for (int i = 0; i < cfg->n_layers; i++) {
    HLayer& L = M->L[i];
    const dsk_layer_spec& s = L.sp;
    if ((s.mixer != DSK_MIX_GQA && s.mixer != DSK_MIX_MLA) || s.rot_dims <= 0) continue;
    const int half = s.rot_dims / 2;
    std::vector<float> f((size_t)half);
    const double base = s.rot_base, dims = s.rot_dims;
    const bool yarn = s.rot_factor > 0.f && (s.mixer != DSK_MIX_GQA || s.rot_scale == DSK_ROTSCALE_YARN);
    const bool bands = s.rot_factor > 0.f && s.mixer == DSK_MIX_GQA && s.rot_scale == DSK_ROTSCALE_BANDS;
    double lo = 0, hi = 0;
    if (yarn) {   // the pair index at which `original` positions hold t turns
      auto at = [&](double t) { return dims * std::log((double)s.rot_original / (2.0 * M_PI * t)) / (2.0 * std::log(base)); };
      lo = std::max(std::floor(at(s.rot_fast)), 0.0);
      hi = std::min(std::ceil(at(s.rot_slow)), dims - 1.0);
      L.rot_mag = (float)(0.1 * std::log((double)s.rot_factor) + 1.0);
    }
    for (int k = 0; k < half; k++) {
      double fr = std::pow(base, -2.0 * k / dims);
      if (yarn) {
        const double ramp = std::min(1.0, std::max(0.0, (k - lo) / std::max(hi - lo, 0.001)));
        fr = fr / s.rot_factor * ramp + fr * (1.0 - ramp);
      }
      if (bands) {   // by wavelength: short ones keep their frequency, long ones are slowed by the factor, a linear blend between
        const double wl = 2.0 * M_PI / fr, orig = s.rot_original;
        if (wl > orig / s.rot_slow) fr = fr / s.rot_factor;
        else if (!(wl < orig / s.rot_fast)) {
          const double sm = (orig / wl - s.rot_slow) / ((double)s.rot_fast - s.rot_slow);
          fr = (1.0 - sm) * fr / s.rot_factor + sm * fr;
        }
      }
      f[k] = (float)fr;
    }
    if (dmalloc(m, (void**)&L.rot_freq, (size_t)half * 4) || cudaMemcpy(L.rot_freq, f.data(), (size_t)half * 4, cudaMemcpyHostToDevice) != cudaSuccess) {
      fail(-2, "rotation table allocation failed"); dsk_model_destroy(m); return nullptr;
    }
  }
  return m;
}

static void model_free(dsk_model* m) { delete m->hy; m->hy = nullptr; }

template <typename ST>
static void launch_convert(const void* src, void* dst, long long rows, long long cols, int tr, bool to_bf16, long long ld) {
  const long long n = rows * cols;
  const unsigned grid = (unsigned)std::max<long long>(1, std::min<long long>((n + 255) / 256, 1 << 16));
  if (to_bf16) convert_kernel<ST, __nv_bfloat16><<<grid, 256>>>((const ST*)src, (__nv_bfloat16*)dst, rows, cols, tr, ld);
  else convert_kernel<ST, float><<<grid, 256>>>((const ST*)src, (float*)dst, rows, cols, tr, ld);
}

// payload (BF16 or F32; host or device) of logical shape rows x cols (cols == 0: a vector) -> dst (fp32 or bf16), optionally
// transposed per head (tr), or with its rows `ld` elements apart (0: packed)
static int put(const char* name, int dtype, const int64_t shape[4], const void* data, size_t nbytes, int on_dev, long long rows,
               long long cols, void* dst, bool to_bf16, int tr, long long ld = 0) {
  if (dtype != DSK_DT_BF16 && dtype != DSK_DT_F32) return fail(-4, "tensor %s: dtype %s unsupported (BF16 or F32)", name, dtype_name(dtype));
  const size_t es = dtype == DSK_DT_BF16 ? 2 : 4;
  const long long n = rows * std::max<long long>(cols, 1);
  if (shape[0] != rows || shape[1] != cols || shape[2] != 0 || nbytes != (size_t)n * es)
    return fail(-4, "tensor mismatch for %s: expected shape=[%lld,%lld], got shape=[%lld,%lld,%lld] (%zu bytes)", name, rows, cols,
                (long long)shape[0], (long long)shape[1], (long long)shape[2], nbytes);
  const void* src = data;
  void* staging = nullptr;
  if (!on_dev) {
    CK(cudaMalloc(&staging, nbytes ? nbytes : 16));
    CK(cudaMemcpy(staging, data, nbytes, cudaMemcpyHostToDevice));
    src = staging;
  }
  if (dtype == DSK_DT_BF16) launch_convert<__nv_bfloat16>(src, dst, rows, std::max<long long>(cols, 1), tr, to_bf16, ld ? ld : std::max<long long>(cols, 1));
  else launch_convert<float>(src, dst, rows, std::max<long long>(cols, 1), tr, to_bf16, ld ? ld : std::max<long long>(cols, 1));
  CK(cudaGetLastError());
  if (staging) { CK(cudaDeviceSynchronize()); CK(cudaFree(staging)); }
  return 0;
}

static int upload(dsk_model* m, const char* name, int dtype, const int64_t shape[4], const void* data, size_t nbytes, int on_dev) {
  Model* M = m->hy;
  const dsk_hybrid_config& c = M->c;
  const bool bf = c.quant == DSK_BF16;
  const std::string nm(name);
  // matrix in the model's quant type
  auto MAT = [&](HTensor& t, long long rows, long long cols, int tr = 0) -> int {
    if (t.present) return fail(-4, "tensor %s uploaded twice", name);
    if (dmalloc(m, &t.p, (size_t)rows * cols * M->wsize + 16)) return -2;
    t.rows = rows; t.cols = cols; t.present = true;
    return put(name, dtype, shape, data, nbytes, on_dev, rows, cols, t.p, bf, tr);
  };
  // fp32 side tensor (norm weights, biases, decays, router)
  auto F32 = [&](float** dst, long long rows, long long cols) -> int {
    if (*dst) return fail(-4, "tensor %s uploaded twice", name);
    if (dmalloc(m, (void**)dst, (size_t)rows * std::max<long long>(cols, 1) * 4)) return -2;
    return put(name, dtype, shape, data, nbytes, on_dev, rows, cols, *dst, false, 0);
  };
  // rows [row0, row0 + rows) of a matrix that stacks several checkpoint tensors (one product instead of several per step)
  auto STACK = [&](HTensor& st, long long total, long long cols, long long row0, long long rows, char* have) -> int {
    if (*have) return fail(-4, "tensor %s uploaded twice", name);
    if (!st.p) {
      if (dmalloc(m, &st.p, (size_t)total * cols * M->wsize + 16)) return -2;
      st.rows = total; st.cols = cols;
    }
    *have = 1;
    return put(name, dtype, shape, data, nbytes, on_dev, rows, cols, (char*)st.p + (size_t)row0 * cols * M->wsize, bf, 0);
  };
  auto STACKV = [&](float** dst, long long total, long long off, long long n, char* have) -> int {   // the same for fp32 vectors
    if (*have) return fail(-4, "tensor %s uploaded twice", name);
    if (!*dst) { if (dmalloc(m, (void**)dst, (size_t)total * 4)) return -2; }
    *have = 1;
    return put(name, dtype, shape, data, nbytes, on_dev, n, 0, *dst + off, false, 0);
  };
  // columns [col0, col0 + cols) of a matrix that holds two output matrices side by side
  auto COLS = [&](HTensor& st, long long rows, long long total, long long col0, long long cols, char* have) -> int {
    if (*have) return fail(-4, "tensor %s uploaded twice", name);
    if (!st.p) {
      if (dmalloc(m, &st.p, (size_t)rows * total * M->wsize + 16)) return -2;
      st.rows = rows; st.cols = total;
    }
    *have = 1;
    return put(name, dtype, shape, data, nbytes, on_dev, rows, cols, (char*)st.p + (size_t)col0 * M->wsize, bf, 0, total);
  };
  // weight of a norm outside the mixers, as it multiplies (1 + the stored one when weights are stored around zero)
  auto NORMW = [&](float** dst) -> int {
    if (int rc = F32(dst, c.dim, 0)) return rc;
    if (!c.norm_one_plus) return 0;
    std::vector<float> v((size_t)c.dim);
    CK(cudaMemcpy(v.data(), *dst, v.size() * 4, cudaMemcpyDeviceToHost));
    for (float& x : v) x += 1.f;
    CK(cudaMemcpy(*dst, v.data(), v.size() * 4, cudaMemcpyHostToDevice));
    return 0;
  };
  // a single number (shape []) -> host float
  auto SCALAR = [&](float* dst, char* have) -> int {
    if (*have) return fail(-4, "tensor %s uploaded twice", name);
    if (dtype != DSK_DT_BF16 && dtype != DSK_DT_F32) return fail(-4, "tensor %s: dtype %s unsupported (BF16 or F32)", name, dtype_name(dtype));
    const size_t es = dtype == DSK_DT_BF16 ? 2 : 4;
    if (shape[0] > 1 || shape[1] != 0 || nbytes != es) return fail(-4, "tensor mismatch for %s: expected a single number, got shape=[%lld,%lld] (%zu bytes)", name, (long long)shape[0], (long long)shape[1], nbytes);
    unsigned char raw[4] = {0, 0, 0, 0};
    if (on_dev) CK(cudaMemcpy(raw, data, es, cudaMemcpyDeviceToHost)); else memcpy(raw, data, es);
    uint32_t bits;
    if (es == 2) bits = ((uint32_t)raw[0] | ((uint32_t)raw[1] << 8)) << 16; else memcpy(&bits, raw, 4);
    memcpy(dst, &bits, 4);
    *have = 1;
    return 0;
  };
  if (nm == "embed") return MAT(M->embed, c.vocab_size, c.dim);
  if (nm == "bigram" && c.bigram_buckets > 0) return MAT(M->bigram, (long long)c.bigram_buckets + 1, c.dim);
  if (nm == "final.norm" && c.norm_scalar) {   // one number for all coordinates: kept as a constant vector, so every norm kernel takes it
    if (M->final_norm) return fail(-4, "tensor %s uploaded twice", name);
    float g = 0.f; char have = 0;
    if (int rc = SCALAR(&g, &have)) return rc;
    std::vector<float> v((size_t)c.dim, g);
    if (dmalloc(m, (void**)&M->final_norm, (size_t)c.dim * 4)) return -2;
    CK(cudaMemcpy(M->final_norm, v.data(), (size_t)c.dim * 4, cudaMemcpyHostToDevice));
    return 0;
  }
  if (nm == "final.norm") return NORMW(&M->final_norm);
  if (nm == "final.norm.b" && c.norm_bias) return F32(&M->final_norm_b, c.dim, 0);
  if (nm == "head") {
    if (c.tie_head) return fail(-4, "tensor %s: this model's LM head is its embedding table", name);
    return MAT(M->head, c.vocab_size, c.dim);
  }
  if (nm == "loop.step") {
    if (c.loop_times < 1) return fail(-4, "tensor %s: the model has no layer loop", name);
    return F32(&M->loop_step, c.loop_times, c.dim);
  }
  if (nm == "loop.in") {
    if (c.loop_times < 1 || !c.loop_in) return fail(-4, "tensor %s: the model has no such layer loop", name);
    return MAT(M->loop_in, c.dim, 2LL * c.dim);
  }
  if (nm == "side.embed") {
    if (c.side_dim <= 0) return fail(-4, "tensor %s: the model has no per-layer token input", name);
    return MAT(M->side_embed, c.vocab_size, (long long)c.side_dim * c.n_layers);
  }
  if (nm.size() < 3 || nm[0] != 'l') return fail(-4, "unknown tensor name %s", name);
  char* end = nullptr;
  const long li = strtol(name + 1, &end, 10);
  if (end == name + 1 || *end != '.' || li < 0 || li >= c.n_layers) return fail(-4, "unknown tensor name %s", name);
  HLayer& L = M->L[li];
  const dsk_layer_spec& s = L.sp;
  const std::string rest(end + 1);
  if (rest == "shift" && c.token_shift) return F32(&L.shift, c.dim, 0);
  if (c.norm_bias) {
    if (rest == "norm1.b") return F32(&L.norm1_bias, c.dim, 0);
    if (rest == "norm2.b" && s.ff_kind != DSK_FF_NONE) return F32(&L.norm2_bias, c.dim, 0);
  }
  if (c.block == DSK_BLOCK_POST) {
    const bool ff = s.ff_kind != DSK_FF_NONE;
    if (rest == "norm1") return c.norm_scalar ? SCALAR(&L.norm1_s, &L.have_n1) : F32(&L.norm1, c.dim, 0);
    if (rest == "norm2" && ff) return c.norm_scalar ? SCALAR(&L.norm2_s, &L.have_n2) : F32(&L.norm2, c.dim, 0);
    if (c.layer_scale) {
      if (rest == "ls1") return F32(&L.ls1, c.dim, 0);
      if (rest == "ls2" && ff) return F32(&L.ls2, c.dim, 0);
    }
    if (c.canon_taps > 0) {
      if (rest == "canon1") return F32(&L.canon1, c.dim, c.canon_taps);
      if (rest == "canon2" && ff) return F32(&L.canon2, c.dim, c.canon_taps);
    }
    if (c.res_gate) {
      if (rest == "rg1") return MAT(L.rg1, c.dim, c.dim);
      if (rest == "rg1.b") return F32(&L.rg1_b, c.dim, 0);
      if (rest == "rg2" && ff) return MAT(L.rg2, c.dim, c.dim);
      if (rest == "rg2.b" && ff) return F32(&L.rg2_b, c.dim, 0);
    }
  } else if (rest == "norm1") return NORMW(&L.norm1);
  if (c.block == DSK_BLOCK_PRE && rest == "norm2" && s.ff_kind != DSK_FF_NONE) return NORMW(&L.norm2);
  if (c.block == DSK_BLOCK_SANDWICH) {
    if (rest == "norm1b") return F32(&L.norm1b, c.dim, 0);
    if (rest == "norm2" && s.ff_kind != DSK_FF_NONE) return F32(&L.norm2, c.dim, 0);
    if (rest == "norm2b" && s.ff_kind != DSK_FF_NONE) return F32(&L.norm2b, c.dim, 0);
    if (rest == "ls1" && c.layer_scale) return F32(&L.ls1, c.dim, 0);
    if (rest == "ls2" && c.layer_scale && s.ff_kind != DSK_FF_NONE) return F32(&L.ls2, c.dim, 0);
  }
  if (rest.rfind("mix.", 0) == 0) {
    std::string k = rest.substr(4);
    bool right = s.mixer == DSK_MIX_GDN;
    if (s.mixer2) {
      if (k.rfind("left.", 0) == 0) k = k.substr(5);
      else if (k.rfind("right.", 0) == 0) { k = k.substr(6); right = true; }
      else return fail(-4, "unknown tensor name %s for two mixers side by side (mix.left.*, mix.right.*)", name);
    }
    if (right) {
      const AttLayout a = att_layout(s);
      const long long KD = gdn_qk(s), RV = gdn_v(s), HV = s.mixer2 ? (long long)s.att_heads * s.att_vdim : 0;
      if (!L.qkv.p) { if (dmalloc(m, &L.qkv.p, (size_t)a.total * c.dim * M->wsize + 16)) return -2; CK(cudaMemset(L.qkv.p, 0, (size_t)a.total * c.dim * M->wsize)); L.qkv.rows = a.total; L.qkv.cols = c.dim; }
      if (k == "q") return STACK(L.qkv, a.total, c.dim, a.dq, KD, &L.have_gdn[0]);
      if (k == "k") return STACK(L.qkv, a.total, c.dim, a.dk, KD, &L.have_gdn[1]);
      if (k == "v") return STACK(L.qkv, a.total, c.dim, a.dv, RV, &L.have_gdn[2]);
      if (k == "g") return STACK(L.qkv, a.total, c.dim, a.dg, RV, &L.have_gdn[3]);
      if (k == "b") return STACK(L.qkv, a.total, c.dim, a.db, s.gdn_heads, &L.have_gdn[4]);
      if (k == "a") return STACK(L.qkv, a.total, c.dim, a.da, s.gdn_heads, &L.have_gdn[5]);
      for (int n = 0; n < 3; n++)
        if (k == std::string(1, "qkv"[n]) + ".conv") {   // taps of the stacked [q | k | v] channels
          if (L.have_conv[n]) return fail(-4, "tensor %s uploaded twice", name);
          if (!L.gdn_conv_w && dmalloc(m, (void**)&L.gdn_conv_w, (size_t)(2 * KD + RV) * s.gdn_conv * 4)) return -2;
          L.have_conv[n] = 1;
          return put(name, dtype, shape, data, nbytes, on_dev, n < 2 ? KD : RV, s.gdn_conv, L.gdn_conv_w + (size_t)n * KD * s.gdn_conv, false, 0);
        }
      if (k == "A_log") return F32(&L.A_log, s.gdn_heads, 0);
      if (k == "dt_bias") return F32(&L.dt_bias, s.gdn_heads, 0);
      if (k == "norm") return F32(&L.lin_norm, s.gdn_vdim, 0);   // one weight vector for all heads
      if (k == "o") return COLS(L.o, c.dim, HV + RV, HV, RV, &L.have_o[1]);
    } else if (s.mixer == DSK_MIX_LIGHTNING) {
      const long long HN = (long long)s.lin_heads * s.lin_dim, HP = (long long)s.lin_heads * s.lin_vdim, tot = 2 * HN + 2 * HP;
      if (k == "q") return STACK(L.lin_in, tot, c.dim, 0, HN, &L.have_lin[0]);
      if (k == "k") return STACK(L.lin_in, tot, c.dim, HN, HN, &L.have_lin[1]);
      if (k == "v") return STACK(L.lin_in, tot, c.dim, 2 * HN, HP, &L.have_lin[2]);
      if (k == "g") return STACK(L.lin_in, tot, c.dim, 2 * HN + HP, HP, &L.have_lin[3]);
      if (k == "norm") return F32(&L.mnorm, HP, 0);
      if (k == "o") return MAT(L.o, c.dim, HP);
    } else if (s.mixer == DSK_MIX_MLSTM) {
      const long long H = s.lin_heads, HN = H * s.lin_dim, HP = H * s.lin_vdim;
      const MlstmLayout a = mlstm_layout(s);
      if (!L.lin_in.p) {
        if (dmalloc(m, &L.lin_in.p, (size_t)a.total * c.dim * M->wsize + 16) || dmalloc(m, (void**)&L.lin_bias, (size_t)a.total * 4)) return -2;
        CK(cudaMemset(L.lin_in.p, 0, (size_t)a.total * c.dim * M->wsize)); CK(cudaMemset(L.lin_bias, 0, (size_t)a.total * 4));
        L.lin_in.rows = a.total; L.lin_in.cols = c.dim;
      }
      if (k == "q") return STACK(L.lin_in, a.total, c.dim, 0, HN, &L.have_lin[0]);
      if (k == "k") return STACK(L.lin_in, a.total, c.dim, a.k, HN, &L.have_lin[1]);
      if (k == "v") return STACK(L.lin_in, a.total, c.dim, a.v, HP, &L.have_lin[2]);
      if (k == "g") return STACK(L.lin_in, a.total, c.dim, a.g, HP, &L.have_lin[3]);
      if (k == "i") return STACK(L.lin_in, a.total, c.dim, a.i, H, &L.have_gate[0]);
      if (k == "f") return STACK(L.lin_in, a.total, c.dim, a.f, H, &L.have_gate[1]);
      if (k == "i.b") return STACKV(&L.lin_bias, a.total, a.i, H, &L.have_gateb[0]);
      if (k == "f.b") return STACKV(&L.lin_bias, a.total, a.f, H, &L.have_gateb[1]);
      if (k == "norm") return F32(&L.mnorm, HP, 0);
      if (k == "o") return MAT(L.o, c.dim, HP);
    } else if (is_ssd(s)) {
      const long long inner = ssd_inner(s), ch = ssd_channels(s);
      if (k == "in") return MAT(L.in, ssd_proj(s), c.dim);
      if (k == "conv") return F32(&L.conv_w, ch, s.ssm_conv);
      if (k == "conv.b") return F32(&L.conv_b, ch, 0);
      if (k == "dt_bias") return F32(&L.dt_bias, s.ssm_heads, 0);
      if (k == "A_log") return F32(&L.A_log, s.ssm_heads, 0);
      if (k == "D") return F32(&L.D, s.ssm_heads, 0);
      if (k == "norm") return F32(&L.mnorm, inner, 0);
      if (k == "o") return MAT(L.o, c.dim, inner);
    } else if (s.mixer == DSK_MIX_HGRN2) {
      const long long HN = (long long)s.lin_heads * s.lin_dim, HP = (long long)s.lin_heads * s.lin_vdim, tot = 2 * HN + HP;
      if (k == "q") return STACK(L.lin_in, tot, c.dim, 0, HN, &L.have_lin[0]);
      if (k == "f") return STACK(L.lin_in, tot, c.dim, HN, HN, &L.have_lin[1]);
      if (k == "v") return STACK(L.lin_in, tot, c.dim, 2 * HN, HP, &L.have_lin[2]);
      if (k == "f.b") {   // the bias of the stacked product: zeros at the q and v rows
        if (!L.lin_bias) { if (dmalloc(m, (void**)&L.lin_bias, (size_t)tot * 4)) return -2; CK(cudaMemset(L.lin_bias, 0, (size_t)tot * 4)); }
        return STACKV(&L.lin_bias, tot, HN, HN, &L.have_linb);
      }
      if (k == "lower") return F32(&L.lower, HN, 0);
      if (k == "o") return MAT(L.o, c.dim, HP);
      if (k == "norm") return F32(&L.lin_norm, s.lin_vdim, 0);   // one weight vector for all heads
    } else if (s.mixer == DSK_MIX_MLA) {
      const long long H = s.att_heads, DK = s.att_dim + s.att_rot_dim, R = s.att_kv_rank, Q = s.att_q_rank, tot = Q + R + s.att_rot_dim;
      if (k == "dq") return STACK(L.in2, tot, c.dim, 0, Q, &L.have_in2[0]);
      if (k == "dkv") return STACK(L.in2, tot, c.dim, Q, R + s.att_rot_dim, &L.have_in2[1]);
      if (k == "dq.norm") return F32(&L.dq_norm, Q, 0);
      if (k == "dkv.norm") return F32(&L.dkv_norm, R, 0);
      if (k == "uq") return MAT(L.uq, H * DK, Q);
      if (k == "uk") { if (int rc = MAT(L.ukT, H * s.att_dim, R, s.att_dim)) return rc; return MAT(L.uk, H * s.att_dim, R); }
      if (k == "uv") return MAT(L.uv, H * s.att_vdim, R);
      if (k == "sink" && s.att_sink == DSK_SINK_HEAD) return F32(&L.sink, H, 0);
      if (k == "g" && s.att_out_gate) return MAT(L.gmat, H * s.att_vdim, c.dim);
      if (k == "o") return MAT(L.o, c.dim, H * s.att_vdim);
    } else if (s.mixer == DSK_MIX_GQA) {
      const long long HD = (long long)s.att_heads * s.att_dim, GD = (long long)s.att_kv_heads * s.att_dim, GV = (long long)s.att_kv_heads * s.att_vdim;
      const AttLayout a = att_layout(s);
      const long long HV = a.gate_rows;
      if (s.att_kv_from >= 0) {   // reads another layer's keys and values: only the query projection (and gate) of its own
        if (k == "q") return STACK(L.qkv, HD + HV, c.dim, 0, HD, &L.have_qkv[0]);
        if (k == "g" && s.att_out_gate) return STACK(L.qkv, HD + HV, c.dim, HD, HV, &L.have_qkv[3]);
      } else if (s.att_value_proj) {
        const long long tot = a.total;
        if (s.mixer2 && !L.qkv.p) { if (dmalloc(m, &L.qkv.p, (size_t)tot * c.dim * M->wsize + 16)) return -2; CK(cudaMemset(L.qkv.p, 0, (size_t)tot * c.dim * M->wsize)); L.qkv.rows = tot; L.qkv.cols = c.dim; }
        if (k == "g" && s.att_out_gate) return STACK(L.qkv, tot, c.dim, a.gate, HV, &L.have_qkv[3]);
        if (k == "q") return STACK(L.qkv, tot, c.dim, 0, HD, &L.have_qkv[0]);
        if (k == "k") return STACK(L.qkv, tot, c.dim, HD, GD, &L.have_qkv[1]);
        if (k == "v") return STACK(L.qkv, tot, c.dim, HD + GD, GV, &L.have_qkv[2]);
        if (s.att_bias) {
          if (!L.qkv_b && (HV > 0 || s.mixer2)) { if (dmalloc(m, (void**)&L.qkv_b, (size_t)tot * 4)) return -2; CK(cudaMemset(L.qkv_b, 0, (size_t)tot * 4)); }   // no bias on the gate's rows
          if (k == "q.b") return STACKV(&L.qkv_b, tot, 0, HD, &L.have_qkvb[0]);
          if (k == "k.b") return STACKV(&L.qkv_b, tot, HD, GD, &L.have_qkvb[1]);
          if (k == "v.b") return STACKV(&L.qkv_b, tot, HD + GD, GV, &L.have_qkvb[2]);
        }
      }
      if (s.att_conv > 0)
        for (int n = 0; n < 3; n++)
          if (k == std::string(1, "qkv"[n]) + ".conv") {
            if (L.have_conv[n]) return fail(-4, "tensor %s uploaded twice", name);
            if (!L.conv_w && dmalloc(m, (void**)&L.conv_w, (size_t)(HD + GD + GV) * s.att_conv * 4)) return -2;
            L.have_conv[n] = 1;
            return put(name, dtype, shape, data, nbytes, on_dev, n == 0 ? HD : n == 1 ? GD : GV, s.att_conv, L.conv_w + (size_t)(n == 0 ? 0 : n == 1 ? HD : HD + GD) * s.att_conv, false, (int)(n == 0 ? HD : n == 1 ? GD : GV));   // stored [taps][channels]
          }
      if (k == "rel" && s.att_rel_max > 0) {   // the number of distance buckets is the tensor's first size
        if (shape[0] < 2 || shape[0] > (1 << 20)) return fail(-4, "tensor %s: %lld distance buckets", name, (long long)shape[0]);
        L.rel_rows = (int)shape[0];
        return F32(&L.rel, shape[0], s.att_heads);
      }
      if (k == "sink" && s.att_sink == DSK_SINK_HEAD) return F32(&L.sink, s.att_heads, 0);
      if (k == "vmix" && s.att_vmix) return SCALAR(&L.vmix, &L.have_vmix);
      if (k == "vmix" || (k == "rel" && s.att_rel_max <= 0)) return 0;   // a checkpoint may carry them for layers that do not use them
      if (k == "q" && !s.att_value_proj) return MAT(L.q, HD, c.dim);
      if (k == "k" && !s.att_value_proj) return MAT(L.kproj, GD, c.dim);
      if (k == "q.norm" && s.att_qk_norm == DSK_QKNORM_HEAD_WEIGHT) return F32(&L.q_norm, s.att_dim, 0);
      if (k == "k.norm" && s.att_qk_norm == DSK_QKNORM_HEAD_WEIGHT) return F32(&L.k_norm, s.att_dim, 0);
      if (k == "q.norm" && s.att_qk_norm == DSK_QKNORM_WHOLE) return F32(&L.q_norm, HD, 0);
      if (k == "k.norm" && s.att_qk_norm == DSK_QKNORM_WHOLE) return F32(&L.k_norm, GD, 0);
      if (k == "talk" && s.att_talk) return F32(&L.talk, s.att_heads, s.att_heads);
      if (k == "o" && s.mixer2) return COLS(L.o, c.dim, (long long)s.att_heads * s.att_vdim + gdn_v(s), 0, (long long)s.att_heads * s.att_vdim, &L.have_o[0]);
      if (k == "o") return MAT(L.o, c.dim, (long long)s.att_heads * s.att_vdim);
    } else {
      const long long H = s.att_heads;
      if (k == "q") return MAT(L.q, H * s.att_dim, c.dim);
      if (k == "uk") { if (int rc = MAT(L.ukT, H * s.att_dim, s.att_kv_rank, s.att_dim)) return rc; return MAT(L.uk, H * s.att_dim, s.att_kv_rank); }
      if (k == "uv") return MAT(L.uv, H * s.att_vdim, s.att_kv_rank);
      if (k == "o") return MAT(L.o, c.dim, H * s.att_vdim);
      if (s.att_kv_from < 0) {
        if (k == "dkv") return MAT(L.dkv, s.att_kv_rank, c.dim);
        if (k == "dkv.norm") return F32(&L.dkv_norm, s.att_kv_rank, 0);
      }
    }
    return fail(-4, "unknown tensor name %s for this layer's mixer", name);
  }
  if (rest.rfind("mlp.", 0) == 0 && s.ff_kind == DSK_FF_DENSE && s.ff_act != DSK_ACT_XIELU) {
    const std::string k = rest.substr(4);
    if (k == "gate") return MAT(L.gate_d, s.ff_hidden, c.dim);
    if (k == "up") return MAT(L.up, s.ff_hidden, c.dim);
    if (k == "down") return MAT(L.down, c.dim, s.ff_hidden);
    return fail(-4, "unknown tensor name %s", name);
  }
  if (rest.rfind("mlp.", 0) == 0 && s.ff_kind == DSK_FF_DENSE) {
    const std::string k = rest.substr(4);
    if (k == "up") return MAT(L.up, s.ff_hidden, c.dim);
    if (k == "up.b") return F32(&L.up_b, s.ff_hidden, 0);
    if (k == "down") return MAT(L.down, c.dim, s.ff_hidden);
    if (k == "down.b") return F32(&L.down_b, c.dim, 0);
    if (k == "act") {   // the activation's two numbers enter as softplus(p) and 1/2 + softplus(q), in fp32
      if (int rc = F32(&L.act, 2, 0)) return rc;
      float pq[2];
      CK(cudaMemcpy(pq, L.act, sizeof(pq), cudaMemcpyDeviceToHost));
      auto softplus = [](float v) { return v > 20.f ? v : log1pf(expf(v)); };
      L.act_a = softplus(pq[0]);
      L.act_b = 0.5f + softplus(pq[1]);
      return 0;
    }
    return fail(-4, "unknown tensor name %s", name);
  }
  if (rest.rfind("mlp.", 0) == 0 && s.ff_kind == DSK_FF_MOE) {
    const std::string k = rest.substr(4);
    const long long E = s.ff_experts, ff = s.ff_hidden;
    if (s.ff_shared > 0) {   // the shared expert's weight row stands behind the router's rows: one product for both
      auto ROWS = [&](long long row0, long long rows, char* have) -> int {
        if (*have) return fail(-4, "tensor %s uploaded twice", name);
        if (!L.router && dmalloc(m, (void**)&L.router, (size_t)(E + 1) * c.dim * 4)) return -2;
        *have = 1;
        return put(name, dtype, shape, data, nbytes, on_dev, rows, c.dim, L.router + row0 * c.dim, false, 0);
      };
      if (k == "router") return ROWS(0, E, &L.have_router[0]);
      if (k == "shared.sg") return ROWS(E, 1, &L.have_router[1]);
      if (k == "shared.gate") return MAT(L.gate_sh, s.ff_shared, c.dim);
      if (k == "shared.up") return MAT(L.up_sh, s.ff_shared, c.dim);
      if (k == "shared.down") return MAT(L.down_sh, c.dim, s.ff_shared);
    }
    if (k == "router") return F32(&L.router, E, c.dim);
    if (k == "correction" && s.ff_router == DSK_ROUTER_SIGMOID) return F32(&L.correction, E, 0);
    if (k == "router.b" && s.ff_router == DSK_ROUTER_TOP_SOFTMAX) return F32(&L.router_b, E, 0);
    if (k.size() > 1 && k[0] == 'e') {
      char* e2 = nullptr;
      const long e = strtol(k.c_str() + 1, &e2, 10);
      if (e2 != k.c_str() + 1 && *e2 == '.' && e >= 0 && e < E) {
        const std::string part(e2 + 1);
        const int which = part == "gate" ? 0 : part == "up" ? 1 : part == "down" ? 2 : -1;
        if (which >= (s.ff_expert == DSK_EXPERT_RELU2 ? 1 : 0)) {
          HTensor& st = which == 0 ? L.gate_s : which == 1 ? L.up_s : L.down_s;
          if (!st.p) {
            if (dmalloc(m, &st.p, (size_t)E * ff * c.dim * M->wsize + 16)) return -2;
            st.rows = which == 2 ? c.dim : ff; st.cols = which == 2 ? ff : c.dim;
          }
          if (L.have[(size_t)which * E + e]) return fail(-4, "tensor %s uploaded twice", name);
          L.have[(size_t)which * E + e] = 1;
          return put(name, dtype, shape, data, nbytes, on_dev, st.rows, st.cols, (char*)st.p + (size_t)e * ff * c.dim * M->wsize, bf, 0);
        }
      }
    }
    return fail(-4, "unknown tensor name %s", name);
  }
  if (rest.rfind("side.", 0) == 0 && c.side_dim > 0) {
    const std::string k = rest.substr(5);
    if (k == "gate") return MAT(L.sgate, c.side_dim, c.dim);
    if (k == "proj") return MAT(L.sproj, c.dim, c.side_dim);
    if (k == "norm") return F32(&L.snorm, c.dim, 0);
  }
  return fail(-4, "unknown tensor name %s", name);
}

static int finalize(dsk_model* m) {
  Model* M = m->hy;
  const dsk_hybrid_config& c = M->c;
  if (!M->embed.present) return fail(-5, "missing tensor embed");
  if (!M->final_norm) return fail(-5, "missing tensor final.norm");
  if (c.norm_bias && !M->final_norm_b) return fail(-5, "missing tensor final.norm.b");
  if (c.side_dim > 0 && !M->side_embed.present) return fail(-5, "missing tensor side.embed");
  if (!c.tie_head && !M->head.present) return fail(-5, "missing tensor head");
  if (c.bigram_buckets > 0 && !M->bigram.present) return fail(-5, "missing tensor bigram");
  // closing norm weight of a post-norm sublayer: (norm weight, a vector or one number) x (layer scale), folded once in fp32
  auto fold = [&](const float* normv, float norm_s, const float* ls, float** out) -> int {
    std::vector<float> a((size_t)c.dim, norm_s), b((size_t)c.dim, 1.f);
    if (normv) CK(cudaMemcpy(a.data(), normv, (size_t)c.dim * 4, cudaMemcpyDeviceToHost));
    if (ls) CK(cudaMemcpy(b.data(), ls, (size_t)c.dim * 4, cudaMemcpyDeviceToHost));
    for (int i = 0; i < c.dim; i++) a[i] *= b[i];
    if (!*out && dmalloc(m, (void**)out, (size_t)c.dim * 4)) return -2;
    CK(cudaMemcpy(*out, a.data(), (size_t)c.dim * 4, cudaMemcpyHostToDevice));
    return 0;
  };
  CK(cudaDeviceSynchronize());
  if (c.loop_times >= 1 && c.loop_stop > c.loop_start && !M->loop_step) return fail(-5, "missing tensor loop.step");
  if (c.loop_in && c.loop_times >= 1 && c.loop_stop > c.loop_start && !M->loop_in.present) return fail(-5, "missing tensor loop.in");
  for (int i = 0; i < c.n_layers; i++) {
    HLayer& L = M->L[i];
    const dsk_layer_spec& s = L.sp;
    if (c.block == DSK_BLOCK_POST) {
      const bool ff = s.ff_kind != DSK_FF_NONE;
      if (c.norm_scalar ? (!L.have_n1 || (ff && !L.have_n2)) : (!L.norm1 || (ff && !L.norm2))) return fail(-5, "layer %d: missing norm tensors (norm1, norm2)", i);
      if (c.layer_scale && (!L.ls1 || (ff && !L.ls2))) return fail(-5, "layer %d: missing layer scale tensors (ls1, ls2)", i);
      if (c.canon_taps > 0 && (!L.canon1 || (ff && !L.canon2))) return fail(-5, "layer %d: missing input convolution tensors (canon1, canon2)", i);
      if (c.res_gate && (!L.rg1.present || !L.rg1_b || (ff && (!L.rg2.present || !L.rg2_b)))) return fail(-5, "layer %d: missing residual gate tensors (rg1, rg1.b, rg2, rg2.b)", i);
      if (fold(L.norm1, L.norm1_s, L.ls1, &L.close1) || (ff && fold(L.norm2, L.norm2_s, L.ls2, &L.close2))) return -2;
    } else if (!L.norm1) return fail(-5, "missing tensor l%d.norm1", i);
    if (c.token_shift && !L.shift) return fail(-5, "missing tensor l%d.shift", i);
    if (c.norm_bias && (!L.norm1_bias || (s.ff_kind != DSK_FF_NONE && !L.norm2_bias))) return fail(-5, "layer %d: missing norm biases (norm1.b, norm2.b)", i);
    if (c.block == DSK_BLOCK_PRE && s.ff_kind != DSK_FF_NONE && !L.norm2) return fail(-5, "missing tensor l%d.norm2", i);
    if (has_gdn(s)) {
      bool all = L.have_conv[0] && L.have_conv[1] && L.have_conv[2] && L.A_log && L.dt_bias && L.lin_norm && L.have_o[1];
      for (char h : L.have_gdn) all = all && h;
      if (!all) return fail(-5, "layer %d: missing delta-rule tensors (q, k, v and their conv, b, a, A_log, dt_bias, g, norm, o)", i);
      L.qkv.present = true;
      L.o.present = s.mixer == DSK_MIX_GDN || L.have_o[0];
    }
    if (c.block == DSK_BLOCK_SANDWICH && (!L.norm1b || (s.ff_kind != DSK_FF_NONE && (!L.norm2 || !L.norm2b))))
      return fail(-5, "layer %d: missing norm tensors (norm1b, norm2, norm2b)", i);
    if (c.block == DSK_BLOCK_SANDWICH) {   // closing norm weights, times the layer scales
      const bool ff = s.ff_kind != DSK_FF_NONE;
      if (c.layer_scale && (!L.ls1 || (ff && !L.ls2))) return fail(-5, "layer %d: missing layer scale tensors (ls1, ls2)", i);
      if (fold(L.norm1b, 1.f, L.ls1, &L.close1) || (ff && fold(L.norm2b, 1.f, L.ls2, &L.close2))) return -2;
    }
    if (s.mixer == DSK_MIX_GDN) {
    } else if (s.mixer == DSK_MIX_MLSTM) {
      L.lin_in.present = L.have_lin[0] && L.have_lin[1] && L.have_lin[2] && L.have_lin[3] && L.have_gate[0] && L.have_gate[1];
      if (!L.lin_in.present || !L.have_gateb[0] || !L.have_gateb[1] || !L.mnorm || !L.o.present) return fail(-5, "layer %d: missing matrix-memory tensors (mix.q, k, v, g, i, i.b, f, f.b, norm, o)", i);
    } else if (s.mixer == DSK_MIX_LIGHTNING) {
      L.lin_in.present = L.have_lin[0] && L.have_lin[1] && L.have_lin[2] && L.have_lin[3];
      if (!L.lin_in.present || !L.mnorm || !L.o.present) return fail(-5, "layer %d: missing lightning-attention tensors (mix.q, k, v, g, norm, o)", i);
    } else if (s.mixer == DSK_MIX_HGRN2) {
      L.lin_in.present = L.have_lin[0] && L.have_lin[1] && L.have_lin[2];
      if (!L.lin_in.present || !L.have_linb || !L.lower || !L.lin_norm || !L.o.present)
        return fail(-5, "layer %d: missing linear-recurrence tensors (mix.q, f, f.b, lower, v, norm, o)", i);
    } else if (s.mixer == DSK_MIX_GQA) {
      if (s.att_out_gate && !L.have_qkv[3]) return fail(-5, "layer %d: missing tensor mix.g", i);
      if (s.att_kv_from >= 0) {
        L.qkv.present = L.have_qkv[0];
        if (!L.qkv.present) return fail(-5, "layer %d: missing tensor mix.q", i);
      } else if (s.att_value_proj) {
        L.qkv.present = L.have_qkv[0] && L.have_qkv[1] && L.have_qkv[2];
        if (!L.qkv.present || (s.att_bias && !(L.have_qkvb[0] && L.have_qkvb[1] && L.have_qkvb[2]))) return fail(-5, "layer %d: missing attention projections (mix.q, k, v and their biases)", i);
      } else if (!L.q.present || !L.kproj.present) return fail(-5, "layer %d: missing attention tensors (mix.q, k)", i);
      if (!L.o.present || (s.att_qk_norm != DSK_QKNORM_HEAD && (!L.q_norm || !L.k_norm)) || (s.att_talk && !L.talk))
        return fail(-5, "layer %d: missing attention tensors (mix.q.norm, k.norm, talk, o)", i);
      if (s.att_conv > 0 && !(L.have_conv[0] && L.have_conv[1] && L.have_conv[2])) return fail(-5, "layer %d: missing convolution taps (mix.q.conv, k.conv, v.conv)", i);
      if ((s.att_sink && !L.sink) || (s.att_rel_max > 0 && !L.rel) || (s.att_vmix && !L.have_vmix && i != M->vmix_first))
        return fail(-5, "layer %d: missing attention tensors (mix.sink, rel, vmix)", i);
      if (s.att_rel_max > 0) {   // distance -> bucket, in double: below half the buckets one distance each, then logarithmic steps up to att_rel_max
        const int B = L.rel_rows, half = B / 2, D = s.att_rel_max;
        if (D <= half) return fail(-5, "layer %d: distance limit %d must exceed half of the %d distance buckets", i, D, B);
        std::vector<int> bk((size_t)D + 1);
        for (int n = 0; n <= D; n++)
          bk[n] = n < half ? n : std::min(B - 1, half + (int)std::floor(std::log((double)n / half) / std::log((double)D / half) * (B - half)));
        if (!L.rel_bucket && dmalloc(m, (void**)&L.rel_bucket, bk.size() * 4)) return -2;
        CK(cudaMemcpy(L.rel_bucket, bk.data(), bk.size() * 4, cudaMemcpyHostToDevice));
      }
    } else if (s.mixer == DSK_MIX_MLA) {
      L.in2.present = L.have_in2[0] && L.have_in2[1];
      if (!L.in2.present || !L.dq_norm || !L.dkv_norm || !L.uq.present || !L.ukT.present || !L.uk.present || !L.uv.present || !L.o.present || (s.att_out_gate && !L.gmat.present) || (s.att_sink && !L.sink))
        return fail(-5, "layer %d: missing latent-attention tensors (mix.dq, dq.norm, uq, dkv, dkv.norm, uk, uv, sink, g, o)", i);
    } else if (is_ssd(s)) {
      if (!L.in.present || !L.o.present || !L.conv_w || !L.conv_b || !L.dt_bias || !L.A_log || !L.D || !L.mnorm)
        return fail(-5, "layer %d: missing state-space mixer tensors (mix.in, conv, conv.b, dt_bias, A_log, D, norm, o)", i);
    } else {
      if (!L.q.present || !L.ukT.present || !L.uk.present || !L.uv.present || !L.o.present) return fail(-5, "layer %d: missing latent-attention tensors (mix.q, uk, uv, o)", i);
      if (s.att_kv_from < 0 && (!L.dkv.present || !L.dkv_norm)) return fail(-5, "layer %d: missing mix.dkv / mix.dkv.norm", i);
    }
    if (s.ff_kind == DSK_FF_DENSE && s.ff_act != DSK_ACT_XIELU) {
      if (!L.gate_d.present || !L.up.present || !L.down.present) return fail(-5, "layer %d: missing feed-forward tensors (mlp.gate, up, down)", i);
    } else if (s.ff_kind == DSK_FF_DENSE && (!L.up.present || !L.down.present || !L.up_b || !L.down_b || !L.act))
      return fail(-5, "layer %d: missing feed-forward tensors (mlp.up, up.b, down, down.b, act)", i);
    if (s.ff_kind == DSK_FF_MOE) {
      if (s.ff_shared > 0 && (!L.have_router[0] || !L.have_router[1] || !L.gate_sh.present || !L.up_sh.present || !L.down_sh.present))
        return fail(-5, "layer %d: missing mlp.router or shared expert tensors (mlp.shared.gate, up, down, sg)", i);
      if (!L.router || (s.ff_router == DSK_ROUTER_SIGMOID && !L.correction) || (s.ff_router == DSK_ROUTER_TOP_SOFTMAX && !L.router_b)) return fail(-5, "layer %d: missing mlp.router / mlp.correction / mlp.router.b", i);
      for (size_t k = s.ff_expert == DSK_EXPERT_RELU2 ? (size_t)s.ff_experts : 0; k < L.have.size(); k++)
        if (!L.have[k]) return fail(-5, "layer %d: missing expert tensor mlp.e%zu.%s", i, k % s.ff_experts, k / s.ff_experts == 0 ? "gate" : k / s.ff_experts == 1 ? "up" : "down");
    }
    if (c.side_dim > 0 && (!L.sgate.present || !L.sproj.present || !L.snorm)) return fail(-5, "layer %d: missing side.gate / side.proj / side.norm", i);
  }
  CK(cudaDeviceSynchronize());
  return 0;
}

// algorithmic weight bytes one decoded token streams
static double active_bytes(const dsk_model* m) {
  const Model* M = m->hy;
  const dsk_hybrid_config& c = M->c;
  const double ws = (double)M->wsize, W = c.dim;
  double tot = W * ws * (c.bigram_buckets > 0 ? 2 : 1) + (double)c.vocab_size * W * ws + W * 4;
  for (const Run& R : M->runs) {
    const HLayer& L = M->L[R.layer];
    const dsk_layer_spec& s = L.sp;
    double mat = 0, f32 = W;
    if (R.pass >= 0) { f32 += W; if (c.loop_in) mat += 2 * W * W; }
    if (c.block == DSK_BLOCK_PRE && s.ff_kind != DSK_FF_NONE) f32 += W;
    if (has_gdn(s)) {
      const double KD = (double)gdn_qk(s), RV = (double)gdn_v(s);
      mat += (2 * KD + 2 * RV + 2 * s.gdn_heads) * W + W * RV;
      f32 += (2 * KD + RV) * s.gdn_conv + 2 * s.gdn_heads + s.gdn_vdim;
    }
    if (c.block == DSK_BLOCK_SANDWICH) f32 += W * (s.ff_kind != DSK_FF_NONE ? 3 : 1);
    if (c.block == DSK_BLOCK_POST) {   // per sublayer: convolution taps, gate matrix and bias (the closing weight is the W counted above)
      const double subs = s.ff_kind != DSK_FF_NONE ? 2 : 1;
      f32 += subs * (W * c.canon_taps + (c.res_gate ? W : 0)) + (subs - 1) * W;
      if (c.res_gate) mat += subs * W * W;
    }
    if (c.token_shift) f32 += W;
    if (c.norm_bias) f32 += W * (s.ff_kind != DSK_FF_NONE ? 2 : 1);
    if (s.mixer == DSK_MIX_GDN) {
    } else if (s.mixer == DSK_MIX_MLSTM) {
      const double H = s.lin_heads, HN = H * s.lin_dim, HP = H * s.lin_vdim;
      mat += (2 * HN + 2 * HP + 2 * H) * W + W * HP;
      f32 += HP + 2 * H;
    } else if (s.mixer == DSK_MIX_LIGHTNING) {
      const double HN = (double)s.lin_heads * s.lin_dim, HP = (double)s.lin_heads * s.lin_vdim;
      mat += (2 * HN + 2 * HP) * W + W * HP;
      f32 += HP;
    } else if (s.mixer == DSK_MIX_HGRN2) {
      const double HN = (double)s.lin_heads * s.lin_dim, HP = (double)s.lin_heads * s.lin_vdim;
      mat += (2 * HN + HP) * W + W * HP;
      f32 += 3 * HN + 2 * HP;
    } else if (s.mixer == DSK_MIX_GQA) {
      const bool reads = s.att_kv_from >= 0;
      const double HD = (double)s.att_heads * s.att_dim, GD = reads ? 0.0 : (double)s.att_kv_heads * s.att_dim, GV = s.att_value_proj && !reads ? (double)s.att_kv_heads * s.att_vdim : 0.0;
      mat += (HD + GD + GV) * W + W * s.att_heads * s.att_vdim + W * (double)att_layout(s).gate_rows;
      f32 += (s.att_qk_norm == DSK_QKNORM_WHOLE ? HD + GD : s.att_qk_norm == DSK_QKNORM_HEAD_WEIGHT ? 2.0 * s.att_dim : 0.0) + (s.att_talk ? (double)s.att_heads * s.att_heads : 0.0) + (s.att_bias ? HD + GD + GV : 0.0) + (s.att_sink == DSK_SINK_HEAD ? s.att_heads : 0) + (HD + GD + GV) * s.att_conv;
    } else if (s.mixer == DSK_MIX_MLA) {
      const double H = s.att_heads, DK = s.att_dim + s.att_rot_dim, Rr = s.att_kv_rank, Q = s.att_q_rank;
      mat += (Q + Rr + s.att_rot_dim) * W + H * DK * Q + H * (s.att_dim + s.att_vdim) * Rr + (s.att_out_gate ? H * s.att_vdim * W : 0.0) + W * H * s.att_vdim;
      f32 += Q + Rr + (s.att_sink == DSK_SINK_HEAD ? H : 0.0);
    } else if (is_ssd(s)) { mat += (double)ssd_proj(s) * W + W * ssd_inner(s); f32 += (double)ssd_channels(s) * (s.ssm_conv + 1) + 3.0 * s.ssm_heads + ssd_inner(s); }
    else {
      mat += (double)s.att_heads * s.att_dim * W + (double)s.att_heads * (s.att_dim + s.att_vdim) * s.att_kv_rank + W * s.att_heads * s.att_vdim;
      if (s.att_kv_from < 0) { mat += (double)s.att_kv_rank * W; f32 += s.att_kv_rank; }
    }
    if (s.ff_kind == DSK_FF_MOE) { mat += (s.ff_expert == DSK_EXPERT_RELU2 ? 2.0 : 3.0) * s.ff_top * s.ff_hidden * W; f32 += (double)s.ff_experts * (W + 1); if (s.ff_shared > 0) { mat += 3.0 * s.ff_shared * W; f32 += W; } }
    if (s.ff_kind == DSK_FF_DENSE && s.ff_act != DSK_ACT_XIELU) mat += 3.0 * s.ff_hidden * W;
    else if (s.ff_kind == DSK_FF_DENSE) { mat += 2.0 * s.ff_hidden * W; f32 += s.ff_hidden + W; }
    if (c.side_dim > 0) { mat += 2.0 * c.side_dim * W + c.side_dim; f32 += W; }
    tot += mat * ws + f32 * 4;
  }
  return tot;
}

// value channels x key rows of a head that one CTA of the token-by-token kernel holds
static bool lin_decode_fits(int N, int P) {
  const int PL = (P + 3) / 4;
  return PL <= kLinDecodeThreads && (N + std::min(kLinDecodeThreads / PL, N) - 1) / std::min(kLinDecodeThreads / PL, N) <= 16;
}

// kernels one decoded token launches (embedding + layers + final norm + LM head + arg-max)
static bool fused_norms(const dsk_hybrid_config& c);
static bool rms_fused(const dsk_hybrid_config& c);
static int launches_per_token(const dsk_model* m) {
  const Model* M = m->hy;
  int n = fused_norms(M->c) ? 3 : 4;
  if (M->c.bigram_buckets > 0) n += 1;
  const bool sandwich = M->c.block == DSK_BLOCK_SANDWICH, post = M->c.block == DSK_BLOCK_POST;
  for (const Run& R : M->runs) {
    const HLayer& L = M->L[R.layer];
    const dsk_layer_spec& s = L.sp;
    if (M->c.token_shift && (&R == &M->runs[0] || !(post && M->c.side_dim > 0 && M->c.canon_taps <= 0))) n += 1;   // later runs: shifted by the previous run's last kernel
    if (post && M->c.canon_taps <= 0) n += (s.ff_kind != DSK_FF_NONE ? 2 : 1) * (1 + (M->c.res_gate ? 1 : 0));   // gate, closing norm
    else if (post) n += (s.ff_kind != DSK_FF_NONE ? 2 : 1) * (1 + (M->c.res_gate ? 1 : 0)) + (&R == &M->runs[0] && M->c.canon_taps > 0 ? 1 : 0);   // gate, closing norm + next convolution in one
    else if (fused_norms(M->c)) n += 1 + (s.ff_kind != DSK_FF_NONE ? 1 : 0) + (&R == &M->runs[0] ? 1 + (R.pass >= 0 ? 1 : 0) : 0);
    else n += 1 + (R.pass >= 0 ? 1 : 0) + (sandwich ? 1 + (s.ff_kind != DSK_FF_NONE ? 2 : 0) : 0);
    if (M->c.block == DSK_BLOCK_PRE && s.ff_kind != DSK_FF_NONE) n += 1;
    if (M->c.block == DSK_BLOCK_PRE && R.pass >= 0) n -= 1;   // the pass vector is added by the opening norm
    if (has_gdn(s)) n += lin_decode_fits(s.gdn_dim, s.gdn_vdim) ? 1 : 3 + (s.gdn_conv > 1 ? 1 : 0);
    if (s.mixer == DSK_MIX_GDN) n += 2;     // stacked projection, o
    else if (s.mixer == DSK_MIX_MLSTM) n += lin_decode_fits(s.lin_dim, s.lin_vdim) ? 3 : 6;   // stacked projection, (gates, records,) recurrence, (norm,) o
    else if (s.mixer == DSK_MIX_LIGHTNING) n += lin_decode_fits(s.lin_dim, s.lin_vdim) ? 4 : 5;   // stacked projection, (records,) recurrence, norm, o
    else if (s.mixer == DSK_MIX_HGRN2) n += 4;   // stacked projection, recurrence, head norm, o
    else if (s.mixer == DSK_MIX_GQA) n += s.att_value_proj ? 5 : 6;   // q, k (or one stacked q / k / v (/ gate) product), norm + rotation, attention, merge, o
    else if (s.mixer == DSK_MIX_MLA) n += 9 + (s.att_out_gate ? 1 : 0);   // down-projections, query norm, query up, latent preparation, absorbed query, attention, merge, value up, (gate,) o
    else n += is_ssd(s) ? 5 : 5 + (s.att_kv_from < 0 ? 2 : 0);
    if (s.ff_kind == DSK_FF_MOE) n += (post && M->c.norm_kind == DSK_NORM_LAYER && !M->c.res_gate && M->c.dim <= 256 * kLnRegs && s.ff_shared == 0) || rms_fused(M->c) ? 4 : 5;
    if (R.pass >= 0 && M->c.loop_in) n += 1 + (&R != &M->runs[0] && fused_norms(M->c) ? 1 : 0);   // product, its norm
    if (s.ff_kind == DSK_FF_DENSE) n += 2;
    if (M->c.side_dim > 0) n += 3;
  }
  return n;
}

// ---------------------------------------------------------------------------------------------------------------------
// state
// ---------------------------------------------------------------------------------------------------------------------
// Asks for a piece of the state's memory; *p is set by salloc_all.  A piece of 1 MB and more takes whole pages of 2 MB, as an allocation of its own does: with all pieces
// packed at 512 bytes, decoded tokens of two designs took 0.6 and 1.7 % longer (where caches, states and rows lie, not what is done with them).
constexpr size_t kStatePage = (size_t)2 << 20;
static int salloc(State* S, void** p, size_t bytes, bool portion = false, bool seq = false) {
  const size_t unit = bytes >= kStatePage / 2 ? kStatePage : 512;
  S->pieces.push_back({p, (std::max<size_t>(bytes, 16) + unit - 1) / unit * unit, portion, seq});
  return 0;
}
// All pieces in one allocation (an allocation and a zeroing for each of 30 to 50 pieces were most of the time that a state took to make and to free), zeroed.
// Where it does not fit with the buffers of the attention of portions, without them.
static int salloc_all(State* S, cudaStream_t st) {
  auto total = [&] { size_t n = 0; for (const State::Piece& q : S->pieces) n += q.bytes; return n; };
  if (cudaMalloc((void**)&S->arena, total()) != cudaSuccess) {
    cudaGetLastError();
    for (State::Piece& q : S->pieces) if (q.portion) { q.bytes = 0; S->prefill_keys = 0; }
    CK(cudaMalloc((void**)&S->arena, total()));
  }
  CK(cudaMemsetAsync(S->arena, 0, total(), st));
  // pages first; what a new sequence finds zeroed stands together, on the pages and behind them (a memset for every piece kept a short prompt waiting for 2 to 4 us each)
  auto place = [](const State::Piece& q) { return q.bytes % kStatePage == 0 ? (q.seq ? 1 : 0) : q.seq ? 2 : 3; };
  std::stable_sort(S->pieces.begin(), S->pieces.end(), [&](const State::Piece& a, const State::Piece& b) { return place(a) < place(b); });
  char* at = S->arena;
  for (const State::Piece& q : S->pieces) {
    *q.at = q.bytes ? at : nullptr;
    if (q.seq) { if (!S->seq) S->seq = at; S->seq_bytes = at + q.bytes - S->seq; }
    at += q.bytes;
  }
  return cudaStreamSynchronize(st) == cudaSuccess ? 0 : -2;
}

static int state_reset(dsk_state* s) {
  State* S = s->hy;
  if (S->seq_bytes) CK(cudaMemsetAsync(S->seq, 0, S->seq_bytes, s->stream));
  S->next_pos = 0;
  s->last_pos = -1;
  s->have_logits = false;
  return 0;
}

static dsk_state* state_create(dsk_model* m) {
  Model* M = m->hy;
  const dsk_hybrid_config& c = M->c;
  dsk_state* s = new dsk_state();
  State* S = new State();
  s->m = m;
  s->hy = S;
  S->chunk = c.chunk;
  S->width = c.dim;
  S->timeline = getenv("DSK_HY_TIMELINE") != nullptr;
  const size_t Tc = c.chunk;
  // the pieces the shared sampling / arg-max code reads
  salloc(S, (void**)&s->ctrl, sizeof(Ctrl));
  if (alloc_host_side(s, (2 * (2 * Tc + 4) + 1) * 4)) return nullptr;
  S->h_in[0] = (int*)(s->h_ctrl + 1); S->h_in[1] = S->h_in[0] + 2 * Tc + 4; S->h_err = S->h_in[1] + 2 * Tc + 4;   // (zeroed)
  s->token_log_cap = 1 << 16;
  salloc(S, (void**)&s->token_log, s->token_log_cap * sizeof(int));
  salloc(S, (void**)&s->step, sizeof(int));
  salloc(S, (void**)&s->sample_out, 4 * sizeof(float));
  salloc(S, (void**)&s->logits, (size_t)c.vocab_size * 4);
  cudaStreamCreateWithFlags(&s->stream, cudaStreamNonBlocking);
  cudaEventCreate(&s->ev0); cudaEventCreate(&s->ev1);
  for (cudaEvent_t& e : S->in_ev) cudaEventCreateWithFlags(&e, cudaEventDisableTiming);
  if (cudaGetLastError() != cudaSuccess) { fail(-2, "state allocation failed"); return nullptr; }
  size_t mx0 = c.dim, mx1 = c.dim, mx2 = c.dim, mx3 = c.dim, mxE = 1, mxTop = 1;
  S->L.resize(M->runs.size());   // one state per layer run
  bool any_talk = false;
  size_t mxLQ = 0, mxLV = 0, mxLH = 0, mxMH = 0, mxShared = 0, mxSeg = 0;
  size_t mxGV = 0;
  for (size_t r = 0; r < M->runs.size(); r++) {
    const int i = M->runs[r].layer;
    const HLayer& L = M->L[i];
    const dsk_layer_spec& sp = L.sp;
    LayerState& ls = S->L[r];
    if (c.block == DSK_BLOCK_POST && c.canon_taps > 1) {
      ls.canon_bytes = (size_t)2 * (c.canon_taps - 1) * c.dim * 4;
      if (salloc(S, (void**)&ls.canon, ls.canon_bytes, false, true)) return nullptr;
    }
    if (c.token_shift) {
      ls.shift_bytes = (size_t)c.dim * 4;
      if (salloc(S, (void**)&ls.shift, ls.shift_bytes, false, true)) return nullptr;
    }
    if (has_gdn(sp)) {
      const size_t KD = gdn_qk(sp), RV = gdn_v(sp), NP = (size_t)sp.gdn_kv_heads * ((sp.gdn_dim + 3) & ~3);
      ls.lin_bytes = (size_t)sp.gdn_heads * sp.gdn_dim * sp.gdn_vdim * 4;
      ls.hist_bytes = (size_t)(sp.gdn_conv - 1 + kConvSpare) * (2 * KD + RV) * 4;
      if (salloc(S, (void**)&ls.lin, ls.lin_bytes, false, true) || salloc(S, (void**)&ls.hist, ls.hist_bytes, false, true)) return nullptr;
      mxLQ = std::max(mxLQ, NP); mxLV = std::max(mxLV, RV); mxLH = std::max<size_t>(mxLH, sp.gdn_heads);
      mx0 = std::max<size_t>(mx0, att_layout(sp).total);
      mx3 = std::max<size_t>(mx3, RV + (sp.mixer2 ? (size_t)sp.att_heads * sp.att_vdim : 0));
    }
    if (sp.mixer == DSK_MIX_GDN) {
    } else if (sp.mixer == DSK_MIX_MLSTM) {
      const size_t H = sp.lin_heads, HN = H * sp.lin_dim, HP = H * sp.lin_vdim;
      ls.lin_bytes = (HN * sp.lin_vdim + HN + H) * 4;   // S, n, m
      if (salloc(S, (void**)&ls.lin, ls.lin_bytes, false, true)) return nullptr;
      mx0 = std::max<size_t>(mx0, mlstm_layout(sp).total); mx3 = std::max<size_t>(mx3, HP);
      mxLV = std::max(mxLV, HP); mxLH = std::max(mxLH, H); mxMH = std::max(mxMH, H);
      mxSeg = std::max(mxSeg, lin_mma_floats((int)H, sp.lin_vdim / 16 + 1, sp.lin_dim, kLmSegs));
    } else if (sp.mixer == DSK_MIX_LIGHTNING) {
      const size_t HN = (size_t)sp.lin_heads * sp.lin_dim, HP = (size_t)sp.lin_heads * sp.lin_vdim;
      ls.lin_bytes = HN * sp.lin_vdim * 4;
      if (salloc(S, (void**)&ls.lin, ls.lin_bytes, false, true)) return nullptr;
      mx0 = std::max<size_t>(mx0, 2 * HN + 2 * HP); mx3 = std::max<size_t>(mx3, HP);
      mxLV = std::max(mxLV, HP); mxLH = std::max<size_t>(mxLH, sp.lin_heads);
      mxSeg = std::max(mxSeg, lin_mma_floats(sp.lin_heads, (sp.lin_vdim + 15) / 16, sp.lin_dim, kLmSegs));
    } else if (sp.mixer == DSK_MIX_HGRN2) {
      const size_t HN = (size_t)sp.lin_heads * sp.lin_dim, HP = (size_t)sp.lin_heads * sp.lin_vdim;
      ls.lin_bytes = HN * sp.lin_vdim * 4;
      if (salloc(S, (void**)&ls.lin, ls.lin_bytes, false, true)) return nullptr;
      mx0 = std::max<size_t>(mx0, 2 * HN + HP); mx2 = std::max<size_t>(mx2, HP); mx3 = std::max<size_t>(mx3, HP);
    } else if (sp.mixer == DSK_MIX_GQA) {
      const size_t HD = (size_t)sp.att_heads * sp.att_dim, GD = (size_t)sp.att_kv_heads * sp.att_dim, GV = (size_t)sp.att_kv_heads * sp.att_vdim;
      if (M->runs[r].owner_run == (int)r) {   // a layer that reads another layer's keys and values caches nothing
        const size_t rows = (size_t)sp.att_keep_first + L.ring;   // the kept first positions have rows of their own in front of the ring
        ls.cache_bytes = rows * GD * 4;
        ls.vcache_bytes = rows * GV * 4;
        if (salloc(S, &ls.cache, ls.cache_bytes, false, true) || salloc(S, &ls.vcache, ls.vcache_bytes, false, true)) return nullptr;
      }
      mx0 = std::max<size_t>(mx0, (sp.att_value_proj ? HD + GD + GV : HD) + (sp.att_out_gate ? (size_t)sp.att_heads * sp.att_vdim : 0)); mx1 = std::max<size_t>(mx1, GD); mx2 = std::max<size_t>(mx2, HD);
      mx3 = std::max<size_t>(mx3, (size_t)sp.att_heads * sp.att_vdim);
      any_talk |= sp.att_talk != 0;
      if (sp.att_conv > 1) {
        ls.hist_bytes = (size_t)(sp.att_conv - 1 + kConvSpare) * (HD + GD + GV) * 4;
        if (salloc(S, (void**)&ls.hist, ls.hist_bytes, false, true)) return nullptr;
      }
      if (sp.att_vmix) mxGV = std::max(mxGV, GV);
    } else if (sp.mixer == DSK_MIX_MLA) {
      const size_t H = sp.att_heads, RW = (size_t)sp.att_kv_rank + sp.att_rot_dim;
      ls.cache_bytes = (size_t)L.ring * RW * 4;
      if (salloc(S, &ls.cache, ls.cache_bytes, false, true)) return nullptr;
      mx0 = std::max<size_t>(mx0, std::max(H * (sp.att_dim + sp.att_rot_dim), H * sp.att_vdim));
      mx1 = std::max<size_t>(mx1, sp.att_q_rank + RW);
      mx2 = std::max<size_t>(mx2, std::max<size_t>(sp.att_q_rank, H * RW));
      mx3 = std::max<size_t>(mx3, std::max(H * RW, H * sp.att_vdim));
    } else if (is_ssd(sp)) {
      ls.ssm_bytes = (size_t)sp.ssm_heads * sp.ssm_vdim * sp.ssm_state * 4;
      ls.hist_bytes = (size_t)std::max(1, sp.ssm_conv - 1) * ssd_channels(sp) * 4;
      if (salloc(S, (void**)&ls.ssm, ls.ssm_bytes, false, true) || salloc(S, (void**)&ls.hist, ls.hist_bytes, false, true)) return nullptr;
      mx0 = std::max<size_t>(mx0, ssd_proj(sp)); mx1 = std::max<size_t>(mx1, ssd_channels(sp));
      mx2 = std::max<size_t>(mx2, ssd_inner(sp)); mx3 = std::max<size_t>(mx3, ssd_inner(sp));
      mxLH = std::max<size_t>(mxLH, sp.ssm_heads);
      mxSeg = std::max(mxSeg, lin_mma_floats(sp.ssm_heads, (sp.ssm_vdim + 15) / 16, sp.ssm_state, kLmSegs));
    } else {
      if (M->runs[r].owner_run == (int)r) {
        ls.cache_bytes = (size_t)L.ring * sp.att_kv_rank * 4;
        if (salloc(S, &ls.cache, ls.cache_bytes, false, true)) return nullptr;
      }
      mx0 = std::max<size_t>(mx0, std::max((size_t)sp.att_heads * sp.att_dim, (size_t)sp.att_heads * sp.att_vdim));
      mx1 = std::max<size_t>(mx1, sp.att_kv_rank);
      mx2 = std::max<size_t>(mx2, (size_t)sp.att_heads * sp.att_kv_rank);
      mx3 = std::max<size_t>(mx3, std::max((size_t)sp.att_heads * sp.att_kv_rank, (size_t)sp.att_heads * sp.att_vdim));
    }
    if (sp.ff_kind == DSK_FF_MOE) {
      mxE = std::max<size_t>(mxE, sp.ff_experts); mxTop = std::max<size_t>(mxTop, sp.ff_top);
      const size_t sh = sp.ff_shared > 0 ? 1 : 0;    // a shared expert's rows stand behind the routed ones'
      mx0 = std::max<size_t>(mx0, sp.ff_experts + sh); mxShared = std::max(mxShared, sh);
      mx2 = std::max<size_t>(mx2, (size_t)sp.ff_top * sp.ff_hidden + sp.ff_shared); mx3 = std::max<size_t>(mx3, (size_t)(sp.ff_top + sh) * c.dim);
    }
    if (sp.ff_kind == DSK_FF_DENSE) mx2 = std::max<size_t>(mx2, sp.ff_hidden);
    mx1 = std::max<size_t>(mx1, c.side_dim);
  }
  S->max_tiles = (int)(Tc * mxTop / 64 + mxE + 1);
  size_t mxHid = 0, mxRouted = 0;   // hidden rows of a feed-forward per token; inputs of routed rows per token
  for (const HLayer& L : M->L) {
    if (L.sp.ff_kind == DSK_FF_MOE) { mxHid = std::max<size_t>(mxHid, (size_t)L.sp.ff_top * L.sp.ff_hidden + L.sp.ff_shared); mxRouted = std::max<size_t>(mxRouted, (size_t)L.sp.ff_top * c.dim); }
    if (L.sp.ff_kind == DSK_FF_DENSE) mxHid = std::max<size_t>(mxHid, L.sp.ff_hidden);
  }
  int rc = 0;
  size_t mxPart = 0;
  for (const HLayer& L : M->L) {
    if (L.sp.mixer == DSK_MIX_LATENT_SWA) mxPart = std::max(mxPart, (size_t)kAttnSplitTokens * L.sp.att_heads * kAttnSplitMax * (L.sp.att_kv_rank + 2));
    if (L.sp.mixer == DSK_MIX_GQA) mxPart = std::max(mxPart, (size_t)kAttnSplitTokens * L.sp.att_heads * kAttnSplitMax * (L.sp.att_vdim + 2));
    if (L.sp.mixer == DSK_MIX_MLA) mxPart = std::max(mxPart, (size_t)kAttnSplitTokens * L.sp.att_heads * kAttnSplitMax * (L.sp.att_kv_rank + L.sp.att_rot_dim + 2));
  }
  rc |= salloc(S, (void**)&S->part, mxPart * 4);
  if ((int)Tc >= kPrefillMin) {   // buffers of the attention of portions, counted for the layers that use them; without them portions run like short steps
    const bool bf16 = c.quant == DSK_BF16;
    auto visible = [&](const dsk_layer_spec& sp, int q) {   // keys that a block of q queries can see
      return (size_t)std::min<long long>((long long)sp.att_window - 1, (long long)c.max_seq_len) + std::min<size_t>(Tc, q) + (sp.mixer == DSK_MIX_GQA ? sp.att_keep_first : 0);
    };
    // layers that run pattn: the visible keys and values split into bf16 parts, behind the up-projected fp32 rows of latent layers
    size_t k16 = 0, v16 = 0, kup = 0, vup = 0, rows = 0, shares = 0;
    auto fused_bytes = [&](int q) {
      k16 = v16 = kup = vup = 0;
      for (const HLayer& L : M->L) {
        if (!takes_pattn(L.sp, bf16)) continue;
        const PattnSize z = pattn_size(L.sp, bf16);
        const size_t n = visible(L.sp, q);
        shares = std::max<size_t>(shares, (size_t)g_sm_count * 128 * (z.V + 2) / (z.Vp / (z.VN * 8)));
        k16 = std::max(k16, n * z.G * z.Dp * z.parts); v16 = std::max(v16, n * z.G * z.Vp * z.parts);
        if (L.sp.mixer != DSK_MIX_GQA) { kup = std::max(kup, n * z.G * L.sp.att_dim); vup = std::max(vup, n * z.G * z.V); }
      }
      return 2 * (k16 + v16) + 4 * (kup + vup);
    };
    // the others, as matrix products between which the scores lie in memory: latent attention up-projects keys and values of all heads (fp32, then packed in
    // the matrix type; with a rotated key part in fp32: its scores are 32-bit products), grouped-query attention packs its cached key / value heads in fp32
    size_t keys = 0, hd = 0, hv = 0, heads = 0, pack_es = 0;
    auto plain_bytes = [&](int q) {
      keys = 0;
      for (const HLayer& L : M->L) {
        if (!has_attn(L.sp) || takes_pattn(L.sp, bf16)) continue;
        const size_t kh = L.sp.mixer == DSK_MIX_GQA ? L.sp.att_kv_heads : L.sp.att_heads;
        if (L.sp.mixer == DSK_MIX_LATENT_SWA) pack_es = std::max(pack_es, M->wsize);
        if (L.sp.mixer == DSK_MIX_MLA) pack_es = 4;
        keys = std::max(keys, visible(L.sp, q));
        hd = std::max<size_t>(hd, kh * (L.sp.att_dim + (L.sp.mixer == DSK_MIX_MLA ? L.sp.att_rot_dim : 0))); hv = std::max<size_t>(hv, kh * L.sp.att_vdim);
        heads = std::max<size_t>(heads, L.sp.att_heads);
      }
      return keys * (hd + hv) * (4 + pack_es) + heads * q * keys * 4;
    };
    // a whole step at a time where its keys take up to 4 GB, else blocks of kPrefillQ queries; layers that mix heads 512 queries at a time where
    // their scores fit (a head's product with the values is then 8 tiles)
    S->pattn_q = (int)Tc;
    size_t fused = fused_bytes(S->pattn_q);
    if (fused > kPortionBytes && S->pattn_q > kPrefillQ) fused = fused_bytes(S->pattn_q = kPrefillQ);
    S->talk_q = any_talk ? 2 * kPrefillQ : kPrefillQ;
    size_t plain = plain_bytes(S->talk_q);
    if (plain > kPortionBytes && any_talk) plain = plain_bytes(S->talk_q = kPrefillQ);
    for (const HLayer& L : M->L) if (has_attn(L.sp)) rows = std::max(rows, visible(L.sp, takes_pattn(L.sp, bf16) ? S->pattn_q : S->talk_q));
    if (rows > 0 && fused <= kPortionBytes + kPortionBytes / 2 && plain <= kPortionBytes) {
      S->prefill_keys = (int)rows;
      if (k16) rc |= salloc(S, (void**)&S->ppart, shares * 4, true) | salloc(S, (void**)&S->k16, k16 * 2, true) | salloc(S, (void**)&S->v16, v16 * 2, true);
      rc |= salloc(S, (void**)&S->kf, std::max(kup, keys * hd) * 4, true) | salloc(S, (void**)&S->vf, std::max(vup, (keys + 3) * hv) * 4, true);
      rc |= salloc(S, (void**)&S->d_rows, rows * 4, true);
      if (pack_es) rc |= salloc(S, &S->kb, keys * hd * pack_es, true) | salloc(S, &S->vt, keys * hv * pack_es, true);
      if (keys) rc |= salloc(S, (void**)&S->sc, heads * S->talk_q * (keys + 3) * 4, true);   // (rows of whole quads)
    }
  }
  rc |= salloc(S, (void**)&S->x, Tc * c.dim * 4) | salloc(S, (void**)&S->h, Tc * c.dim * 4);
  if (c.loop_embed && c.loop_times > 1) rc |= salloc(S, (void**)&S->emb, Tc * c.dim * 4);
  if (mxSeg && Tc >= 64) rc |= salloc(S, (void**)&S->lseg, mxSeg * 4);
  if (mxLH) rc |= salloc(S, (void**)&S->lrec, (Tc + kLinBlk - 1) / kLinBlk * mxLH * kRecFloats * 4) | salloc(S, (void**)&S->lout, Tc * mxLV * 4);
  for (const HLayer& L : M->L)
    if (L.sp.mixer2 && !S->side && (cudaStreamCreateWithFlags(&S->side, cudaStreamNonBlocking) != cudaSuccess || cudaEventCreateWithFlags(&S->ev_fork, cudaEventDisableTiming) != cudaSuccess ||
                                    cudaEventCreateWithFlags(&S->ev_join, cudaEventDisableTiming) != cudaSuccess)) { fail(-2, "stream creation failed"); return nullptr; }
  if (c.loop_in && c.loop_times >= 1) rc |= salloc(S, (void**)&S->xin, Tc * 2 * c.dim * 4);
  if (mxMH) rc |= salloc(S, (void**)&S->lgate, 3 * (Tc + 1) * mxMH * 4) | salloc(S, (void**)&S->lden, Tc * mxMH * 4);
  if (mxShared) rc |= salloc(S, (void**)&S->wsh, Tc * 4);
  if (mxLQ) rc |= salloc(S, (void**)&S->lq, Tc * mxLQ * 4) | salloc(S, (void**)&S->lk, Tc * mxLQ * 4) | salloc(S, (void**)&S->lv, Tc * mxLV * 4);
  if (c.block == DSK_BLOCK_SANDWICH || c.block == DSK_BLOCK_POST) rc |= salloc(S, (void**)&S->y, Tc * c.dim * 4);
  if (c.token_shift) rc |= salloc(S, (void**)&S->hs, Tc * c.dim * 4);
  if (mxGV) rc |= salloc(S, (void**)&S->vfirst, Tc * mxGV * 4);
  rc |= salloc(S, (void**)&S->d_prev, 16);
  rc |= salloc(S, (void**)&S->b0, Tc * mx0 * 4) | salloc(S, (void**)&S->b1, Tc * mx1 * 4) | salloc(S, (void**)&S->b2, Tc * mx2 * 4) | salloc(S, (void**)&S->b3, Tc * mx3 * 4);
  rc |= salloc(S, (void**)&S->wgt, Tc * mxTop * 4) | salloc(S, (void**)&S->d_idx, Tc * mxTop * 4) | salloc(S, (void**)&S->d_perm, Tc * mxTop * 4);
  rc |= salloc(S, (void**)&S->d_tiles, (size_t)S->max_tiles * sizeof(int4)) | salloc(S, (void**)&S->d_ntiles, 16);
  rc |= salloc(S, (void**)&S->d_ctl, (2 * Tc + 4) * 4);
  S->head_rows = (int)std::min<size_t>(Tc, 256);
  if (c.quant == DSK_BF16 && Tc > 4) {
    // a product's input is one of b0 .. b3, a row of 2 x width values (loop products), or latents of the visible keys
    size_t rank = 0;
    for (const HLayer& L : M->L) rank = std::max<size_t>(rank, has_attn(L.sp) && L.sp.mixer != DSK_MIX_GQA ? L.sp.att_kv_rank : 0);
    S->a16_elems = std::max(Tc * std::max({mx0, mx1, mx2, mx3, (size_t)2 * c.dim, mxRouted}), (size_t)S->prefill_keys * rank);
    S->hid16_elems = Tc * mxHid;
    rc |= salloc(S, (void**)&S->a16, S->a16_elems * 2) | salloc(S, (void**)&S->hid16, S->hid16_elems * 2) | salloc(S, (void**)&S->h16, Tc * c.dim * 2);
  }
  rc |= salloc(S, (void**)&S->logits, (size_t)S->head_rows * c.vocab_size * 4);
  if (rc || salloc_all(S, s->stream)) { fail(-2, "state allocation failed"); return nullptr; }
  S->d_tok = S->d_ctl + 4; S->d_want = S->d_tok + Tc;
  s->logits_src = s->logits;
  m->n_states++;
  return s;
}

static void state_free(dsk_state* s) {
  State* S = s->hy;
  if (!S) return;
  if (S->step_graph) cudaGraphExecDestroy(S->step_graph);
  if (S->side) { cudaStreamSynchronize(S->side); cudaStreamDestroy(S->side); cudaEventDestroy(S->ev_fork); cudaEventDestroy(S->ev_join); }
  for (cudaEvent_t e : S->tl_events) cudaEventDestroy(e);
  for (cudaEvent_t e : S->in_ev) if (e) cudaEventDestroy(e);
  cudaFree(S->arena);
  s->ctrl = nullptr; s->token_log = s->step = nullptr; s->sample_out = s->logits = nullptr;   // (pieces of it)
  delete S;
  s->hy = nullptr;
}

// ---------------------------------------------------------------------------------------------------------------------
// the chunk step
// ---------------------------------------------------------------------------------------------------------------------
// marks the end of a group of launches (timeline mode only; never inside a captured step)
static void mark(State* S, const char* label, cudaStream_t st) {
  if (!S->timeline) return;
  if (S->tl_used == S->tl_events.size()) { cudaEvent_t e; cudaEventCreate(&e); S->tl_events.push_back(e); S->tl_labels.push_back(label); }
  S->tl_labels[S->tl_used] = label;
  cudaEventRecord(S->tl_events[S->tl_used++], st);
}
static void timeline_report(State* S, int T) {
  if (!S->timeline || S->tl_used < 2) { S->tl_used = 0; return; }
  cudaEventSynchronize(S->tl_events[S->tl_used - 1]);
  std::map<std::string, double> sum;
  double tot = 0;
  for (size_t i = 1; i < S->tl_used; i++) {
    float ms = 0;
    cudaEventElapsedTime(&ms, S->tl_events[i - 1], S->tl_events[i]);
    sum[S->tl_labels[i]] += ms; tot += ms;
  }
  fprintf(stderr, "[dsk timeline] step of %d tokens: %.3f ms |", T, tot);
  for (auto& kv : sum) fprintf(stderr, " %s %.3f", kv.first.c_str(), kv.second);
  fprintf(stderr, "\n");
  S->tl_used = 0;
}

// Launches a kernel as a programmatic dependent of the one ahead of it in the stream: it is set up, and runs up to its grid_wait, while
// that one still runs.  Only in short steps (chain_step): their kernels take a few microseconds, about what a launch takes.  bf16, six models of two or three
// layers (widths 1024 and 2048), with against without: 5 tokens 15 - 18 % less, 45 tokens 11 - 17, 100 tokens 11 - 17, 256 tokens 6 - 13, and from
// there on not in all of them (400 and 512 tokens 0 to 14 % less, 1024 tokens 10 % less to 5 % more): 256 is the line.  fp32: up to 4 tokens 10 - 15 %
// less; 5 to 45 tokens 3 - 7 % less, 100 tokens 5 % less to 8 % more, 600 tokens 36 % more (1.88 to 2.56 ms: its products are about one CTA per SM, and waiting
// CTAs take the places that the running kernel leaves): 4 is the line.  plain_next: the coming launch waits
// as usual (it joins another stream).
static thread_local bool chain_step = false, plain_next = false;
template <typename... KA> struct Launch {
  void (*kernel)(KA...);
  cudaLaunchConfig_t cfg;
  unsigned cluster;   // CTAs of a cluster, along x
  template <typename... A> void operator()(A&&... a) const {
    static_assert(sizeof...(A) == sizeof...(KA), "every argument of a kernel is given");
    cudaLaunchAttribute at[2]{};
    cudaLaunchConfig_t c = cfg;
    c.attrs = at;
    c.numAttrs = 0;
    if (chain_step && !plain_next) {
      at[c.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
      at[c.numAttrs++].val.programmaticStreamSerializationAllowed = 1;
    }
    if (cluster > 1) {
      at[c.numAttrs].id = cudaLaunchAttributeClusterDimension;
      at[c.numAttrs].val.clusterDim.x = cluster; at[c.numAttrs].val.clusterDim.y = 1; at[c.numAttrs++].val.clusterDim.z = 1;
    }
    plain_next = false;
    cudaLaunchKernelEx(&c, kernel, static_cast<KA>(a)...);
  }
};
template <typename... KA>
static Launch<KA...> launch_next(void (*kernel)(KA...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, unsigned cluster = 1) {
  cudaLaunchConfig_t c{};
  c.gridDim = grid; c.blockDim = block; c.dynamicSmemBytes = smem; c.stream = st;
  return {kernel, c, cluster};
}

static GemmP gp(const float* A, int lda, const void* W, int ldw, float* C, int ldc, int M, int N, int K) {
  GemmP P{};
  P.A = A; P.lda = lda; P.W = W; P.ldw = ldw; P.C = C; P.ldc = ldc; P.M = M; P.N = N; P.K = K;
  P.a_div = 1; P.z_adiv = 1; P.z_wdiv = 1; P.alpha = 1.f;
  return P;
}

static void launch_gemm_mma(int epi, const GemmP& P, int Z, int tile_cap, cudaStream_t st) {
  const int bn = epi_dual(epi) ? 64 : 128;
  const dim3 grid((unsigned)((P.N + bn - 1) / bn), (unsigned)(P.tiles ? tile_cap : (P.M + 127) / 128), (unsigned)Z);
  switch (epi) {
    case HEPI_STORE: launch_next(gemm_mma<HEPI_STORE>, grid, 256, kMmaSmem, st)(P); break;
    case HEPI_ADD: launch_next(gemm_mma<HEPI_ADD>, grid, 256, kMmaSmem, st)(P); break;
    case HEPI_GLU: launch_next(gemm_mma<HEPI_GLU>, grid, 256, kMmaSmem, st)(P); break;
    case HEPI_XIELU: launch_next(gemm_mma<HEPI_XIELU>, grid, 256, kMmaSmem, st)(P); break;
    case HEPI_GEGLU: launch_next(gemm_mma<HEPI_GEGLU>, grid, 256, kMmaSmem, st)(P); break;
    case HEPI_SIGMUL: launch_next(gemm_mma<HEPI_SIGMUL>, grid, 256, kMmaSmem, st)(P); break;
    case HEPI_RELU2: launch_next(gemm_mma<HEPI_RELU2>, grid, 256, kMmaSmem, st)(P); break;
    case HEPI_LINGATE: launch_next(gemm_mma<HEPI_LINGATE>, grid, 256, kMmaSmem, st)(P); break;
    case HEPI_SILU_SIG: launch_next(gemm_mma<HEPI_SILU_SIG>, grid, 256, kMmaSmem, st)(P); break;
    case HEPI_SOFTCAP: launch_next(gemm_mma<HEPI_SOFTCAP>, grid, 256, kMmaSmem, st)(P); break;
    case HEPI_SWIGLU: launch_next(gemm_mma<HEPI_SWIGLU>, grid, 256, kMmaSmem, st)(P); break;
    default: launch_next(gemm_mma<HEPI_GELU_MUL>, grid, 256, kMmaSmem, st)(P); break;
  }
}

// ---- portions on the tensor cores (gemm_tc5) ----
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*, const cuuint32_t*,
                                  CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
static EncodeTiledFn encode_tiled() {
  static EncodeTiledFn fn = [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess || q != cudaDriverEntryPointSuccess) p = nullptr;
    return (EncodeTiledFn)p;
  }();
  return fn;
}
// bf16 rows x cols matrix of pitch ld, copied in boxes of box_rows x 64 (elements past its edges read as zeros)
static bool tile_map(CUtensorMap* m, const void* p, long long rows, long long cols, long long ld, int box_rows) {
  const cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows}, strides[1] = {(cuuint64_t)ld * 2};
  const cuuint32_t box[2] = {(cuuint32_t)kTcDepth, (cuuint32_t)box_rows}, one[2] = {1, 1};
  return encode_tiled()(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(p), dims, strides, box, one, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                        CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}
// Whether a product of more than four rows runs on gemm_tc5: bf16 matrices whose rows TMA can address (16-byte base and pitch), one batch,
// and room for the rounded activations.  gemm_mma takes the others (odd sizes, per-head batches).
static bool tc_ok(const State* S, bool bf16, int epi, const GemmP& P, int Z) {
  auto al = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; };
  if (!bf16 || Z != 1 || P.z_expert || (!P.tiles && (P.M <= 4 || P.N <= 96)) || !encode_tiled()) return false;
  if (P.K % 8 || P.ldw % 8 || !al(P.W) || (epi_dual(epi) && (!al(P.W2) || P.bias))) return false;
  if (P.tiles && P.sW % P.ldw) return false;
  return P.A16 || (size_t)P.M * P.K <= S->a16_elems;
}
static void launch_tc5(State* S, int epi, const GemmP& P, int tile_cap, cudaStream_t st) {
  const __nv_bfloat16* A16 = P.A16;
  if (!A16 && P.A == S->mirror && P.lda == S->width && P.K == S->width) {
    A16 = S->h16;
    if (P.a_map) {
      launch_next(gather_rows16, (unsigned)std::min<long long>(((long long)P.M * (P.K / 8) + 255) / 256, g_sm_count * 8), 256, 0, st)(S->h16, P.a_map, P.a_div, S->a16, P.M, P.K);
      S->launches++;
      A16 = S->a16;
    }
  }
  if (!A16) {
    const int vec = P.lda % 4 == 0 && (reinterpret_cast<uintptr_t>(P.A) & 15) == 0;
    const long long n = (long long)P.M * (P.K / 8);
    launch_next(bf16_rows, (unsigned)std::min<long long>((n + 255) / 256, g_sm_count * 8), 256, 0, st)(P.A, P.lda, P.a_map, P.a_div, S->a16, P.M, P.K, vec);
    S->launches++;
    A16 = S->a16;
  }
  // column tile: rounds of the grid times (columns + what a slice of the activations costs, about 64 columns)
  const bool dual = epi_dual(epi);
  const int mt = P.tiles ? tile_cap : (P.M + kTcRows - 1) / kTcRows;
  TcP T{};
  long long best = -1, grid = 1;
  for (int bn = 256; bn >= 32; bn /= 2) {
    if (dual && bn < 64) break;
    const int cols = dual ? bn / 2 : bn;
    const long long tiles = (long long)mt * ((P.N + cols - 1) / cols), cost = (tiles + g_sm_count - 1) / g_sm_count * (bn + 64);
    if (best < 0 || cost < best) { best = cost; T.bn = bn; grid = std::min<long long>(tiles, g_sm_count); }
  }
  T.stages = std::min(kTcMaxStages, kTcRing / ((kTcRows + T.bn) * kTcDepth * 2));
  T.n_mt = mt; T.rows_per_expert = P.tiles ? (int)(P.sW / P.ldw) : 0;
  T.C16 = P.C16; T.ldc16 = P.N; T.err = S->h_err;
  T.wide = P.C16 ? P.N % 4 == 0 && (reinterpret_cast<uintptr_t>(P.C16) & 7) == 0 : P.ldc % 4 == 0 && (reinterpret_cast<uintptr_t>(P.C) & 15) == 0;
  const int brows = dual ? T.bn / 2 : T.bn;
  const long long wrows = P.tiles ? (long long)T.rows_per_expert * P.n_expert : P.N;
  CUtensorMap mA, mB, mB2;
  if (!tile_map(&mA, A16, P.M, P.K, P.K, kTcRows) || !tile_map(&mB, P.W, wrows, P.K, P.ldw, brows) || !tile_map(&mB2, dual ? P.W2 : P.W, wrows, P.K, P.ldw, brows)) {
    *S->h_err = 2;
    return;
  }
#define DSK_TC5(E) case E: launch_next(gemm_tc5<E>, (unsigned)grid, kTcThreads, kTcSmem, st)(P, T, mA, mB, mB2); break
  switch (epi) {
    DSK_TC5(HEPI_STORE); DSK_TC5(HEPI_ADD); DSK_TC5(HEPI_GLU); DSK_TC5(HEPI_XIELU); DSK_TC5(HEPI_GEGLU); DSK_TC5(HEPI_SIGMUL);
    DSK_TC5(HEPI_RELU2); DSK_TC5(HEPI_LINGATE); DSK_TC5(HEPI_SILU_SIG); DSK_TC5(HEPI_SOFTCAP); DSK_TC5(HEPI_SWIGLU); DSK_TC5(HEPI_GELU_MUL);
  }
#undef DSK_TC5
}

template <typename WT>
// products of up to four rows
static void launch_gemv(int epi, const GemmP& P, int Z, cudaStream_t st) {
  if (gemv_one_ok<WT>(P)) {
    const int n = std::max(P.N, P.n_shared > 0 ? P.sN : 0);
    const int R = (long long)n * Z >= (Z == 1 ? 16384 : g_sm_count * 64) ? 2 : 1;   // rows per warp: two where one each would be more warps than the chip holds at a time
    const dim3 grid((unsigned)std::max(1, std::min((n + 8 * R - 1) / (8 * R), g_sm_count * 8)), (unsigned)Z);
#define DSK_GEMV1(E) do { if (R == 2) launch_next(gemv_one<WT, E, 2>, grid, 256, 0, st)(P); else launch_next(gemv_one<WT, E, 1>, grid, 256, 0, st)(P); } while (0)
    switch (epi) {
      case HEPI_STORE: DSK_GEMV1(HEPI_STORE); break;
      case HEPI_ADD: DSK_GEMV1(HEPI_ADD); break;
      case HEPI_GLU: DSK_GEMV1(HEPI_GLU); break;
      case HEPI_XIELU: DSK_GEMV1(HEPI_XIELU); break;
      case HEPI_GEGLU: DSK_GEMV1(HEPI_GEGLU); break;
      case HEPI_SIGMUL: DSK_GEMV1(HEPI_SIGMUL); break;
      case HEPI_RELU2: DSK_GEMV1(HEPI_RELU2); break;
      case HEPI_LINGATE: DSK_GEMV1(HEPI_LINGATE); break;
      case HEPI_SILU_SIG: DSK_GEMV1(HEPI_SILU_SIG); break;
      case HEPI_SOFTCAP: DSK_GEMV1(HEPI_SOFTCAP); break;
      case HEPI_SWIGLU: DSK_GEMV1(HEPI_SWIGLU); break;
      default: DSK_GEMV1(HEPI_GELU_MUL); break;
    }
#undef DSK_GEMV1
  } else {
    const dim3 grid((unsigned)std::max(1, std::min((std::max(P.N, P.n_shared > 0 ? P.sN : 0) + 7) / 8, g_sm_count * 8)), (unsigned)Z);
    switch (epi) {
      case HEPI_STORE: launch_next(gemv_rows<WT, HEPI_STORE>, grid, 256, 0, st)(P); break;
      case HEPI_ADD: launch_next(gemv_rows<WT, HEPI_ADD>, grid, 256, 0, st)(P); break;
      case HEPI_GLU: launch_next(gemv_rows<WT, HEPI_GLU>, grid, 256, 0, st)(P); break;
      case HEPI_XIELU: launch_next(gemv_rows<WT, HEPI_XIELU>, grid, 256, 0, st)(P); break;
      case HEPI_GEGLU: launch_next(gemv_rows<WT, HEPI_GEGLU>, grid, 256, 0, st)(P); break;
      case HEPI_SIGMUL: launch_next(gemv_rows<WT, HEPI_SIGMUL>, grid, 256, 0, st)(P); break;
      case HEPI_RELU2: launch_next(gemv_rows<WT, HEPI_RELU2>, grid, 256, 0, st)(P); break;
      case HEPI_LINGATE: launch_next(gemv_rows<WT, HEPI_LINGATE>, grid, 256, 0, st)(P); break;
      case HEPI_SILU_SIG: launch_next(gemv_rows<WT, HEPI_SILU_SIG>, grid, 256, 0, st)(P); break;
      case HEPI_SOFTCAP: launch_next(gemv_rows<WT, HEPI_SOFTCAP>, grid, 256, 0, st)(P); break;
      case HEPI_SWIGLU: launch_next(gemv_rows<WT, HEPI_SWIGLU>, grid, 256, 0, st)(P); break;
      default: launch_next(gemv_rows<WT, HEPI_GELU_MUL>, grid, 256, 0, st)(P); break;
    }
  }
}
// fp32 products of more than four rows, routed ones in tiles of 128 (gemm_split)
static void launch_split(State* state, int epi, const GemmP& P, int Z, int tile_cap, cudaStream_t st) {
  const int bn = epi_dual(epi) ? kSplitN / 2 : kSplitN;
  const int mt = P.tiles ? tile_cap : (P.M + kTcRows - 1) / kTcRows, nt = (P.N + bn - 1) / bn, slices = (P.K + kSplitDepth - 1) / kSplitDepth;
  // Shares of the depth, a cluster of CTAs a tile: rounds of CTAs x (slices of 2000 cycles + what a tile takes besides, joining included).  45 x 1024 x 4096: 59 us by tiles
  // alone, 27 with four CTAs a tile; 37 x 130 x 8192 108 and 26 with eight; 600 x 1024 x 2816, 80 tiles, 56 and 70 with two.
  static const std::array<int, 9> room = [] {   // CTAs of clusters of c that run at a time (not all SMs are in a group of eight)
    std::array<int, 9> r{};
    for (int c = 2; c <= 8; c *= 2) {
      cudaLaunchConfig_t cfg{};
      cudaLaunchAttribute at{};
      at.id = cudaLaunchAttributeClusterDimension;
      at.val.clusterDim.x = (unsigned)c; at.val.clusterDim.y = at.val.clusterDim.z = 1;
      cfg.gridDim = dim3((unsigned)c * 32); cfg.blockDim = dim3(kSplitThreads); cfg.dynamicSmemBytes = split_smem(kSplitStages); cfg.attrs = &at; cfg.numAttrs = 1;
      int n = 0;
      if (cudaOccupancyMaxActiveClusters(&n, gemm_split<HEPI_STORE, true>, &cfg) != cudaSuccess) { cudaGetLastError(); n = 0; }
      r[c] = n * c;
    }
    return r;
  }();
  int S = 1;
  long long best = 0;
  for (int c = 1; c <= 8 && c <= slices && (c == 1 || (!P.band && room[c])); c *= 2) {
    const long long ctas = (long long)mt * nt * Z * c, at_once = c == 1 ? g_sm_count : room[c];
    const long long cost = (ctas + at_once - 1) / at_once * ((slices + c - 1) / c * 2000LL + (c > 1 ? 8000 : 5500));
    if (c == 1 || cost < best) { best = cost; S = c; }
  }
  const dim3 grid((unsigned)(nt * S), (unsigned)mt, (unsigned)Z);
  // (a short depth takes no more shared memory than it has slices, the rest is L1: a prompt of 1500 tokens with mixed heads 1594 -> 1589 us, fp32 prompts and 45 tokens the same)
  const int stages = std::max(1, std::min(kSplitStages, (slices + S - 1) / S));
#define DSK_SPLIT(E) case E: if (S > 1) launch_next(gemm_split<E, true>, grid, kSplitThreads, split_smem(stages), st, (unsigned)S)(P, stages, S, state->h_err); \
    else launch_next(gemm_split<E, false>, grid, kSplitThreads, split_smem(stages), st)(P, stages, 1, state->h_err); break
  switch (epi) {
    DSK_SPLIT(HEPI_STORE); DSK_SPLIT(HEPI_ADD); DSK_SPLIT(HEPI_GLU); DSK_SPLIT(HEPI_XIELU); DSK_SPLIT(HEPI_GEGLU); DSK_SPLIT(HEPI_SIGMUL);
    DSK_SPLIT(HEPI_RELU2); DSK_SPLIT(HEPI_LINGATE); DSK_SPLIT(HEPI_SILU_SIG); DSK_SPLIT(HEPI_SOFTCAP); DSK_SPLIT(HEPI_SWIGLU); DSK_SPLIT(HEPI_GELU_MUL);
  }
#undef DSK_SPLIT
}
// many rows, few columns (gemm_narrow); the epilogues such products have
static void launch_narrow(bool bf16, int epi, const GemmP& P, cudaStream_t st) {
  const dim3 grid((unsigned)((P.M + kNarrowRows - 1) / kNarrowRows), (unsigned)((P.N + 31) / 32));
#define DSK_NARROW(E) case E: if (bf16) launch_next(gemm_narrow<__nv_bfloat16, E>, grid, 256, 0, st)(P); else launch_next(gemm_narrow<float, E>, grid, 256, 0, st)(P); break
  switch (epi) {
    DSK_NARROW(HEPI_STORE); DSK_NARROW(HEPI_ADD); DSK_NARROW(HEPI_XIELU); DSK_NARROW(HEPI_RELU2); DSK_NARROW(HEPI_LINGATE); DSK_NARROW(HEPI_SILU_SIG);
    DSK_NARROW(HEPI_SOFTCAP); DSK_NARROW(HEPI_GELU_MUL);
  }
#undef DSK_NARROW
}
// C = A W^T (+ epilogue).  Z > 1: per-head batches or (gemv) one batch per routed (token, slot) pair.
static void linear(State* S, bool bf16, int epi, const GemmP& P, int Z, cudaStream_t st, int tile_cap = 0) {
  struct Over { State* S; const float* C; ~Over() { if (C == S->mirror) S->mirror = nullptr; } } over{S, P.C};   // (its operand may be the mirror until then)
  const bool small = P.z_expert != nullptr || (!P.tiles && P.M <= 4);
  if (!small && !P.tiles && Z == 1 && P.N <= 96) {   // narrow output (router, token-input gate): warp-per-row products over batches of 4 rows
    // (a CTA of gemm_narrow has 16 rows: under 448 they are too few.  Steps of 256 / 384 / 512 / 1024 tokens, two layers with 64 experts and a token input of
    // 32, width 2048: 714 / 819 / 873 / 1126 us with it, 650 / 806 / 895 / 1221 with the products of warps; width 1024: 519 / 669 / 738 / 786 and 506 / 654 / 749 / 832)
    // (fp32 ones of some more are faster in three parts, their depth shared by a cluster.  64 columns, us, gemm_narrow and gemm_split: 2048 rows 2048 deep 31 and 19, 448 rows
    // 2048 deep 21 and 14, 777 rows 1024 deep 12 and 12.  Error against 64 bits, depth 512 / 1024 / 2048: normal operands 15.6, 21.1, 29.4e-8 and 8.9, 10.3, 12.6e-8, all of one sign 6.0,
    // 7.2, 9.1e-8 and 8.4, 9.2, 10.8e-8)
    if (!bf16 && P.M >= kNarrowMin && (long long)P.M * P.K >= 900000) {
      launch_split(S, epi, P, 1, 0, st);
      S->launches++;
      return;
    }
    if (epi != HEPI_SIGMUL && P.M >= kNarrowMin && !epi_dual(epi)) {
      launch_narrow(bf16, epi, P, st);
      S->launches++;
      return;
    }
    GemmP Q = P;
    Q.z_rows = P.M;
    const int zb = (P.M + 3) / 4;
    if (bf16) launch_gemv<__nv_bfloat16>(epi, Q, zb, st);
    else launch_gemv<float>(epi, Q, zb, st);
    S->launches++;
    return;
  }
  if (tc_ok(S, bf16, epi, P, Z)) launch_tc5(S, epi, P, tile_cap, st);
  else if (bf16 && !small) launch_gemm_mma(epi, P, Z, tile_cap, st);
  else if (!small) launch_split(S, epi, P, Z, tile_cap, st);
  else if (bf16) launch_gemv<__nv_bfloat16>(epi, P, Z, st);
  else launch_gemv<float>(epi, P, Z, st);
  S->launches++;
}

// A feed-forward whose two products both run on gemm_tc5 keeps its hidden rows in bf16, in the row order of the products (the second one
// would round them anyway).
static void hidden16(State* S, bool bf16, int epi_up, GemmP& up, int epi_down, GemmP& down, __nv_bfloat16* buf) {
  if (!S->hid16 || (reinterpret_cast<uintptr_t>(buf) & 15) || !tc_ok(S, bf16, epi_up, up, 1)) return;
  GemmP d = down;
  d.A16 = buf;
  if (!tc_ok(S, bf16, epi_down, d, 1)) return;
  up.C16 = buf;
  down.A16 = buf;
}

static void launch_scan(const dsk_layer_spec& sp, const float* proj, int ld_proj, const float* xbc, int ld_xbc, const HLayer& L,
                        float* state, float* out, int T, cudaStream_t st) {
  const int H = sp.ssm_heads, P = sp.ssm_vdim, N = sp.ssm_state, G = sp.ssm_groups;
  const int inner = H * P;
  int PB = std::min(P, 64);   // value channels per CTA: fewer when the heads alone would leave most SMs idle
  while (PB > 32 && H * ((P + PB - 1) / PB) < g_sm_count) PB /= 2;   // (measured: 32 channels per CTA is the best split at 64 heads x 64)
  if (const char* e = getenv("DSK_SCAN_PB")) PB = std::max(1, std::min(std::min(P, 64), atoi(e)));   // A/B switch
  const dim3 grid((unsigned)H, (unsigned)((P + PB - 1) / PB));
  const int threads = ((PB * 8 + 31) / 32) * 32;
  const int TB = T >= 64 ? 64 : 16;   // tokens staged per round
  const int NP = (N + 3) & ~3;
  const size_t smem = (size_t)TB * (2 + 2 * NP + 2 * PB) * 4;
  const int need = (N + 31) / 32;     // float4 groups of state per thread
#define DSK_SCAN(RQ) launch_next(ssd_scan<RQ>, grid, threads, smem, st)(proj, ld_proj, 0, inner + (int)ssd_channels(sp), xbc, ld_xbc, 0, inner, inner + G * N, \
                                                               L.dt_bias, L.A_log, L.D, state, out, inner, T, H, P, N, G, PB, TB)
  if (need <= 1) DSK_SCAN(1); else if (need <= 2) DSK_SCAN(2); else if (need <= 3) DSK_SCAN(3); else if (need <= 4) DSK_SCAN(4);
  else if (need <= 6) DSK_SCAN(6); else DSK_SCAN(8);
#undef DSK_SCAN
}

static void launch_hgrn2(const dsk_layer_spec& sp, const float* proj, int ld, float* state, float* out, int T, cudaStream_t st) {
  const int H = sp.lin_heads, N = sp.lin_dim, P = sp.lin_vdim;
  // threads per value channel (measured at 16 heads x 128 x 128 and x 64 x 64: 16 threads and 16 channels per CTA are the best split; fewer
  // channels per CTA repeat the staging of a head's gates and queries in more CTAs, more leave SMs idle)
  int TPC = N >= 256 ? 32 : N >= 64 ? 16 : 8;
  if (const char* e = getenv("DSK_LIN_TPC")) { const int v = atoi(e); if ((v == 8 || v == 16 || v == 32) && N >= 4 * v) TPC = v; }   // A/B switch
  int PB = std::min(P, 512 / TPC);   // value channels per CTA
  while (PB > 16 && H * ((P + PB - 1) / PB) < g_sm_count) PB /= 2;
  if (PB == 16 && H * ((P + 15) / 16) < 74) PB = 8;
  if (const char* e = getenv("DSK_LIN_PB")) PB = std::max(1, std::min(std::min(P, 512 / TPC), atoi(e)));   // A/B switch
  const dim3 grid((unsigned)H, (unsigned)((P + PB - 1) / PB));
  const int threads = ((PB * TPC + 31) / 32) * 32;
  const int NP = (N + 3) & ~3;
  int TB = T >= 64 ? 64 : 16;         // tokens staged per round, in two buffers
  while (TB > 16 && (size_t)2 * TB * (2 * NP + PB) * 4 > 160 * 1024) TB /= 2;
  const size_t smem = (size_t)2 * TB * (2 * NP + PB) * 4;
  const int need = (N + 4 * TPC - 1) / (4 * TPC);     // float4 groups of state per thread
#define DSK_LIN(RQ, C) launch_next(hgrn2_scan<RQ, C>, grid, threads, smem, st)(proj, ld, 0, H * N, 2 * H * N, state, out, H * P, T, H, N, P, PB, TB)
  if (TPC == 32) { if (need <= 1) DSK_LIN(1, 32); else DSK_LIN(2, 32); }
  else if (TPC == 16) { if (need <= 1) DSK_LIN(1, 16); else if (need <= 2) DSK_LIN(2, 16); else if (need <= 3) DSK_LIN(3, 16); else DSK_LIN(4, 16); }
  else if (need <= 1) DSK_LIN(1, 8); else if (need <= 2) DSK_LIN(2, 8); else if (need <= 3) DSK_LIN(3, 8); else if (need <= 4) DSK_LIN(4, 8);
  else if (need <= 6) DSK_LIN(6, 8); else DSK_LIN(8, 8);
#undef DSK_LIN
}

static size_t ssd_gram_smem(const dsk_layer_spec& s) {
  return ((size_t)2 * kLinBlk * (((s.ssm_state + 3) & ~3) + 4) + (size_t)2 * kLinBlk * (s.ssm_heads / s.ssm_groups)) * 4;
}
// lin_scan: warps of a CTA and CTAs, by value channels that a warp has (CW) and by how many CTAs there are; extra: a column more, the normaliser
struct LinScanShape { int warps, ctas; };
static LinScanShape lin_scan_shape(int H, int P, bool extra, int CW) {
  int warps = std::max(1, std::min(8, (P + CW - 1) / CW));
  while (warps > 2 && H * ((P + warps * CW - 1) / (warps * CW)) < g_sm_count) warps = (warps + 1) / 2;
  return {warps, H * ((P + (extra ? 1 : 0) + warps * CW - 1) / (warps * CW))};
}
// Whether lin_mma walks a portion, and in how many segments (0: lin_scan does).  us: lin_scan 8 for the launch, and a block by the warps w that an SM has, 0.95 for 2, 1.1 for 4,
// 1.4 for 8, 2.4 for 16, 4.8 for 32; lin_mma, 128 (64) key entries, a block walked for results 1.95 (1.25), for the end state alone 1.1 (0.6), a round of CTAs each, 6 for the launch, 11
// for two, 0.8 a segment that states are joined over.  Measured over 4 to 64 heads of 32 to 128 channels, 64 and 128 entries, with and without the normaliser, 48 to 2048 tokens (354
// walks): what this takes is 0.3 % above the fastest on average, once 4 % above lin_scan.  2048 tokens, lin_scan and lin_mma: 64 heads of 64 channels 312 and 222 (two segments), 16 of
// 128 186 and 116 (four), 16 of 128 with the normaliser, whose column takes a third CTA, 188 and 152 (three), 4 of 64 with 64 entries 134 and 46 (eight), 64 of 128 with the normaliser 637
// and 532 (three); 600 tokens, 16 of 64 with 64 entries 46 and 23; 100 tokens, 8 of 128 with 128 entries 17 and 21: not taken; 48 tokens, 32 of 64 with 64 entries 12.8 and 10.1 (one walk).
// In chained steps launches hide under one another: a set of numbers of their own, over 256 walks of 33 to 256 tokens between the kernels around them 0.6 % above the fastest on average.
static int lin_mma_segments(const float* q, const float* k, int ldq, int hs, const float* v, int ldv, int T, int H, int N, int P, bool extra, const float* seg) {
  auto al = [](const float* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; };
  if (!seg || (N != 64 && N != 128) || P % 4 || ldq % 4 || hs % 4 || ldv % 4 || !al(q) || !al(k) || !al(v)) return 0;
  const int nb = (T + kLinBlk - 1) / kLinBlk, ctas = H * ((P + (extra ? 1 : 0) + kLmCh - 1) / kLmCh);
  const LinScanShape scan = lin_scan_shape(H, P, extra, N == 64 ? 4 : 2);
  const bool chained = chain_step;
  const double full = N == 128 ? (chained ? 2.1 : 1.95) : chained ? 1.15 : 1.25, ends = N == 128 ? 1.1 : 0.6, w = scan.warps * ((scan.ctas + g_sm_count - 1) / g_sm_count);
  double best = (chained ? 7 : 8) + nb * std::max(0.8 + 0.075 * w, 0.15 * w);
  int segs = 0;
  for (int n = 1; n <= kLmSegs; n++) {
    const int per = (nb + n - 1) / n, rounds = (ctas * n + g_sm_count - 1) / g_sm_count, first = (ctas * (n - 1) + g_sm_count - 1) / g_sm_count;
    const double cost = per * (rounds * full + first * ends) + (chained ? (n > 1 ? 9 + 0.5 * n : 5) : n > 1 ? 11 + 0.8 * n : 6);
    if ((nb + per - 1) / per == n && cost < best) { best = cost; segs = n; }
  }
  return segs;
}
static void launch_lin_mma(LinMmaP p, int N, int nseg, cudaStream_t st) {
  const int nb = (p.T + kLinBlk - 1) / kLinBlk, cg = (p.groups + kLmGroups - 1) / kLmGroups;
  p.nseg = nseg; p.per = (nb + nseg - 1) / nseg;
  auto* kernel = N == 64 ? lin_mma<8> : lin_mma<16>;
  const size_t smem = N == 64 ? LinMma<8>::SMEM : LinMma<16>::SMEM;
  for (p.mode = nseg > 1 ? 0 : 1; p.mode < 2; p.mode++) launch_next(kernel, dim3((unsigned)p.H, (unsigned)cg, (unsigned)(p.mode ? nseg : nseg - 1)), kLmThreads, smem, st)(p);
}

// the walk over the blocks of a step (lin_scan): lanes per channel group by the key size, warps per CTA by how many CTAs there are
static void launch_lin_scan(bool delta, const float* q, const float* k, int ldq, int hs, int rep, const float* v, int ldv, const float* rec, float* state,
                            float* out, int ldo, int T, int H, int N, int P, cudaStream_t st, State* S, float* nst = nullptr, float* den = nullptr, int sn = 0, int sp = 1) {
  if (!sn) sn = P;                    // state rows [N][P] of a head, unless said otherwise
  if (const int n = delta ? 0 : lin_mma_segments(q, k, ldq, hs, v, ldv, T, H, N, P, nst != nullptr, S->lseg)) {
    if (n > 1) S->launches++;                // (callers count one)
    launch_lin_mma(LinMmaP{q, k, v, rec, state, out, nst, den, S->lseg, ldq, hs, rep, ldv, ldo, T, H, P, sn, sp, (P + (nst ? 1 : 0) + 15) / 16, n, 0, 0}, N, n, st);
    return;
  }
  const int TPC = N <= 32 ? 8 : N <= 64 ? 16 : 32, RQ = N <= 128 ? 1 : 2;
  int CPT = N > 128 ? 4 : 2;          // value channels per lane
  if (const char* e = getenv("DSK_LIN_CPT")) CPT = atoi(e) == 4 || N > 128 ? 4 : 2;   // A/B switch
  const int CW = CPT * (32 / TPC);
  int warps = lin_scan_shape(H, P, nst != nullptr, CW).warps;
  if (const char* e = getenv("DSK_LIN_WARPS")) warps = std::max(1, std::min(8, atoi(e)));   // A/B switch
  const int PB = warps * CW;
  const dim3 grid((unsigned)H, (unsigned)((P + (nst ? 1 : 0) + PB - 1) / PB));
  const size_t smem = lin_scan_smem(4 * TPC * RQ, PB, warps, CW);
  if (!delta) plain_next = true;   // (its CTAs, few and long, would double up on the SMs that the kernel ahead leaves first: 200 tokens of 16 heads of 64 channels and entries with the normaliser 31 and 27 us)
#define DSK_LSCAN(D, A, B, C) launch_next(lin_scan<D, A, B, C>, grid, 32 * (warps + kLinStage), smem, st)(q, k, ldq, hs, rep, v, ldv, rec, state, out, ldo, T, H, N, P, PB, nst, den, sn, sp)
#define DSK_LSCANS(D) do { if (N > 128) DSK_LSCAN(D, 32, 2, 4); else if (CPT == 2) { if (N <= 32) DSK_LSCAN(D, 8, 1, 2); else if (N <= 64) DSK_LSCAN(D, 16, 1, 2); else DSK_LSCAN(D, 32, 1, 2); } \
  else { if (N <= 32) DSK_LSCAN(D, 8, 1, 4); else if (N <= 64) DSK_LSCAN(D, 16, 1, 4); else DSK_LSCAN(D, 32, 1, 4); } } while (0)
  if (delta) DSK_LSCANS(true); else DSK_LSCANS(false);
#undef DSK_LSCANS
#undef DSK_LSCAN
}

static void launch_lin_decode(int mode, const GdnP& D, const float* decay, float* state, const float* norm_w, float eps, int gate_off, float alpha,
                              float* out, int ldo, cudaStream_t st, const MlstmP& memory = MlstmP{1.f, nullptr, nullptr}) {
  const int NG = std::min(kLinDecodeThreads / ((D.P + 3) / 4), D.N), need = (D.N + NG - 1) / NG;
  const size_t smem = lin_decode_smem(D.N, D.P);
#define DSK_LDEC(X, R) launch_next(lin_decode<X, R>, D.H, kLinDecodeThreads, smem, st)(D, decay, state, norm_w, eps, gate_off, alpha, out, ldo, memory)
#define DSK_LDECS(X) do { if (need <= 1) DSK_LDEC(X, 1); else if (need <= 2) DSK_LDEC(X, 2); else if (need <= 4) DSK_LDEC(X, 4); else if (need <= 8) DSK_LDEC(X, 8); else DSK_LDEC(X, 16); } while (0)
  if (mode == LIN_DELTA) DSK_LDECS(LIN_DELTA); else if (mode == LIN_MLSTM) DSK_LDECS(LIN_MLSTM); else DSK_LDECS(LIN_PLAIN);
#undef DSK_LDECS
#undef DSK_LDEC
}

// gated delta rule of T tokens from the raw projections in S->b0 (columns of att_layout) -> out rows (pitch ldo), times alpha
static void gdn_forward(State* S, const HLayer& L, LayerState& ls, int ldp, const AttLayout& a, float* out, int ldo, float alpha, float eps, int T, cudaStream_t st, __nv_bfloat16* out16 = nullptr) {
  const dsk_layer_spec& sp = L.sp;
  const int H = sp.gdn_heads, G = sp.gdn_kv_heads, N = sp.gdn_dim, P = sp.gdn_vdim, RV = H * P, NP = (N + 3) & ~3, CH = 2 * G * N + RV;
  const GdnP D{S->b0, ldp, (int)a.dq, (int)a.db, (int)a.da, L.gdn_conv_w, L.A_log, L.dt_bias, ls.hist, sp.gdn_conv - 1 + kConvSpare, sp.gdn_conv, T, H, G, N, P, S->d_ctl};
  if (T <= kLinDecodeTokens && lin_decode_fits(N, P)) {
    launch_lin_decode(LIN_DELTA, D, nullptr, ls.lin, L.lin_norm, eps, (int)a.dg, alpha, out, ldo, st);
    S->launches++;
    return;
  }
  const int nb = (T + kLinBlk - 1) / kLinBlk;
  const size_t smem = (size_t)(2 * kLinBlk * (NP + 4) + 2 * kLinBlk * kLinBlk + 8 * kLinBlk * kLinBlk) * 4;
  launch_next(gdn_prepare, dim3((unsigned)nb, (unsigned)(G + (RV + 255) / 256)), 256, smem, st)(D, S->lq, S->lk, S->lv, NP, S->lrec);
  launch_lin_scan(true, S->lq, S->lk, G * NP, NP, H / G, S->lv, RV, S->lrec, ls.lin, S->lout, RV, T, H, N, P, st, S);
  if (sp.gdn_conv > 1) { launch_next(conv_ring_store, (CH + 127) / 128, 128, 0, st)(S->b0, ldp, (int)a.dq, ls.hist, D.ring, T, CH, sp.gdn_conv, S->d_ctl); S->launches++; }
  launch_next(head_rmsnorm, (unsigned)(((long long)T * H + 7) / 8), 256, 0, st)(S->lout, RV, L.lin_norm, out, ldo, T, H, P, eps, S->b0 + a.dg, ldp, alpha, 0, 0, nullptr, nullptr, out16);
  S->launches += 3;
}

// lightning attention of T tokens from [silu q | silu k | silu v | sigmoid g] rows in S->b0 -> S->lout (ahead of the norm)
static void lightning_forward(State* S, const HLayer& L, LayerState& ls, int ldp, int T, cudaStream_t st) {
  const dsk_layer_spec& sp = L.sp;
  const int H = sp.lin_heads, N = sp.lin_dim, P = sp.lin_vdim, HN = H * N, HP = H * P;
  if (T <= kLinDecodeTokens && lin_decode_fits(N, P)) {
    const GdnP D{S->b0, ldp, 0, 0, 0, nullptr, nullptr, nullptr, nullptr, 1, 1, T, H, H, N, P, S->d_ctl};
    launch_lin_decode(LIN_PLAIN, D, L.decay, ls.lin, nullptr, 0.f, 0, 1.f, S->lout, HP, st);
    S->launches++;
    return;
  }
  launch_next(lin_gram, dim3((unsigned)((T + kLinBlk - 1) / kLinBlk), (unsigned)H), 256, (size_t)2 * kLinBlk * (((N + 3) & ~3) + 4) * 4, st)(S->b0, S->b0 + HN, ldp, L.log_decay, T, H, N, S->lrec);
  launch_lin_scan(false, S->b0, S->b0 + HN, ldp, N, 1, S->b0 + 2 * HN, ldp, S->lrec, ls.lin, S->lout, HP, T, H, N, P, st, S);
  S->launches += 2;
}

// mLSTM of T tokens from the stacked projection in S->b0 (columns of mlstm_layout) -> normed and gated heads in out [T][H P]
static void mlstm_forward(State* S, const HLayer& L, LayerState& ls, int ldp, const MlstmLayout& a, float* out, float eps, int T, cudaStream_t st, __nv_bfloat16* out16) {
  const dsk_layer_spec& sp = L.sp;
  const int H = sp.lin_heads, N = sp.lin_dim, P = sp.lin_vdim, HN = H * N, HP = H * P;
  float *nst = ls.lin + (size_t)HN * P, *mst = nst + HN;
  if (T <= kLinDecodeTokens && lin_decode_fits(N, P)) {
    const GdnP D{S->b0, ldp, 0, (int)a.i, (int)a.f, nullptr, nullptr, nullptr, nullptr, 1, 1, T, H, H, N, P, S->d_ctl};
    launch_lin_decode(LIN_MLSTM, D, nullptr, ls.lin, L.mnorm, eps, (int)a.g, 1.f, out, HP, st, MlstmP{sp.lin_gate_cap, nst, mst});
    S->launches++;
    return;
  }
  float *gi = S->lgate, *gf = gi + (size_t)H * T, *gm = gf + (size_t)H * T;
  launch_next(mlstm_gates, H, 256, 0, st)(S->b0, ldp, (int)a.i, (int)a.f, sp.lin_gate_cap, T, H, gi, gf, gm, mst);
  launch_next(mlstm_gram, dim3((unsigned)((T + kLinBlk - 1) / kLinBlk), (unsigned)H), 256, (size_t)2 * kLinBlk * (((N + 3) & ~3) + 4) * 4, st)(S->b0, S->b0 + HN, ldp, gi, gf, gm, T, H, N, S->lrec);
  launch_lin_scan(false, S->b0, S->b0 + HN, ldp, N, 1, S->b0 + 2 * HN, ldp, S->lrec, ls.lin, S->lout, HP, T, H, N, P, st, S, nst, S->lden);
  launch_next(head_rmsnorm, (unsigned)(((long long)T * H + 7) / 8), 256, 0, st)(S->lout, HP, L.mnorm, out, HP, T, H, P, eps, S->b0 + a.g, ldp, 1.f, P, 1, S->lden, gm, out16);
  S->launches += 4;
}

static int R0(const Model* M, size_t ri) { return M->runs[ri].owner_run; }

// whether a tile of 32 keys and values fits decode_attn (gqa_attn takes larger heads, and mixed ones)
static bool decode_attn_fits(int D, int Dv) { return Dv <= 1024 && decode_attn_floats(D, Dv, false) * 4 <= 200 * 1024; }
// decode-sized attention (P.T, sizes, caches, mask and gate given): the split of rows and keys over CTAs, and the merge of key shares
static void launch_decode_attn(State* S, DecodeAttn P, bool latent, cudaStream_t st) {
  const int T = P.T, rep = P.H / P.G;
  P.TQ = T >= 8 ? 8 : T >= 4 ? 4 : T >= 2 ? 2 : 1;
  P.HB = std::min(rep, 8 / P.TQ);
  P.NS = 1;
  if (T <= kAttnSplitTokens) {   // the widest key range a CTA can meet is span + kept + TQ - 1 keys
    const int tiles = (std::min(P.span, P.ring) + P.mods.keep + P.TQ - 1 + 31) / 32;
    // Shares of the keys: one a tile, but no more CTAs than run at a time (three an SM).  With a CTA per tile and key head, 16 key heads behind a window of 4096
    // were 1024 CTAs, waiting for a place and mostly without a key of theirs: two such layers (width 1024) and their head took 120 us a token behind 30 keys and
    // 150 behind 2000, gqa_attn with its four key heads a CTA 117 and 139, this 109 and 135.
    const int rows = (T + P.TQ - 1) / P.TQ * P.G * ((rep + P.HB - 1) / P.HB), most = std::max(1, std::min(kAttnSplitMax, 3 * g_sm_count / rows)), per = (tiles + most - 1) / most;
    P.NS = (tiles + per - 1) / per;
  }
  P.part = S->part;
  const dim3 grid((unsigned)((T + P.TQ - 1) / P.TQ), (unsigned)(P.G * ((rep + P.HB - 1) / P.HB)), (unsigned)P.NS);
  const size_t smem = decode_attn_floats(P.D, P.Dv, latent) * 4;
  const int cv = P.Dv <= 256 ? 1 : P.Dv <= 512 ? 2 : 4;
#define DSK_DECODE_ATTN(KV, CV) do { if (P.TQ > 1) launch_next(decode_attn<KV, CV, true>, grid, 256, smem, st)(P); else launch_next(decode_attn<KV, CV, false>, grid, 256, smem, st)(P); } while (0)
  if (latent) {
    if (cv == 1) DSK_DECODE_ATTN(true, 1);
    else if (cv == 2) DSK_DECODE_ATTN(true, 2);
    else DSK_DECODE_ATTN(true, 4);
  } else if (cv == 1) DSK_DECODE_ATTN(false, 1);
  else if (cv == 2) DSK_DECODE_ATTN(false, 2);
  else DSK_DECODE_ATTN(false, 4);
#undef DSK_DECODE_ATTN
  S->launches++;
  if (P.NS > 1) {
    launch_next(latent_swa_merge, dim3((unsigned)(T * P.H), (unsigned)((P.Dv + 127) / 128)), 128, 0, st)(S->part, P.out, P.Dv, P.NS, P.gate, P.ld_gate, P.H, P.gate_head,
                                                                                                        P.ld_out, P.alpha);
    S->launches++;
  }
}
// the same over cached latents with absorbed queries qa [T][H][R]
static void launch_latent_attn(State* S, const float* qa, const float* cache, float* out, int T, int H, int R, int mask, int window, int ring, float scale, const float* sink,
                               cudaStream_t st) {
  DecodeAttn P{};
  P.q = qa; P.kc = P.vc = cache; P.out = out; P.ctl = S->d_ctl; P.T = T; P.H = H; P.G = 1; P.D = P.Dv = P.ldk = P.ldv = R; P.mask = mask; P.span = window; P.ring = ring;
  P.scale = scale; P.alpha = 1.f; P.ld_out = H * R; P.mods.sink = sink;
  launch_decode_attn(S, P, true, st);
}

// rows x cols bf16 matrices, `count` of them behind one another, copied in boxes of 32 rows x 64 columns (rows past a matrix read as zeros)
static bool box_map(CUtensorMap* m, const void* p, long long cols, long long rows, long long count) {
  const cuuint64_t dims[3] = {(cuuint64_t)cols, (cuuint64_t)rows, (cuuint64_t)count}, strides[2] = {(cuuint64_t)cols * 2, (cuuint64_t)rows * cols * 2};
  const cuuint32_t box[3] = {64, (cuuint32_t)kP5Keys, 1}, one[3] = {1, 1, 1};
  return encode_tiled()(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(p), dims, strides, box, one, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                        CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}
// Heads that pattn5 takes: queries and two pieces of keys in shared memory, whole 64-entry rows (smaller heads would be half padding), scores' accumulators in TMEM
static bool pattn5_takes(const PattnSize& z) {
  const int nch = (z.Dp + 63) / 64;
  return encode_tiled() && z.Dp >= 64 && nch <= kP5MaxChunks && p5_smem(z.parts, nch, z.VN / 8, 2, 1) <= kPattn5SmemMax;
}
static void launch_pattn5(State* S, const PattnSize& z, PattnP& A, cudaStream_t st) {
  const int nch = (z.Dp + 63) / 64, vb = z.VN / 8, vst = p5_smem(z.parts, nch, vb, 4, 2) <= kPattn5SmemMax ? 2 : 1;
  int kst = 2;
  while (kst < std::min(kP5MaxK, 3 * nch) && p5_smem(z.parts, nch, vb, kst + 1, vst) <= kPattn5SmemMax) kst++;
  const int smem = p5_smem(z.parts, nch, vb, kst, vst), qb = (A.T + kP5Rows - 1) / kP5Rows, zc = z.Vp / (vb * 64);
  // shares of the keys where the query blocks leave SMs idle, of at least four tiles (joining them takes about as long as three)
  const long long ctas = (long long)qb * A.H * zc, tiles = (std::min<long long>(A.Lk, (long long)A.span + kP5Rows) + kP5Keys - 1) / kP5Keys;
  const long long most = std::min({g_sm_count / ctas, tiles / 4, (long long)kAttnSplitMax});
  A.NS = most > 1 && (tiles + most - 1) / most + 3 < tiles ? (int)most : 1;
  A.part = S->ppart;
  CUtensorMap mK, mV;
  if (!box_map(&mK, A.kb, z.Dp, A.Lk, (long long)z.parts * z.G) || !box_map(&mV, A.vb, z.Vp, A.Lk, (long long)z.parts * z.G)) { *S->h_err = 2; return; }
  const dim3 grid((unsigned)A.H, (unsigned)qb, (unsigned)(zc * A.NS));
  auto* kernel = z.parts == 1 ? (vb == 1 ? pattn5<1, 1> : pattn5<1, 2>) : vb == 1 ? pattn5<3, 1> : pattn5<3, 2>;
  launch_next(kernel, grid, kP5Threads, smem, st)(A, mK, mV, kst, vst, S->h_err);
}

static void launch_pattn(State* S, const PattnSize& z, const PackP& K, PattnP& A, cudaStream_t st) {
  // 16 query rows per warp, a CTA an SM, tiles of 16 keys where 32 do not fit.  Four warps are one on each of an SM's tensor cores; with eight a tile of keys takes about 1.2 times
  // as long (two a core hide one another's waits, and more threads copy the tile), with two 1.4 times.  Where the query blocks leave SMs idle, the keys are cut into shares of
  // at least four tiles, one CTA each, and latent_swa_merge joins them.  What costs least, rounds of CTAs x time of a tile x tiles, is taken.  Two layers of width 2048, 16 heads of 128, behind
  // 8000 keys, steps of 32 / 128 / 256 / 512 tokens take 0.68 / 0.83 / 1.6 / 3.3 ms; with warps halved until the SMs had a CTA each they took 4.3 / 5.0 / 6.1 / 13.4, as products between
  // which scores lie in memory 2.2 / 3.1 / 4.5 / 9.3
  const int zc = z.Vp / (z.VN * 8);
  int w = 0, nk = 0;
  A.NS = 1;
  long long best = 0;
  for (int cw = 8; cw >= 2; cw /= 2) {
    const int ck = pattn_smem(z.parts, cw, z.Dp, z.VN, 4) <= (size_t)kPattnSmemMax ? 4 : 2;
    if (pattn_smem(z.parts, cw, z.Dp, z.VN, ck) > (size_t)kPattnSmemMax) continue;
    const long long ctas = (long long)((A.T + 16 * cw - 1) / (16 * cw)) * A.H * zc, tiles = (std::min<long long>(K.Lk, (long long)A.span + 16 * cw) + 8 * ck - 1) / (8 * ck);
    const long long most = std::max<long long>(1, std::min({g_sm_count / ctas, tiles / 4, (long long)kAttnSplitMax}));
    for (long long ns = 1; ns <= most; ns += std::max<long long>(1, most - 1)) {   // (joining shares takes about as long as a tile)
      const long long cost = (ctas * ns + g_sm_count - 1) / g_sm_count * (cw == 8 ? 6 : cw == 4 ? 5 : 7) * ((tiles + ns - 1) / ns + (ns > 1)) * ck;
      if (!w || cost < best) { best = cost; w = cw; nk = ck; A.NS = (int)ns; }
    }
  }
  A.part = S->ppart;
  const dim3 grid((unsigned)A.H, (unsigned)((A.T + 16 * w - 1) / (16 * w)), (unsigned)(zc * A.NS));
  const size_t smem = pattn_smem(z.parts, w, z.Dp, z.VN, nk);
  auto run = [&](auto* k4, auto* k2) { launch_next(nk == 4 ? k4 : k2, grid, 32 * w, smem, st)(A); };
#define DSK_PATTN(A_, B_) do { if (A.NS > 1) run(pattn<A_, B_, 4, true>, pattn<A_, B_, 2, true>); else run(pattn<A_, B_, 4, false>, pattn<A_, B_, 2, false>); } while (0)
  if (z.parts == 1 && z.VN == 8) DSK_PATTN(1, 8);
  else if (z.parts == 1) DSK_PATTN(1, 16);
  else if (z.VN == 8) DSK_PATTN(3, 8);
  else DSK_PATTN(3, 16);
#undef DSK_PATTN
}

// Attention of Tq queries in one kernel: K (keys, values and the visible range given) is split into bf16 parts, then A runs over it.
static void portion_attn(State* S, const PattnSize& z, PackP K, PattnP A, cudaStream_t st) {
  K.V = z.V; K.Dp = z.Dp; K.Vp = z.Vp; K.G = z.G; K.kb = S->k16; K.vb = S->v16;
  A.kb = S->k16; A.vb = S->v16; A.G = z.G; A.D = z.D; A.Dp = z.Dp; A.V = z.V; A.Vp = z.Vp; A.Lk = K.Lk; A.nk = K.nk; A.first = K.first; A.mods.keep = K.keep;
  if (z.parts == 1) launch_next(pattn_pack<1>, K.Lk, 256, 0, st)(K);
  else launch_next(pattn_pack<3>, K.Lk, 256, 0, st)(K);
  if (pattn5_takes(z)) launch_pattn5(S, z, A, st);
  else launch_pattn(S, z, K, A, st);
  if (A.NS > 1) {
    launch_next(latent_swa_merge, dim3((unsigned)(A.T * A.H), (unsigned)((A.V + 127) / 128)), 128, 0, st)(S->ppart, A.out, A.V, A.NS, A.gate, A.ld_gate, A.H, A.gate_head, A.ld_out, A.alpha);
    S->launches++;
  }
  S->launches += 2;
}

// LM head on the wanted rows [first, first + count) of the chunk whose normalised rows are in S->h -> S->logits [count][vocab]
static void enqueue_head(dsk_model* m, dsk_state* s, int first, int count, float* logits, cudaStream_t st) {
  Model* M = m->hy;
  State* S = s->hy;
  const dsk_hybrid_config& c = M->c;
  GemmP P = gp(S->h, c.dim, c.tie_head ? M->embed.p : M->head.p, c.dim, logits, c.vocab_size, count, c.vocab_size, c.dim);
  P.a_map = S->d_want + first; P.alpha = c.logit_scale; P.lim = c.logit_softcap;
  linear(S, c.quant == DSK_BF16, c.logit_softcap > 0.f ? HEPI_SOFTCAP : HEPI_STORE, P, 1, st);
}

// where a kernel that makes rows of the width for the products of a portion puts them rounded (those products read bf16 rows; short steps' read fp32)
static __nv_bfloat16* mirror16(State* S, int T) { return T > 4 ? S->h16 : nullptr; }
// RMS norm in groups, stored.  A warp a group where the groups are more than the CTAs that the chip holds at a time (eight of 256 threads an SM).
// out16 (nullable): packed bf16 rows, with the warps' form beside the others (out may be null), else instead of them.  Returns whether both were written.
static bool rms_groups(const float* in, int ld_in, const float* w, float* out, int ld_out, int T, int n, int groups, float eps, cudaStream_t st, __nv_bfloat16* out16 = nullptr) {
  const bool rows = n / groups <= 1024 && (long long)T * groups > 8ll * g_sm_count;
  if (rows)
    launch_next(group_rmsnorm_rows, (unsigned)(((long long)T * groups + 7) / 8), 256, 0, st)(in, ld_in, w, out, ld_out, T, n, groups, eps, out16);
  else launch_next(group_rmsnorm<float>, dim3((unsigned)T, (unsigned)groups), 256, 0, st)(in, ld_in, w, out, ld_out, n, groups, eps, 0, 0.f, nullptr, 0, nullptr, 0, out ? nullptr : out16);
  return rows;
}
// the model's norm over the T rows of `in` (width values each): stored into `out`, or added into it times alpha (mode 1)
static void norm_rows(const dsk_hybrid_config& c, State* S, const float* in, const float* w, const float* b, float* out, int T, int mode, float alpha, cudaStream_t st) {
  __nv_bfloat16* m16 = mirror16(S, T);
  S->mirror = m16 ? out : nullptr;
  if (c.norm_kind == DSK_NORM_LAYER) launch_next(layer_norm, T, 256, 0, st)(in, c.dim, w, b, out, c.dim, c.dim, c.norm_eps, mode, alpha, nullptr, 0, m16);
  else if (mode == 0 && c.norm_groups == 1) launch_next(rms_open, T, 256, 0, st)(const_cast<float*>(in), nullptr, nullptr, w, out, c.dim, c.norm_eps, m16);   // (adds nothing: the row is only read)
  else if (mode == 0) { if (!rms_groups(in, c.dim, w, out, c.dim, T, c.dim, c.norm_groups, c.norm_eps, st, m16)) S->mirror = nullptr; }
  else {
    S->mirror = nullptr;
    launch_next(group_rmsnorm<float>, dim3((unsigned)T, (unsigned)c.norm_groups), 256, 0, st)(in, c.dim, w, out, c.dim, c.dim, c.norm_groups, c.norm_eps, mode, alpha, nullptr, 0, nullptr, 0, nullptr);
  }
  S->launches++;
}

template <typename... A>
static void launch_rms_add_norm(int T, int n, cudaStream_t st, A... a) {
  if (T <= kAttnSplitTokens) launch_next(rms_add_norm<1024, kLnRegs / 4>, T, 1024, 0, st)(a...);
  else if (n <= 256 * 8) launch_next(rms_add_norm<256, 8>, T, 256, 0, st)(a...);
  else launch_next(rms_add_norm<256, kLnRegs>, T, 256, 0, st)(a...);
}

static bool fused_norms(const dsk_hybrid_config& c) {
  return c.block == DSK_BLOCK_SANDWICH && (c.norm_kind == DSK_NORM_LAYER || c.norm_groups == 1) && c.dim <= 256 * kLnRegs && c.side_dim == 0;
}
static bool rms_fused(const dsk_hybrid_config& c) { return fused_norms(c) && c.norm_kind == DSK_NORM_RMS; }

// where a sublayer's last product goes: added into the residual stream (parallel blocks), or stored for the closing norm
struct Sink { int epi; float* C; float alpha; };

// Enqueues the kernels of one chunk of T <= chunk tokens (ids in S->d_tok, first position in S->d_ctl) on `st`.
// n_want > 0: the LM head runs on the rows listed in S->d_want -> S->logits [n_want][vocab].  trace (device, nullable):
// [layer runs][T][width] copies of the residual stream after every layer run.
// pos0 >= 0: the first position as the host knows it (portions may then take the matrix-product attention path); -1 inside a
// captured step, where positions live in device memory only.
static int enqueue_chunk(dsk_model* m, dsk_state* s, int T, int n_want, float* trace, cudaStream_t st, int pos0 = -1) {
  Model* M = m->hy;
  State* S = s->hy;
  const dsk_hybrid_config& c = M->c;
  const bool bf = c.quant == DSK_BF16;
  chain_step = T <= kAttnSplitTokens || (bf && T <= 256);
  const bool sandwich = c.block == DSK_BLOCK_SANDWICH, post = c.block == DSK_BLOCK_POST, pre = c.block == DSK_BLOCK_PRE;
  const int W = c.dim;
  const float mult = c.residual_mult;
  const float es = c.embed_scale != 0.f ? c.embed_scale : 1.f;
  const int nb = c.bigram_buckets;
  float* keep_emb = S->xin ? S->xin + W : S->emb;   // the embedding output again, for a layer loop
  const int ld_keep = S->xin ? 2 * W : W;
  S->mirror = nullptr;
  if (bf) launch_next(embed_rows<__nv_bfloat16>, T, 256, 0, st)(S->d_tok, (const __nv_bfloat16*)M->embed.p, W, S->x, es, nb > 0 ? (const __nv_bfloat16*)M->bigram.p : nullptr,
                                                       nb, c.bigram_mul_prev, c.bigram_mul_cur, S->d_ctl, S->d_prev, keep_emb, ld_keep);
  else launch_next(embed_rows<float>, T, 256, 0, st)(S->d_tok, (const float*)M->embed.p, W, S->x, es, nb > 0 ? (const float*)M->bigram.p : nullptr, nb, c.bigram_mul_prev,
                                            c.bigram_mul_cur, S->d_ctl, S->d_prev, keep_emb, ld_keep);
  S->launches++;
  if (nb > 0) { launch_next(carry_token, 1, 1, 0, st)(S->d_tok, T, S->d_prev); S->launches++; }   // the next step's first token pairs with this step's last
  if (pos0 < 0) S->tl_used = 0;   // a captured step records no events
  const bool tl = S->timeline && pos0 >= 0;
  auto MK = [&](const char* label) { if (tl) mark(S, label, st); };
  MK("embed");
  // a product whose input the kernel ahead of it may write rounded: where to
  auto rounded = [&](int epi, GemmP& P) -> __nv_bfloat16* { return T > 4 && bf && tc_ok(S, bf, epi, P, 1) ? const_cast<__nv_bfloat16*>(P.A16 = S->a16) : nullptr; };
  const Sink to_x{HEPI_ADD, S->x, mult}, to_y{HEPI_STORE, S->y, 1.f};
  // sandwich blocks: "x += norm(y); h = norm(x)" runs as one kernel (not while the residual stream is being recorded)
  const bool fuse = fused_norms(c) && !trace, frms = fuse && rms_fused(c);
  bool xin_ready = false; // the stream already stands in S->xin (the coming run opens a loop pass with a product)
  bool h_ready = false;   // S->h already holds the norm that opens the coming run (or the final norm)
  bool hs_ready = false;  // S->hs already holds the token-shifted input of the coming run's mixer
  for (size_t ri = 0; ri < M->runs.size(); ri++) {
    const Run& run = M->runs[ri];
    const int li = run.layer;
    const HLayer& L = M->L[li];
    const dsk_layer_spec& sp = L.sp;
    LayerState& ls = S->L[ri];
    // post-norm blocks: a sublayer reads u = x + conv(x) (S->h; the stream itself without a convolution); afterwards its result y is gated
    // by sigmoid(rg x + b), normalised with the folded weight (norm x layer scale) and added to the stream
    auto open_post = [&](const float* taps, int which) -> const float* {
      if (c.canon_taps <= 0) return S->x;
      float* ring = ls.canon ? ls.canon + (size_t)which * (c.canon_taps - 1) * W : nullptr;
      const int ty = (T + kCanonTokens - 1) / kCanonTokens;
      S->mirror = nullptr;
      launch_next(canon_conv, dim3((unsigned)((W + 127) / 128), (unsigned)ty), 128, 0, st)(S->x, W, taps, ring, S->h, W, T, W, c.canon_taps, S->d_ctl);
      S->launches++;
      if (ty > 1 && c.canon_taps > 1) { launch_next(canon_history, (W + 127) / 128, 128, 0, st)(S->x, W, ring, T, W, c.canon_taps, S->d_ctl); S->launches++; }
      return S->h;
    };
    auto close_post = [&](const HTensor& rg, const float* rg_b, const float* close_w, const float* close_b) {
      if (c.res_gate) {
        GemmP G = gp(S->x, W, rg.p, W, S->y, W, T, W, W);
        G.bias = rg_b;
        linear(S, bf, HEPI_SIGMUL, G, 1, st);
      }
      norm_rows(c, S, S->y, close_w, close_b, S->x, T, 1, mult, st);
    };
    // decode-sized steps: the closing norm and the next sublayer's input convolution as one kernel (not while the stream is recorded);
    // next_taps / next_ring: the convolution that follows (the feed-forward's, or the next layer's mixer's)
    const bool small_post = post && c.canon_taps > 0 && T <= kCloseOpenTokens && !trace;
    auto close_open = [&](const HTensor& rg, const float* rg_b, const float* close_w, const float* next_taps, float* next_ring) {
      if (c.res_gate) {
        GemmP G = gp(S->x, W, rg.p, W, S->y, W, T, W, W);
        G.bias = rg_b;
        linear(S, bf, HEPI_SIGMUL, G, 1, st);
      }
      S->mirror = nullptr;
      launch_next(close_open_small, (W + 127) / 128, 128, 0, st)(S->y, close_w, mult, c.norm_eps, S->x, W, next_taps, next_ring, S->h, T, W, c.canon_taps, S->d_ctl);
      S->launches++;
    };
    auto ring_of = [&](size_t run_i, int which) { return S->L[run_i].canon ? S->L[run_i].canon + (size_t)which * (c.canon_taps - 1) * W : nullptr; };
    const bool has_next = ri + 1 < M->runs.size();
    const float* hin = S->h;   // what the mixer reads
    if (post) { if (!h_ready) hin = open_post(L.canon1, 0); }
    else if (pre) {   // a pass of the layer loop opens with its vector (and, but for the first, the embedding) added to the stream
      const bool again = c.loop_embed && run.pass > 0;
      launch_next(rms_open, T, 256, 0, st)(S->x, again ? S->emb : nullptr, run.pass >= 0 ? M->loop_step + (size_t)run.pass * W : nullptr, L.norm1, S->h, W, c.norm_eps, mirror16(S, T));
      S->mirror = mirror16(S, T) ? S->h : nullptr;
      S->launches++;
    } else if (!h_ready) {
      if (run.pass >= 0 && c.loop_in) {   // a pass of the layer loop opens with a product over [stream | embedding], its vector as the bias
        if (!xin_ready) { launch_next(copy_rows, T, 256, 0, st)(S->x, W, S->xin, 2 * W, W); S->launches++; }
        xin_ready = false;
        GemmP In = gp(S->xin, 2 * W, M->loop_in.p, 2 * W, S->x, W, T, W, 2 * W);
        In.bias = M->loop_step + (size_t)run.pass * W;
        linear(S, bf, HEPI_STORE, In, 1, st);
        MK("loop.in");
      } else if (run.pass >= 0) {   // a pass of the layer loop opens with its own vector added to the residual stream
        if (S->mirror == S->x) S->mirror = nullptr;
        launch_next(add_row, T, 256, 0, st)(S->x, W, M->loop_step + (size_t)run.pass * W, W);
        S->launches++;
      }
      norm_rows(c, S, S->x, L.norm1, L.norm1_bias, S->h, T, 0, 0.f, st);
    }
    h_ready = false;
    const float* hff = hin;   // what a feed-forward of a parallel block reads: the mixer's input ahead of the token shift
    if (c.token_shift && hs_ready) { hin = S->hs; hs_ready = false; }   // the previous run's last kernel shifted already
    else if (c.token_shift) {      // the mixer reads its input blended with the previous token's; the step's last row is carried on
      const int ty = (T + kCanonTokens - 1) / kCanonTokens;
      launch_next(token_shift, dim3((unsigned)((W + 127) / 128), (unsigned)ty), 128, 0, st)(hin, W, L.shift, ls.shift, S->hs, W, T, W, S->d_ctl, mirror16(S, T));
      S->mirror = mirror16(S, T) ? S->hs : nullptr;
      S->launches++;
      if (ty > 1) { launch_next(shift_carry, (W + 127) / 128, 128, 0, st)(hin, W, ls.shift, T, W); S->launches++; }
      hin = S->hs;
    }
    // the closing norm of this run's last sublayer, fused with what opens the next run (its pass vector and first norm) or the head
    auto close_run = [&](const float* wb, int routed = 0) {   // routed > 0: the sublayer's output is the weighted sum of the routed rows in S->b3
      if (!fuse) { norm_rows(c, S, S->y, wb, nullptr, S->x, T, 1, mult, st); return; }
      __nv_bfloat16* m16 = mirror16(S, T);
      const Run* next = ri + 1 < M->runs.size() ? &M->runs[ri + 1] : nullptr;
      if (frms) {
        const bool to_xin = next && next->pass >= 0;   // the pass opens with a product: its norm follows that
        const bool product = to_xin && c.loop_in;
        const bool shared = routed && sp.ff_shared > 0;
        launch_rms_add_norm(T, W, st, routed ? S->b3 : S->y, routed ? S->wgt : nullptr, routed, shared ? S->b3 + (size_t)T * routed * W : nullptr, S->wsh, wb, S->x,
                                        product ? S->xin : S->x, product ? 2 * W : W, to_xin ? nullptr : next ? M->L[next->layer].norm1 : M->final_norm, S->h, W, c.norm_eps, mult, m16);
        S->mirror = !to_xin && m16 ? S->h : nullptr;
        S->launches++;
        xin_ready = product;
        h_ready = !to_xin;
        return;
      }
      const float* row = next && next->pass >= 0 ? M->loop_step + (size_t)next->pass * W : nullptr;
      launch_next(layer_norm_add_norm, T, 256, 0, st)(S->y, wb, S->x, row, next ? M->L[next->layer].norm1 : M->final_norm, S->h, W, c.norm_eps, mult, m16);
      S->mirror = m16 ? S->h : nullptr;
      S->launches++;
      h_ready = true;
    };
    const Sink sink = (sandwich || post) ? to_y : to_x;
    // a routed feed-forward that closes with a layer norm and no gate: no separate pass for the weighted sum of the experts' outputs
    const bool combine_in_norm = post && sp.ff_kind == DSK_FF_MOE && c.norm_kind == DSK_NORM_LAYER && !c.res_gate && W <= 256 * kLnRegs && sp.ff_shared == 0;
    if (sp.mixer == DSK_MIX_GQA) {
      const int H = sp.att_heads, G = sp.att_kv_heads, D = sp.att_dim, V = sp.att_vdim, HD = H * D, GD = G * D, GV = G * V, rep = H / G;
      const int keep = sp.att_keep_first;
      const bool reads = sp.att_kv_from >= 0;   // keys and values of another layer: its caches, written earlier in this step
      const int ring = M->L[L.owner].ring;
      float *kc = (float*)S->L[R0(M, ri)].cache, *vc = (float*)S->L[R0(M, ri)].vcache;
      const ScoreMods sm{sp.att_softcap, sp.att_rel_max > 0 ? L.rel : nullptr, L.rel_bucket, sp.att_rel_max, sp.att_sink ? L.sink : nullptr, keep};
      MK("norm");
      const AttLayout lay = att_layout(sp);
      const int HV = (int)lay.gate_rows;   // the output gate's raw values come out of the stacked product
      const int ldp = reads ? HD + HV : (int)lay.total;
      const float* gate = HV ? S->b0 + (reads ? HD : (int)lay.gate) : nullptr;
      const int gate_head = sp.att_out_gate == DSK_GATE_HEAD;
      const int ldo = H * V + (sp.mixer2 ? (int)gdn_v(sp) : 0);   // a second mixer's heads stand behind this one's
      const float lscale = sp.mixer2 ? sp.mix_scale : 1.f;
      // a decoded token's heads over several CTAs, where each head has a norm of its own
      const dim3 qk_grid((unsigned)T, (unsigned)(sp.att_qk_norm != DSK_QKNORM_WHOLE && T <= kAttnSplitTokens ? (H + (reads ? 0 : G) + 7) / 8 : 1));
      if (reads) {
        linear(S, bf, HEPI_STORE, gp(hin, W, L.qkv.p, W, S->b0, ldp, T, ldp, W), 1, st);
        MK("att.qk");
        launch_next(qk_norm_rope, qk_grid, 256, 0, st)(S->b0, S->b2, HD, nullptr, nullptr, GD, GV, ldp, 0, 0, L.q_norm, nullptr, c.norm_eps, D, sp.rot_dims, L.rot_freq,
                                        L.rot_mag, S->d_ctl, nullptr, nullptr, ring, keep, nullptr, 0.f, nullptr, sp.rot_layout, sp.att_qk_norm, ConvP{nullptr, nullptr, 0, 1, 0});
      } else if (sp.att_value_proj) {   // one product for the stacked q / k / v rows; the first value-mixing layer keeps its values for the later ones
        const int ld = ldp;
        GemmP P = gp(hin, W, L.qkv.p, W, S->b0, ld, T, ld, W);
        P.bias = sp.att_bias ? L.qkv_b : nullptr;
        linear(S, bf, HEPI_STORE, P, 1, st);
        MK("att.qk");
        if (sp.mixer2 == DSK_MIX_GDN && !tl) {   // the second mixer on its own stream: it shares nothing with the first but the projections
          CKL(cudaEventRecord(S->ev_fork, st));
          CKL(cudaStreamWaitEvent(S->side, S->ev_fork, 0));
          plain_next = true;
          gdn_forward(S, L, ls, ldp, lay, S->b3 + H * V, ldo, sp.mix2_scale, c.norm_eps, T, S->side);
          CKL(cudaEventRecord(S->ev_join, S->side));
          plain_next = true;
        }
        const bool blend = sp.att_vmix && li != M->vmix_first;
        ConvP cv{nullptr, nullptr, 0, 1, 0};
        if (sp.att_conv > 0) cv = ConvP{L.conv_w, ls.hist, sp.att_conv, sp.att_conv - 1 + kConvSpare, sp.att_conv > 1 && T <= kConvSpare};
        launch_next(qk_norm_rope, qk_grid, 256, cv.w ? (size_t)8 * D * 4 : 0, st)(S->b0, S->b2, HD, S->b0 + HD, S->b0 + HD + GD, GD, GV, ld, ld, ld, L.q_norm, L.k_norm, c.norm_eps, D, sp.rot_dims,
                                        L.rot_freq, L.rot_mag, S->d_ctl, kc, vc, ring, keep, blend ? S->vfirst : nullptr, L.vmix,
                                        sp.att_vmix && li == M->vmix_first ? S->vfirst : nullptr, sp.rot_layout, sp.att_qk_norm, cv);
        if (sp.att_conv > 1 && !cv.store) {   // a long step stores its last inputs after its convolutions
          launch_next(conv_ring_store, (HD + GD + GV + 127) / 128, 128, 0, st)(S->b0, ld, 0, ls.hist, cv.ring, T, HD + GD + GV, sp.att_conv, S->d_ctl);
          S->launches++;
        }
      } else {
        linear(S, bf, HEPI_STORE, gp(hin, W, L.q.p, W, S->b0, HD, T, HD, W), 1, st);
        linear(S, bf, HEPI_STORE, gp(hin, W, L.kproj.p, W, S->b1, GD, T, GD, W), 1, st);
        MK("att.qk");
        launch_next(qk_norm_rope, qk_grid, 256, 0, st)(S->b0, S->b2, HD, S->b1, nullptr, GD, GV, HD, GD, GD, L.q_norm, L.k_norm, c.norm_eps, D, sp.rot_dims, L.rot_freq,
                                        L.rot_mag, S->d_ctl, kc, vc, ring, keep, nullptr, 0.f, nullptr, sp.rot_layout, sp.att_qk_norm, ConvP{nullptr, nullptr, 0, 1, 0});
      }
      S->launches++;
      MK("att.norm+rot");
      if (pos0 >= 0 && T >= kPrefillMin && S->prefill_keys > 0) {
        if (takes_pattn(sp, bf)) {
          const PattnSize z = pattn_size(sp, bf);
          for (int t0 = 0; t0 < T; t0 += S->pattn_q) {
            const int Tq = std::min(S->pattn_q, T - t0), qpos0 = pos0 + t0;
            PackP K{};
            K.first = mask_first(sp.att_mask, sp.att_window, qpos0); K.nk = std::min(keep, K.first); K.Lk = K.nk + qpos0 + Tq - K.first; K.keep = keep; K.ring = ring;
            K.k = kc; K.v = vc; K.ldk = GD; K.ldv = GV; K.D0 = D; K.kv_cached = 1;
            PattnP A{};
            A.q = S->b2 + (size_t)t0 * HD; A.ldq = HD; A.out = S->b3 + (size_t)t0 * ldo; A.ld_out = ldo; A.gate = gate ? gate + (size_t)t0 * ldp : nullptr; A.ld_gate = ldp;
            A.gate_head = gate_head; A.T = Tq; A.H = H; A.pos0 = qpos0; A.mask = sp.att_mask; A.span = sp.att_window; A.scale = sp.att_scale; A.alpha = lscale; A.mods = sm;
            portion_attn(S, z, K, A, st);
          }
          MK("att.fused");
        } else {
        // a portion: blocks of queries, each as  scores = q k^T per head (fp32);  mixing of the heads and masked softmax;  o = P v
        const int block_q = sp.att_talk ? S->talk_q : kPrefillQ;
        for (int t0 = 0; t0 < T; t0 += block_q) {
          const int Tq = std::min(block_q, T - t0), qpos0 = pos0 + t0;
          const int first = mask_first(sp.att_mask, sp.att_window, qpos0), nk = std::min(keep, first), Lk = nk + qpos0 + Tq - first;
          const int LP = (Lk + 3) & ~3;   // rows of scores and of transposed values take 16-byte loads
          launch_next(pack_ring_kv<float>, Lk, 256, 0, st)(kc, vc, S->kf, S->vf, first, Lk, LP, ring, G, D, V, nk, keep);
          S->launches++;
          MK("att.pack");
          GemmP Sc = gp(S->b2 + (size_t)t0 * HD, HD, S->kf, D, S->sc, LP, Tq, Lk, D);
          Sc.w_made = 1;
          Sc.sA = D; Sc.sW = (long long)Lk * D; Sc.z_wdiv = rep; Sc.sC = (long long)Tq * LP; Sc.alpha = sp.att_scale;
          Sc.band = BAND_COLS; Sc.band_first = first - nk; Sc.band_pos = qpos0; Sc.band_mask = sp.att_mask; Sc.band_window = sp.att_window; Sc.band_keep = keep;
          linear(S, false, HEPI_STORE, Sc, H, st);
          MK("att.scores");
          if (sp.att_talk) {
            const int hr = H <= 16 ? 16 : H <= 32 ? 32 : 0, nt = hr ? 512 : 128;
            const size_t base = ((size_t)(H * (hr ? hr : H) + 3) / 4 * 4 + (hr ? 0 : (size_t)H * nt)) * 4, all = base + (size_t)H * Lk * 4;
            const int staged = all <= (size_t)200 * 1024;
            auto* kernel = hr == 16 ? mix_softmax<16> : hr == 32 ? mix_softmax<32> : mix_softmax<0>;
            launch_next(kernel, (unsigned)Tq, (unsigned)nt, staged ? all : base, st)(S->sc, L.talk, H, Tq, Lk, LP, first, qpos0, sp.att_mask, sp.att_window, nk, sm, staged);
          } else {
            launch_next(softmax_band, dim3((unsigned)Tq, (unsigned)H), 128, 0, st)(S->sc, Tq, Lk, LP, first, qpos0, sp.att_mask, sp.att_window, nk, sm);
          }
          S->launches++;
          MK("att.softmax");
          GemmP Ov = gp(S->sc, LP, S->vf, LP, S->b3 + (size_t)t0 * ldo, ldo, Tq, V, Lk);
          Ov.w_made = 1;
          Ov.sA = (long long)Tq * LP; Ov.sW = (long long)V * LP; Ov.z_wdiv = rep; Ov.sC = V; Ov.alpha = lscale;
          Ov.band = BAND_DEPTH; Ov.band_first = Sc.band_first; Ov.band_pos = qpos0; Ov.band_mask = sp.att_mask; Ov.band_window = sp.att_window; Ov.band_keep = Sc.band_keep;
          linear(S, false, HEPI_STORE, Ov, H, st);
          MK("att.pv");
        }
        if (gate) { launch_next(gate_rows, T, 256, 0, st)(S->b3, ldo, gate, ldp, H * V, gate_head ? V : 1); S->launches++; }   // heads *= sigmoid(g h)
        }
      } else if (!sp.att_talk && decode_attn_fits(D, V)) {
        DecodeAttn A{};
        A.q = S->b2; A.kc = kc; A.vc = vc; A.out = S->b3; A.ctl = S->d_ctl; A.gate = gate; A.T = T; A.H = H; A.G = G; A.D = D; A.Dv = V; A.ldk = GD; A.ldv = GV;
        A.mask = sp.att_mask; A.span = sp.att_window; A.ring = ring; A.ld_gate = ldp; A.gate_head = gate_head; A.ld_out = ldo; A.scale = sp.att_scale; A.alpha = lscale; A.mods = sm;
        launch_decode_attn(S, A, false, st);
        MK("att.decode");
      } else {
        int NS = 1;
        if (T <= kAttnSplitTokens) NS = std::max(1, std::min((std::min(sp.att_window, ring) + keep + 31) / 32, kAttnSplitMax));
        const int GL = gqa_key_heads(H, G, sp.att_talk != 0);   // without score mixing the key heads are dealt over CTAs
        launch_next(gqa_attn, dim3((unsigned)T, (unsigned)NS, (unsigned)(G / GL)), 256, gqa_attn_smem_floats(GL * rep, GL, D, V, sp.att_talk != 0) * 4, st)(
            S->b2, kc, vc, S->b3, sp.att_talk ? L.talk : nullptr, T, H, G, D, V, S->d_ctl, sp.att_mask, sp.att_window, ring, sp.att_scale, NS, S->part, sm,
            NS > 1 ? nullptr : gate, ldp, gate_head, ldo, lscale);
        if (NS > 1) launch_next(latent_swa_merge, dim3((unsigned)(T * H), (unsigned)((V + 127) / 128)), 128, 0, st)(S->part, S->b3, V, NS, gate, ldp, H, gate_head, ldo, lscale);
        S->launches += NS > 1 ? 2 : 1;
        MK("att.decode");
      }
      if (sp.mixer2 == DSK_MIX_GDN && !tl) { CKL(cudaStreamWaitEvent(st, S->ev_join, 0)); plain_next = true; }
      else if (sp.mixer2 == DSK_MIX_GDN) {   // timeline: one after the other
        gdn_forward(S, L, ls, ldp, lay, S->b3 + H * V, ldo, sp.mix2_scale, c.norm_eps, T, st);
        MK("gdn");
      }
      GemmP P = gp(S->b3, ldo, L.o.p, ldo, sink.C, W, T, W, ldo);   // both mixers' output matrices in one product
      P.alpha = sink.alpha;
      linear(S, bf, sink.epi, P, 1, st);
      MK("att.o");
    } else if (sp.mixer == DSK_MIX_MLA) {
      const int H = sp.att_heads, D = sp.att_dim, Rd = sp.att_rot_dim, DK = D + Rd, V = sp.att_vdim, R = sp.att_kv_rank, RW = R + Rd, Q = sp.att_q_rank;
      float* cache = (float*)ls.cache;
      const int ldi = Q + RW;
      MK("norm");
      linear(S, bf, HEPI_STORE, gp(hin, W, L.in2.p, W, S->b1, ldi, T, ldi, W), 1, st);              // [query latent | key / value latent | rotated key part]
      GemmP Uq = gp(S->b2, Q, L.uq.p, Q, S->b0, H * DK, T, H * DK, Q);                             // q [T][H][D | Rd]
      __nv_bfloat16* q16 = rounded(HEPI_STORE, Uq);
      rms_groups(S->b1, ldi, L.dq_norm, q16 ? nullptr : S->b2, Q, T, Q, 1, c.norm_eps, st, q16);
      S->launches++;
      linear(S, bf, HEPI_STORE, Uq, 1, st);
      const bool portion = pos0 >= 0 && T >= kPrefillMin && S->prefill_keys > 0;
      launch_next(mla_prepare, T, 256, 0, st)(S->b1 + Q, ldi, L.dkv_norm, c.norm_eps, S->b0, portion ? nullptr : S->b2, H, D, Rd, R, sp.rot_dims, L.rot_freq,
                                     L.rot_mag, sp.rot_layout, S->d_ctl, cache, L.ring);
      S->launches++;
      MK("att.q+latent");
      float* ov = S->b3;   // [T][H*V] heads' outputs
      ScoreMods sm{};
      sm.sink = sp.att_sink ? L.sink : nullptr;
      if (portion && takes_pattn(sp, bf)) {   // plain keys and values up-projected from the visible latents, the rotated key part shared by the heads
        const PattnSize z = pattn_size(sp, bf);
        for (int t0 = 0; t0 < T; t0 += S->pattn_q) {
          const int Tq = std::min(S->pattn_q, T - t0), qpos0 = pos0 + t0;
          PackP P{};
          P.first = mask_first(sp.att_mask, sp.att_window, qpos0); P.Lk = qpos0 + Tq - P.first; P.ring = L.ring;
          launch_next(ring_rows, (P.Lk + 255) / 256, 256, 0, st)(P.first, P.Lk, L.ring, S->d_rows);
          GemmP K = gp(cache, RW, L.uk.p, R, S->kf, H * D, P.Lk, H * D, R);
          K.a_map = S->d_rows;
          linear(S, bf, HEPI_STORE, K, 1, st);
          GemmP Vp = gp(cache, RW, L.uv.p, R, S->vf, H * V, P.Lk, H * V, R);
          Vp.a_map = S->d_rows;
          linear(S, bf, HEPI_STORE, Vp, 1, st);
          MK("att.kv_up");
          P.k = S->kf; P.v = S->vf; P.krot = cache + R; P.ldk = H * D; P.ldv = H * V; P.ldr = RW; P.D0 = D; P.Rd = Rd;
          PattnP A{};
          A.q = S->b0 + (size_t)t0 * H * DK; A.ldq = H * DK; A.out = S->b3 + (size_t)t0 * H * V; A.ld_out = H * V; A.T = Tq; A.H = H; A.pos0 = qpos0; A.mask = sp.att_mask;
          A.span = sp.att_window; A.scale = sp.att_scale; A.alpha = 1.f; A.mods = sm;
          portion_attn(S, z, P, A, st);
          S->launches++;
        }
        MK("att.fused");
      } else if (portion) {
        // blocks of kPrefillQ queries: plain keys and values up-projected from the visible latents, the rotated key part appended to every
        // head's keys; scores, softmax and the value product in fp32
        for (int t0 = 0; t0 < T; t0 += kPrefillQ) {
          const int Tq = std::min(kPrefillQ, T - t0), qpos0 = pos0 + t0;
          const int first = mask_first(sp.att_mask, sp.att_window, qpos0), Lk = qpos0 + Tq - first;
          launch_next(ring_rows, (Lk + 255) / 256, 256, 0, st)(first, Lk, L.ring, S->d_rows);
          GemmP K = gp(cache, RW, L.uk.p, R, S->kf, H * D, Lk, H * D, R);
          K.a_map = S->d_rows;
          linear(S, bf, HEPI_STORE, K, 1, st);
          GemmP Vp = gp(cache, RW, L.uv.p, R, S->vf, H * V, Lk, H * V, R);
          Vp.a_map = S->d_rows;
          linear(S, bf, HEPI_STORE, Vp, 1, st);
          MK("att.kv_up");
          launch_next(pack_mla_kv, Lk, 256, 0, st)(S->kf, S->vf, cache, S->d_rows, (float*)S->kb, (float*)S->vt, Lk, H, D, Rd, R, V);
          MK("att.pack");
          GemmP Sc = gp(S->b0 + (size_t)t0 * H * DK, H * DK, S->kb, DK, S->sc, Lk, Tq, Lk, DK);
          Sc.w_made = 1;
          Sc.sA = DK; Sc.sW = (long long)Lk * DK; Sc.sC = (long long)Tq * Lk; Sc.alpha = sp.att_scale;
          linear(S, false, HEPI_STORE, Sc, H, st);
          MK("att.scores");
          launch_next(softmax_band, dim3((unsigned)Tq, (unsigned)H), 128, 0, st)(S->sc, Tq, Lk, Lk, first, qpos0, sp.att_mask, sp.att_window, 0, sm);
          MK("att.softmax");
          GemmP Ov = gp(S->sc, Lk, S->vt, Lk, S->b3 + (size_t)t0 * H * V, H * V, Tq, V, Lk);
          Ov.w_made = 1;
          Ov.sA = (long long)Tq * Lk; Ov.sW = (long long)V * Lk; Ov.sC = V;
          linear(S, false, HEPI_STORE, Ov, H, st);
          MK("att.pv");
          S->launches += 3;
        }
      } else {
        {   // absorbed query: qa[t][h][0:R] = W_uk[h]^T q_plain[t][h]  (mla_prepare put the rotated part behind it)
          GemmP P = gp(S->b0, H * DK, L.ukT.p, D, S->b2, H * RW, T, R, D);
          P.sA = DK; P.sW = (long long)R * D; P.sC = RW;
          linear(S, bf, HEPI_STORE, P, H, st);
        }
        launch_latent_attn(S, S->b2, cache, S->b3, T, H, RW, sp.att_mask, sp.att_window, L.ring, sp.att_scale, sm.sink, st);
        {  // value up-projection per head from the first R entries of the weighted cache rows
          GemmP P = gp(S->b3, H * RW, L.uv.p, R, S->b0, H * V, T, V, R);
          P.sA = RW; P.sW = (long long)V * R; P.sC = V;
          linear(S, bf, HEPI_STORE, P, H, st);
        }
        ov = S->b0;
        MK("att.absorbed");
      }
      if (sp.att_out_gate) linear(S, bf, HEPI_SIGMUL, gp(hin, W, L.gmat.p, W, ov, H * V, T, H * V, W), 1, st);   // heads *= sigmoid(g u)
      GemmP P = gp(ov, H * V, L.o.p, H * V, sink.C, W, T, W, H * V);
      P.alpha = sink.alpha;
      linear(S, bf, sink.epi, P, 1, st);
      MK("att.o");
    } else if (sp.mixer == DSK_MIX_GDN) {
      const AttLayout lay = att_layout(sp);
      const int ldp = (int)lay.total, RV = (int)gdn_v(sp);
      MK("norm");
      linear(S, bf, HEPI_STORE, gp(hin, W, L.qkv.p, W, S->b0, ldp, T, ldp, W), 1, st);
      MK("gdn.in");
      GemmP P = gp(S->b3, RV, L.o.p, RV, sink.C, W, T, W, RV);
      P.alpha = sink.alpha;
      gdn_forward(S, L, ls, ldp, lay, S->b3, RV, 1.f, c.norm_eps, T, st, rounded(sink.epi, P));
      MK("gdn");
      linear(S, bf, sink.epi, P, 1, st);
      MK("gdn.o");
    } else if (sp.mixer == DSK_MIX_MLSTM) {
      const MlstmLayout lay = mlstm_layout(sp);
      const int HP = sp.lin_heads * sp.lin_vdim, pw = (int)lay.total;
      MK("norm");
      GemmP In = gp(hin, W, L.lin_in.p, W, S->b0, pw, T, pw, W);
      In.bias = L.lin_bias;
      linear(S, bf, HEPI_STORE, In, 1, st);
      MK("lin.in");
      GemmP P = gp(S->b3, HP, L.o.p, HP, sink.C, W, T, W, HP);
      P.alpha = sink.alpha;
      mlstm_forward(S, L, ls, pw, lay, S->b3, c.norm_eps, T, st, rounded(sink.epi, P));
      MK("lin.scan");
      linear(S, bf, sink.epi, P, 1, st);
      MK("lin.o");
    } else if (sp.mixer == DSK_MIX_LIGHTNING) {
      const int HN = sp.lin_heads * sp.lin_dim, HP = sp.lin_heads * sp.lin_vdim, pw = 2 * HN + 2 * HP;
      MK("norm");
      GemmP In = gp(hin, W, L.lin_in.p, W, S->b0, pw, T, pw, W);   // [silu q | silu k | silu v | sigmoid g]: the activations run in the product's epilogue
      In.aux_off = 2 * HN + HP;
      linear(S, bf, HEPI_SILU_SIG, In, 1, st);
      MK("lin.in");
      lightning_forward(S, L, ls, pw, T, st);
      MK("lin.scan");
      GemmP P = gp(S->b3, HP, L.o.p, HP, sink.C, W, T, W, HP);
      P.alpha = sink.alpha;
      launch_next(group_rmsnorm<float>, T, 256, 0, st)(S->lout, HP, L.mnorm, S->b3, HP, HP, 1, c.norm_eps, 0, 0.f, nullptr, 0, S->b0 + 2 * HN + HP, pw, rounded(sink.epi, P));
      S->launches++;
      MK("lin.norm");
      linear(S, bf, sink.epi, P, 1, st);
      MK("lin.o");
    } else if (sp.mixer == DSK_MIX_HGRN2) {
      const int H = sp.lin_heads, HN = H * sp.lin_dim, HP = H * sp.lin_vdim, pw = 2 * HN + HP;
      MK("norm");
      GemmP In = gp(hin, W, L.lin_in.p, W, S->b0, pw, T, pw, W);   // [silu(q) | forget gate | v]: the activations run in the product's epilogue, in fp32
      In.bias = L.lin_bias; In.aux = L.lower; In.aux_off = HN;
      linear(S, bf, HEPI_LINGATE, In, 1, st);
      MK("lin.in");
      launch_hgrn2(sp, S->b0, pw, ls.lin, S->b2, T, st);
      MK("lin.scan");
      GemmP P = gp(S->b3, HP, L.o.p, HP, sink.C, W, T, W, HP);
      P.alpha = sink.alpha;
      launch_next(head_rmsnorm, (unsigned)(((long long)T * H + 7) / 8), 256, 0, st)(S->b2, HP, L.lin_norm, S->b3, HP, T, H, sp.lin_vdim, c.norm_eps, nullptr, 0, 1.f, 0, 0, nullptr, nullptr,
                                                                                    rounded(sink.epi, P));
      S->launches += 2;
      MK("lin.norm");
      linear(S, bf, sink.epi, P, 1, st);
      MK("lin.o");
    } else if (is_ssd(sp)) {
      const int inner = (int)ssd_inner(sp), ch = (int)ssd_channels(sp), pw = (int)ssd_proj(sp);
      MK("norm");
      linear(S, bf, HEPI_STORE, gp(hin, W, L.in.p, W, S->b0, pw, T, pw, W), 1, st);
      MK("ssd.in");
      if (T <= kConvShort) launch_next(causal_conv_silu_short, (ch + 127) / 128, 128, 0, st)(S->b0 + inner, pw, L.conv_w, L.conv_b, ls.hist, S->b1, ch, T, ch, sp.ssm_conv);
      else {
        launch_next(causal_conv_silu, dim3((unsigned)((ch + 127) / 128), (unsigned)((T + kConvTokens - 1) / kConvTokens)), 128, 0, st)(S->b0 + inner, pw, L.conv_w, L.conv_b, ls.hist, S->b1, ch, T, ch, sp.ssm_conv);
        if (sp.ssm_conv > 1) launch_next(conv_history_update, (ch + 127) / 128, 128, 0, st)(S->b0 + inner, pw, ls.hist, T, ch, sp.ssm_conv);
      }
      MK("ssd.conv");
      if (T > kLinDecodeTokens && ssd_gram_smem(sp) <= 200 * 1024) {   // blocks of 16 tokens at once (ssd_scan: a chain over single tokens, 0.47 us each)
        const int H = sp.ssm_heads, N = sp.ssm_state, P = sp.ssm_vdim, G = sp.ssm_groups;
        launch_next(ssd_gram, dim3((unsigned)((T + kLinBlk - 1) / kLinBlk), (unsigned)G), 256, ssd_gram_smem(sp), st)(
            S->b1 + inner + G * N, S->b1 + inner, ch, S->b0 + inner + ch, pw, L.dt_bias, L.A_log, T, H, N, H / G, S->lrec);
        launch_lin_scan(false, S->b1 + inner + G * N, S->b1 + inner, ch, N, H / G, S->b1, ch, S->lrec, ls.ssm, S->b2, inner, T, H, N, P, st, S, nullptr, nullptr, 1, N);
        if (inner % 4 == 0 && ch % 4 == 0 && pw % 4 == 0 && P % 4 == 0)
          launch_next(ssd_gate<4>, dim3((unsigned)T, (unsigned)((inner + 1023) / 1024)), 256, 0, st)(S->b2, S->b1, ch, S->b0, pw, L.D, inner, P);
        else launch_next(ssd_gate<1>, dim3((unsigned)T, (unsigned)((inner + 255) / 256)), 256, 0, st)(S->b2, S->b1, ch, S->b0, pw, L.D, inner, P);
        S->launches += 2;
      } else launch_scan(sp, S->b0, pw, S->b1, ch, L, ls.ssm, S->b2, T, st);
      MK("ssd.scan");
      GemmP P = gp(S->b3, inner, L.o.p, inner, sink.C, W, T, W, inner);
      P.alpha = sink.alpha;
      __nv_bfloat16* o16 = rounded(sink.epi, P);
      rms_groups(S->b2, inner, L.mnorm, o16 ? nullptr : S->b3, inner, T, inner, sp.ssm_norm_groups, c.norm_eps, st, o16);
      S->launches += 4;
      MK("ssd.norm");
      linear(S, bf, sink.epi, P, 1, st);
      MK("ssd.o");
    } else {
      const int H = sp.att_heads, D = sp.att_dim, V = sp.att_vdim, R = sp.att_kv_rank;
      const HLayer& O = M->L[L.owner];
      float* cache = (float*)S->L[R0(M, ri)].cache;
      MK("norm");
      linear(S, bf, HEPI_STORE, gp(hin, W, L.q.p, W, S->b0, H * D, T, H * D, W), 1, st);
      if (L.owner == li) {
        linear(S, bf, HEPI_STORE, gp(hin, W, L.dkv.p, W, S->b1, R, T, R, W), 1, st);
        launch_next(group_rmsnorm<float>, T, 256, 0, st)(S->b1, R, L.dkv_norm, cache, R, R, 1, c.norm_eps, 0, 0.f, S->d_ctl, O.ring, nullptr, 0, nullptr);
        S->launches++;
      }
      MK("att.q+latent");
      const float* ov = S->b0;   // [T][H*V] heads' outputs
      if (pos0 >= 0 && T >= kPrefillMin && S->prefill_keys > 0) {
        // a portion: blocks of kPrefillQ queries, each as  k, v = up-projections of the visible latents;  P = softmax_band(q k^T);  o = P v
        ov = S->b3;
        if (takes_pattn(sp, bf)) {
          const PattnSize z = pattn_size(sp, bf);
          for (int t0 = 0; t0 < T; t0 += S->pattn_q) {
            const int Tq = std::min(S->pattn_q, T - t0), qpos0 = pos0 + t0;
            PackP P{};
            P.first = mask_first(sp.att_mask, sp.att_window, qpos0); P.Lk = qpos0 + Tq - P.first; P.ring = O.ring;
            launch_next(ring_rows, (P.Lk + 255) / 256, 256, 0, st)(P.first, P.Lk, O.ring, S->d_rows);
            GemmP K = gp(cache, R, L.uk.p, R, S->kf, H * D, P.Lk, H * D, R);
            K.a_map = S->d_rows;
            linear(S, bf, HEPI_STORE, K, 1, st);
            GemmP Vp = gp(cache, R, L.uv.p, R, S->vf, H * V, P.Lk, H * V, R);
            Vp.a_map = S->d_rows;
            linear(S, bf, HEPI_STORE, Vp, 1, st);
            MK("att.kv_up");
            P.k = S->kf; P.v = S->vf; P.ldk = H * D; P.ldv = H * V; P.D0 = D;
            PattnP A{};
            A.q = S->b0 + (size_t)t0 * H * D; A.ldq = H * D; A.out = S->b3 + (size_t)t0 * H * V; A.ld_out = H * V; A.T = Tq; A.H = H; A.pos0 = qpos0; A.mask = sp.att_mask;
            A.span = sp.att_window; A.scale = sp.att_scale; A.alpha = 1.f;
            portion_attn(S, z, P, A, st);
            S->launches++;
          }
          MK("att.fused");
        } else
        for (int t0 = 0; t0 < T; t0 += kPrefillQ) {
          const int Tq = std::min(kPrefillQ, T - t0), qpos0 = pos0 + t0;
          const int first = mask_first(sp.att_mask, sp.att_window, qpos0), Lk = qpos0 + Tq - first;
          launch_next(ring_rows, (Lk + 255) / 256, 256, 0, st)(first, Lk, O.ring, S->d_rows);
          GemmP K = gp(cache, R, L.uk.p, R, S->kf, H * D, Lk, H * D, R);
          K.a_map = S->d_rows;
          linear(S, bf, HEPI_STORE, K, 1, st);
          GemmP Vp = gp(cache, R, L.uv.p, R, S->vf, H * V, Lk, H * V, R);
          Vp.a_map = S->d_rows;
          linear(S, bf, HEPI_STORE, Vp, 1, st);
          MK("att.kv_up");
          if (bf) launch_next(pack_keys_values<__nv_bfloat16>, Lk, 256, 0, st)(S->kf, S->vf, (__nv_bfloat16*)S->kb, (__nv_bfloat16*)S->vt, Lk, H, D, V);
          else launch_next(pack_keys_values<float>, Lk, 256, 0, st)(S->kf, S->vf, (float*)S->kb, (float*)S->vt, Lk, H, D, V);
          GemmP Sc = gp(S->b0 + (size_t)t0 * H * D, H * D, S->kb, D, S->sc, Lk, Tq, Lk, D);
          Sc.w_made = 1;
          Sc.sA = D; Sc.sW = (long long)Lk * D; Sc.sC = (long long)Tq * Lk; Sc.alpha = sp.att_scale;
          MK("att.pack");
          linear(S, bf, HEPI_STORE, Sc, H, st);
          MK("att.scores");
          launch_next(softmax_band, dim3((unsigned)Tq, (unsigned)H), 128, 0, st)(S->sc, Tq, Lk, Lk, first, qpos0, sp.att_mask, sp.att_window, 0, ScoreMods{});
          GemmP Ov = gp(S->sc, Lk, S->vt, Lk, S->b3 + (size_t)t0 * H * V, H * V, Tq, V, Lk);
          Ov.w_made = 1;
          Ov.sA = (long long)Tq * Lk; Ov.sW = (long long)V * Lk; Ov.sC = V;
          MK("att.softmax");
          linear(S, bf, HEPI_STORE, Ov, H, st);
          MK("att.pv");
          S->launches += 3;
        }
      } else {
        {  // absorbed query: qa[t][h][:] = W_uk[h]^T q[t][h][:]
          GemmP P = gp(S->b0, H * D, L.ukT.p, D, S->b2, H * R, T, R, D);
          P.sA = D; P.sW = (long long)R * D; P.sC = R;
          linear(S, bf, HEPI_STORE, P, H, st);
        }
        launch_latent_attn(S, S->b2, cache, S->b3, T, H, R, sp.att_mask, sp.att_window, O.ring, sp.att_scale, nullptr, st);
        {  // value up-projection per head: ov[t][h][:] = W_uv[h] o[t][h][:]
          GemmP P = gp(S->b3, H * R, L.uv.p, R, S->b0, H * V, T, V, R);
          P.sA = R; P.sW = (long long)V * R; P.sC = V;
          linear(S, bf, HEPI_STORE, P, H, st);
        }
      }
      MK("att.absorbed");
      GemmP P = gp(ov, H * V, L.o.p, H * V, sink.C, W, T, W, H * V);
      P.alpha = sink.alpha;
      linear(S, bf, sink.epi, P, 1, st);
      MK("att.o");
    }
    if (!post) hin = hff;
    if (post) {   // the mixer's result closes; the feed-forward (or, without one, the next layer's mixer) opens on the new stream
      if (small_post && sp.ff_kind != DSK_FF_NONE) { close_open(L.rg1, L.rg1_b, L.close1, L.canon2, ring_of(ri, 1)); hin = S->h; }
      else if (small_post && has_next) { close_open(L.rg1, L.rg1_b, L.close1, M->L[M->runs[ri + 1].layer].canon1, ring_of(ri + 1, 0)); h_ready = true; }
      else {
        close_post(L.rg1, L.rg1_b, L.close1, L.norm1_bias);
        if (sp.ff_kind != DSK_FF_NONE) hin = open_post(L.canon2, 1);
      }
      MK("norm");
    }
    if (sandwich) {   // x += norm1b(mixer output); the feed-forward then reads norm2 of the new x
      if (sp.ff_kind == DSK_FF_NONE) close_run(L.close1);
      else if (frms) {
        launch_rms_add_norm(T, W, st, S->y, nullptr, 0, nullptr, nullptr, L.close1, S->x, S->x, W, L.norm2, S->h, W, c.norm_eps, mult, mirror16(S, T));
        S->mirror = mirror16(S, T) ? S->h : nullptr;
        S->launches++;
      } else if (fuse) {
        launch_next(layer_norm_add_norm, T, 256, 0, st)(S->y, L.close1, S->x, nullptr, L.norm2, S->h, W, c.norm_eps, mult, mirror16(S, T));
        S->mirror = mirror16(S, T) ? S->h : nullptr;
        S->launches++;
      } else {
        norm_rows(c, S, S->y, L.close1, nullptr, S->x, T, 1, mult, st);
        norm_rows(c, S, S->x, L.norm2, nullptr, S->h, T, 0, 0.f, st);
      }
      MK("norm");
    }
    if (pre && sp.ff_kind != DSK_FF_NONE) {
      launch_next(rms_open, T, 256, 0, st)(S->x, nullptr, nullptr, L.norm2, S->h, W, c.norm_eps, mirror16(S, T));
      S->mirror = mirror16(S, T) ? S->h : nullptr;
      S->launches++;
      hin = S->h;
      MK("norm");
    }
    if (sp.ff_kind == DSK_FF_DENSE && sp.ff_act != DSK_ACT_XIELU) {
      const int ff = sp.ff_hidden;
      GemmP U = gp(hin, W, L.gate_d.p, W, S->b2, ff, T, ff, W);
      U.W2 = L.up.p; U.lim = sp.ff_limit;
      GemmP Dn = gp(S->b2, ff, L.down.p, ff, sink.C, W, T, W, ff);
      Dn.alpha = sink.alpha;
      const int act = sp.ff_act == DSK_ACT_GLU_CLAMPED ? HEPI_GLU : sp.ff_act == DSK_ACT_SWIGLU ? HEPI_SWIGLU : HEPI_GEGLU;
      hidden16(S, bf, act, U, sink.epi, Dn, S->hid16);
      linear(S, bf, act, U, 1, st);
      MK("ff.up");
      linear(S, bf, sink.epi, Dn, 1, st);
      MK("ff.down");
    } else if (sp.ff_kind == DSK_FF_DENSE) {
      const int ff = sp.ff_hidden;
      GemmP U = gp(hin, W, L.up.p, W, S->b2, ff, T, ff, W);
      U.bias = L.up_b; U.act_a = L.act_a; U.act_b = L.act_b;
      GemmP Dn = gp(S->b2, ff, L.down.p, ff, sink.C, W, T, W, ff);
      Dn.bias = L.down_b; Dn.alpha = sink.alpha;
      hidden16(S, bf, HEPI_XIELU, U, sink.epi, Dn, S->hid16);
      linear(S, bf, HEPI_XIELU, U, 1, st);
      MK("ff.up");
      linear(S, bf, sink.epi, Dn, 1, st);
      MK("ff.down");
    }
    if (sp.ff_kind == DSK_FF_MOE) {
      const int E = sp.ff_experts, top = sp.ff_top, ff = sp.ff_hidden, pairs = T * top;
      const bool shared = sp.ff_shared > 0;
      const int ffs = sp.ff_shared, ldz = E + (shared ? 1 : 0), groups = std::max(1, sp.ff_groups);
      GemmP Rt = gp(hin, W, L.router, W, S->b0, ldz, T, ldz, W);   // router: fp32 weights in every mode (and the shared expert's weight)
      Rt.bias = sp.ff_router == DSK_ROUTER_TOP_SOFTMAX ? L.router_b : nullptr;
      linear(S, false, HEPI_STORE, Rt, 1, st);
      launch_next(moe_route, T, 128, (size_t)(2 * E + top + groups) * 4, st)(S->b0, ldz, sp.ff_router == DSK_ROUTER_SIGMOID ? L.correction : nullptr, E, top, sp.ff_router_scale,
                                                                    S->d_idx, S->wgt, sp.ff_router == DSK_ROUTER_SOFTMAX_GROUPS ? 2 : sp.ff_router == DSK_ROUTER_TOP_SOFTMAX ? 1 : 0,
                                                                    groups, sp.ff_groups > 0 ? sp.ff_groups_keep : 1, shared ? S->wsh : nullptr);
      S->launches++;
      MK("moe.router");
      const bool relu2 = sp.ff_expert == DSK_EXPERT_RELU2;   // one up matrix per expert instead of a gated pair
      const int epi_up = relu2 ? HEPI_RELU2 : sp.ff_expert == DSK_EXPERT_SWIGLU ? HEPI_SWIGLU : HEPI_GLU;
      GemmP G = gp(hin, W, relu2 ? L.up_s.p : L.gate_s.p, W, S->b2, ff, pairs, ff, W);
      G.W2 = relu2 ? nullptr : L.up_s.p; G.sW = (long long)ff * W; G.lim = sp.ff_limit;
      GemmP Dn = gp(S->b2, ff, L.down_s.p, ff, S->b3, W, pairs, W, ff);
      Dn.sW = (long long)ff * W;
      float *hsh = S->b2 + (size_t)pairs * ff, *ysh = S->b3 + (size_t)pairs * W;   // the shared expert's hidden rows and outputs, behind the routed ones'
      if (T <= 4) {
        G.z_expert = S->d_idx; G.z_adiv = top; Dn.z_expert = S->d_idx; Dn.z_adiv = 1;
        if (shared) {   // its rows ride in the same launches
          G.z_shared = pairs; G.n_shared = T; G.sN = ffs; G.sK = W; G.s_lda = W; G.s_ldc = ffs; G.sW1 = L.gate_sh.p; G.sW2 = L.up_sh.p; G.As = hin; G.Cs = hsh;
          Dn.z_shared = pairs; Dn.n_shared = T; Dn.sN = W; Dn.sK = ffs; Dn.s_lda = ffs; Dn.s_ldc = W; Dn.sW1 = L.down_sh.p; Dn.As = hsh; Dn.Cs = ysh;
        }
        linear(S, bf, epi_up, G, pairs + (shared ? T : 0), st);
        MK("moe.glu");
        linear(S, bf, HEPI_STORE, Dn, pairs + (shared ? T : 0), st);
        MK("moe.down");
      } else {
        constexpr int bm = 128;   // rows per tile of the product kernels that follow (gemm_tc5, gemm_mma, gemm_split)
        launch_next(moe_plan, 1, 1024, (size_t)3 * E * 4, st)(S->d_idx, pairs, E, bm, S->d_perm, S->d_tiles, S->d_ntiles);
        S->launches++;
        G.tiles = S->d_tiles; G.n_tiles = S->d_ntiles; G.a_map = S->d_perm; G.a_div = top; G.c_map = S->d_perm;
        Dn.tiles = S->d_tiles; Dn.n_tiles = S->d_ntiles; Dn.a_map = S->d_perm; Dn.a_div = 1; Dn.c_map = S->d_perm;
        const int cap = std::min(S->max_tiles, pairs / bm + E + 1);
        G.n_expert = Dn.n_expert = E;
        hidden16(S, bf, epi_up, G, HEPI_STORE, Dn, S->hid16);
        MK("moe.plan");
        linear(S, bf, epi_up, G, 1, st, cap);
        MK("moe.glu");
        linear(S, bf, HEPI_STORE, Dn, 1, st, cap);
        MK("moe.down");
        if (shared) {
          GemmP Us = gp(hin, W, L.gate_sh.p, W, hsh, ffs, T, ffs, W);
          Us.W2 = L.up_sh.p; Us.lim = sp.ff_limit;
          GemmP Ds = gp(hsh, ffs, L.down_sh.p, ffs, ysh, W, T, W, ffs);
          hidden16(S, bf, epi_up, Us, HEPI_STORE, Ds, S->hid16 + (size_t)pairs * ff);
          linear(S, bf, epi_up, Us, 1, st);
          linear(S, bf, HEPI_STORE, Ds, 1, st);
          MK("moe.shared");
        }
      }
      if (combine_in_norm) {   // x += ln(sum_k w_k y_k): the weighted sum of the experts' outputs is taken by the closing layer norm as it reads its row
        launch_next(layer_norm, T, 256, 0, st)(S->b3, W, L.close2, L.norm2_bias, S->x, W, W, c.norm_eps, 1, mult, S->wgt, top, mirror16(S, T));
        S->mirror = mirror16(S, T) ? S->x : nullptr;
        S->launches++;
      } else if (!frms) {   // (sandwich blocks of RMS norms combine as they close)
        if (S->mirror == sink.C) S->mirror = nullptr;
        launch_next(moe_combine, dim3((unsigned)T, (unsigned)((W + (W % 4 ? 255 : 1023)) / (W % 4 ? 256 : 1024))), 256, 0, st)(sink.C, W, S->b3, S->wgt, top, W, sink.alpha, sink.epi == HEPI_ADD ? 1 : 0, shared ? ysh : nullptr, S->wsh);
        S->launches++;
      }
      MK("moe.combine");
    }
    if (sandwich && sp.ff_kind != DSK_FF_NONE) {
      close_run(L.close2, frms && sp.ff_kind == DSK_FF_MOE ? sp.ff_top : 0);
      MK("norm");
    }
    if (post && sp.ff_kind != DSK_FF_NONE && !combine_in_norm) {
      if (small_post && has_next) { close_open(L.rg2, L.rg2_b, L.close2, M->L[M->runs[ri + 1].layer].canon1, ring_of(ri + 1, 0)); h_ready = true; }
      else close_post(L.rg2, L.rg2_b, L.close2, L.norm2_bias);
      MK("norm");
    }
    if (c.side_dim > 0) {
      const int sd = c.side_dim;
      GemmP P = gp(S->x, W, L.sgate.p, W, S->b1, sd, T, sd, W);
      P.aux = M->side_embed.p; P.aux_row = S->d_tok; P.aux_ld = sd * c.n_layers; P.aux_off = li * sd;
      linear(S, bf, HEPI_GELU_MUL, P, 1, st);
      linear(S, bf, HEPI_STORE, gp(S->b1, sd, L.sproj.p, sd, S->h, W, T, W, sd), 1, st);
      // decode-sized steps of post-norm blocks: the normed addition and the next layer's token shift in one launch over 128-channel CTAs
      if (post && c.canon_taps <= 0 && T <= kCloseOpenTokens && !trace) {
        const bool next_shift = c.token_shift && has_next;
        S->mirror = nullptr;
        launch_next(rms_add_shift_small, (W + 127) / 128, 128, 0, st)(S->h, L.snorm, mult, c.norm_eps, S->x, W, next_shift ? M->L[M->runs[ri + 1].layer].shift : nullptr,
                                                             next_shift ? S->L[ri + 1].shift : nullptr, S->hs, T, W, S->d_ctl);
        hs_ready = next_shift;
      } else {
        if (S->mirror == S->x) S->mirror = nullptr;
        launch_next(group_rmsnorm<float>, T, 256, 0, st)(S->h, W, L.snorm, S->x, W, W, 1, c.norm_eps, 1, mult, nullptr, 0, nullptr, 0, nullptr);
      }
      S->launches++;
      MK("side");
    }
    if (trace) CKL(cudaMemcpyAsync(trace + ri * (size_t)T * W, S->x, (size_t)T * W * 4, cudaMemcpyDeviceToDevice, st));
  }
  if (n_want > 0) {   // final norm of every row, LM head on the first group of wanted rows (enqueue_head does the others)
    if (pre) { launch_next(rms_open, T, 256, 0, st)(S->x, nullptr, nullptr, M->final_norm, S->h, W, c.norm_eps, mirror16(S, T)); S->mirror = mirror16(S, T) ? S->h : nullptr; S->launches++; }
    else if (!h_ready) norm_rows(c, S, S->x, M->final_norm, M->final_norm_b, S->h, T, 0, 0.f, st);
    enqueue_head(m, s, 0, std::min(n_want, S->head_rows), pos0 < 0 ? s->logits : S->logits, st);   // a captured step leaves its one row in the state
    MK("head");
  }
  CKL(cudaGetLastError());
  return 0;
}

// arg-max of the state's logits into Ctrl::argmax_key, which is 0 ahead of it; a few CTAs: one takes 13 us for 100 k logits, mostly waiting
static void launch_argmax(dsk_state* s, int vocab) {
  launch_next(argmax_row, (unsigned)std::max(1, std::min(vocab / 4096, 32)), 256, 0, s->stream)(s->logits, vocab, s->ctrl);
}

// tokens [n] at positions pos0.. of the state's sequence; want: ascending indices into tokens whose logits go to host_logits
// [n_want][vocab]; host_layers (nullable): [layers][n][width] residual stream after every layer.
static int run_chunks(dsk_model* m, dsk_state* s, const int32_t* tokens, int n, int pos0, const int32_t* want, int n_want, float* host_logits, float* host_layers) {
  Model* M = m->hy;
  State* S = s->hy;
  const dsk_hybrid_config& c = M->c;
  if (n <= 0) return fail(-4, "empty chunk");
  if (pos0 == 0) { if (state_reset(s)) return -2; }
  else if (pos0 < 0 || pos0 != S->next_pos) return fail(-4, "chunk starts at position %d but the state's sequence is at %d (recurrent state cannot be rewound; position 0 starts a new sequence)", pos0, S->next_pos);
  for (int i = 0; i < n; i++) if (tokens[i] < 0 || tokens[i] >= c.vocab_size) return fail(-4, "token %d out of range", tokens[i]);
  for (int i = 0; i < n_want; i++) if (want[i] < 0 || want[i] >= n || (i && want[i] <= want[i - 1])) return fail(-4, "wanted rows must be ascending indices into the chunk");
  for (const HLayer& L : M->L)   // a ring cache shortened to max_seq_len holds no position beyond it
    if (L.owner >= 0 && M->L[L.owner].ring < L.sp.att_window - 1 + S->chunk && pos0 + n > M->L[L.owner].ring)
      return fail(-4, "position %d does not fit the attention cache (max_seq_len %d)", pos0 + n - 1, c.max_seq_len);
  float* d_trace = nullptr;
  int wi = 0;
  for (int o = 0; o < n; o += S->chunk) {
    const int T = std::min(S->chunk, n - o);
    // one copy brings the chunk in (position, tokens and rows apart, behind a wait for the chunk ahead, kept the GPU idle for some 15 us a chunk)
    const int slot = (o / S->chunk) & 1;
    int *in = S->h_in[slot], *in_want = in + 4 + S->chunk;
    CK(cudaEventSynchronize(S->in_ev[slot]));   // the copy that had this staging buffer before
    in[0] = pos0 + o;
    memcpy(in + 4, tokens + o, (size_t)T * 4);
    int nw = 0;
    while (wi + nw < n_want && want[wi + nw] < o + T) { in_want[nw] = want[wi + nw] - o; nw++; }
    const bool apart = S->chunk - T > 4096;     // (rows far behind the tokens of a short chunk)
    CK(cudaMemcpyAsync(S->d_ctl, in, (size_t)(nw && !apart ? 4 + S->chunk + nw : 4 + T) * 4, cudaMemcpyHostToDevice, s->stream));
    if (nw && apart) CK(cudaMemcpyAsync(S->d_want, in_want, (size_t)nw * 4, cudaMemcpyHostToDevice, s->stream));
    CK(cudaEventRecord(S->in_ev[slot], s->stream));
    if (host_layers) { CK(cudaMalloc((void**)&d_trace, M->runs.size() * (size_t)T * c.dim * 4)); }
    if (enqueue_chunk(m, s, T, nw, d_trace, s->stream, pos0 + o)) { if (d_trace) cudaFree(d_trace); return -2; }
    for (int g0 = 0; g0 < nw; g0 += S->head_rows) {   // the LM head in groups of head_rows wanted rows
      const int gn = std::min(S->head_rows, nw - g0);
      if (g0 > 0) enqueue_head(m, s, g0, gn, S->logits, s->stream);
      if (g0 + gn == nw) {   // the last wanted row stays in the state for the samplers
        CK(cudaMemcpyAsync(s->logits, S->logits + (size_t)(gn - 1) * c.vocab_size, (size_t)c.vocab_size * 4, cudaMemcpyDeviceToDevice, s->stream));
        CK(cudaMemsetAsync(&s->ctrl->argmax_key, 0, sizeof(s->ctrl->argmax_key), s->stream));
        launch_argmax(s, c.vocab_size);
        CK(cudaMemcpyAsync(s->h_ctrl, s->ctrl, sizeof(Ctrl), cudaMemcpyDeviceToHost, s->stream));
      }
      if (host_logits && copy_to_host(s, host_logits + (size_t)(wi + g0) * c.vocab_size, S->logits, (size_t)gn * c.vocab_size * 4, false)) return -2;   // (the call waits at its end)
    }
    timeline_report(S, T);
    if (host_layers) {
      CK(cudaStreamSynchronize(s->stream));
      for (size_t l = 0; l < M->runs.size(); l++)
        CK(cudaMemcpy(host_layers + ((size_t)l * n + o) * c.dim, d_trace + (size_t)l * T * c.dim, (size_t)T * c.dim * 4, cudaMemcpyDeviceToHost));
      cudaFree(d_trace); d_trace = nullptr;
    }
    wi += nw;
  }
  CK(cudaStreamSynchronize(s->stream));
  CK(cudaGetLastError());
  // (a step that lacks a product has gone into caches and recurrences: the sequence is not to be continued)
  if (*(volatile int*)S->h_err) { const int e = *S->h_err; *S->h_err = 0; S->next_pos = -1; return fail(-2, e == 2 ? "a product's tensor map was refused" : "a wait inside a matrix product gave up"); }
  S->next_pos = pos0 + n;
  s->last_pos = pos0 + n - 1;
  s->have_logits = n_want > 0 && want[n_want - 1] == n - 1;
  return 0;
}

static int forward_chunk(dsk_model* m, dsk_state* s, const int32_t* tokens, int n, int pos0, const int32_t* want, int n_want, float* host_logits, float* host_layers) {
  const int rc = run_chunks(m, s, tokens, n, pos0, want, n_want, host_logits, host_layers);
  if (rc) cudaStreamSynchronize(s->stream);   // nothing is on its way into the caller's memory, nor out of the staging buffers
  return rc;
}

// greedy loop on the device: arg-max of the logits in the state -> next token -> one-token chunk -> logits, n_steps times,
// without a host round trip.  The step is captured once per state as a CUDA graph (positions advance in device memory).
static int decode_greedy(dsk_model* m, dsk_state* s, int start_pos, int n_steps, int32_t* out_tokens, float* elapsed_ms) {
  Model* M = m->hy;
  State* S = s->hy;
  const dsk_hybrid_config& c = M->c;
  if (start_pos < 0 || start_pos != S->next_pos) return fail(-4, "dsk_decode_greedy: start_pos %d must follow the state's sequence (at %d)", start_pos, S->next_pos);
  const int one = 0;
  CK(cudaMemcpyAsync(S->d_want, &one, 4, cudaMemcpyHostToDevice, s->stream));
  launch_next(set_ctl, 1, 1, 0, s->stream)(S->d_ctl, start_pos - 1);   // (greedy_feed moves on)
  CK(cudaMemsetAsync(s->step, 0, sizeof(int), s->stream));
  CK(cudaStreamSynchronize(s->stream));
  if (!S->step_graph) {
    cudaGraph_t g = nullptr;
    CK(cudaStreamBeginCapture(s->stream, cudaStreamCaptureModeThreadLocal));
    launch_next(greedy_feed, 1, 1, 0, s->stream)(s->ctrl, S->d_tok, s->token_log, s->step, S->d_ctl);
    int rc = enqueue_chunk(m, s, 1, 1, nullptr, s->stream);
    launch_argmax(s, c.vocab_size);
    cudaError_t e = cudaStreamEndCapture(s->stream, &g);
    if (rc || e != cudaSuccess) return fail(-2, "capturing the decode step failed: %s", cudaGetErrorString(e));
    CK(cudaGraphInstantiate(&S->step_graph, g, 0));
    cudaGraphDestroy(g);
  }
  CK(cudaEventRecord(s->ev0, s->stream));
  for (int i = 0; i < n_steps; i++) CK(cudaGraphLaunch(S->step_graph, s->stream));
  CK(cudaEventRecord(s->ev1, s->stream));
  CK(cudaStreamSynchronize(s->stream));
  if (elapsed_ms) CK(cudaEventElapsedTime(elapsed_ms, s->ev0, s->ev1));
  if (out_tokens) CK(cudaMemcpy(out_tokens, s->token_log, (size_t)n_steps * 4, cudaMemcpyDeviceToHost));
  S->next_pos = start_pos + n_steps;
  s->last_pos = S->next_pos - 1;
  s->have_logits = true;
  return 0;
}

}  // namespace hyb

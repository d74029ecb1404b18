// dsk_decode_host.cuh — plans and launches the token chain of dsk_decode.cuh for one dsk_state.  Included by dsk_engine.cu.
#pragma once

namespace dk {

enum Kind { EMBED, GEMV, ATTN };
struct Launch {
  Kind kind;
  int layer, grid, smem, at;   // at: index into the plan's parameters of that kind
  int form;                    // 0, 1: kDkWarpsA, kDkWarpsB warps
  const char* name;
  DkLists lists;
};
// Which token's graph: fed by the host with / without logits, fed by the arg-max.
enum { HOST_LOGITS = 0, HOST_HYDRATE = 1, GREEDY = 2 };

struct Plan {
  int quant = 0;
  std::vector<Launch> L;
  std::vector<DkGemv> gemv;
  DkGemv* told = nullptr;                // the same on the device
  unsigned char* staged = nullptr;       // a feed-forward's staged input, for the launch of its routed experts
  std::vector<DkAttn> attn;
  DkEmbed embed{};
  cudaGraphExec_t graph[3] = {nullptr, nullptr, nullptr};
  bool ran[3] = {false, false, false};   // a variant is captured when it comes a second time: its first pass is plain launches
  ~Plan() {
    for (cudaGraphExec_t g : graph) if (g) cudaGraphExecDestroy(g);
    cudaFree(told);
    cudaFree(staged);
  }
};

static constexpr int kSmemLimit = 200 * 1024;
// dynamic shared memory of the two forms: together within an SM's 228 KB, the second not twice; rings are as deep as that allows.  A dk_gemv has kSmemFixed beside it
// (its static variables and the kilobyte that a CTA costs).  A launch whose inputs and shallowest rings take more than kSmemA comes to its SMs when the one ahead has gone.
static constexpr int kSmemFixed = 9344 + 1024;
static constexpr int kSmemB = 108 * 1024, kSmemA = 228 * 1024 - kSmemB - 2 * kSmemFixed, kSmemAttnB = 114 * 1024;
static_assert(sizeof(DkGemv) + (kDkSegs + 1) * sizeof(DkRun) + 3 * 256 * 2 + 32 * 4 + sizeof(DkRouteSmem) + 8 + 1024 <= kSmemFixed, "dk_gemv's static variables");
static_assert(2 * (kSmemB + kSmemFixed) > 228 * 1024 && 2 * (kSmemAttnB + 1024) > 228 * 1024 && kSmemA + kSmemAttnB + kSmemFixed + 2048 <= 228 * 1024, "two forms beside one another, the second not twice");

static int slot_bytes(int q) { return q == DSK_Q2_K ? DkTraits<Q_Q2K>::slot : DkTraits<Q_F32>::slot; }

// `count` matrices as the file has them -> tiles
template <int Q>
static void tile_q(const unsigned char* src, uint8_t* dst, int rows, int cols, int count, cudaStream_t st) {
  const long long tiles = (long long)cdiv(rows, DkTraits<Q>::rows) * count, units = tiles * dk_units(Q, cols);
  if (units == 0) return;
  if constexpr (DkTraits<Q>::kq)
    dk_tile_kq<Q><<<(unsigned)std::min<long long>(tiles * cdiv(cols, 2048), 1 << 16), 256, 0, st>>>(src, dst, rows, cols, tiles, disk_row_bytes(Q, cols) * rows * count);
  else
    dk_tile_kernel<Q><<<(unsigned)std::min<long long>((units + 31) / 32, 1 << 16), 256, 0, st>>>(src, dst, rows, cols, units);
}
static int tile(int quant, const unsigned char* src, uint8_t* dst, int rows, int cols, int count, cudaStream_t st, bool wait) {
  switch (quant) {
    case DSK_F32: tile_q<Q_F32>(src, dst, rows, cols, count, st); break;
    case DSK_F16: tile_q<Q_F16>(src, dst, rows, cols, count, st); break;
    case DSK_F8E5M2: tile_q<Q_F8>(src, dst, rows, cols, count, st); break;
    case DSK_Q2_K: tile_q<Q_Q2K>(src, dst, rows, cols, count, st); break;
    default: tile_q<Q_Q3K>(src, dst, rows, cols, count, st); break;
  }
  CK(cudaGetLastError());
  if (wait) CK(cudaDeviceSynchronize());
  return 0;
}
// the router: tiles of its own in a quantised model
static size_t router_bytes(const dsk_config& c) {
  const int E = c.n_routed_experts;
  return c.quant == DSK_F32 ? dk_matrix_bytes(DSK_F32, E, c.dim) : (size_t)cdiv(E, kDkF32Rows) * cdiv(c.dim, kDkF32Cols) * kDkF32Unit;
}
static int tile_router(const dsk_config& c, const float* src, float* dst, cudaStream_t st, bool wait) {
  const int E = c.n_routed_experts, n = c.dim;
  if (c.quant == DSK_F32) return tile(DSK_F32, (const unsigned char*)src, (uint8_t*)dst, E, n, 1, st, wait);
  const int units = (int)(router_bytes(c) / kDkF32Unit);
  if (units > 0) dk_tile_router<<<(unsigned)((units + 7) / 8), 256, 0, st>>>(src, (unsigned char*)dst, E, n, units);
  CK(cudaGetLastError());
  if (wait) CK(cudaDeviceSynchronize());
  return 0;
}

// Whether the kernels take a model of these shapes
static bool takes(const dsk_config& c) {
  if (c.use_mla) return false;
  const int hd = c.qk_nope_head_dim + c.qk_rope_head_dim, sh = c.n_shared_experts * c.moe_intermediate_size, att = c.n_heads * c.v_head_dim;
  if ((c.quant == DSK_Q2_K || c.quant == DSK_Q3_K) && (c.dim > 8192 || c.q_lora_rank > 8192 || c.kv_lora_rank > 8192)) return false;   // (one pass of the norm)
  if (hd % 8 || c.v_head_dim % 8 || c.v_head_dim > 8 * 32 * kDkWarpsB || hd > 4096) return false;
  const bool moe = c.n_routed_experts > 0 && c.first_k_dense_replace < c.n_layers;
  const int mi = moe ? c.moe_intermediate_size : 0, K = moe ? c.n_active_routed : 0;
  const int unit = c.quant == DSK_F8E5M2 ? 64 : (c.quant == DSK_Q2_K || c.quant == DSK_Q3_K) ? 256 : c.quant == DSK_F16 ? 16 : 4;   // columns a row is made of
  for (int n : {c.dim, c.q_lora_rank, c.kv_lora_rank, att, mi, moe ? sh : 0, c.hidden_dim}) if (n % unit) return false;
  auto pow2 = [](int v) { return v > 0 && (v & (v - 1)) == 0; };
  if (c.quant == DSK_F8E5M2 && (c.bs1 < 64 || !pow2(c.bs1) || !pow2(c.bs0))) return false;   // a group of 64 columns has one scale
  if (c.hidden_dim <= 0 && !(moe && c.first_k_dense_replace <= 0)) return false;
  if (moe && (c.n_active_routed < 1 || c.n_active_routed > 8 || mi <= 0)) return false;
  for (int n : {c.dim, c.q_lora_rank, c.kv_lora_rank, att, mi, moe ? sh : 0, c.hidden_dim}) if (dk_units(c.quant, n) > 255) return false;
  if (dk_whole(DSK_F32, c.dim) / kDkF32Cols > 255) return false;
  auto bytes = [&](int n, int times) { return dk_x_bytes(c.quant, times * dk_whole(c.quant, n)); };
  const int most = std::max(std::max(bytes(c.dim, 1) + dk_whole(DSK_F32, c.dim) * 4, bytes(att, 1)),
                            std::max(bytes(c.q_lora_rank, 1) + bytes(c.kv_lora_rank, 1), std::max(bytes(mi, K) + bytes(moe ? sh : 0, 1), bytes(c.hidden_dim, 1))));
  return most <= 96 * 1024;   // (whether sums and rings fit beside the staged inputs, arrange() says launch by launch)
}

// A launch in the making: matrices in order, each with the row tiles it has
struct Draft {
  DkGemv g{};
  std::vector<int> tiles;   // row tiles of a matrix
  bool even = false;        // every matrix is cut at the same rows (down projection)
};
// what a shape's plan consists of
struct Arranged {
  std::vector<DkRun> runs;
  std::vector<DkWarp> warps;
  std::vector<DkItem> items;
  std::vector<int> first, even, kind;   // kind: of a matrix
  std::vector<unsigned short> units;
  int max_runs, part_at, raw_at, ring_at, depth, smem;
  DkInput in[2];
  DkLists lists;                        // the above on the device (then they are empty here)
};
// The plans of a model, worked out and placed when it is made (layers are alike: one a shape); its states only read them
struct Shapes {
  std::map<std::vector<int>, Arranged> of;
  void* mem = nullptr;
  ~Shapes() { cudaFree(mem); }
};

// Row tiles to CTAs: by bytes, a tile to the CTA in whose share of the whole it begins; a pair's halves alike.
static void deal(const Draft& D, int q, int G, std::vector<std::vector<DkRun>>* out) {
  const DkGemv& g = D.g;
  long long total = 0;
  std::vector<long long> before(g.nsegs), cost(g.nsegs);
  for (int j = 0; j < g.nsegs; j++) {
    const long long b = (long long)g.seg[j].nb * (g.seg[j].f32 && q != DSK_F32 ? kDkF32Unit : dk_unit_bytes(q));
    cost[j] = b; before[j] = total;
    if (j > 0 && g.seg[j - 1].pair) { before[j] = before[j - 1]; cost[j] = cost[j - 1]; }   // (as its other half)
    else { if (g.seg[j].pair) cost[j] = 2 * b; total += cost[j] * D.tiles[j]; }
  }
  out->assign(G, {});
  for (int c = 0; c < G; c++) {
    auto& R = (*out)[c];
    for (int j = 0; j < g.nsegs; j++) {
      auto at = [&](int cc) {
        if (D.even) return (int)((long long)D.tiles[j] * cc / G);
        const long long lim = (total * cc + G - 1) / G - before[j];
        return (int)std::min<long long>(D.tiles[j], lim <= 0 ? 0 : (lim + cost[j] - 1) / cost[j]);
      };
      const int a = at(c), b = at(c + 1);
      if (a >= b) continue;
      R.push_back(DkRun{j, a, b - a, 0});
    }
  }
}
// The places of a tile of nb units cut into `pieces`: what DkLists::units holds; false: a piece would have none.  K-quants: branches of the tree of classes; the
// router: a class a piece; else equal lengths
static bool places(int quant, bool router, int nb, int pieces, unsigned short* out) {
  const bool pairs = dk_kq(quant) && !router, classes = pairs || router;
  if (pieces < 1 || pieces > nb || (pairs && (pieces > 8 || (pieces & (pieces - 1)))) || (router && pieces != std::min(8, nb))) return false;
  int k = 0;
  if (!classes) {
    for (int i = 0; i < pieces; i++) {
      const int end = nb * (i + 1) / pieces;
      for (; k < end; k++) out[k] = (unsigned short)(k | (k + 1 == end ? kDkPieceEnds : 0));
    }
    return true;
  }
  const int per = 8 / (pairs ? pieces : 8);   // classes of a piece
  for (int p = 0; p < 8 / per; p++) {
    int last = -1;
    for (int i = 0; i < per; i++) {
      const int c = dk_class(pairs, p * per + i), n = dk_class_units(nb, c);
      if (n <= 0) { if (last >= 0) out[last] += 1 << 12; continue; }
      for (int j = 0; j < n; j++, k++) out[k] = (unsigned short)((c + 8 * j) | (j + 1 == n ? kDkClassEnds | (i << 9) : 0));
      last = k - 1;
    }
    if (last < 0) { if (router) continue; return false; }
    out[last] |= kDkPieceEnds;
  }
  return true;
}
// The units [u, v) of a CTA's stream to each of its NW warps, by whole pieces (first units of them and of the end): a piece to the warp in whose share its middle lies
static void share(const std::vector<int>& piece, int NW, std::vector<int>* first_piece) {
  const int n = (int)piece.size() - 1, total = piece[n], busy = std::min(NW, std::max(1, n));
  first_piece->assign(NW + 1, n);
  int p = 0;
  for (int w = 0; w < busy; w++) {
    (*first_piece)[w] = p;
    while (p < n && ((long long)piece[p] + piece[p + 1]) * busy < 2ll * (w + 1) * total) p++;
    if (w + 1 == busy) p = n;
  }
}
// The plan of a shape, and shared memory: staged inputs | sums of pieces, ahead of them x as it comes | rings as deep as leaves room for a CTA of the other form.
// false: it does not fit
static bool arrange(const Draft& D, int q, int G, int form, Arranged* out) {
  const DkGemv& g = D.g;
  const int NW = form ? kDkWarpsB : kDkWarpsA, TR = dk_rows(q), PS = dk_part(q);
  std::vector<std::vector<DkRun>> runs;
  Arranged& L = *out;
  deal(D, q, G, &runs);
  L.max_runs = 1;
  for (auto& r : runs) L.max_runs = std::max(L.max_runs, (int)r.size());
  // kinds of matrices (columns, router), and for each the ways to cut a tile into pieces
  std::vector<std::pair<int, int>> kinds;
  L.kind.clear();
  for (int j = 0; j < g.nsegs; j++) {
    const std::pair<int, int> k{g.seg[j].nb, g.seg[j].f32 && q != DSK_F32};
    auto it = std::find(kinds.begin(), kinds.end(), k);
    L.kind.push_back((int)(it - kinds.begin()));
    if (it == kinds.end()) kinds.push_back(k);
  }
  if (kinds.size() > 3) return false;
  struct Cut { int pieces = 1; std::vector<unsigned short> units; std::vector<int> len; };   // len: units of its pieces
  std::vector<Cut> cuts[3];
  const int nk = (int)kinds.size();
  for (int k = 0; k < nk; k++) {
    std::vector<int> ways{1, 2, 3, 4, 5, 6, 8, 11, 12, 16};
    if (kinds[k].second) ways = {std::min(8, kinds[k].first)};   // (the router has no choice)
    for (int n : ways) {
      Cut c;
      c.pieces = n; c.units.assign(256, 0);
      if (!places(q, kinds[k].second, kinds[k].first, n, c.units.data())) continue;
      for (int u = 0, len = 1; u < kinds[k].first; u++, len++) if (c.units[u] & kDkPieceEnds) { c.len.push_back(len); len = 0; }
      cuts[k].push_back(c);
    }
  }
  for (int k = nk; k < 3; k++) cuts[k].resize(1);
  std::vector<std::vector<int>> shapes;   // of CTAs: (kind, tiles) in order
  for (auto& R : runs) {
    std::vector<int> v;
    for (auto& r : R) { v.push_back(L.kind[r.seg]); v.push_back(r.tiles); }
    if (std::find(shapes.begin(), shapes.end(), v) == shapes.end()) shapes.push_back(v);
  }
  // the choice with the least loaded busiest warp; a piece costs about a unit more than it has
  const Cut* pick[3] = {};
  long long best = 1ll << 60;
  int most_pieces = 0;
  std::vector<int> ends, fp;
  auto add_tiles = [&](const Cut& c, int tiles) { for (int t = 0; t < tiles; t++) for (int n : c.len) ends.push_back(ends.back() + n); };
  for (const Cut& a : cuts[0])
    for (const Cut& b : cuts[1])
      for (const Cut& d : cuts[2]) {
        const Cut* c[3] = {&a, &b, &d};
        long long worst = 0;
        int pieces = 0;
        for (auto& v : shapes) {
          ends.assign(1, 0);
          for (size_t i = 0; i < v.size(); i += 2) add_tiles(*c[v[i]], v[i + 1]);
          pieces = std::max(pieces, (int)ends.size() - 1);
          share(ends, NW, &fp);
          for (int w = 0; w < NW; w++) worst = std::max(worst, (long long)(ends[fp[w + 1]] - ends[fp[w]]) * 2 + (fp[w + 1] - fp[w]));
        }
        if (pieces * PS * 4 > 32 * 1024 && best < 1ll << 60) continue;   // (the first choice, uncut tiles, is there for shapes that need more)
        if (worst < best) { best = worst; most_pieces = pieces; std::copy(c, c + 3, pick); }
      }
  if (best == 1ll << 60 || most_pieces * PS > 65535) return false;   // (DkItem::parts)
  L.units.assign(3 * 256, 0);
  for (int k = 0; k < nk; k++) std::copy(pick[k]->units.begin(), pick[k]->units.end(), L.units.begin() + 256 * k);
  L.runs.assign((size_t)G * L.max_runs, DkRun{-1, 0, 0, 0});
  L.warps.assign((size_t)G * NW, DkWarp{});
  size_t rows = 0;
  for (int j = 0; j < g.nsegs; j++) rows += (size_t)D.tiles[j] * TR;
  L.items.reserve(rows);
  for (int cta = 0; cta < G; cta++) {
    auto& R = runs[cta];
    std::vector<int> start(R.size() + 1, 0), piece0(R.size() + 1, 0);   // first units, first pieces of the runs
    ends.assign(1, 0);
    for (size_t i = 0; i < R.size(); i++) {
      add_tiles(*pick[L.kind[R[i].seg]], R[i].tiles);
      start[i + 1] = start[i] + R[i].tiles * g.seg[R[i].seg].nb; piece0[i + 1] = (int)ends.size() - 1;
      R[i].piece = piece0[i];
    }
    std::copy(R.begin(), R.end(), L.runs.begin() + (size_t)cta * L.max_runs);
    share(ends, NW, &fp);
    for (int w = 0; w < NW; w++) {
      DkWarp& W = L.warps[(size_t)cta * NW + w];
      W.u0 = ends[fp[w]]; W.u1 = ends[fp[w + 1]]; W.piece = fp[w];
      if (W.u0 >= W.u1) { W.u0 = W.u1 = 0; continue; }
      while (W.u0 >= start[W.run + 1]) W.run++;
      const int nb = g.seg[R[W.run].seg].nb;
      W.start = start[W.run]; W.tile = (W.u0 - W.start) / nb; W.kb = W.u0 - W.start - W.tile * nb;
    }
    L.first.push_back((int)L.items.size());
    for (size_t i = 0; i < R.size(); i++) {
      const DkSeg& S = g.seg[R[i].seg];
      const bool router = S.f32 && q != DSK_F32;
      const int tr = router ? kDkF32Rows : TR, n = pick[L.kind[R[i].seg]]->pieces;
      for (int t = 0; t < R[i].tiles; t++)
        for (int r = 0; r < tr; r++) {   // a row's place in the sums of its tile's first piece
          const int place = t * n * PS + (dk_kq(q) && !router ? (r >> 3) * 32 + (r & 7) * 4 : r);
          DkItem I{};
          I.r = (R[i].tile0 + t) * tr + r;
          I.seg = (short)(I.r < S.rows ? R[i].seg : -1);
          I.n = (short)n;
          I.parts = (unsigned short)(piece0[i] * PS + place);
          if (S.pair) I.parts2 = (unsigned short)(piece0[i + 1] * PS + place);
          L.items.push_back(I);
        }
      if (S.pair) i++;
    }
  }
  L.first.push_back((int)L.items.size());
  if (D.even) for (int cta = 0; cta <= G; cta++) L.even.push_back((int)((long long)D.tiles[0] * cta / G));
  int off = 0;
  for (int i = 0; i < g.nin; i++) {
    DkInput& I = L.in[i] = g.in[i];
    I.at = off; I.f32_at = -1;
    I.stride = I.seg ? dk_whole(q, I.seg) : 0;
    I.len = I.seg ? I.n / I.seg * I.stride : dk_whole(q, I.n);
    if (I.stride == I.seg) I.seg = I.stride = 0;
    I.bytes = dk_x_bytes(q, I.len);
    off += I.bytes;
  }
  for (int j = 0; j < g.nsegs; j++)
    if (g.seg[j].f32 && (q == DSK_F8E5M2 || kq_quant(q)) && L.in[0].f32_at < 0) { L.in[0].f32_at = off; off += dk_whole(DSK_F32, L.in[0].n) * 4; }
  L.part_at = off;
  // (x as it comes is read before the first sum is written; for the router it becomes the fp32 copy)
  L.raw_at = g.nin > 0 && L.in[0].f32_at >= 0 ? L.in[0].f32_at : off;
  int raw = 0;
  if (kq_quant(q) && g.in[0].norm && L.in[0].f32_at < 0) for (int i = 0; i < g.nin; i++) raw += g.in[i].n * 4;
  off = (int)align_up((size_t)off + std::max(raw, most_pieces * PS * 4), 128);
  L.ring_at = off;
  const int ring = NW * slot_bytes(q), room = form ? kSmemB : kSmemA;
  L.depth = 2;
  while (L.depth < 4 && off + (L.depth + 1) * ring <= room) L.depth++;
  L.smem = off + L.depth * ring;
  if (form) L.smem = std::max(L.smem, kSmemB);
  return L.smem <= kSmemLimit;
}
// all lists on the device, one behind another
static int place(Shapes& S) {
  std::vector<char> all;
  auto put = [&](const auto& v) {
    const size_t at = all.size(), n = v.size() * sizeof(v[0]);
    all.resize(align_up(at + n, 128));
    if (n) memcpy(all.data() + at, v.data(), n);
    return at;
  };
  std::vector<std::array<size_t, 6>> at;
  for (auto& s : S.of) { Arranged& A = s.second; at.push_back({put(A.runs), put(A.warps), put(A.items), put(A.first), put(A.units), put(A.even)}); }
  CK(cudaMalloc(&S.mem, all.size()));
  CK(cudaMemcpy(S.mem, all.data(), all.size(), cudaMemcpyHostToDevice));
  const char* d = (const char*)S.mem;
  size_t i = 0;
  for (auto& s : S.of) {
    Arranged& A = s.second;
    const std::array<size_t, 6>& o = at[i++];
    A.lists = DkLists{(const DkRun*)(d + o[0]), (const DkWarp*)(d + o[1]), (const DkItem*)(d + o[2]), (const int*)(d + o[3]), (const unsigned short*)(d + o[4]), (const int*)(d + o[5]), A.max_runs};
    A.runs = {}; A.warps = {}; A.items = {}; A.first = {}; A.units = {}; A.even = {};
  }
  return 0;
}

// The launches of a token.  Without `out` only their shapes are worked out, into `shapes`; -1 there: one does not fit
static int build(const dsk_model* m, const dsk_state* s, Shapes& shapes, Plan* out) {
  const dsk_config& c = m->c;
  const int q = c.quant, G = g_sm_count, mi = c.moe_intermediate_size, hd = m->head_dim;
  Plan none;
  Plan& P = out ? *out : none;
  P.quant = q;
  auto log2i = [](int v) { int sh = 0; while ((1 << sh) < v) sh++; return sh; };
  auto draft = [&] {
    Draft D;
    DkGemv& g = D.g;
    g.eps = c.norm_eps; g.bs0_shift = log2i(c.bs0); g.bs1_shift = log2i(c.bs1); g.silu = c.act_silu; g.ctrl = s->ctrl; g.x = s->x;
    g.nope = c.qk_nope_head_dim; g.vh = c.v_head_dim; g.hd = hd; g.heads = c.n_heads;
    return D;
  };
  auto input = [&](Draft& D, const float* x, const float* norm, int n, int seg = 0) {
    DkInput& I = D.g.in[D.g.nin++];
    I.x = x; I.norm = norm; I.n = n; I.inv_n = 1.0f / (float)n; I.seg = seg;
  };
  // a matrix; in: its input, xa: the place of its columns in it, in segments (resolved when the inputs have been placed)
  auto matrix = [&](Draft& D, const uint8_t* w, const float* scale, int rows, int n, float* o, int in, int segment = 0) -> DkSeg& {
    DkSeg& S = D.g.seg[D.g.nsegs++];
    S = DkSeg{};
    S.w = w; S.s = scale; S.out = o; S.rows = rows; S.slot = -1; S.nb = dk_units(q, n); S.ncb = c.bs1 > 0 ? cdiv(n, c.bs1) : 0;
    S.xa = in; S.xb = segment; S.in = in;
    D.tiles.push_back(cdiv(rows, dk_rows(q)));
    return S;
  };
  auto tensor = [&](Draft& D, const DTensor& t, float* o, int in, int segment = 0) -> DkSeg& { return matrix(D, t.w, t.scale, t.rows, t.cols, o, in, segment); };
  auto expert = [&](DkSeg& S, const DTensor& t, int k) { S.slot = k; S.w_stride = (long long)t.expert_bytes; S.s_stride = (long long)t.scale_expert; };
  auto planned = [&](const Draft& D, int form) -> const Arranged* {
    std::vector<int> key{form, D.g.nsegs, D.g.nin, D.even};   // (all that arrange() reads)
    for (const DkInput& I : D.g.in) { key.push_back(I.n); key.push_back(I.seg); key.push_back(I.norm != nullptr); }
    for (int j = 0; j < D.g.nsegs; j++) { key.push_back(D.g.seg[j].rows); key.push_back(D.g.seg[j].nb); key.push_back((D.g.seg[j].f32 << 1) | D.g.seg[j].pair); }
    auto it = shapes.of.find(key);
    if (it != shapes.of.end()) return &it->second;
    if (out) { fail(-4, "token chain: a launch without a plan"); return nullptr; }
    Arranged& A = shapes.of[key];
    return arrange(D, q, G, form, &A) ? &A : nullptr;
  };
  int form = 0;
  auto add = [&](Draft& D, int layer, const char* name, const int* down_tiles = nullptr) -> int {
    form ^= 1;
    const Arranged* L = planned(D, form);
    if (!L) return -1;
    if (!out) return 0;
    DkGemv& g = D.g;
    g.part_at = L->part_at; g.raw_at = L->raw_at; g.ring_at = L->ring_at; g.depth = L->depth;
    for (int i = 0; i < g.nin; i++) { const DkInput o = g.in[i]; g.in[i] = L->in[i]; g.in[i].x = o.x; g.in[i].norm = o.norm; g.in[i].ready = o.ready; }
    for (int j = 0; j < g.nsegs; j++) {
      DkSeg& S = g.seg[j];
      S.kind = L->kind[j];
      const DkInput& I = g.in[S.xa];
      const int col = S.xb * (I.stride ? I.stride : mi);
      if (kq_quant(q)) { S.xa = I.at + col; S.xb = I.at + I.n + (col >> 8) * 4; S.xc = I.at + I.n + dk_q8_scales(I.n) + (col >> 8) * 32; }
      else if (q == DSK_F8E5M2) { S.xa = I.at + col * 2; S.xb = I.at + I.len * 2 + col * 2; S.xc = I.at + I.len * 4 + (col >> 6) * 4; }
      else { S.xa = I.at + col * 4; S.xb = 0; }
      if (S.f32 && I.f32_at >= 0) S.xa = I.f32_at;
    }
    P.L.push_back(Launch{GEMV, layer, G, L->smem, (int)P.gemv.size(), form, name, L->lists});
    P.L.back().lists.down_tiles = down_tiles;
    P.gemv.push_back(g);
    return 0;
  };
  if (out) CK(cudaMalloc((void**)&P.staged, (size_t)dk_x_bytes(q, dk_whole(q, c.dim)) + 16));   // (and the norm's factor)
  {
    DkEmbed& e = P.embed;
    e.table = m->embed.w; e.scale = m->embed.scale; e.x = s->x; e.ctrl = s->ctrl; e.log = s->token_log; e.step = s->step;
    e.dim = c.dim; e.bs0 = std::max(1, c.bs0); e.bs1 = std::max(1, c.bs1); e.original_max = c.original_max_position; e.vocab = c.vocab_size;
    P.L.push_back(Launch{EMBED, -1, cdiv(c.dim, 256), 0, 0, 0, "embed", DkLists{}});
  }
  for (int l = 0; l < c.n_layers; l++) {
    const Layer& L = m->layers[l];
    {
      Draft D = draft();
      input(D, s->x, L.rms_att, c.dim);
      if (c.q_lora_rank > 0) tensor(D, L.wq_a, s->q_a, 0); else tensor(D, L.wq, s->q, 0);
      tensor(D, L.wkv_a, s->kv_a, 0);
      D.g.epi = EPI_STORE;
      if (l == 0) D.g.reset = &s->ctrl->argmax_key;
      if (add(D, l, "proj")) return -1;
    }
    {   // query up-projection beside keys and values: both wait for the same launch
      Draft D = draft();
      if (c.q_lora_rank > 0) { input(D, s->q_a, L.rms_q_a, c.q_lora_rank); tensor(D, L.wq_b, s->q, 0); }
      input(D, s->kv_a, L.rms_kv_a, c.kv_lora_rank);
      tensor(D, L.wkv_b, s->kv_b, D.g.nin - 1);
      D.g.epi = EPI_KVB; D.g.kcache = L.kcache; D.g.vcache = L.vcache;
      if (add(D, l, "q_b+kv_b")) return -1;
    }
    {
      DkAttn a{};
      a.q = s->q; a.kv_a = s->kv_a; a.freq = m->rope_freq; a.out = s->xb2; a.kcache = L.kcache; a.vcache = L.vcache; a.scratch = s->att_scratch; a.ctrl = s->ctrl;
      a.scratch_len = c.max_seq_len + kConsumers + 8;
      a.heads = c.n_heads; a.hd = hd; a.nope = c.qk_nope_head_dim; a.rope = c.qk_rope_head_dim; a.vh = c.v_head_dim; a.kv_lora = c.kv_lora_rank; a.is_v3 = c.is_v3;
      form ^= 1;
      const int room = form ? kSmemAttnB : kSmemA, row = 2 * (hd + c.v_head_dim);
      const int parts = dk_attn_parts(c.v_head_dim) * 4;
      a.hold = std::max(0, (room - hd * 4) / (row + 4)) & ~3;
      if (a.hold * 2 * hd < parts) a.hold = 0;
      const int bytes = std::max(std::max(hd * 4 + a.hold * (row + 4), hd * 4 + parts + 4096), form ? kSmemAttnB : 0);
      a.max_att = (bytes - hd * 4 - parts) / 4;
      P.L.push_back(Launch{ATTN, l, c.n_heads, bytes, (int)P.attn.size(), form, "attn", DkLists{}});
      P.attn.push_back(a);
    }
    {
      Draft D = draft();
      input(D, s->xb2, nullptr, c.n_heads * c.v_head_dim);
      tensor(D, L.wo, s->x, 0);
      D.g.epi = EPI_RESID;
      if (add(D, l, "wo")) return -1;
    }
    const int sh = L.is_moe ? c.n_shared_experts * mi : c.hidden_dim, K = L.is_moe ? c.n_active_routed : 0;
    {   // router logits and the feed-forward that every token takes (shared experts, or the dense layer)
      Draft D = draft();
      input(D, s->x, L.rms_ffn, c.dim);
      if (L.is_moe) {
        DkSeg& S = matrix(D, (const uint8_t*)L.gate, nullptr, c.n_routed_experts, c.dim, s->moe_logits, 0);
        if (q != DSK_F32) { S.f32 = 1; S.nb = cdiv(c.dim, kDkF32Cols); D.tiles.back() = cdiv(c.n_routed_experts, kDkF32Rows); }
        D.g.publish = P.staged;
      }
      if (sh > 0) { tensor(D, L.is_moe ? L.sw1 : L.w1, s->hbs, 0).pair = 1; tensor(D, L.is_moe ? L.sw3 : L.w3, nullptr, 0); }
      D.g.epi = EPI_STORE;
      if (D.g.nsegs > 0 && add(D, l, L.is_moe ? "gate+shared" : "glu")) return -1;
    }
    DkRoute r{};
    r.logits = s->moe_logits; r.bias = L.gate_bias; r.scores = s->moe_scores; r.act_w = s->act_w; r.act = s->act;
    r.E = c.n_routed_experts; r.K = K; r.norm_topk = c.norm_topk_prob; r.sigmoid = c.scoring_sigmoid; r.scale = c.routed_scaling_factor;
    r.groups = c.topk_method == 1 ? std::max(1, c.n_group) : 0; r.keep = c.topk_group;
    r.group = c.n_routed_experts / std::max(1, c.n_group);
    // down projection: the segment that every token takes, then the routed ones
    Draft down = draft();
    if (K) input(down, s->hbk, nullptr, K * mi, mi);
    if (sh > 0) { input(down, s->hbs, nullptr, sh); tensor(down, L.is_moe ? L.sw2 : L.w2, s->x, down.g.nin - 1); }
    for (int k = 0; k < K; k++) expert(tensor(down, L.w2, s->x, 0, k), L.w2, k);
    down.g.epi = EPI_DOWN; down.even = true; down.g.route = K ? ROUTE_READ : ROUTE_NONE; down.g.r = r;
    if (K) {   // routing + routed experts
      const Arranged* dl = planned(down, form);   // (the form after next)
      if (!dl) return -1;
      Draft D = draft();
      input(D, nullptr, nullptr, c.dim);
      D.g.in[0].ready = P.staged;
      for (int k = 0; k < K; k++) {
        DkSeg& a = tensor(D, L.w1, s->hbk + (size_t)k * mi, 0);
        a.pair = 1;
        expert(a, L.w1, k);
        expert(tensor(D, L.w3, nullptr, 0), L.w3, k);
      }
      D.g.epi = EPI_STORE; D.g.route = ROUTE_MAKE; D.g.r = r;
      D.g.r.w2 = L.w2.w; D.g.r.w2_stride = (long long)L.w2.expert_bytes; D.g.r.w2_tile = (long long)dk_units(q, mi) * dk_unit_bytes(q);
      if (add(D, l, "glu", dl->lists.down_tiles)) return -1;
    }
    if (add(down, l, "down")) return -1;
  }
  {
    Draft D = draft();
    input(D, s->x, m->rms_final, c.dim);
    tensor(D, m->wcls, s->logits, 0);
    D.g.epi = EPI_LOGITS; D.g.argmax = &s->ctrl->argmax_key;
    if (add(D, -1, "lm_head")) return -1;
  }
  if (!out) return 0;
  CK(cudaMalloc((void**)&P.told, P.gemv.size() * sizeof(DkGemv)));
  CK(cudaMemcpy(P.told, P.gemv.data(), P.gemv.size() * sizeof(DkGemv), cudaMemcpyHostToDevice));
  return 0;
}

// The plans of a model of these shapes, or null: the interpreter runs it (decided when the model is made, since matrices are laid out for the chain)
static std::shared_ptr<Shapes> fits(const dsk_config& c, int n_ranks) {
  if (n_ranks != 1 || !takes(c)) return nullptr;
  // a model of these sizes and a state, neither with any memory
  static float there;   // (a norm)
  const int hd = c.qk_nope_head_dim + c.qk_rope_head_dim, mi = c.moe_intermediate_size, sh = c.n_shared_experts * mi;
  auto sized = [](int rows, int cols) { DTensor t; t.rows = rows; t.cols = cols; return t; };
  dsk_model m;
  m.c = c; m.head_dim = hd; m.rms_final = &there; m.wcls = sized(c.vocab_size, c.dim);
  m.layers.resize(c.n_layers);
  for (int l = 0; l < c.n_layers; l++) {
    Layer& L = m.layers[l];
    L.is_moe = c.n_routed_experts > 0 && l >= c.first_k_dense_replace;
    L.rms_att = L.rms_ffn = L.rms_q_a = L.rms_kv_a = &there;
    const int ff = L.is_moe ? mi : c.hidden_dim;
    L.wq = sized(c.n_heads * hd, c.dim); L.wq_a = sized(c.q_lora_rank, c.dim); L.wq_b = sized(c.n_heads * hd, c.q_lora_rank);
    L.wkv_a = sized(c.kv_lora_rank + c.qk_rope_head_dim, c.dim); L.wkv_b = sized(c.n_heads * (c.qk_nope_head_dim + c.v_head_dim), c.kv_lora_rank);
    L.wo = sized(c.dim, c.n_heads * c.v_head_dim);
    L.w1 = L.w3 = sized(ff, c.dim); L.w2 = sized(c.dim, ff);
    L.sw1 = L.sw3 = sized(sh, c.dim); L.sw2 = sized(c.dim, sh);
  }
  dsk_state s;
  Ctrl ctrl;
  s.ctrl = &ctrl;
  auto shapes = std::make_shared<Shapes>();
  return build(&m, &s, *shapes, nullptr) ? nullptr : shapes;
}

template <int Q>
static cudaError_t launch_one(const Plan& P, const Launch& L, int from_argmax, bool chained, cudaStream_t st) {
  cudaLaunchConfig_t cfg{};
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cfg.gridDim = dim3((unsigned)L.grid); cfg.dynamicSmemBytes = (size_t)L.smem; cfg.stream = st;
  if (chained) { cfg.attrs = &at; cfg.numAttrs = 1; }
  switch (L.kind) {
    case EMBED: cfg.blockDim = dim3(256); return cudaLaunchKernelEx(&cfg, dk_embed<Q>, P.embed, from_argmax);
    case GEMV:
      cfg.blockDim = dim3(32 * (L.form ? kDkWarpsB : kDkWarpsA));
      return cudaLaunchKernelEx(&cfg, L.form ? dk_gemv<Q, kDkWarpsB> : dk_gemv<Q, kDkWarpsA>, (const DkGemv*)(P.told + L.at), L.lists);
    default: cfg.blockDim = dim3(32 * (L.form ? kDkWarpsB : kDkWarpsA)); return cudaLaunchKernelEx(&cfg, L.form ? dk_attn<kDkWarpsB> : dk_attn<kDkWarpsA>, P.attn[L.at]);
  }
}
static cudaError_t launch_one(const Plan& P, const Launch& L, int from_argmax, bool chained, cudaStream_t st) {
  switch (P.quant) {
    case DSK_F32: return launch_one<Q_F32>(P, L, from_argmax, chained, st);
    case DSK_F16: return launch_one<Q_F16>(P, L, from_argmax, chained, st);
    case DSK_F8E5M2: return launch_one<Q_F8>(P, L, from_argmax, chained, st);
    case DSK_Q2_K: return launch_one<Q_Q2K>(P, L, from_argmax, chained, st);
    default: return launch_one<Q_Q3K>(P, L, from_argmax, chained, st);
  }
}
// (one split of an SM's memory for all kernels of a token: another one would wait until the SM is empty)
template <typename K>
static cudaError_t attributes(K kernel) {
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
  return e == cudaSuccess ? cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemLimit) : e;
}
template <int Q>
static cudaError_t attributes_of() {
  cudaError_t e = attributes(dk_gemv<Q, kDkWarpsA>);
  if (e == cudaSuccess) e = attributes(dk_gemv<Q, kDkWarpsB>);
  return e == cudaSuccess ? attributes(dk_embed<Q>) : e;
}
static int set_attributes() {
  CK(attributes_of<Q_F32>()); CK(attributes_of<Q_F16>()); CK(attributes_of<Q_F8>()); CK(attributes_of<Q_Q2K>()); CK(attributes_of<Q_Q3K>());
  CK(attributes(dk_attn<kDkWarpsA>)); CK(attributes(dk_attn<kDkWarpsB>));
  return 0;
}

// launches [b, e) of the plan, one behind another
static int run(const Plan& P, int b, int e, int from_argmax, cudaStream_t st) {
  for (int i = b; i < e; i++) CKL(launch_one(P, P.L[i], from_argmax, i > b, st));
  g_launch_count += e - b;
  return 0;
}
// one token
static int token(Plan& P, int variant, cudaStream_t st) {
  const int n = (int)P.L.size() - (variant == HOST_HYDRATE ? 1 : 0), feed = variant == GREEDY ? 1 : 0;
  if (!P.ran[variant]) { P.ran[variant] = true; return run(P, 0, n, feed, st); }
  if (!P.graph[variant]) {
    cudaGraph_t g = nullptr;
    CK(cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal));
    const int rc = run(P, 0, n, feed, st);
    const cudaError_t e = cudaStreamEndCapture(st, &g);
    if (rc || e != cudaSuccess) return fail(-2, "capturing a token failed: %s", cudaGetErrorString(e));
    const cudaError_t ei = cudaGraphInstantiate(&P.graph[variant], g, 0);
    cudaGraphDestroy(g);
    CK(ei);
    g_launch_count -= n;
  }
  CKL(cudaGraphLaunch(P.graph[variant], st));
  g_launch_count += n;
  return 0;
}
static int layer_range(const Plan& P, int layer, int* b, int* e) {
  *b = 0; *e = 0;
  for (int i = 0; i < (int)P.L.size(); i++) if (P.L[i].layer == layer) { if (!*e) *b = i; *e = i + 1; }
  return 0;
}

}  // namespace dk

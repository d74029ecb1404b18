// dsk_decode.cuh — the kernels of a token on one GPU (MHA blocks): embedding, products, routing, attention, down projection, LM head.
//
// A token is a chain of launches (planned in dsk_decode_host.cuh), the phases of Model::_forward_cpu / Block::_block_cpu /
// BlockMHA::_attention_impl (src/infer.cpp:810-1049, 1265-1317):
//     dk_embed | per layer: dk_gemv q(+q_a), kv_a | dk_gemv q_b, kv_b -> KV cache | dk_attn | dk_gemv wo + residual |
//     dk_gemv router logits, shared w1, w3 | dk_gemv routing, routed w1, w3 | dk_gemv w2 + weighted sum | dk_gemv LM head + arg-max
// What bounds it is latency: a layer of V2-Lite moves 86 MB (13 us) through seven dependent phases.  So every launch is a programmatic dependent
// of the one ahead: its CTAs come to their SMs while that one still runs (two fit an SM), read what they are told, ask for the first weights of every
// warp, and only then wait; the stream of weights from HBM goes on through the dependencies, and what a phase costs beyond it is one launch, one
// activation vector staged, one reduction.
//
//   * one CTA an SM; a CTA owns whole row tiles of every matrix (runs, dealt out by bytes when the chain is planned).  A matrix lies in memory as its tiles do, unit of
//     columns behind unit, so that a run is one stream of units, which the CTA's warps cut into equal lengths; partial sums meet in shared memory
//     in a fixed order, one thread a row ends the row.
//   * a lane copies the words that it will multiply itself (cp.async) into a ring of `depth` units in shared memory: bytes in flight
//     cost no registers, need no barrier, and start ahead of the wait.
//   * K-quants: a unit is 16 rows x 256 columns in the order in which mma.sync m16n8k32 takes them: the 2-bit (3-bit)
//     fields are masked, not shifted, and multiplied as unsigned bytes; the eight columns of an instruction hold the eight sub-blocks of half a block,
//     each under its own mask, so that four instructions give 16 rows x 8 sub-block sums (whole numbers, as the reference's) at 64 weights a lane.
//   * F8E5M2: a unit is 16 rows x 128 columns; mma.sync m16n8k16 on the exact fp16 split of the activations, as in the interpreter (mma_rows_f8).
//     fp16, fp32: a unit is four rows (router: two) x 32 16-byte words.
// dsk_mega.cuh's interpreter runs what this chain does not: several ranks, true-MLA blocks, and the shapes that dk::fits refuses.
// Against it (B200, whole calls): V2 shape in Q2_K, three layers and the LM head, a token behind 144 positions 470 -> 374 us; V3 shape in Q3_K, two layers, behind 40
// 592 -> 427 us; V2-Lite shape in F8E5M2, eight layers, 16 tokens 13.6 -> 9.4 ms (these read 83, 139 and 150 us of bytes a token).
#pragma once

#include "dsk_mega.cuh"

namespace dsk {

// ---- how matrices lie in memory -----------------------------------------------------------------------------------------
// [matrix][row tile][unit of columns][what the 32 lanes copy].  Lane (g, t) = (lane / 4, lane % 4) holds of the tile's rows g and g + 8:
//   Q2_K, 1344 bytes (16 x 84): [half h][lane] 16 bytes: fields of row g, columns 4t.., row g + 8, row g columns 16 + 4t.., row g + 8 (of the half's 32 bytes);
//     1024: [lane] 8 bytes: the four scale | min bytes of quarter t of row g, of row g + 8; 1280: [g] d, dmin of row g, of row g + 8.
//   Q3_K, 1760 bytes (16 x 110): weights u = 0..7 of s = 0..3 (32 columns apart) make a byte u0 | u1 << 3 | (u2 >> 1) << 6 and a nibble (u2 & 1) | u3 << 1:
//     [half][lane] 16 bytes of such bytes; 1024: [lane] 16 bytes, low nibble half 0, high nibble half 1; 1536: [lane] 4 + 1664: [lane] 2 bytes: the four six-bit
//     scales of quarter t of row g, of row g + 8; 1728: [g] d of row g, of row g + 8.
//   F8E5M2, 2048 bytes: [columns 0.., 64..][row g, g + 8][lane] 16 bytes at column 16t.
//   fp16, fp32, 2048 bytes: [row 0..3][lane] 16 bytes; the router in a quantised model: [row 0..1][lane].
// Quarter t = 2h + c of a block: sub-blocks 8h + 2s + c, s = 0..3.  Rows and columns that fill up a last tile or unit are zeros.
//
// K-quant units do not lie in the order of their columns.  A last bit of an activation can turn the rounding of its 8-bit form, so the sums have one order, which
// is the interpreter's (kq_tile_rows): quarters of blocks 8 apart one after another, then the eight classes of blocks (b mod 8) in pairs 4, 2 and 1 apart, then the quarters.
// Units of a class lie side by side, and the classes as the pairs meet (0 4 2 6 1 5 3 7): a half, a quarter or an eighth of a tile's units is a branch of
// that tree, which a warp sums by itself.  The router's rows likewise: words 8 units apart, then the classes 0 to 7 (gate_f32_stage).
template <int Q> struct DkTraits {
  static constexpr bool kq = QTraits<Q>::kq;
  static constexpr int rows = kq || Q == Q_F8 ? 16 : 4;
  static constexpr int cols = kq ? 256 : Q == Q_F8 ? 128 : Q == Q_F16 ? 256 : 128;
  static constexpr int unit = Q == Q_Q2K ? 1344 : Q == Q_Q3K ? 1760 : 2048;
  static constexpr int slot = Q == Q_Q2K ? 1536 : 2048;   // its place in a ring: 16 bytes a lane three or four times
  static constexpr int part = kq ? 64 : rows;             // floats of a piece's sums: K-quants a row's four quarters
};
constexpr int kDkF32Rows = 2, kDkF32Cols = 128, kDkF32Unit = 1024;   // router of a quantised model
__host__ __device__ inline bool dk_kq(int quant) { return quant == Q_Q2K || quant == Q_Q3K; }
__host__ __device__ inline int dk_rows(int quant) { return quant == Q_F32 || quant == Q_F16 ? 4 : 16; }
__host__ __device__ inline int dk_part(int quant) { return dk_kq(quant) ? 64 : dk_rows(quant); }
__host__ __device__ inline int dk_cols(int quant) { return quant == Q_F32 || quant == Q_F8 ? 128 : 256; }
__host__ __device__ inline int dk_unit_bytes(int quant) { return quant == Q_Q2K ? DkTraits<Q_Q2K>::unit : quant == Q_Q3K ? DkTraits<Q_Q3K>::unit : 2048; }
__host__ __device__ inline int dk_units(int quant, int n) { return (n + dk_cols(quant) - 1) / dk_cols(quant); }
__host__ inline size_t dk_matrix_bytes(int quant, int rows, int cols) {
  return (size_t)((rows + dk_rows(quant) - 1) / dk_rows(quant)) * (size_t)dk_units(quant, cols) * (size_t)dk_unit_bytes(quant);
}
// the class at place i of a tile: pairs as they meet (K-quants), or in order (router); units of class c of nb
__host__ __device__ inline int dk_class(bool pairs, int i) { return pairs ? ((i & 1) << 2) | (i & 2) | ((i >> 2) & 1) : i; }
__host__ __device__ inline int dk_class_units(int nb, int c) { return (nb - c + 7) >> 3; }   // (c < 8; 0 where nb <= c)
// the unit of columns at place k of a tile of nb, and the other way round
__host__ __device__ inline int dk_unit_at(bool pairs, int nb, int k) {
  int i = 0;
  for (; i < 7; i++) { const int n = dk_class_units(nb, dk_class(pairs, i)); if (k < n) break; k -= n; }
  return dk_class(pairs, i) + 8 * k;
}
__host__ __device__ inline int dk_place_of(bool pairs, int nb, int unit) {
  int at = unit >> 3;
  for (int i = 0; dk_class(pairs, i) != (unit & 7); i++) at += dk_class_units(nb, dk_class(pairs, i));
  return at;
}

// rows as the file has them -> tiles.  src: `bytes` on a 16-byte boundary, matrices of `rows` rows of n values, one behind another; `tiles`: row tiles of all of them.
// K-quants: a CTA takes eight blocks side by side of a tile's 16 rows.  Blocks of 110 bytes begin on any even address, so the rows come as whole words into shared
// memory, every block there on a boundary of four bytes, and a warp makes a unit with word operations.  Bound by memory: 1.61 GB of Q3_K from the device,
// allocation of the tiles included, 2.2 ms (a lane that gathered its unit byte by byte 5.0; laid out as before the chain 2.4).
template <int Q>
__global__ void __launch_bounds__(256) dk_tile_kq(const unsigned char* __restrict__ src, unsigned char* __restrict__ dst, int rows, int n, long long tiles, size_t bytes) {
  constexpr int BB = Q == Q_Q2K ? kQ2Bytes : kQ3Disk, SB = (BB + 3) / 4 * 4, RW = (8 * BB + 5) / 4;   // words that hold eight blocks at any even address
  __shared__ __align__(16) unsigned char blk[16][8][SB];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3, h = t >> 1, c = t & 1;   // (h, c: the lane's quarter)
  const int nb = n >> 8, per = (rows + 15) / 16, chunks = (nb + 7) / 8;
  for (long long job = blockIdx.x; job < tiles * chunks; job += gridDim.x) {
    const long long rt = job / chunks, mat = rt / per;
    const int b0 = (int)(job - rt * chunks) * 8, blocks = min(8, nb - b0), r0 = (int)(rt - mat * per) * 16, nr = min(16, rows - r0);
    __syncthreads();
    const long long base = ((mat * rows + r0) * nb + b0) * BB;   // the first row's blocks; row r's `pitch` bytes further on
    const int pitch = nb * BB, len = blocks * BB;
    for (int i0 = tid; i0 < nr * RW; i0 += 256 * 4) {   // (four loads under way)
      uint32_t v[4];
      int row[4], p[4];   // of a word: its row, the place in it that the word begins at (-2 where that is a boundary ahead of it)
#pragma unroll
      for (int j = 0; j < 4; j++) {
        const int i = i0 + 256 * j;
        row[j] = i / RW;
        const long long from = base + (long long)row[j] * pitch, at = (from & ~3ll) + 4 * (i - row[j] * RW);
        p[j] = i < nr * RW && at < from + len ? (int)(at - from) : len;
        v[j] = 0u;
        if (p[j] < len) v[j] = at + 4 <= (long long)bytes ? *reinterpret_cast<const uint32_t*>(src + at) : *reinterpret_cast<const unsigned short*>(src + at);
      }
#pragma unroll
      for (int j = 0; j < 4; j++) {
        if constexpr (BB % 4 == 0) { if (p[j] < len) *reinterpret_cast<uint32_t*>(&blk[row[j]][p[j] / BB][p[j] % BB]) = v[j]; }
        else {
#pragma unroll
          for (int k = 0; k < 2; k++) {
            const int at = p[j] + 2 * k;
            if (at >= 0 && at < len) *reinterpret_cast<unsigned short*>(&blk[row[j]][at / BB][at % BB]) = (unsigned short)(v[j] >> (16 * k));
          }
        }
      }
    }
    __syncthreads();
    if (warp >= blocks) continue;
    unsigned char* o = dst + (size_t)(rt * nb + dk_place_of(true, nb, b0 + warp)) * DkTraits<Q>::unit;
    auto word = [&](int half, int at) { return g + 8 * half < nr ? *reinterpret_cast<const uint32_t*>(&blk[g + 8 * half][warp][at]) : 0u; };   // of row g, g + 8
    const int pick = c ? 0x7531 : 0x6420;   // bytes c, c + 2, c + 4, c + 6 of eight
    if constexpr (Q == Q_Q2K) {
#pragma unroll
      for (int hh = 0; hh < 2; hh++) {
        const int at = 16 + 32 * hh + 4 * t;
        *reinterpret_cast<uint4*>(o + 512 * hh + 16 * lane) = make_uint4(word(0, at), word(1, at), word(0, at + 16), word(1, at + 16));
      }
      *reinterpret_cast<uint2*>(o + 1024 + 8 * lane) = make_uint2(__byte_perm(word(0, 8 * h), word(0, 8 * h + 4), pick), __byte_perm(word(1, 8 * h), word(1, 8 * h + 4), pick));
      if (t < 2) *reinterpret_cast<uint32_t*>(o + 1280 + 8 * g + 4 * t) = word(t, 80);
    } else {
      uint32_t nib[4] = {0u, 0u, 0u, 0u};
#pragma unroll
      for (int hh = 0; hh < 2; hh++) {
        uint32_t b[4];
#pragma unroll
        for (int w = 0; w < 4; w++) {   // row g + 8 (w & 1), columns 4t + 16 (w >> 1)
          const int at = 4 * t + 16 * (w >> 1);
          const uint32_t q = word(w & 1, 32 + 32 * hh + at), hm = word(w & 1, at) >> (4 * hh);
          uint32_t u[4];
#pragma unroll
          for (int s = 0; s < 4; s++) u[s] = ((q >> (2 * s)) & 0x03030303u) | (((hm >> s) & 0x01010101u) << 2);
          b[w] = u[0] | (u[1] << 3) | ((u[2] & 0x06060606u) << 5);
          nib[w] |= ((u[2] & 0x01010101u) | (u[3] << 1)) << (4 * hh);
        }
        *reinterpret_cast<uint4*>(o + 512 * hh + 16 * lane) = make_uint4(b[0], b[1], b[2], b[3]);
      }
      *reinterpret_cast<uint4*>(o + 1024 + 16 * lane) = make_uint4(nib[0], nib[1], nib[2], nib[3]);
      unsigned long long sc = 0;
#pragma unroll
      for (int i = 0; i < 2; i++) {
        const uint32_t lo = (__byte_perm(word(i, 96), word(i, 100), pick) >> (4 * h)) & 0x0F0F0F0Fu, hi = word(i, 104);
#pragma unroll
        for (int k = 0; k < 4; k++)   // sub-block 8h + 2k + c
          sc |= (unsigned long long)(((lo >> (8 * k)) & 15u) | (((hi >> (8 * ((2 * k + c) & 3) + 4 * h + 2 * (k >> 1))) & 3u) << 4)) << (24 * i + 6 * k);
      }
      *reinterpret_cast<uint32_t*>(o + 1536 + 4 * lane) = (uint32_t)sc;
      *reinterpret_cast<unsigned short*>(o + 1664 + 2 * lane) = (unsigned short)(sc >> 32);
      if (t < 2) *reinterpret_cast<unsigned short*>(o + 1728 + 4 * g + 2 * t) = (unsigned short)word(t, 108);
    }
  }
}
// the rest, 16-byte words (n is a multiple of 16, 16 or 4 values: whole words), a warp a unit
template <int Q>
__global__ void __launch_bounds__(256) dk_tile_kernel(const unsigned char* __restrict__ src, unsigned char* __restrict__ dst, int rows, int n, long long units) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  constexpr int R = DkTraits<Q>::rows, ES = Q == Q_F8 ? 1 : Q == Q_F16 ? 2 : 4;
  const int nb = (n + DkTraits<Q>::cols - 1) / DkTraits<Q>::cols, per = (rows + R - 1) / R;
  // (four units side by side a warp: one division for them, sixteen loads under way)
  for (long long u0 = 4 * ((long long)blockIdx.x * 8 + (threadIdx.x >> 5)); u0 < units; u0 += (long long)gridDim.x * 32) {
    long long rt = u0 / nb;
    int b = (int)(u0 - rt * nb), tile = (int)(rt % per);
    long long row0 = rt / per * rows;   // the matrix's first row
    uint4 v[4][4];
#pragma unroll
    for (int j = 0; j < 4; j++) {
#pragma unroll
      for (int k = 0; k < 4; k++) {
        const int r = tile * R + (Q == Q_F8 ? g + 8 * (k & 1) : k), col = b * DkTraits<Q>::cols + (Q == Q_F8 ? 64 * (k >> 1) + 16 * t : lane * (16 / ES));
        v[j][k] = make_uint4(0u, 0u, 0u, 0u);
        if (u0 + j < units && r < rows && col < n) v[j][k] = *reinterpret_cast<const uint4*>(src + ((size_t)(row0 + r) * n + col) * ES);
      }
      if (++b == nb) { b = 0; if (++tile == per) { tile = 0; row0 += rows; } }
    }
#pragma unroll
    for (int j = 0; j < 4; j++)
      if (u0 + j < units) {
        unsigned char* o = dst + (size_t)(u0 + j) * DkTraits<Q>::unit;
#pragma unroll
        for (int k = 0; k < 4; k++) *reinterpret_cast<uint4*>(o + 512 * k + 16 * lane) = v[j][k];
      }
  }
}
__global__ void __launch_bounds__(256) dk_tile_router(const float* __restrict__ src, unsigned char* __restrict__ dst, int rows, int n, int units) {
  const int lane = threadIdx.x & 31, nb = (n + kDkF32Cols - 1) / kDkF32Cols;
  for (int unit = blockIdx.x * 8 + (threadIdx.x >> 5); unit < units; unit += gridDim.x * 8)
    for (int k = 0; k < kDkF32Rows; k++) {
      const int r = unit / nb * kDkF32Rows + k, col = dk_unit_at(false, nb, unit % nb) * kDkF32Cols + 4 * lane;
      float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
      if (r < rows && col < n) v = *reinterpret_cast<const float4*>(src + (size_t)r * n + col);
      *reinterpret_cast<float4*>(dst + (size_t)unit * kDkF32Unit + 512 * k + 16 * lane) = v;
    }
}

// (No "memory" on what follows: what a launch is told lies in shared memory and would be read again behind each of them.  What they store is read by
// volatile loads, behind a barrier.)
// ---- copies of weights ---------------------------------------------------------------------------------------------------
__device__ __forceinline__ void cp16(uint32_t dst, const void* src) { asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src)); }
__device__ __forceinline__ void cp8(uint32_t dst, const void* src) { asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst), "l"(src)); }
__device__ __forceinline__ void cp4(uint32_t dst, const void* src) { asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src)); }
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
// the 128-byte lines of [p, p + bytes) into L2, one a thread (a bulk prefetch instead took 5 to 10 us to issue)
__device__ __forceinline__ void l2_prefetch(const uint8_t* p, long long bytes, int t, int nt) {
  for (long long o = (long long)t * 128; o < bytes; o += (long long)nt * 128) asm volatile("prefetch.global.L2 [%0];" ::"l"(p + o));
}

// ---- what a launch is told ----------------------------------------------------------------------------------------------
// Launches alternate between two forms that fit an SM beside one another but not twice: the first is kept from it by its registers (13 warps of 80: two are
// 66560), the second by its shared memory.  A launch that comes while the one ahead still holds its SMs then has one CTA on every SM; where two of
// a launch could share an SM they did, and took twice as long as the others.
constexpr int kDkWarpsA = 13, kDkWarpsB = 12;
constexpr int kDkAhead = 16;           // units that a warp asks L2 for ahead of its ring
constexpr int kDkSegs = 18;            // matrices of a launch: pairs of up to eight routed experts; router and shared pair
enum { EPI_DOWN = 6 };   // beside EPI_STORE .. EPI_LOGITS: rows of all matrices add up, weighted by the routing, onto x
enum { ROUTE_NONE = 0, ROUTE_MAKE = 1, ROUTE_READ = 2 };
struct DkSeg {                 // a matrix
  const uint8_t* w;
  const float* s;              // f8 block scales
  float* out;
  long long w_stride, s_stride;   // between experts (bytes, floats)
  int rows, slot;              // slot: -1, or the place in the list of routed experts
  int nb, f32, pair;           // units of a row tile; router of a quantised model; the next matrix is its `up` half
  int xa, xb, xc;              // its staged input: K-quant bytes, scales, block sums; f8: high halves, low halves, group scales; else fp32 (bytes from the start)
  int ncb, in, kind;           // f8: block scales of a row; which input; which places (DkLists::units)
};
struct DkRun { int seg, tile0, tiles, piece; };   // row tiles [tile0, tile0 + tiles) of a matrix are a CTA's own, their pieces numbered from `piece` on there
// What a plan works out for a warp: its units of the CTA's stream (whole pieces of row tiles); the run, that run's first unit, tile and place in it that the
// first lies in; its first piece of the CTA's
struct __align__(16) DkWarp { int u0, u1, run, start, tile, kb, piece, pad; };
// for a row that a CTA ends: where its first piece's sum lies (floats), of the `up` half; how many pieces (side by side, DkTraits::part apart); matrix; row
struct __align__(16) DkItem { unsigned short parts, parts2; short n, seg; int r, pad; };
// and for a unit's place in a tile: its unit of columns; K-quants: whether a class ends with it, that class's place in the piece, classes without a unit behind it; whether
// a piece ends with it
enum { kDkClassEnds = 1 << 8, kDkPieceEnds = 1 << 15 };
struct DkLists {               // of a shape, by CTA
  const DkRun* runs;           // [max_runs], a matrix of -1 ends a list
  const DkWarp* warps;         // [form's warps]
  const DkItem* items;         // from first[cta] to first[cta + 1]
  const int* first;
  const unsigned short* units; // [3][256]: places of a tile of each kind of matrix
  const int* down_tiles;       // [CTA + 1] row tiles of the down projection behind it
  int max_runs;
};
struct DkInput {
  const float *x, *norm;
  const unsigned char* ready;  // staged already by the launch ahead: bytes to copy
  float inv_n;                 // 1 / length
  int n, at, bytes, f32_at;    // length, where it is staged, how many bytes, where an fp32 copy goes (-1: none)
  int len, seg, stride;        // staged values (whole units); segments of `seg` values lie `stride` apart (0: one)
};
struct DkRoute {
  const float *logits, *bias;
  float *scores, *act_w;
  int* act;
  int E, K, norm_topk, sigmoid, groups, keep;   // groups: 0 = none
  float scale;
  int group;                   // experts of a group
  const uint8_t* w2;           // the down projection behind it: routed rows that this CTA's share of it will read
  long long w2_stride, w2_tile;   // bytes of an expert, of a row tile
};
struct __align__(16) DkGemv {
  DkSeg seg[kDkSegs];
  DkInput in[2];
  DkRoute r;
  int nsegs, nin, epi, route;
  int depth, ring_at, part_at, raw_at;       // units a warp has under way; where rings, sums of pieces, inputs as they come (K-quants with a norm) lie
  float eps;
  int bs0_shift, bs1_shift, silu;
  int nope, vh, hd, heads;
  __half *kcache, *vcache;     // EPI_KVB
  float* x;                    // EPI_DOWN, EPI_RESID: the residual rows
  const Ctrl* ctrl;
  unsigned long long* argmax;  // EPI_LOGITS
  unsigned long long* reset;   // the arg-max key that this launch clears (the token has been read), or null
  unsigned char* publish;      // the staged input goes here too (for the launch behind), or null
};
static_assert(sizeof(DkGemv) % 16 == 0 && sizeof(DkGemv) / 16 <= 32 * kDkWarpsB, "copied in 16-byte words, one a thread");
struct DkAttn {
  float* q;
  const float *kv_a, *freq;
  float* out;
  __half *kcache, *vcache;
  float* scratch;              // [heads][scratch_len] scores of long contexts
  long long scratch_len;
  const Ctrl* ctrl;
  int heads, hd, nope, rope, vh, kv_lora, is_v3;
  int max_att, hold;           // scores that fit shared memory, positions (a multiple of 4) that fit with keys and values
};
struct DkEmbed {
  const uint8_t* table;
  const float* scale;
  float* x;
  Ctrl* ctrl;
  int *log, *step;
  int dim, bs0, bs1, original_max, vocab;
};

// ---- staging --------------------------------------------------------------------------------------------------------------
__device__ __forceinline__ void bar_group(int id, int n) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(n) : "memory"); }

// staged bytes of n values; all but K-quants rounded up to whole units, the rest zeros
__host__ __device__ inline int dk_whole(int quant, int n) { return dk_units(quant, n) * dk_cols(quant); }
// (K-quants: len 8-bit values, a scale a block, then 16 block sums a block on an 8-byte boundary)
__host__ __device__ inline int dk_q8_scales(int len) { return ((len >> 8) * 4 + 7) & ~7; }
__host__ __device__ inline int dk_x_bytes(int quant, int len) {
  return (int)(dk_kq(quant) ? align_up((size_t)len + dk_q8_scales(len) + (len >> 8) * 32, 128) : quant == Q_F8 ? x16_bytes(len) : align_up((size_t)len * 4, 128));
}
__device__ __forceinline__ float4 mul4(float4 v, float4 w) { return make_float4(__fmul_rn(v.x, w.x), __fmul_rn(v.y, w.y), __fmul_rn(v.z, w.z), __fmul_rn(v.w, w.w)); }
__device__ __forceinline__ float sq4(float4 v, float s) { s = fmaf(v.x, v.x, s); s = fmaf(v.y, v.y, s); s = fmaf(v.z, v.z, s); return fmaf(v.w, v.w, s); }
// (Warp operations under a mask of half the warp split it: everything here is done by whole warps, halves told apart by shuffles.)
// Maximum and minimum over the 16 lanes of a half warp
__device__ __forceinline__ void half_range(float& hi, float& lo) {
#pragma unroll
  for (int o = 8; o; o >>= 1) { hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, o)); lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, o)); }
}
// quantize_row_q8_K_ref (src/quant.cpp:616-653) of one 256-block by half a warp, 16 values a lane: the whole numbers of q8_block_nf.  qs, d, bsums: shared
// addresses of the block's, sums of sub-blocks quarter by quarter.  660 cycles with the value of largest magnitude found by a scan, 400 from maximum and minimum.
__device__ __forceinline__ void q8_half_block(const float4 (&x)[4], bool on, uint32_t qs, uint32_t d, uint32_t bsums) {
  const int l = threadIdx.x & 15, hb = threadIdx.x & 16;
  const float v[16] = {x[0].x, x[0].y, x[0].z, x[0].w, x[1].x, x[1].y, x[1].z, x[1].w, x[2].x, x[2].y, x[2].z, x[2].w, x[3].x, x[3].y, x[3].z, x[3].w};
  float h4[4], l4[4];
#pragma unroll
  for (int k = 0; k < 4; k++) {
    h4[k] = fmaxf(fmaxf(v[4 * k], v[4 * k + 1]), fmaxf(v[4 * k + 2], v[4 * k + 3]));
    l4[k] = fminf(fminf(v[4 * k], v[4 * k + 1]), fminf(v[4 * k + 2], v[4 * k + 3]));
  }
  float hi = fmaxf(fmaxf(h4[0], h4[1]), fmaxf(h4[2], h4[3])), lo = fminf(fminf(l4[0], l4[1]), fminf(l4[2], l4[3]));
  half_range(hi, lo);
  float mx = hi > -lo ? hi : lo;   // the value of largest magnitude, with its sign
  if (__any_sync(0xffffffffu, hi == -lo && hi != 0.f)) {   // both signs: the first of them (the order of the reference's scan)
    float f = 0.f;
    bool has = false;
#pragma unroll
    for (int j = 15; j >= 0; j--) if (fabsf(v[j]) == hi) { f = v[j]; has = true; }
    const unsigned who = (__ballot_sync(0xffffffffu, has) >> hb) & 0xffffu;
    f = __shfl_sync(0xffffffffu, f, hb + (who ? __ffs(who) - 1 : 0));
    if (hi == -lo) mx = f;
  }
  const bool zero = !(fabsf(mx) > 0.f);   // (also a block of NaN alone: the reference's scan finds no largest value in it)
  const float iscale = zero ? 0.f : __fdiv_rn(-127.f, mx);
  uint32_t w[4];
#pragma unroll
  for (int k = 0; k < 4; k++) {
    int qv[4];
#pragma unroll
    for (int j = 0; j < 4; j++) qv[j] = min(127, __float_as_int(__fadd_rn(__fmul_rn(iscale, v[4 * k + j]), 12582912.f)) - 0x4B400000);
    w[k] = zero ? 0u : __byte_perm(__byte_perm((uint32_t)qv[0], (uint32_t)qv[1], 0x0040), __byte_perm((uint32_t)qv[2], (uint32_t)qv[3], 0x0040), 0x5410);
  }
  int s = 0;
#pragma unroll
  for (int k = 0; k < 4; k++) s = __dp4a((int)w[k], 0x01010101, s);
  if (!on) return;
  if (l == 0) asm volatile("st.shared.f32 [%0], %1;" ::"r"(d), "f"(zero ? 0.f : __fmul_rn(mx, -1.0f / 127.0f)));
  asm volatile("st.shared.u16 [%0], %1;" ::"r"(bsums + 2u * (4 * (2 * (l >> 3) + (l & 1)) + ((l >> 1) & 3))), "h"((short)s));   // (quarter by quarter)
  asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(qs + 16u * l), "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]));
}
// four f8 columns in the two fp16 parts of x16_store_nf; am: the largest magnitude of the 16 lanes' 64 columns
__device__ __forceinline__ void x16_put(const X16& x, int f, float4 v, float am) {
  const unsigned eb = (__float_as_uint(am) >> 23) & 0xffu;
  const unsigned sb = am > 0.f ? min(max(267u - eb, 1u), 254u) : 127u;
  const float sc = __uint_as_float(sb << 23), inv = __uint_as_float((254u - sb) << 23);
  const float a0 = v.x * sc, a1 = v.y * sc, a2 = v.z * sc, a3 = v.w * sc;
  const __half2 h01 = __floats2half2_rn(a0, a1), h23 = __floats2half2_rn(a2, a3);
  const float2 f01 = __half22float2(h01), f23 = __half22float2(h23);
  const __half2 l01 = __floats2half2_rn(a0 - f01.x, a1 - f01.y), l23 = __floats2half2_rn(a2 - f23.x, a3 - f23.y);
  const uint32_t hw0 = *reinterpret_cast<const uint32_t*>(&h01), hw1 = *reinterpret_cast<const uint32_t*>(&h23);
  const uint32_t lw0 = *reinterpret_cast<const uint32_t*>(&l01), lw1 = *reinterpret_cast<const uint32_t*>(&l23);
  asm volatile("st.shared.v2.u32 [%0], {%1,%2};" ::"r"(x.hi + (uint32_t)f * 8u), "r"(hw0), "r"(hw1));
  asm volatile("st.shared.v2.u32 [%0], {%1,%2};" ::"r"(x.lo + (uint32_t)f * 8u), "r"(lw0), "r"(lw1));
  if ((f & 15) == 0) asm volatile("st.shared.f32 [%0], %1;" ::"r"(x.gs + (uint32_t)(f >> 4) * 4u), "f"(inv));
}
// Both inputs of a launch one behind the other, 16 values a thread and step (6144 in all): K-quants half a warp a block; else four float4s,
// a CTA's threads apart.  All but K-quants: what is staged is x times the norm's weights: the root of the mean square is one factor of all columns, and the
// rows are multiplied by it when they are ended, so that the staging does not wait for the sum of squares (1 us a launch).
// K-quants: the factor is part of what is rounded to 8 bits; x lies in shared memory first, and its squares are summed in the interpreter's order (stage_q8; for the
// router gate_f32_stage).
template <int Q, int NW>
struct DkStage {
  const DkGemv& P;
  const int t, n0, all;   // float4s (K-quants: blocks) of the first input, of both
  __device__ __forceinline__ DkStage(const DkGemv& p, int tid)
      : P(p), t(tid), n0(QTraits<Q>::kq ? p.in[0].n >> 8 : p.in[0].n >> 2), all(n0 + (p.nin > 1 ? (QTraits<Q>::kq ? p.in[1].n >> 8 : p.in[1].n >> 2) : 0)) {}
  __device__ __forceinline__ int steps() const { return QTraits<Q>::kq ? (all + 2 * NW - 1) / (2 * NW) : (all + 4 * (32 * NW) - 1) / (4 * (32 * NW)); }
  // K-quants: where a thread's share of step i comes from and goes to (worked out ahead of the wait for the first)
  struct At { const float4 *x, *w; uint32_t qs, d, bsums, f32; bool on, second; };
  __device__ __forceinline__ At at(uint32_t smem, int i) const {
    At A{};
    if constexpr (QTraits<Q>::kq) {
      const int b = (t >> 4) + 2 * NW * i, in = b >= n0, bl = in ? b - n0 : b;
      const DkInput& I = P.in[in];
      A.on = b < all; A.second = in;
      A.x = A.on ? reinterpret_cast<const float4*>(I.x) + (bl << 6) + 4 * (t & 15) : nullptr;
      A.w = A.on && I.norm ? reinterpret_cast<const float4*>(I.norm) + (bl << 6) + 4 * (t & 15) : nullptr;
      A.qs = smem + (uint32_t)(I.at + (bl << 8)); A.d = smem + (uint32_t)(I.at + I.n + bl * 4); A.bsums = smem + (uint32_t)(I.at + I.n + dk_q8_scales(I.n) + bl * 32);
      A.f32 = I.f32_at >= 0 ? smem + (uint32_t)(I.f32_at + (bl << 10) + 64 * (t & 15)) : 0u;
    }
    return A;
  }
  __device__ __forceinline__ void hold(float4 (&H)[4], bool norm, int i, const At& A) const {
    if constexpr (QTraits<Q>::kq) {
      const float4* p = norm ? A.w : A.x;
#pragma unroll
      for (int k = 0; k < 4; k++) H[k] = p ? p[k] : make_float4(0.f, 0.f, 0.f, 0.f);
    } else {
      const float4 *x0 = reinterpret_cast<const float4*>(norm ? P.in[0].norm : P.in[0].x), *x1 = reinterpret_cast<const float4*>(norm ? P.in[1].norm : P.in[1].x);
#pragma unroll
      for (int k = 0; k < 4; k++) {
        const int f = 4 * (32 * NW) * i + (32 * NW) * k + t;
        const float4* p = f < n0 ? x0 : x1;
        H[k] = f < all && p ? p[f < n0 ? f : f - n0] : make_float4(0.f, 0.f, 0.f, 0.f);
      }
    }
  }
  __device__ __forceinline__ void squares(const float4 (&H)[4], int i, const At& A, float (&ss)[2]) const {
    if constexpr (QTraits<Q>::kq) {
      const float q = sq4(H[3], sq4(H[2], 0.f)) + sq4(H[1], sq4(H[0], 0.f));
      if (A.second) ss[1] += q; else ss[0] += q;
    } else {
#pragma unroll
      for (int k = 0; k < 4; k++) { const float q = sq4(H[k], 0.f); if (4 * (32 * NW) * i + (32 * NW) * k + t >= n0) ss[1] += q; else ss[0] += q; }
    }
  }
  // K-quants with a norm: this thread's squares of both inputs and, for the router, of the first (256 threads)
  __device__ __forceinline__ void raw_squares(uint32_t raw, float (&ss)[3]) const {
    const int lane = t & 31, warp = t >> 5;
    auto chain = [](uint4 v, float s) {
      s = fmaf(__uint_as_float(v.x), __uint_as_float(v.x), s); s = fmaf(__uint_as_float(v.y), __uint_as_float(v.y), s);
      s = fmaf(__uint_as_float(v.z), __uint_as_float(v.z), s); return fmaf(__uint_as_float(v.w), __uint_as_float(v.w), s);
    };
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const int b = warp + 8 * k;
      if (b < n0) { const uint32_t p = raw + (uint32_t)(b << 10) + 32u * lane; ss[0] = chain(lds128(p + 16u), chain(lds128(p), ss[0])); }
      if (b < all - n0) { const uint32_t p = raw + (uint32_t)((n0 + b) << 10) + 32u * lane; ss[1] = chain(lds128(p + 16u), chain(lds128(p), ss[1])); }
    }
    if (P.in[0].f32_at >= 0) {
#pragma unroll
      for (int k = 0; k < 8; k++) if (t + 256 * k < n0 << 6) ss[2] = chain(lds128(raw + 16u * (t + 256 * k)), ss[2]);
    }
  }
  // X: the values as they come; w: the norm's weights
  __device__ __forceinline__ void put_normed(const float4 (&X)[4], const float4 (&W)[4], const At& A, const float (&sc)[3]) const {
    if (!__any_sync(0xffffffffu, A.on)) return;
    const float s = A.second ? sc[1] : sc[0];
    auto times = [](float4 v, float f, float4 w) {
      return make_float4(__fmul_rn(__fmul_rn(v.x, f), w.x), __fmul_rn(__fmul_rn(v.y, f), w.y), __fmul_rn(__fmul_rn(v.z, f), w.z), __fmul_rn(__fmul_rn(v.w, f), w.w));
    };
    float4 v[4];
#pragma unroll
    for (int k = 0; k < 4; k++) v[k] = times(X[k], s, W[k]);
    q8_half_block(v, A.on, A.qs, A.d, A.bsums);
    if (A.f32 && A.on) {
#pragma unroll
      for (int k = 0; k < 4; k++) {
        const float4 r = times(X[k], sc[2], W[k]);
        asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(A.f32 + 16u * k), "f"(r.x), "f"(r.y), "f"(r.z), "f"(r.w));
      }
    }
  }
  __device__ __forceinline__ void put(unsigned char* smem, const float4 (&X)[4], const float4 (&W)[4], int i, const At& A, bool norm) const {
    float4 v[4];
#pragma unroll
    for (int k = 0; k < 4; k++) v[k] = norm ? mul4(X[k], W[k]) : X[k];
    if constexpr (QTraits<Q>::kq) {
      if (!__any_sync(0xffffffffu, A.on)) return;
      q8_half_block(v, A.on, A.qs, A.d, A.bsums);
    } else {
      float am[4];
      if constexpr (Q == Q_F8) {   // (lengths are multiples of 64: half warps are whole; lanes past the end hold zeros)
#pragma unroll
        for (int k = 0; k < 4; k++) am[k] = fmaxf(fmaxf(fabsf(v[k].x), fabsf(v[k].y)), fmaxf(fabsf(v[k].z), fabsf(v[k].w)));
#pragma unroll
        for (int o = 8; o; o >>= 1)
#pragma unroll
          for (int k = 0; k < 4; k++) am[k] = fmaxf(am[k], __shfl_xor_sync(0xffffffffu, am[k], o));
      }
#pragma unroll
      for (int k = 0; k < 4; k++) {
        const int f = 4 * (32 * NW) * i + (32 * NW) * k + t, in = f >= n0;
        if (f < all) {
          const DkInput& I = P.in[in];
          int fl = in ? f - n0 : f;
          if (I.seg) fl += fl / (I.seg >> 2) * ((I.stride - I.seg) >> 2);
          if constexpr (Q == Q_F8) {
            x16_put(carve_x16(smem + I.at, I.len), fl, v[k], am[k]);
            if (I.f32_at >= 0) reinterpret_cast<float4*>(smem + I.f32_at)[fl] = v[k];
          } else reinterpret_cast<float4*>(smem + I.at)[fl] = v[k];
        }
      }
    }
  }
  // zeros from the end of an input, of its segments, up to a whole unit
  __device__ __forceinline__ void pad(unsigned char* smem) const {
    if constexpr (!QTraits<Q>::kq) {
      for (int i = 0; i < P.nin; i++) {
        const DkInput& I = P.in[i];
        const int seg = I.seg ? I.seg : I.n, stride = I.seg ? I.stride : I.len, gap = (stride - seg) >> 2;   // (float4s)
        if (gap == 0) continue;
        for (int j = t; j < I.len / stride * gap; j += (32 * NW)) {
          const int k = j / gap, f = ((k * stride + seg) >> 2) + j - k * gap;
          if constexpr (Q == Q_F8) {
            const X16 x = carve_x16(smem + I.at, I.len);
            asm volatile("st.shared.v2.u32 [%0], {%1,%1};" ::"r"(x.hi + f * 8u), "r"(0u));
            asm volatile("st.shared.v2.u32 [%0], {%1,%1};" ::"r"(x.lo + f * 8u), "r"(0u));
            if ((f & 15) == 0) asm volatile("st.shared.u32 [%0], %1;" ::"r"(x.gs + (f >> 4) * 4u), "r"(0u));
          } else reinterpret_cast<float4*>(smem + I.at)[f] = make_float4(0.f, 0.f, 0.f, 0.f);
        }
      }
    }
    if (P.in[0].f32_at >= 0) {
      const int n = P.in[0].n, w = (n + kDkF32Cols - 1) / kDkF32Cols * kDkF32Cols, f = (n >> 2) + t;
      if (f < (w >> 2)) reinterpret_cast<float4*>(smem + P.in[0].f32_at)[f] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
  }
};

// ---- routing: softmax | sigmoid (+ bias) and greedy / group-limited top-K (moe_gate, src/infer.cpp:493-599) -----------------------
// 256 threads, one an expert.  Every warp holds all logits and forms their sum by itself; then scores and indices are compared as one whole number (larger
// score, or the same and a lower index: the order of the reference's K scans), and the K selected are those that fewer than K candidates
// beat, four threads counting for a candidate.
// GROUP_LIMITED_GREEDY keeps, inside each group, the `keep` best experts with a score above zero (the reference compares the first candidate
// with x[-1], 0.0f in its heap layout).  A slot with no expert left gets -1 and weight 0.  Every CTA routes for itself; CTA 0 writes the results out.
struct __align__(16) DkRouteSmem { unsigned long long key[256], cand[256]; float score[256]; unsigned mask[8]; int act[16]; float sel[16], w[16]; };
__device__ __forceinline__ void dk_route(const DkRoute R, DkRouteSmem& S, int g0, float bias, bool publish) {
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5, E = R.E;
  const bool mine = t < E;
  float v[8], s;
#pragma unroll
  for (int i = 0; i < 8; i++) v[i] = 32 * i + lane < E ? R.logits[32 * i + lane] : -3.402823466e38f;
  float own = v[0];
#pragma unroll
  for (int i = 1; i < 8; i++) own = warp == i ? v[i] : own;
  if (R.sigmoid) {
    s = 1.0f / (1.0f + expf(-own));
  } else {
    float m = v[0];
#pragma unroll
    for (int i = 1; i < 8; i++) m = fmaxf(m, v[i]);
    m = warp_max(m);
#pragma unroll
    for (int i = 0; i < 8; i++) v[i] = 32 * i + lane < E ? expf(v[i] - m) : 0.f;
    own = v[0];
#pragma unroll
    for (int i = 1; i < 8; i++) own = warp == i ? v[i] : own;
#pragma unroll
    for (int o = 16; o; o >>= 1)
#pragma unroll
      for (int i = 0; i < 8; i++) if (32 * i < E) v[i] += __shfl_xor_sync(0xffffffffu, v[i], o);
    s = own / (v[0] + v[1] + v[2] + v[3] + v[4] + v[5] + v[6] + v[7]);   // (32 experts at a time, the interpreter's order)
  }
  if (R.bias && mine) s += bias;
  const unsigned long long key = ((unsigned long long)orderable(s + 0.0f) << 32) | (unsigned)(255 - t);   // (+ 0: -0 and 0 tie)
  S.score[t] = s;
  S.key[t] = key;
  if (t < 16) { S.act[t] = -1; S.sel[t] = 0.f; }
  bool cand = mine;
  if (R.groups > 0) {
    bar_group(2, 256);
    const int gs = R.group;
    int rank = 0;
    if (mine) {
#pragma unroll 8
      for (int j = 0; j < gs; j++) rank += S.key[g0 + j] > key ? 1 : 0;
    }
    cand = mine && s > 0.0f && rank < R.keep;
  }
  const unsigned bal = __ballot_sync(0xffffffffu, cand);
  if (lane == 0) S.mask[warp] = bal;
  bar_group(2, 256);
  int n = 0, before = 0;   // candidates side by side
#pragma unroll
  for (int w = 0; w < 8; w++) { const int c = __popc(S.mask[w]); before += w < warp ? c : 0; n += c; }
  if (cand) S.cand[before + __popc(bal & ((1u << lane) - 1u))] = key;
  bar_group(2, 256);
  for (int i0 = 0; i0 < n; i0 += 64) {
    const int i = i0 + (t >> 2);
    const unsigned long long k = i < n ? S.cand[i] : 0ull;
    int rank = 0;
#pragma unroll 8
    for (int j = t & 3; j < n; j += 4) rank += S.cand[j] > k ? 1 : 0;
    rank += __shfl_xor_sync(0xffffffffu, rank, 1);
    rank += __shfl_xor_sync(0xffffffffu, rank, 2);
    if ((t & 3) == 0 && i < n && rank < R.K) { const int e = 255 - (int)(k & 255u); S.act[rank] = e; S.sel[rank] = S.score[e]; }
  }
  bar_group(2, 256);
  if (t < 16) {
    const int e = S.act[t];
    float wsum = 1.0f;
    if (R.norm_topk) {
      wsum = 0.f;
      for (int k = 0; k < R.K; k++) if (S.act[k] >= 0) wsum += S.sel[k];
    }
    const float w = t < R.K && e >= 0 ? S.sel[t] / wsum * R.scale : 0.f;
    S.w[t] = w;
    if (publish && t < R.K) { R.act[t] = e; R.act_w[t] = w; }
  }
  if (publish && mine) R.scores[t] = s;   // state buffer for the host (moe_weights after softmax | sigmoid + bias)
}

// ---- units of columns -------------------------------------------------------------------------------------------------------
__device__ __forceinline__ void imma(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// this lane's words of the unit at p into its place of the ring
template <int Q>
__device__ __forceinline__ void dk_issue(const uint8_t* p, uint32_t place, bool f32) {
  const int lane = threadIdx.x & 31;
  const uint32_t d = place + 16u * lane;
  p += 16 * lane;
  if (Q == Q_F32 || !f32) {
    if constexpr (Q == Q_Q2K) {
      cp16(d, p); cp16(d + 512u, p + 512); cp8(d + 1024u, p + 1024 - 8 * lane); cp8(d + 1032u, p + 1280 + 8 * (lane >> 2) - 16 * lane);
    } else if constexpr (Q == Q_Q3K) {
      cp16(d, p); cp16(d + 512u, p + 512); cp16(d + 1024u, p + 1024);
      cp4(d + 1536u, p + 1536 - 12 * lane); cp4(d + 1540u, p + 1664 + 4 * (lane >> 1) - 16 * lane); cp4(d + 1544u, p + 1728 + 4 * (lane >> 2) - 16 * lane);
    } else {
      cp16(d, p); cp16(d + 512u, p + 512); cp16(d + 1024u, p + 1024); cp16(d + 1536u, p + 1536);
    }
  } else {
    cp16(d, p); cp16(d + 512u, p + 512);
  }
}

// What unit u adds to the sums of a piece; acc: K-quant: quarter t of rows g, g + 8; f8: rows g, g + 8, high and low halves; else one a row.
// K-quants: the instructions' columns 2t and 2t + 1 are quarter t's sub-blocks s = 0, 1 in one set of sums and s = 2, 3 in another.  About 105 instructions for the 1344 bytes
// of a Q2_K unit (13 bytes each; a lane a quarter block with dp4a, as in the interpreter, 5.3), 8 of them mma at 8 cycles of a sub-partition.  In a launch
// they are a third of what a warp issues (ncu, V2's routed w1 and w3: 3740 instructions for 12 units, 34 % of the issue slots; staging and routing have the rest).
template <int Q>
__device__ __forceinline__ void dk_unit(float (&acc)[4], uint32_t src, uint32_t xa, uint32_t xb, uint32_t xc, int u, float f0, float f1) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const uint32_t d = src + 16u * lane;
  if constexpr (QTraits<Q>::kq) {
    const uint4 h0 = lds128(d), h1 = lds128(d + 512u), e = lds128(d + 1024u);
    uint4 e2 = make_uint4(0u, 0u, 0u, 0u);
    if constexpr (Q == Q_Q3K) e2 = lds128(d + 1536u);
    // activations: lane (g = 4h + 2c + s', t) feeds word t of sub-blocks (h, c) s' and s' + 2
    const uint32_t ya = xa + 256u * u + 128u * (g >> 2) + 32u * (g & 1) + 16u * ((g >> 1) & 1) + 4u * t;
    const uint32_t y0 = lds32(ya), y1 = lds32(ya + 64u);
    uint32_t bs01, bs23;   // block sums of quarter t's sub-blocks
    asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(bs01), "=r"(bs23) : "r"(xc + 32u * u + 8u * t));
    const float yd = __uint_as_float(lds32(xb + 4u * u));
    int c01[4] = {0, 0, 0, 0}, c23[4] = {0, 0, 0, 0};
#pragma unroll
    for (int hh = 0; hh < 2; hh++) {
      const uint4 w = hh ? h1 : h0;
#pragma unroll
      for (int s = 0; s < 4; s++) {
        const uint32_t y = s < 2 ? y0 : y1, b0 = g == 4 * hh + (s & 1) ? y : 0u, b1 = g == 4 * hh + 2 + (s & 1) ? y : 0u;
        int(&c)[4] = s < 2 ? c01 : c23;
        if constexpr (Q == Q_Q2K) {
          const uint32_t mk = 0x03030303u << (2 * s);
          imma(c, w.x & mk, w.y & mk, w.z & mk, w.w & mk, b0, b1);
        } else {
          auto f = [&](uint32_t b8, uint32_t n4) -> uint32_t {
            return s == 0 ? b8 & 0x07070707u : s == 1 ? b8 & 0x38383838u : s == 2 ? (b8 & 0xC0C0C0C0u) | ((n4 << (hh ? 1 : 5)) & 0x20202020u) : n4 & (hh ? 0xE0E0E0E0u : 0x0E0E0E0Eu);
          };
          imma(c, f(w.x, e.x), f(w.y, e.y), f(w.z, e.z), f(w.w, e.w), b0, b1);
        }
      }
    }
    if constexpr (Q == Q_Q2K) {   // sums of s are 4^s times too large
#pragma unroll
      for (int r = 0; r < 2; r++) {
        const uint32_t sb = r ? e.y : e.x, dm = r ? e.w : e.z;
        const uint32_t sc4 = sb & 0x0F0F0F0Fu, m4 = (sb >> 4) & 0x0F0F0F0Fu;
        const int isum = (int)__byte_perm(sc4, 0u, 0x4440u) * c01[2 * r] + (int)__byte_perm(sc4, 0u, 0x4441u) * (c01[2 * r + 1] >> 2) +
                         (int)__byte_perm(sc4, 0u, 0x4442u) * (c23[2 * r] >> 4) + (int)__byte_perm(sc4, 0u, 0x4443u) * (c23[2 * r + 1] >> 6);
        int summs = __dp2a_lo((int)bs01, (int)m4, 0);
        summs = __dp2a_hi((int)bs23, (int)m4, summs);
        const float o = fmaf(yd * h2f((uint16_t)(dm & 0xffff)), (float)isum, -__fmul_rn(yd * h2f((uint16_t)(dm >> 16)), (float)summs));   // (rounded as kq_quarter does)
        acc[r] = __fadd_rn(acc[r], o);
      }
    } else {
      const int sh3 = t < 2 ? 1 : 5;
      const int bv[4] = {4 * (int)(short)(bs01 & 0xffffu), 4 * ((int)bs01 >> 16), 4 * (int)(short)(bs23 & 0xffffu), 4 * ((int)bs23 >> 16)};
      const uint32_t s1 = lane & 1 ? e2.y >> 16 : e2.y & 0xffffu;
#pragma unroll
      for (int r = 0; r < 2; r++) {
        const uint32_t sc = r ? (e2.x >> 24) | (s1 << 8) : e2.x & 0xffffffu;   // four six-bit scales
        const int v0 = c01[2 * r] - bv[0], v1 = (c01[2 * r + 1] >> 3) - bv[1], v2 = (c23[2 * r] >> 5) - bv[2], v3 = (c23[2 * r + 1] >> sh3) - bv[3];
        const int isum = (int)(sc & 63u) * v0 + (int)((sc >> 6) & 63u) * v1 + (int)((sc >> 12) & 63u) * v2 + (int)((sc >> 18) & 63u) * v3 - 32 * (v0 + v1 + v2 + v3);
        acc[r] = __fadd_rn(acc[r], __fmul_rn(h2f((uint16_t)(r ? e2.z >> 16 : e2.z & 0xffffu)) * yd, (float)isum));
      }
    }
  } else if constexpr (Q == Q_F8) {
    const uint32_t bp = g < 2 ? 1u : 0u, pb = (g == 1 ? xb : xa) + (uint32_t)(u * 128 + 16 * t) * 2u, pg = xc + 8u * u;
#pragma unroll
    for (int k = 0; k < 2; k++) {
      const uint4 a = lds128(d + 1024u * k), b = lds128(d + 1024u * k + 512u);
      const uint4 b0 = lds128_pred(pb + 128u * k, bp), b1 = lds128_pred(pb + 128u * k + 16u, bp);
      const float f = (k ? f1 : f0) * __uint_as_float(lds32(pg + 4u * k));
      float ca[4], cb[4];
      mma_f16_zero(ca, DSK_A4(a.x, b.x), b0.x, b0.y);
      mma_f16_zero(cb, DSK_A4(a.z, b.z), b1.x, b1.y);
      mma_f16(ca, DSK_A4(a.y, b.y), b0.z, b0.w);
      mma_f16(cb, DSK_A4(a.w, b.w), b1.z, b1.w);
#pragma unroll
      for (int i = 0; i < 4; i++) acc[i] = fmaf(ca[i] + cb[i], f, acc[i]);
    }
  } else {
    constexpr int EPC = Q == Q_F16 ? 8 : 4;
    float xv[EPC];
#pragma unroll
    for (int q = 0; q < EPC / 4; q++) {
      const uint4 v = lds128(xa + (uint32_t)((u * 32 + lane) * (EPC / 4) + q) * 16u);
      xv[4 * q] = __uint_as_float(v.x); xv[4 * q + 1] = __uint_as_float(v.y); xv[4 * q + 2] = __uint_as_float(v.z); xv[4 * q + 3] = __uint_as_float(v.w);
    }
#pragma unroll
    for (int r = 0; r < 4; r++) acc[r] += chunk_dot<Q>(lds128(d + 512u * r), xv);
  }
}
__device__ __forceinline__ void dk_unit_f32(float (&acc)[4], uint32_t src, uint32_t xa, int u) {
  const int lane = threadIdx.x & 31;
  const uint4 v = lds128(xa + (uint32_t)(u * 32 + lane) * 16u);
  const float xv[4] = {__uint_as_float(v.x), __uint_as_float(v.y), __uint_as_float(v.z), __uint_as_float(v.w)};
#pragma unroll
  for (int r = 0; r < kDkF32Rows; r++) {   // (one chain over a class: gate_f32_stage)
    const uint4 w = lds128(src + 16u * lane + 512u * r);
    acc[r] = fmaf(__uint_as_float(w.x), xv[0], acc[r]); acc[r] = fmaf(__uint_as_float(w.y), xv[1], acc[r]);
    acc[r] = fmaf(__uint_as_float(w.z), xv[2], acc[r]); acc[r] = fmaf(__uint_as_float(w.w), xv[3], acc[r]);
  }
}
// The pairs of classes: v, the sum of the class at place `pos` of a piece, and `empty` classes of no unit behind it, into the branches held in b; v becomes the
// sum of all that the last of them completes
struct DkBranch { float b[3][2]; };
__device__ __forceinline__ void dk_pair(DkBranch& B, float (&v)[2], int pos, int empty) {
#pragma unroll 1
  for (;;) {
#pragma unroll
    for (int r = 0; r < 2; r++) {
      if (!(pos & 1)) { B.b[0][r] = v[r]; continue; }
      v[r] = B.b[0][r] + v[r];
      if (!(pos & 2)) { B.b[1][r] = v[r]; continue; }
      v[r] = B.b[1][r] + v[r];
      if (!(pos & 4)) { B.b[2][r] = v[r]; continue; }
      v[r] = B.b[2][r] + v[r];
    }
    if (empty == 0) return;
    empty--; pos++; v[0] = v[1] = 0.f;
  }
}
// the sums of a piece -> part
template <int Q>
__device__ __forceinline__ void dk_sums(const float (&acc)[4], float* part, bool f32) {
  const int lane = threadIdx.x & 31;
  if (Q != Q_F32 && Q != Q_F16 && f32) {
    const float a = warp_sum(acc[0]), b = warp_sum(acc[1]);
    if (lane == 0) { part[0] = a; part[1] = b; }
    return;
  }
  if constexpr (QTraits<Q>::kq) {
    part[lane] = acc[0]; part[32 + lane] = acc[1];
  } else if constexpr (Q == Q_F8) {   // (columns 0 and 1 of the product are in the lanes with t == 0)
    if ((lane & 3) == 0) { part[lane >> 2] = acc[0] + acc[1]; part[8 + (lane >> 2)] = acc[2] + acc[3]; }
  } else {
    float v[4];
#pragma unroll
    for (int r = 0; r < 4; r++) v[r] = warp_sum(acc[r]);
    if (lane == 0) { part[0] = v[0]; part[1] = v[1]; part[2] = v[2]; part[3] = v[3]; }
  }
}

// ---- the products of a launch -------------------------------------------------------------------------------------------------
// Ahead of the wait everything is worked out that does not hang on the launches ahead: the warp's first units asked for, where a thread's share of the input
// comes from and goes to, which rows it will end and where their parts will lie.
template <int Q, int NW>
__global__ void __maxnreg__(80) dk_gemv(const DkGemv* __restrict__ told, const __grid_constant__ DkLists lists) {
  extern __shared__ __align__(128) unsigned char dsk_dyn_smem[];
  __shared__ __align__(16) DkGemv P;
  __shared__ DkRun s_run[kDkSegs + 1];
  __shared__ __align__(16) unsigned short s_unit[3][256];
  __shared__ __align__(16) float s_red[32];
  __shared__ DkRouteSmem s_route;
  __shared__ unsigned long long s_best;
  constexpr bool KQ = QTraits<Q>::kq;
  constexpr int NT = 32 * NW, PS = DkTraits<Q>::part, TR = DkTraits<Q>::rows, SLOT = DkTraits<Q>::slot, UB = DkTraits<Q>::unit;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  unsigned char* smem = dsk_dyn_smem;
  const uint32_t base = smem_u32(smem);
  // (all of it asked for at once: it has gone from L2 since the last token)
  if (tid < (int)(sizeof(DkGemv) / 16)) reinterpret_cast<uint4*>(&P)[tid] = reinterpret_cast<const uint4*>(told)[tid];
  if (tid >= NT - 32 && lane <= lists.max_runs) s_run[lane] = lane < lists.max_runs ? lists.runs[blockIdx.x * lists.max_runs + lane] : DkRun{-1, 0, 0, 0};
  if (tid < (int)(sizeof(s_unit) / 16)) reinterpret_cast<uint4*>(s_unit)[tid] = reinterpret_cast<const uint4*>(lists.units)[tid];
  const DkWarp mine = lists.warps[blockIdx.x * NW + warp];
  const int item0 = lists.first[blockIdx.x], rows = lists.first[blockIdx.x + 1] - item0;   // rows that this CTA ends
  const DkItem* items = lists.items + item0;
  DkItem first{0, 0, 0, -1, 0, 0};
  if (tid < rows) first = items[tid];
  if (tid == 0) s_best = 0ull;
  __syncthreads();
  const int depth = P.depth, epi = P.epi, u0 = mine.u0, u1 = mine.u1;   // this warp's units of the stream over the CTA's runs
  const uint32_t ring = base + (uint32_t)(P.ring_at + warp * depth * SLOT);
  bool routed = P.route == ROUTE_NONE;   // rows of chosen experts are known only behind the wait
  int run_p = mine.run, start_p = mine.start, at_p = u0, left_p = 0, ub = UB;   // what is asked for next: run, its first unit, unit, units left of the run
  const uint8_t* p = nullptr;
  // the next unit into a place of the ring; false: it has to wait for the routing
  auto issue = [&](int place) {
    while (left_p == 0 && at_p < u1) {
      const DkRun R = s_run[run_p];
      const DkSeg& S = P.seg[R.seg];
      const int end = start_p + R.tiles * S.nb;
      if (at_p < end) {
        if (!routed && S.slot >= 0) return false;
        const int e = S.slot >= 0 ? s_route.act[S.slot] : 0, n = min(end, u1) - at_p;
        if (e >= 0) {
          ub = Q != Q_F32 && S.f32 ? kDkF32Unit : UB;
          p = S.w + (size_t)e * S.w_stride + (size_t)(R.tile0 * S.nb + at_p - start_p) * ub;
          left_p = n;
          l2_prefetch(p, (long long)min(n, kDkAhead) * ub, lane, 32);
        }
        at_p += n;
      }
      start_p = end; run_p++;
    }
    if (left_p > 0) {
      dk_issue<Q>(p, ring + (uint32_t)(place * SLOT), ub != UB);
      p += ub; left_p--;
    }
    cp_commit();
    return true;
  };
  int filled = 0;
  while (filled < depth && issue(filled)) filled++;
  const DkStage<Q, NW> stage(P, tid);
  const bool norm = P.in[0].norm != nullptr;
  const int steps = stage.steps();
  typename DkStage<Q, NW>::At A = stage.at(base, 0);
  float4 w[4], x[4];
  if (norm) stage.hold(w, true, 0, A);   // (norm weights and biases are weights too)
  const int group0 = P.route == ROUTE_MAKE && P.r.groups > 0 ? tid / P.r.group * P.r.group : 0;
  const float bias = P.route == ROUTE_MAKE && P.r.bias && tid < P.r.E ? P.r.bias[tid] : 0.f;
  const float* part = reinterpret_cast<const float*>(smem + P.part_at);
  grid_wait();
  if (P.reset && blockIdx.x == 0 && tid == 0) *P.reset = 0ull;
  if (P.in[0].ready) {   // staged by the launch ahead
    for (int i = tid; i < (P.in[0].bytes >> 4); i += NT) cp16(base + (uint32_t)P.in[0].at + 16u * i, P.in[0].ready + 16 * i);
    cp_commit();
    if (warp < 8) dk_route(P.r, s_route, group0, bias, blockIdx.x == 0);
    cp_wait<0>();
    __syncthreads();
  } else {
    if (P.route == ROUTE_READ && tid < P.r.K) { s_route.act[tid] = P.r.act[tid]; s_route.w[tid] = P.r.act_w[tid]; }
    if (KQ && norm) {
      const uint32_t raw = base + (uint32_t)P.raw_at;
      const int f0 = P.in[0].n >> 2, f1 = f0 + (P.nin > 1 ? P.in[1].n >> 2 : 0);
      for (int f = tid; f < f1; f += NT) cp16(raw + 16u * f, f < f0 ? P.in[0].x + 4 * f : P.in[1].x + 4 * (f - f0));
      cp_commit();
      cp_wait<0>();
      __syncthreads();
      const bool router = P.in[0].f32_at >= 0;
      if (warp < 8) {
        float ss[3] = {0.f, 0.f, 0.f};
        stage.raw_squares(raw, ss);
#pragma unroll
        for (int o = 16; o; o >>= 1)
#pragma unroll
          for (int i = 0; i < 3; i++) ss[i] += __shfl_xor_sync(0xffffffffu, ss[i], o);
        if (lane == 0) { s_red[warp] = ss[0]; s_red[8 + warp] = ss[1]; s_red[16 + warp] = ss[2]; }
      }
      __syncthreads();
      float sc[3];
#pragma unroll
      for (int i = 0; i < 3; i++) {
        if ((i == 1 && P.nin < 2) || (i == 2 && !router)) { sc[i] = 0.f; continue; }
        const float4 a = reinterpret_cast<const float4*>(s_red)[2 * i], b = reinterpret_cast<const float4*>(s_red)[2 * i + 1];
        const float ss = a.x + a.y + a.z + a.w + b.x + b.y + b.z + b.w;
        sc[i] = 1.0f / sqrtf(ss / (float)P.in[i & 1].n + P.eps);
      }
#pragma unroll 1
      for (int i = 0;;) {
        const uint32_t src = raw + (uint32_t)(((tid >> 4) + 2 * NW * i) << 10) + 64u * (tid & 15);
        if (A.on) {
#pragma unroll
          for (int k = 0; k < 4; k++) { const uint4 v = lds128(src + 16u * k); x[k] = make_float4(__uint_as_float(v.x), __uint_as_float(v.y), __uint_as_float(v.z), __uint_as_float(v.w)); }
        } else {
#pragma unroll
          for (int k = 0; k < 4; k++) x[k] = make_float4(0.f, 0.f, 0.f, 0.f);
        }
        stage.put_normed(x, w, A, sc);
        if (++i >= steps) break;
        A = stage.at(base, i);
        stage.hold(w, true, i, A);
      }
      __syncthreads();
    } else {
    stage.hold(x, false, 0, A);
    if (!norm && steps > 1) stage.hold(w, false, 1, stage.at(base, 1));
    float ss[2] = {0.f, 0.f};
#pragma unroll 1
    for (int i = 0;;) {
      if (norm) stage.squares(x, i, A, ss);
      stage.put(smem, x, w, i, A, norm);
      if (++i >= steps) break;
      A = stage.at(base, i);
      if (norm) { stage.hold(x, false, i, A); stage.hold(w, true, i, A); }
      else {
#pragma unroll
        for (int k = 0; k < 4; k++) x[k] = w[k];
        if (i + 1 < steps) stage.hold(w, false, i + 1, stage.at(base, i + 1));
      }
    }
    stage.pad(smem);
    if (norm) {
#pragma unroll
      for (int o = 16; o; o >>= 1) { ss[0] += __shfl_xor_sync(0xffffffffu, ss[0], o); ss[1] += __shfl_xor_sync(0xffffffffu, ss[1], o); }
      if (lane == 0) { s_red[warp] = ss[0]; s_red[16 + warp] = ss[1]; }
    }
    __syncthreads();
    }
  }
  // (only here: the CTAs of the launch behind come where room is, and each SM has room for one of them once the launch ahead has gone)
  grid_release();
  routed = true;
  while (filled < depth && issue(filled)) filled++;
  // the norms' factors, in every thread (1 / sqrt rounded once)
  float sc[2] = {1.f, 1.f};
  if constexpr (KQ) {
  } else if (norm) {
    float a = lane < NW ? s_red[lane] : 0.f, b = lane < NW ? s_red[16 + lane] : 0.f;
#pragma unroll
    for (int o = 8; o; o >>= 1) { a += __shfl_xor_sync(0xffffffffu, a, o); b += __shfl_xor_sync(0xffffffffu, b, o); }
    sc[0] = __frsqrt_rn(fmaf(__shfl_sync(0xffffffffu, a, 0), P.in[0].inv_n, P.eps));
    if (P.nin > 1) sc[1] = __frsqrt_rn(fmaf(__shfl_sync(0xffffffffu, b, 0), P.in[1].inv_n, P.eps));
  } else if (P.in[0].ready) sc[0] = *reinterpret_cast<const volatile float*>(P.in[0].ready + P.in[0].bytes);
  if (P.publish && blockIdx.x == gridDim.x - 1) {
    for (int i = tid; i < (P.in[0].bytes >> 4); i += NT) reinterpret_cast<uint4*>(P.publish)[i] = reinterpret_cast<const uint4*>(smem + P.in[0].at)[i];
    if (!KQ && tid == 0) *reinterpret_cast<float*>(P.publish + P.in[0].bytes) = sc[0];
  }
  // residual row and cache position ahead of their use
  float xres = 0.f;
  int kv_pos = 0;
  if (first.seg >= 0 && (epi == EPI_DOWN || epi == EPI_RESID)) xres = P.x[first.r];
  if (epi == EPI_KVB) kv_pos = P.ctrl->kv_pos;
  int place = 0, at = u0, run_c = mine.run, start_c = mine.start, tile_c = mine.tile, kb_c = mine.kb;
  float* out = const_cast<float*>(part) + mine.piece * PS;
  while (at < u1) {
    const DkRun R = s_run[run_c];
    const DkSeg& S = P.seg[R.seg];
    const int nb = S.nb, end = start_c + R.tiles * nb, stop = min(end, u1), e = S.slot >= 0 ? s_route.act[S.slot] : 0;
    const unsigned short* places = s_unit[S.kind];
    if (e >= 0) {
      const uint32_t xa = base + (uint32_t)S.xa, xb = base + (uint32_t)S.xb, xc = base + (uint32_t)S.xc;
      const bool jf = Q != Q_F32 && S.f32;
      int tile = tile_c, kb = kb_c;
      unsigned ent = places[kb];
      const float* bs = nullptr;
      float f0 = 0.f, f1 = 0.f;
      auto scales = [&] {   // f8: of the next unit
        if constexpr (Q == Q_F8) if (!jf) { f0 = bs[(kb * 128) >> P.bs1_shift]; f1 = bs[min((kb * 128 + 64) >> P.bs1_shift, S.ncb - 1)]; }
      };
      auto scale_row = [&] { if constexpr (Q == Q_F8) bs = S.s + (size_t)e * S.s_stride + (size_t)(((R.tile0 + tile) * 16) >> P.bs0_shift) * S.ncb; };
      scale_row();
      scales();
      float acc[4] = {0.f, 0.f, 0.f, 0.f};
      DkBranch B;
#pragma unroll 1
      for (; at < stop; at++) {
        if (depth == 2) cp_wait<1>(); else if (depth == 3) cp_wait<2>(); else cp_wait<3>();
        const float g0 = f0, g1 = f1;
        const unsigned now = ent;
        if (++kb == nb) { kb = 0; tile++; if (at + 1 < stop) scale_row(); }
        if (at + 1 < stop) { ent = places[kb]; scales(); }
        if (jf) dk_unit_f32(acc, ring + (uint32_t)(place * SLOT), xa, now & 255u);
        else dk_unit<Q>(acc, ring + (uint32_t)(place * SLOT), xa, xb, xc, now & 255u, g0, g1);
        issue(place);
        place = place + 1 == depth ? 0 : place + 1;
        if constexpr (KQ) {
          if (!jf && (now & kDkClassEnds)) {
            float v[2] = {acc[0], acc[1]};
            dk_pair(B, v, (now >> 9) & 7, (now >> 12) & 7);
            if (now & kDkPieceEnds) { acc[0] = v[0]; acc[1] = v[1]; }
            else acc[0] = acc[1] = 0.f;
          }
        }
        if (now & kDkPieceEnds) {
          dk_sums<Q>(acc, out, jf);
          out += PS;
#pragma unroll
          for (int k = 0; k < 4; k++) acc[k] = 0.f;
        }
      }
    }
    at = stop; start_c = end; run_c++; tile_c = kb_c = 0;
    out = const_cast<float*>(part) + s_run[run_c].piece * PS;
  }
  if (P.route == ROUTE_MAKE) {   // rows of the chosen experts that this CTA multiplies in the launch behind
    const int ta = lists.down_tiles[blockIdx.x], tb = lists.down_tiles[blockIdx.x + 1];
    for (int k = warp; k < P.r.K; k += NW)
      if (s_route.act[k] >= 0) l2_prefetch(P.r.w2 + (size_t)s_route.act[k] * P.r.w2_stride + (size_t)ta * P.r.w2_tile, (long long)(tb - ta) * P.r.w2_tile, lane, 32);
  }
  __syncthreads();
  auto sum = [&](int parts, int n, bool f32) {   // a row's pieces
    if constexpr (KQ) {
      if (!f32) {   // the rest of the pairs, then the quarters
        auto at = [&](int k) { return *reinterpret_cast<const float4*>(part + parts + k * PS); };
        auto add = [](float4 a, float4 b) { return make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w); };
        float4 v = at(0);
        if (n > 1) v = add(v, at(1));
        if (n > 2) v = add(v, add(at(2), at(3)));
        if (n > 4) v = add(v, add(add(at(4), at(5)), add(at(6), at(7))));
        return (v.x + v.z) + (v.y + v.w);
      }
    }
    float v = part[parts];   // in order
#pragma unroll 1
    for (int k = 1; k < n; k += 4) {
      float q[4];
#pragma unroll
      for (int i = 0; i < 4; i++) q[i] = k + i < n ? part[parts + (k + i) * PS] : 0.f;
#pragma unroll
      for (int i = 0; i < 4; i++) v += q[i];
    }
    return v;
  };
  if (epi == EPI_DOWN) {   // x += sum_k w_k (w2_k . h_k) + shared, in the reference's order (src/infer.cpp:873-877, 899-903, 926-930)
    // a thread a row of a run; then a thread a row
    float* d = reinterpret_cast<float*>(smem);   // (the staged input has been read)
    for (int i = tid; i < rows; i += NT) {
      const DkItem I = i == tid ? first : items[i];
      if (I.seg < 0) continue;
      const int slot = P.seg[I.seg].slot;
      d[i] = slot < 0 || s_route.act[slot] >= 0 ? sum(I.parts, I.n, false) : 0.f;
    }
    __syncthreads();
    const int n = s_run[0].seg >= 0 ? s_run[0].tiles * TR : 0;
    for (int i = tid; i < n; i += NT) {
      const int r = s_run[0].tile0 * TR + i;
      if (r >= P.seg[0].rows) continue;
      float v = i == tid ? xres : P.x[r], all = 0.f;
      bool shared = false;
      for (int j = 0; j * n < rows; j++) {
        const int slot = P.seg[s_run[j].seg].slot;
        const float q = d[j * n + i];
        if (slot < 0) { all = q; shared = true; }   // (the segment every token takes comes first, its sum last)
        else if (s_route.act[slot] >= 0) v = fmaf(q, s_route.w[slot], v);
      }
      P.x[r] = shared ? v + all : v;
    }
    return;
  }
  unsigned long long best = 0ull;
  for (int i = tid; i < rows; i += NT) {
    const DkItem I = i == tid ? first : items[i];
    if (I.seg < 0) continue;
    const DkSeg& S = P.seg[I.seg];
    if (S.slot >= 0 && s_route.act[S.slot] < 0) continue;
    const float f = S.in ? sc[1] : sc[0];
    float val = f * sum(I.parts, I.n, Q != Q_F32 && S.f32);
    if (S.pair) val = (P.silu ? silu_f(val) : gelu_f(val)) * (f * sum(I.parts2, I.n, false));
    if (epi == EPI_RESID) val += i == tid ? xres : P.x[I.r];
    S.out[I.r] = val;
    if (epi == EPI_KVB && I.seg == P.nsegs - 1) {   // (the query rows ahead of it are only stored)
      const int pr = P.nope + P.vh, h = I.r / pr, ii = I.r - h * pr;
      if (ii < P.nope) P.kcache[((size_t)kv_pos * P.heads + h) * P.hd + ii] = __float2half_rn(val);
      else P.vcache[((size_t)kv_pos * P.heads + h) * P.vh + (ii - P.nope)] = __float2half_rn(val);
    }
    if (epi == EPI_LOGITS) {
      const unsigned long long key = ((unsigned long long)orderable(val) << 32) | (unsigned long long)(0xFFFFFFFFu - (unsigned)I.r);
      if (key > best) best = key;
    }
  }
  if (epi == EPI_LOGITS) {
#pragma unroll
    for (int o = 16; o; o >>= 1) { const unsigned long long ob = __shfl_xor_sync(0xffffffffu, best, o); if (ob > best) best = ob; }
    if (lane == 0 && best) atomicMax(&s_best, best);
    __syncthreads();
    if (tid == 0 && s_best) atomicMax(P.argmax, s_best);
  }
}

// ---- rope + attention of one head (src/infer.cpp:648-762, 956-1045): one CTA a head ------------------------------------------------------
// The head's older keys and values come into shared memory ahead of the wait: they were written launches ago (a launch begins when the one ahead of it
// is past its own wait, so only the one ahead may still run, and that writes row kv_pos).  What is left behind the wait is the new row, one pass over
// shared memory for the scores and one for the values.  Contexts that do not fit (156 or 180 positions of 192 + 128 halves), those whose first rows
// turn in place (sinks) and those that the new row lies behind are read from global memory in the same passes.
// Shared memory: query | scores of `hold` positions | their keys (later partial sums of the values) | their values; or query | partial sums | scores
__host__ __device__ inline int dk_attn_parts(int vh) { return (vh <= 256 ? 256 / vh : 1) * vh; }
template <int NW>
__global__ void __maxnreg__(80) dk_attn(const __grid_constant__ DkAttn P) {
  extern __shared__ __align__(128) unsigned char dsk_dyn_smem[];
  __shared__ float s_red[32];
  constexpr int NT = 32 * NW;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, h = blockIdx.x;
  float* qs = reinterpret_cast<float*>(dsk_dyn_smem);
  const size_t kstride = (size_t)P.heads * P.hd, vstride = (size_t)P.heads * P.vh;
  const __half *kh = P.kcache + (size_t)h * P.hd, *vh = P.vcache + (size_t)h * P.vh;
  const volatile int* cw = reinterpret_cast<const volatile int*>(P.ctrl);   // (set launches ago; not out of L1)
  const int pos = cw[offsetof(Ctrl, pos) / 4], kv_pos = cw[offsetof(Ctrl, kv_pos) / 4], kv_len = cw[offsetof(Ctrl, kv_len) / 4], kv_sink = cw[offsetof(Ctrl, kv_sink) / 4];
  const int nc = P.hd >> 3, nv = P.vh >> 3, half_r = P.rope >> 1;   // (16-byte words of a row)
  const bool held = kv_len <= P.hold && kv_pos < kv_len && kv_sink == 0;   // (a block call may put its row behind those that it reads)
  float* att = qs + P.hd;
  __half *ks = reinterpret_cast<__half*>(att + P.hold), *vs = ks + (size_t)P.hold * P.hd;
  float* part = held ? reinterpret_cast<float*>(ks) : att;
  if (!held) att = kv_len <= P.max_att ? att + dk_attn_parts(P.vh) : P.scratch + (size_t)h * P.scratch_len;
  const uint32_t ks_u = smem_u32(ks), vs_u = smem_u32(vs);
  auto copy_rows = [&](int t0, int t1, int but) {   // positions [t0, t1) but one
    for (int i = t0 * nc + tid; i < t1 * nc; i += NT) { const int t = i / nc, c = i - t * nc; if (t != but) cp16(ks_u + 16u * i, kh + (size_t)t * kstride + 8 * c); }
    for (int i = t0 * nv + tid; i < t1 * nv; i += NT) { const int t = i / nv, c = i - t * nv; if (t != but) cp16(vs_u + 16u * i, vh + (size_t)t * vstride + 8 * c); }
  };
  if (held) { copy_rows(0, kv_len, kv_pos); cp_commit(); }
  float cs = 0.f, sn = 0.f;
  if (tid < half_r) rope_cs(P.freq, tid, pos, cs, sn);
  else if (tid >= 64 && tid < 64 + half_r) rope_cs(P.freq, tid - 64, pos, cs, sn);
  grid_wait();
  grid_release();
  float* qh = P.q + (size_t)h * P.hd;
  if (held) { copy_rows(kv_pos, kv_pos + 1, -1); cp_commit(); }
  for (int i = tid; i < P.nope; i += NT) qs[i] = qh[i];
  __half r0h = __half(), r1h = __half();
  if (tid < half_r) {
    const float v0 = qh[P.nope + 2 * tid], v1 = qh[P.nope + 2 * tid + 1];
    const float r0 = fmaf(v0, cs, -(v1 * sn)), r1 = fmaf(v1, cs, v0 * sn);
    if (P.is_v3) { qs[P.nope + 2 * tid] = r0; qs[P.nope + 2 * tid + 1] = r1; }
    else { qs[P.nope + tid] = r0; qs[P.nope + tid + half_r] = r1; }
  } else if (tid >= 64 && tid < 64 + half_r) {
    const int t = tid - 64;
    const float v0 = P.kv_a[P.kv_lora + 2 * t], v1 = P.kv_a[P.kv_lora + 2 * t + 1];
    r0h = __float2half_rn(fmaf(v0, cs, -(v1 * sn))); r1h = __float2half_rn(fmaf(v1, cs, v0 * sn));
    __half* kr = P.kcache + (size_t)kv_pos * kstride + (size_t)h * P.hd + P.nope;
    if (P.is_v3) { kr[2 * t] = r0h; kr[2 * t + 1] = r1h; }
    else { kr[t] = r0h; kr[t + half_r] = r1h; }
  }
  if (kv_pos < kv_sink) __syncthreads();   // (a block call whose new row is a sink: it turns too)
  const int rows_at_once = NT / half_r;   // sink rows turn by one position, in place: read, then write
  for (int r0 = 0; r0 < kv_sink; r0 += rows_at_once) {
    const int r = r0 + tid / half_r, t = tid - (tid / half_r) * half_r;
    const bool on = tid < rows_at_once * half_r && r < kv_sink;
    __half* kr = P.kcache + (size_t)(on ? r : 0) * kstride + (size_t)h * P.hd + P.nope;
    float a = 0.f, b = 0.f;
    if (on) {
      float c1, s1; rope_cs(P.freq, t, 1, c1, s1);
      const float v0 = __half2float(kr[2 * t]), v1 = __half2float(kr[2 * t + 1]);
      a = fmaf(v0, c1, -(v1 * s1)); b = fmaf(v1, c1, v0 * s1);
    }
    __syncthreads();
    if (on) {
      if (P.is_v3) { kr[2 * t] = __float2half_rn(a); kr[2 * t + 1] = __float2half_rn(b); }
      else { kr[t] = __float2half_rn(a); kr[t + half_r] = __float2half_rn(b); }
    }
  }
  cp_wait<0>();
  __syncthreads();
  if (held) {   // (over what came with the row: its rotated part of the token before)
    if (tid >= 64 && tid < 64 + half_r) {
      const int t = tid - 64;
      __half* kr = ks + (size_t)kv_pos * P.hd + P.nope;
      if (P.is_v3) { kr[2 * t] = r0h; kr[2 * t + 1] = r1h; }
      else { kr[t] = r0h; kr[t + half_r] = r1h; }
    }
    __syncthreads();
  }
  if (tid < P.rope) qh[P.nope + tid] = qs[P.nope + tid];   // the reference rotates the query in place
  const float inv = sqrtf((float)P.hd);
  float m = -3.402823466e38f;
  // (sums over a key, over the probabilities and over the values in the interpreter's order: c_attention)
  auto scores = [&](const __half* k, size_t stride) {
    for (int t0 = warp * 8; t0 < kv_len; t0 += NW * 8) {   // eight positions a warp, two values a lane and step
      float a[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
      for (int c = lane * 2; c < P.hd; c += 64) {
        const float2 q = *reinterpret_cast<const float2*>(qs + c);
        float2 f[8];
#pragma unroll
        for (int u = 0; u < 8; u++) f[u] = __half22float2(*reinterpret_cast<const __half2*>(k + (size_t)min(t0 + u, kv_len - 1) * stride + c));
#pragma unroll
        for (int u = 0; u < 8; u++) { a[u] = fmaf(q.x, f[u].x, a[u]); a[u] = fmaf(q.y, f[u].y, a[u]); }
      }
#pragma unroll
      for (int o = 16; o; o >>= 1)
#pragma unroll
        for (int u = 0; u < 8; u++) a[u] += __shfl_xor_sync(0xffffffffu, a[u], o);
      float own = a[0];
#pragma unroll
      for (int u = 1; u < 8; u++) own = lane == u ? a[u] : own;
      if (lane < 8 && t0 + lane < kv_len) { own = own / inv; att[t0 + lane] = own; m = fmaxf(m, own); }
    }
  };
  if (held) scores(ks, P.hd); else scores(kh, kstride);
  m = warp_max(m);
  if (lane == 0) s_red[warp] = m;
  __syncthreads();
  m = warp_max(lane < NW ? s_red[lane] : -3.402823466e38f);
  float sum = 0.f;
  if (tid < 256) for (int t = tid; t < kv_len; t += 256) { const float e = expf(att[t] - m); att[t] = e; sum += e; }
  sum = warp_sum(sum);
  if (lane == 0 && warp < 8) s_red[16 + warp] = sum;
  __syncthreads();
  sum = s_red[16] + s_red[17] + s_red[18] + s_red[19] + s_red[20] + s_red[21] + s_red[22] + s_red[23];
  for (int t = tid; t < kv_len; t += NT) att[t] = att[t] / sum;
  __syncthreads();
  const int groups = max(1, 256 / P.vh);   // positions apart that a thread adds up
  auto values = [&](const __half* v0, size_t stride) {
    for (int i = tid; i < groups * P.vh; i += NT) {
      const int g = i / P.vh;
      const __half* v = v0 + (i - g * P.vh);
      float acc = 0.f;
#pragma unroll 16
      for (int t = g; t < kv_len; t += groups) acc = fmaf(att[t], __half2float(v[(size_t)t * stride]), acc);
      part[i] = acc;
    }
  };
  if (held) values(vs, P.vh); else values(vh, vstride);
  __syncthreads();
  for (int i = tid; i < P.vh; i += NT) {
    float o = 0.f;
    for (int k = 0; k < groups; k++) o += part[k * P.vh + i];
    P.out[(size_t)h * P.vh + i] = o;
  }
}

// ---- embedding row: token feed, step counters, dequantised row.  A CTA 256 columns; CTA 0 also moves the control words on ----------------
// from_argmax: the token is the previous launch's arg-max (every CTA reads it from the key; the LM head's successor clears the key later).
template <int Q>
__global__ void __launch_bounds__(256) dk_embed(const __grid_constant__ DkEmbed P, int from_argmax) {
  grid_wait();
  grid_release();
  const int tid = threadIdx.x, dim = P.dim;
  // (a key that no LM head has set gives index 2^32 - 1: the host refuses such a call)
  const int token = from_argmax ? (int)min(0xFFFFFFFFu - (unsigned)(P.ctrl->argmax_key & 0xFFFFFFFFull), (unsigned)P.vocab - 1u) : P.ctrl->token;
  if (from_argmax && blockIdx.x == 0 && tid == 0) {
    Ctrl* c = P.ctrl;
    const int pos = c->pos + 1, sink = pos >= P.original_max ? 2 : 0;
    c->token = token; c->pos = pos; c->kv_sink = sink;
    c->kv_pos = sink + (pos - sink) % (P.original_max - sink);
    c->kv_len = pos >= P.original_max ? P.original_max : pos + 1;
    if (P.log && P.step) { P.log[*P.step] = token; *P.step = *P.step + 1; }
  }
  const int i = blockIdx.x * 256 + tid;
  if (i >= dim) return;
  float val;
  const int nb = (dim + DkTraits<Q>::cols - 1) / DkTraits<Q>::cols, r = token % DkTraits<Q>::rows, unit = i / DkTraits<Q>::cols;
  const uint8_t* o = P.table + ((size_t)(token / DkTraits<Q>::rows) * nb + (QTraits<Q>::kq ? dk_place_of(true, nb, unit) : unit)) * DkTraits<Q>::unit;
  if constexpr (Q == Q_F32) val = *reinterpret_cast<const float*>(o + 512 * r + 4 * (i & 127));
  else if constexpr (Q == Q_F16) val = __half2float(*reinterpret_cast<const __half*>(o + 512 * r + 2 * (i & 255)));
  else if constexpr (Q == Q_F8) {
    const int ncb = (dim + P.bs1 - 1) / P.bs1, c = i & 127;
    val = h2f((uint16_t)((uint16_t)o[1024 * (c >> 6) + 512 * (r >> 3) + 16 * (4 * (r & 7) + ((c >> 4) & 3)) + (c & 15)] << 8)) * P.scale[(size_t)(token / P.bs0) * ncb + i / P.bs1];
  } else {
    // column i of the row in its tile: half h, s, byte l of the half's 32, lane (g, t) and byte of the lane's 16
    const int w = i & 255, h = w >> 7, s = (w >> 5) & 3, l = w & 31;
    const int g = r & 7, t = (l & 15) >> 2, lane = 4 * g + t, at = 16 * lane + 8 * (l >> 4) + 4 * (r >> 3) + (l & 3);
    const int sl = 4 * g + 2 * h + (l >> 4);   // the lane that has the scale: quarter 2h + (l >> 4)
    if constexpr (Q == Q_Q2K) {
      const int sc = o[1024 + 8 * sl + 4 * (r >> 3) + s], qv = (o[512 * h + at] >> (2 * s)) & 3;
      const uint16_t* dm = reinterpret_cast<const uint16_t*>(o + 1280 + 8 * g + 4 * (r >> 3));
      val = fmaf(h2f(dm[0]) * (float)(sc & 0xF), (float)qv, -__fmul_rn(h2f(dm[1]), (float)(sc >> 4)));
    } else {
      const int byte = o[512 * h + at], nib = (o[1024 + at] >> (4 * h)) & 15;
      const int u = s == 0 ? byte & 7 : s == 1 ? (byte >> 3) & 7 : s == 2 ? ((byte >> 6) << 1) | (nib & 1) : nib >> 1;
      const uint32_t s0 = *reinterpret_cast<const uint32_t*>(o + 1536 + 4 * sl), s1 = *reinterpret_cast<const uint16_t*>(o + 1664 + 2 * sl);
      const unsigned long long sc48 = (unsigned long long)s0 | ((unsigned long long)s1 << 32);
      const int sc = (int)((sc48 >> (6 * (4 * (r >> 3) + s))) & 63u);
      const uint16_t d = *reinterpret_cast<const uint16_t*>(o + 1728 + 4 * g + 2 * (r >> 3));
      val = (h2f(d) * (float)(sc - 32)) * (float)(u - 4);
    }
  }
  P.x[i] = val;
}

}  // namespace dsk

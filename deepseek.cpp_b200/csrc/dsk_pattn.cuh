// dsk_pattn.cuh — softmax attention of portions (layer-list models without mixing of the heads' scores) in one kernel: scores, mask, softmax and
// the weighted values of a block of queries against all of their keys, nothing of it in global memory.
//
// Products run on mma.sync (bf16 x bf16 -> fp32, m16n8k16).  PARTS = 3 (designs with 32-bit scores and weights): every fp32 operand is the sum
// of three bf16 numbers (8 + 8 + 8 bits of mantissa, fp32's exponent range), and a product takes the six pairs whose order is at least 2^-16 of
// the leading one; what is left out is below an fp32 rounding.  The sum over 16 elements comes out of the tensor core and is added in fp32
// registers (rounded to nearest), so that a sum of n elements sees n / 16 roundings where a chain of FMAs sees n: the error against 64 bits is not
// larger than that of the fp32 products it replaces.  PARTS = 1: operands rounded to bf16 (latent attention of bf16 models, whose products
// always took them so).
// pattn_pack splits the visible keys and values once per step; a CTA (16 query rows per warp) streams them in tiles of 32 or 16 through two
// buffers (cp.async); where the query blocks of all heads are fewer than the SMs, shares of the keys are CTAs of their own.  Bound: issue slots - six products per element, their operands from shared memory, softmax.  Before, a block of 256
// queries wrote its scores, read them for the softmax and again for the values, all three in kernels of their own on the fp32 pipe.
#pragma once

#include "dsk_hybrid.cuh"

namespace dsk {
namespace hy {

struct PackP {
  const float *k, *krot, *v;     // key rows [..][G][D0] (+ a part shared by the groups: krot, Rd values), value rows [..][G][V]
  int ldk, ldr, ldv, D0, Rd, V, Dp, Vp, G, Lk, nk, first, keep, ring;
  int kv_cached;                 // k and v rows are cache rows (else row j belongs to the j-th visible key); krot rows always are
  __nv_bfloat16 *kb, *vb;        // [parts][G][Lk][Dp], [parts][G][Lk][Vp], zeros behind D0 + Rd and V
};

template <int PARTS>
__device__ __forceinline__ void split_bf16(float x, __nv_bfloat16 (&o)[PARTS]) {
#pragma unroll
  for (int i = 0; i < PARTS; i++) {
    o[i] = __float2bfloat16_rn(x);
    if (i + 1 < PARTS) {   // exact: the rest has fewer bits (an infinity stays in the first part; a finite number has finite parts)
      if (isinf(__bfloat162float(o[i])) && isfinite(x)) o[i] = __ushort_as_bfloat16(x > 0.f ? 0x7F7F : 0xFF7F);
      x = isfinite(x) ? x - __bfloat162float(o[i]) : 0.f;
    }
  }
}

template <int PARTS>
__global__ void __launch_bounds__(256) pattn_pack(const PackP P) {
  grid_enter();
  const int j = blockIdx.x;
  const size_t crow = (size_t)cache_row(j < P.nk ? j : P.first + j - P.nk, P.keep, P.ring), row = P.kv_cached ? crow : (size_t)j;
  const int kq = P.Dp / 4, vq = P.Vp / 4;
  for (int e = threadIdx.x; e < P.G * (kq + vq); e += 256) {
    const bool key = e < P.G * kq;
    const int q = key ? e : e - P.G * kq, per = key ? kq : vq, g = q / per, c = (q - g * per) * 4;
    float x[4];
#pragma unroll
    for (int u = 0; u < 4; u++) {
      const int d = c + u;
      if (key) x[u] = d < P.D0 ? P.k[row * P.ldk + g * P.D0 + d] : d < P.D0 + P.Rd ? P.krot[crow * P.ldr + d - P.D0] : 0.f;
      else x[u] = d < P.V ? P.v[row * P.ldv + g * P.V + d] : 0.f;
    }
    __nv_bfloat16 s[4][PARTS];
#pragma unroll
    for (int u = 0; u < 4; u++) split_bf16<PARTS>(x[u], s[u]);
    __nv_bfloat16* dst = key ? P.kb + ((size_t)g * P.Lk + j) * P.Dp + c : P.vb + ((size_t)g * P.Lk + j) * P.Vp + c;
    const size_t part = (size_t)P.G * P.Lk * (key ? P.Dp : P.Vp);
#pragma unroll
    for (int i = 0; i < PARTS; i++) {
      __nv_bfloat162 lo, hi;
      lo.x = s[0][i]; lo.y = s[1][i]; hi.x = s[2][i]; hi.y = s[3][i];
      *reinterpret_cast<uint2*>(dst + i * part) = make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
    }
  }
}

struct PattnP {
  const float* q;                // query rows: token t, head h at q + t * ldq + h * D
  const __nv_bfloat16 *kb, *vb;  // (pattn_pack)
  float* out;                    // token t, head h at out + t * ld_out + h * V
  const float* gate;             // (see gqa_attn)
  float* part;                   // NS > 1: results of a share of the keys (see latent_swa_merge)
  int T, H, G, D, Dp, V, Vp, ldq, ld_out, ld_gate, gate_head, Lk, nk, first, pos0, mask, span, NS;
  float scale, alpha;
  ScoreMods mods;
};

// NK: 8-key groups of a tile
__host__ __device__ inline size_t pattn_smem(int parts, int warps, int Dp, int VN, int NK) {
  return (size_t)parts * 2 * ((size_t)warps * 16 * (Dp + 8) + 2 * NK * 8 * ((Dp + 8) + (VN * 8 + 8)));
}

__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void ldmatrix_x4_at(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void mma_bf16_first(float (&c)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {   // c = a b
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
               : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]), "f"(0.f));
}
// two fp32 values as PARTS pairs of bf16, for finite values (see plain_dot for the others)
template <int PARTS>
__device__ __forceinline__ void split_pair(float x, float y, uint32_t (&o)[PARTS]) {
#pragma unroll
  for (int i = 0; i < PARTS; i++) {
    const __nv_bfloat162 p = __floats2bfloat162_rn(x, y);
    o[i] = *reinterpret_cast<const uint32_t*>(&p);
    if (i + 1 < PARTS) { x -= __uint_as_float(o[i] << 16); y -= __uint_as_float(o[i] & 0xffff0000u); }
  }
}
// acc[n] += sum over 16 elements of a b[n] for N tiles: the six leading pairs of the operands' parts, joined in the tensor core and then added.  A
// step of all N sums comes before the next step of any: a sum's products wait for one another (some 24 cycles each), the N sums do not.
// load(part, b) brings the tiles' b operands of a part.
template <int PARTS, int N, typename Load>
__device__ __forceinline__ void mma_parts(float (*acc)[4], const uint32_t (&a)[PARTS][4], Load load) {
  uint32_t b[N][2];
  auto step = [&](float (*t)[4], const uint32_t (&x)[4]) {
#pragma unroll
    for (int n = 0; n < N; n++) mma_bf16_16816(t[n], x[0], x[1], x[2], x[3], b[n][0], b[n][1]);
  };
  if constexpr (PARTS == 1) {
    load(0, b);
    step(acc, a[0]);
  } else {
    float t[N][4];
    load(2, b);
#pragma unroll
    for (int n = 0; n < N; n++) mma_bf16_first(t[n], a[0], b[n]);
    load(1, b);
    step(t, a[1]);
    step(t, a[0]);
    load(0, b);
    step(t, a[2]);
    step(t, a[1]);
    step(t, a[0]);
#pragma unroll
    for (int n = 0; n < N; n++)
#pragma unroll
      for (int i = 0; i < 4; i++) acc[n][i] += t[n][i];
  }
}

template <int PARTS>
__device__ __forceinline__ float joined(const __nv_bfloat16* x, size_t part) {   // the number whose parts lie `part` apart
  float v = __bfloat162float(x[(PARTS - 1) * part]);
#pragma unroll
  for (int i = PARTS - 2; i >= 0; i--) v += __bfloat162float(x[i * part]);
  return v;
}
// The key tiles (KT keys) that a CTA with queries q0 .. q0 + BM - 1 meets: those of the kept keys, then from the first key of its first query to its last query.  Share `s` of
// NS has the tiles begin .. end - 1 of them.
struct KeyTiles { int kept, t0, begin, end; };
__device__ __forceinline__ KeyTiles key_tiles(const PattnP& P, int q0, int BM, int KT, int s, int NS) {
  const int last = min(P.T, q0 + BM) - 1;
  const int lo_v = P.nk + mask_first(P.mask, P.span, P.pos0 + q0) - P.first, hi_v = P.nk + P.pos0 + last - P.first;
  KeyTiles k;
  k.kept = (min(P.mods.keep, hi_v + 1) + KT - 1) / KT;   // (kept positions are keys 0 .. keep - 1 whether or not they lie in the range)
  k.t0 = max(k.kept, lo_v / KT);
  const int n = k.kept + max(0, hi_v / KT - k.t0 + 1), per = (n + NS - 1) / NS;
  k.begin = s * per;
  k.end = min(n, k.begin + per);
  return k;
}
__device__ __forceinline__ int tile_key(const KeyTiles& k, int i, int KT) { return (i < k.kept ? i : k.t0 + i - k.kept) * KT; }
// Query t of head h again, by one warp and from its visible keys alone, into columns v0 .. v0 + VN * 8 - 1 of the output: for rows whose result is not
// finite.  In the products of a tile a key out of sight has the weight 0, and 0 x Inf is NaN; an infinity times the parts of a number is NaN.
template <int PARTS, int VN, int KT, bool SHARES>
__device__ __noinline__ void pattn_row(const PattnP& P, int t, int h, int v0, KeyTiles tiles, int share) {
  constexpr int CL = VN / 4;           // columns per lane
  const int lane = threadIdx.x & 31, g = h / (P.H / P.G), pos = P.pos0 + t, lo = mask_first(P.mask, P.span, pos), last = P.nk + pos - P.first;
  const float* q = P.q + (size_t)t * P.ldq + (size_t)h * P.D;
  const size_t kpart = (size_t)P.G * P.Lk * P.Dp, vpart = (size_t)P.G * P.Lk * P.Vp;
  float m = -1e30f, l = 0.f, acc[CL];
#pragma unroll
  for (int k = 0; k < CL; k++) acc[k] = 0.f;
  for (int i = tiles.begin; i < tiles.end && !isnan(l); i++) {
    const int j0 = tile_key(tiles, i, KT), v = j0 + lane, p = v < P.nk ? v : P.first + v - P.nk;
    const bool ok = lane < KT && v <= last && (p < P.mods.keep || p >= lo);
    if (!__any_sync(0xffffffffu, ok)) continue;
    float s = 0.f;
    if (ok) {
      const __nv_bfloat16* kr = P.kb + ((size_t)g * P.Lk + v) * P.Dp;
      for (int d = 0; d < P.D; d++) s = fmaf(PARTS == 1 ? __bfloat162float(__float2bfloat16_rn(q[d])) : q[d], joined<PARTS>(kr + d, kpart), s);
      s = mod_score(P.mods, s * P.scale, pos - p, h, P.H);
    }
    s = ok ? s : -1e30f;
    const float m_new = fmaxf(m, warp_max(s)), c = expf(m - m_new), pr = ok ? expf(s - m_new) : 0.f;
    l = l * c + warp_sum(pr);
    m = m_new;
#pragma unroll
    for (int k = 0; k < CL; k++) acc[k] *= c;
    for (int jj = 0; jj < KT; jj++) {
      const float pj = __shfl_sync(0xffffffffu, pr, jj);
      if (pj == 0.f) continue;
      const __nv_bfloat16* vr = P.vb + ((size_t)g * P.Lk + j0 + jj) * P.Vp + v0 + lane;
#pragma unroll
      for (int k = 0; k < CL; k++) acc[k] = fmaf(pj, joined<PARTS>(vr + 32 * k, vpart), acc[k]);
    }
  }
  float f = 1.f;
  if (P.mods.sink && share == 0) {
    const float sk = P.mods.sink[h], m_new = fmaxf(m, sk);
    f = expf(m - m_new);
    l = l * f + expf(sk - m_new);
    m = m_new;
  }
  const float inv = f / l * P.alpha;
  float* pp = SHARES ? P.part + (((size_t)t * P.H + h) * P.NS + share) * (P.V + 2) : nullptr;
  if (SHARES && v0 == 0 && lane == 0) { pp[0] = m; pp[1] = l; }
#pragma unroll
  for (int k = 0; k < CL; k++) {
    const int c = v0 + lane + 32 * k;
    if (c >= P.V) continue;
    if (SHARES) { pp[2 + c] = acc[k] * f; continue; }
    const float gt = P.gate ? sigmoid_f(P.gate[(size_t)t * P.ld_gate + (P.gate_head ? (size_t)h : (size_t)h * P.V + c)]) : 1.f;
    P.out[(size_t)t * P.ld_out + (size_t)h * P.V + c] = acc[k] * inv * gt;
  }
}

// VN: 8-column groups of values in a CTA (blockIdx.z picks the columns and, with SHARES, the share of the keys: a form of its own, prompts that fill the chip ran 3 % longer on one for both)
template <int PARTS, int VN, int NK, bool SHARES>
__global__ void __launch_bounds__(256, 1) pattn(const __grid_constant__ PattnP P) {
  constexpr int KT = NK * 8;                                           // keys of a tile
  extern __shared__ __align__(16) unsigned char pa_raw[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nthr = blockDim.x, BM = nthr / 2;
  const int Dp = P.Dp, pq = Dp + 8;
  constexpr int pvt = VN * 8 + 8;                                      // row pitches (ldmatrix rows on distinct banks)
  const uint32_t qs = smem_u32(pa_raw), qpart = (uint32_t)(BM * pq * 2);
  const uint32_t kpart = (uint32_t)(KT * pq * 2), vpart = (uint32_t)(KT * pvt * 2), buf = PARTS * (kpart + vpart);
  const uint32_t ks0 = qs + PARTS * qpart;
  const int qb = (int)gridDim.y - 1 - (int)blockIdx.y, q0 = qb * BM;   // late queries, which see most keys, first for every head
  const int zc = SHARES ? (int)gridDim.z / P.NS : 1, share = SHARES ? (int)blockIdx.z / zc : 0;
  const int h = blockIdx.x, g = h / (P.H / P.G), v0 = ((int)blockIdx.z - share * zc) * VN * 8;
  grid_enter();
  // query rows, split
  for (int e = threadIdx.x; e < BM * (Dp / 4); e += nthr) {
    const int r = e / (Dp / 4), c = (e - r * (Dp / 4)) * 4;
    __nv_bfloat16 s[4][PARTS];
#pragma unroll
    for (int u = 0; u < 4; u++) split_bf16<PARTS>(q0 + r < P.T && c + u < P.D ? P.q[(size_t)(q0 + r) * P.ldq + (size_t)h * P.D + c + u] : 0.f, s[u]);
#pragma unroll
    for (int i = 0; i < PARTS; i++) {
      __nv_bfloat162 lo, hi;
      lo.x = s[0][i]; lo.y = s[1][i]; hi.x = s[2][i]; hi.y = s[3][i];
      *reinterpret_cast<uint2*>(pa_raw + i * qpart + (size_t)(r * pq + c) * 2) = make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
    }
  }
  const KeyTiles tiles = key_tiles(P, q0, BM, KT, share, SHARES ? P.NS : 1);
  const int chunks = Dp / 8 + VN;
  auto fetch = [&](int i) {   // a warp copies rows (part, key) warp, warp + warps, ..: a lane per 16 bytes of the key row and the value row
    const int key0 = tile_key(tiles, i, KT);
    const uint32_t kd = ks0 + (uint32_t)(i & 1) * buf, vd = kd + PARTS * kpart;
    for (int r = warp; r < PARTS * KT; r += nthr >> 5) {
      const int part = r / KT, j = r - part * KT, v = key0 + j;
      const bool in = v < P.Lk;
      const size_t row = ((size_t)part * P.G + g) * P.Lk + (in ? v : 0);
      for (int c = lane; c < chunks; c += 32) {
        const bool key = c < chunks - VN;
        const int cc = (key ? c : c - (chunks - VN)) * 8;
        const __nv_bfloat16* src = key ? P.kb + row * Dp + cc : P.vb + row * P.Vp + v0 + cc;
        const uint32_t dst = key ? kd + part * kpart + (uint32_t)(j * pq + cc) * 2 : vd + part * vpart + (uint32_t)(j * pvt + cc) * 2;
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(in ? 16 : 0) : "memory");
      }
    }
    cp_async_commit();
  };
  if (tiles.begin < tiles.end) fetch(tiles.begin);
  const int row_lo = q0 + warp * 16 + (lane >> 2);                      // this thread's query rows: row_lo and row_lo + 8
  const int first_lo[2] = {mask_first(P.mask, P.span, P.pos0 + row_lo), mask_first(P.mask, P.span, P.pos0 + row_lo + 8)};
  // a tile whose keys every query of the warp sees needs no mask
  const int w_pos = P.pos0 + q0 + warp * 16, w_lo = mask_first(P.mask, P.span, w_pos + 15);
  const bool capped = P.mods.cap > 0.f;
  const float s_mul = capped ? P.scale / P.mods.cap : P.scale;
  float o[VN][4], m[2] = {-1e30f, -1e30f}, l[2] = {0.f, 0.f};
#pragma unroll
  for (int n = 0; n < VN; n++)
#pragma unroll
    for (int i = 0; i < 4; i++) o[n][i] = 0.f;
  const uint32_t qa = qs + (uint32_t)((warp * 16 + (lane & 7) + ((lane >> 3) & 1) * 8) * pq + (lane >> 4) * 8) * 2;
  for (int it = tiles.begin; it < tiles.end; it++) {
    cp_async_wait<0>();
    __syncthreads();                                                     // tile it is there; everyone is through tile it - 1
    if (it + 1 < tiles.end) fetch(it + 1);
    const uint32_t kt = ks0 + (uint32_t)(it & 1) * buf, vt = kt + PARTS * kpart;
    float s[NK][4];
#pragma unroll
    for (int n = 0; n < NK; n++)
#pragma unroll
      for (int i = 0; i < 4; i++) s[n][i] = 0.f;
    const uint32_t kaddr = kt + (uint32_t)(((lane & 7) + (lane >> 4) * 8) * pq + ((lane >> 3) & 1) * 8) * 2;
#pragma unroll 2
    for (int k = 0; k < Dp; k += 16) {
      uint32_t a[PARTS][4];
#pragma unroll
      for (int i = 0; i < PARTS; i++) ldmatrix_x4_at(a[i], qa + i * qpart + k * 2);
      mma_parts<PARTS, NK>(s, a, [&](int part, uint32_t (&bb)[NK][2]) {
#pragma unroll
        for (int np = 0; np < NK / 2; np++) {
          uint32_t r[4];
          ldmatrix_x4_at(r, kaddr + part * kpart + (uint32_t)(np * 16 * pq + k) * 2);
          bb[2 * np][0] = r[0]; bb[2 * np][1] = r[1]; bb[2 * np + 1][0] = r[2]; bb[2 * np + 1][1] = r[3];
        }
      });
    }
    // scale, cap, bias and mask: rows row_lo (entries 0, 1) and row_lo + 8 (entries 2, 3); keys n * 8 + (lane & 3) * 2 + {0, 1}
    const int key0 = tile_key(tiles, it, KT);
#pragma unroll
    for (int n = 0; n < NK; n++)
#pragma unroll
      for (int i = 0; i < 4; i++) s[n][i] *= s_mul;
    if (capped) {
#pragma unroll
      for (int n = 0; n < NK; n++)
#pragma unroll
        for (int i = 0; i < 4; i++) s[n][i] = P.mods.cap * tanhf(s[n][i]);
    }
    const int p_lo = P.first + key0 - P.nk, p_hi = p_lo + KT - 1;        // positions of a tile behind the kept rows
    if (P.mods.rel || key0 < P.nk || p_hi > w_pos || p_lo < w_lo || key0 + KT > P.Lk) {
#pragma unroll
      for (int n = 0; n < NK; n++)
#pragma unroll
        for (int i = 0; i < 4; i++) {
          const int pos = P.pos0 + row_lo + (i >> 1) * 8, v = key0 + n * 8 + (lane & 3) * 2 + (i & 1), p = v < P.nk ? v : P.first + v - P.nk;
          const bool ok = v < P.Lk && p <= pos && (p < P.mods.keep || p >= first_lo[i >> 1]);
          if (ok && P.mods.rel) s[n][i] += P.mods.rel[(size_t)P.mods.bucket[min(pos - p, P.mods.rel_max)] * P.H + h];
          if (!ok) s[n][i] = -INFINITY;
        }
    }
    float c[2], sum[2] = {0.f, 0.f};
#pragma unroll
    for (int r = 0; r < 2; r++) {
      float mx = fmaxf(s[0][2 * r], s[0][2 * r + 1]);
#pragma unroll
      for (int n = 1; n < NK; n++) mx = fmaxf(mx, fmaxf(s[n][2 * r], s[n][2 * r + 1]));
      mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
      mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
      const float m_new = fmaxf(m[r], mx);
      c[r] = expf(m[r] - m_new);
      m[r] = m_new;
    }
#pragma unroll
    for (int n = 0; n < NK; n++)
#pragma unroll
      for (int i = 0; i < 4; i++) { s[n][i] = expf(s[n][i] - m[i >> 1]); sum[i >> 1] += s[n][i]; }   // (a key out of sight: e^-inf = 0)
#pragma unroll
    for (int r = 0; r < 2; r++) {
      sum[r] += __shfl_xor_sync(0xffffffffu, sum[r], 1);
      sum[r] += __shfl_xor_sync(0xffffffffu, sum[r], 2);
      l[r] = fmaf(l[r], c[r], sum[r]);
    }
    if (__any_sync(0xffffffffu, c[0] != 1.f || c[1] != 1.f)) {
#pragma unroll
      for (int n = 0; n < VN; n++) { o[n][0] *= c[0]; o[n][1] *= c[0]; o[n][2] *= c[1]; o[n][3] *= c[1]; }
    }
    const uint32_t vaddr = vt + (uint32_t)(((lane & 7) + ((lane >> 3) & 1) * 8) * pvt + (lane >> 4) * 8) * 2;
#pragma unroll
    for (int kk = 0; kk < NK / 2; kk++) {
      uint32_t a[PARTS][4];
#pragma unroll
      for (int q = 0; q < 4; q++) {   // fragment registers: {row, keys 0-7}, {row + 8, keys 0-7}, {row, keys 8-15}, {row + 8, keys 8-15}
        const int n = 2 * kk + (q >> 1), i0 = (q & 1) * 2;
        uint32_t x[PARTS];
        split_pair<PARTS>(s[n][i0], s[n][i0 + 1], x);
#pragma unroll
        for (int i = 0; i < PARTS; i++) a[i][q] = x[i];
      }
#pragma unroll
      for (int n = 0; n < VN; n += 4)
        mma_parts<PARTS, 4>(o + n, a, [&](int part, uint32_t (&bb)[4][2]) {
#pragma unroll
          for (int np = 0; np < 2; np++) {
            uint32_t r[4];
            ldmatrix_x4_trans(r, vaddr + part * vpart + (uint32_t)(kk * 16 * pvt + (n + 2 * np) * 8) * 2);
            bb[2 * np][0] = r[0]; bb[2 * np][1] = r[1]; bb[2 * np + 1][0] = r[2]; bb[2 * np + 1][1] = r[3];
          }
        });
    }
  }
  uint32_t again = 0;   // rows of the warp whose result is not finite
#pragma unroll
  for (int r = 0; r < 2; r++) {
    float any = l[r];   // (finite as long as everything is)
#pragma unroll
    for (int n = 0; n < VN; n++) any = fmaf(0.f, o[n][2 * r], fmaf(0.f, o[n][2 * r + 1], any));
    uint32_t lanes = __ballot_sync(0xffffffffu, !isfinite(any));
    lanes |= lanes >> 1; lanes |= lanes >> 2;
#pragma unroll
    for (int i = 0; i < 8; i++) again |= ((lanes >> (4 * i)) & 1u) << (i + 8 * r);
  }
#pragma unroll
  for (int r = 0; r < 2; r++) {
    const int t = row_lo + r * 8;
    if (t >= P.T || ((again >> ((lane >> 2) + 8 * r)) & 1u)) continue;
    float f = 1.f;
    if (P.mods.sink && share == 0) {   // a key with a zero value vector
      const float sk = P.mods.sink[h], m_new = fmaxf(m[r], sk);
      f = expf(m[r] - m_new);
      l[r] = l[r] * f + expf(sk - m_new);
      m[r] = m_new;
    }
    const float inv = f / l[r] * P.alpha;
    float* pp = SHARES ? P.part + (((size_t)t * P.H + h) * P.NS + share) * (P.V + 2) : nullptr;
    if (SHARES && v0 == 0 && (lane & 3) == 0) { pp[0] = m[r]; pp[1] = l[r]; }
#pragma unroll
    for (int n = 0; n < VN; n++)
#pragma unroll
      for (int i = 0; i < 2; i++) {
        const int c = v0 + n * 8 + (lane & 3) * 2 + i;
        if (c >= P.V) continue;
        if (SHARES) { pp[2 + c] = o[n][r * 2 + i] * f; continue; }
        const float gt = P.gate ? sigmoid_f(P.gate[(size_t)t * P.ld_gate + (P.gate_head ? (size_t)h : (size_t)h * P.V + c)]) : 1.f;
        P.out[(size_t)t * P.ld_out + (size_t)h * P.V + c] = o[n][r * 2 + i] * inv * gt;
      }
  }
  for (; again; again &= again - 1) {
    const int t = q0 + warp * 16 + __ffs(again) - 1;
    if (t < P.T) pattn_row<PARTS, VN, KT, SHARES>(P, t, h, v0, tiles, share);
  }
}

}  // namespace hy
}  // namespace dsk

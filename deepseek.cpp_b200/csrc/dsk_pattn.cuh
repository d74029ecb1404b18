// dsk_pattn.cuh — softmax attention of portions (layer-list models without mixing of the heads' scores) in one kernel: scores, mask, softmax and
// the weighted values of a block of queries against all of their keys, nothing of it in global memory.
//
// Products run on mma.sync (bf16 x bf16 -> fp32, m16n8k16).  PARTS = 3 (designs with 32-bit scores and weights): every fp32 operand is the sum
// of three bf16 numbers (8 + 8 + 8 bits of mantissa, fp32's exponent range), and a product takes the six pairs whose order is at least 2^-16 of
// the leading one; what is left out is below an fp32 rounding.  The sum over 16 elements comes out of the tensor core and is added in fp32
// registers (rounded to nearest), so that a sum of n elements sees n / 16 roundings where a chain of FMAs sees n: the error against 64 bits is not
// larger than that of the fp32 products it replaces.  PARTS = 1: operands rounded to bf16 (latent attention of bf16 models, whose products
// always took them so).
// pattn_pack splits the visible keys and values once per step; a CTA (16 query rows per warp) streams them in tiles of 32 through two buffers
// (cp.async).  Bound: the tensor pipe at six products per element, then shared-memory reads of the query fragments.  Before, a block of 256
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
    if (i + 1 < PARTS) x = isfinite(x) ? x - __bfloat162float(o[i]) : 0.f;   // exact: the rest has fewer bits (an infinity stays in the first part)
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
  int T, H, G, D, Dp, V, Vp, ldq, ld_out, ld_gate, gate_head, Lk, nk, first, pos0, mask, span;
  float scale, alpha;
  ScoreMods mods;
};

constexpr int kPattnKeys = 32;
__host__ __device__ inline size_t pattn_smem(int parts, int warps, int Dp, int VN) {
  return (size_t)parts * 2 * ((size_t)warps * 16 * (Dp + 8) + 2 * kPattnKeys * ((Dp + 8) + (VN * 8 + 8)));
}

__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void ldmatrix_x4_at(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
// acc += sum over 16 elements of a b: the six leading pairs of the operands' parts, small ones first, joined in the tensor core
template <int PARTS>
__device__ __forceinline__ void mma_parts(float (&acc)[4], const uint32_t (&a)[PARTS][4], const uint32_t (&b)[PARTS][2]) {
  if constexpr (PARTS == 1) {
    mma_bf16_16816(acc, a[0][0], a[0][1], a[0][2], a[0][3], b[0][0], b[0][1]);
  } else {
    float t[4] = {0.f, 0.f, 0.f, 0.f};
    mma_bf16_16816(t, a[2][0], a[2][1], a[2][2], a[2][3], b[0][0], b[0][1]);
    mma_bf16_16816(t, a[0][0], a[0][1], a[0][2], a[0][3], b[2][0], b[2][1]);
    mma_bf16_16816(t, a[1][0], a[1][1], a[1][2], a[1][3], b[1][0], b[1][1]);
    mma_bf16_16816(t, a[1][0], a[1][1], a[1][2], a[1][3], b[0][0], b[0][1]);
    mma_bf16_16816(t, a[0][0], a[0][1], a[0][2], a[0][3], b[1][0], b[1][1]);
    mma_bf16_16816(t, a[0][0], a[0][1], a[0][2], a[0][3], b[0][0], b[0][1]);
#pragma unroll
    for (int i = 0; i < 4; i++) acc[i] += t[i];
  }
}

template <int PARTS, int VN>   // VN: 8-column groups of values in a CTA (blockIdx.z picks the columns)
__global__ void __launch_bounds__(256, 1) pattn(const PattnP P) {
  extern __shared__ __align__(16) unsigned char pa_raw[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nthr = blockDim.x, BM = nthr / 2;
  const int Dp = P.Dp, pq = Dp + 8, pvt = VN * 8 + 8;                 // row pitches (ldmatrix rows on distinct banks)
  const uint32_t qs = smem_u32(pa_raw), qpart = (uint32_t)(BM * pq * 2);
  const uint32_t kpart = (uint32_t)(kPattnKeys * pq * 2), vpart = (uint32_t)(kPattnKeys * pvt * 2), buf = PARTS * (kpart + vpart);
  const uint32_t ks0 = qs + PARTS * qpart;
  const int qb = (int)gridDim.x - 1 - (int)blockIdx.x, q0 = qb * BM;   // late queries, which see most keys, first
  const int h = blockIdx.y, g = h / (P.H / P.G), v0 = (int)blockIdx.z * VN * 8;
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
  // tiles this CTA meets: those of the kept keys, then from the first key of its first query to its last query
  const int last = min(P.T, q0 + BM) - 1;
  const int lo_v = P.nk + mask_first(P.mask, P.span, P.pos0 + q0) - P.first, hi_v = P.nk + P.pos0 + last - P.first;
  // (kept positions are keys 0 .. keep - 1 whether or not they lie in the range)
  const int kept = (min(P.mods.keep, hi_v + 1) + kPattnKeys - 1) / kPattnKeys, t0 = max(kept, lo_v / kPattnKeys), n_tiles = kept + max(0, hi_v / kPattnKeys - t0 + 1);
  auto tile_key = [&](int i) { return (i < kept ? i : t0 + i - kept) * kPattnKeys; };
  auto fetch = [&](int i) {
    const int key0 = tile_key(i);
    const uint32_t kd = ks0 + (uint32_t)(i & 1) * buf, vd = kd + PARTS * kpart;
    const int kc = Dp / 8;
    for (int e = threadIdx.x; e < PARTS * kPattnKeys * (kc + VN); e += nthr) {
      const bool key = e < PARTS * kPattnKeys * kc;
      const int q = key ? e : e - PARTS * kPattnKeys * kc, per = key ? kc : VN, r = q / per, c = (q - r * per) * 8, part = r / kPattnKeys, j = r - part * kPattnKeys;
      const int v = key0 + j;
      const bool in = v < P.Lk;
      const size_t row = ((size_t)part * P.G + g) * P.Lk + (in ? v : 0);
      const __nv_bfloat16* src = key ? P.kb + row * Dp + c : P.vb + row * P.Vp + v0 + c;
      const uint32_t dst = key ? kd + part * kpart + (uint32_t)(j * pq + c) * 2 : vd + part * vpart + (uint32_t)(j * pvt + c) * 2;
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(in ? 16 : 0) : "memory");
    }
    cp_async_commit();
  };
  if (n_tiles > 0) fetch(0);
  const int row_lo = q0 + warp * 16 + (lane >> 2);                      // this thread's query rows: row_lo and row_lo + 8
  const int first_lo[2] = {mask_first(P.mask, P.span, P.pos0 + row_lo), mask_first(P.mask, P.span, P.pos0 + row_lo + 8)};
  float o[VN][4], m[2] = {-1e30f, -1e30f}, l[2] = {0.f, 0.f};
#pragma unroll
  for (int n = 0; n < VN; n++)
#pragma unroll
    for (int i = 0; i < 4; i++) o[n][i] = 0.f;
  const uint32_t qa = qs + (uint32_t)((warp * 16 + (lane & 7) + ((lane >> 3) & 1) * 8) * pq + (lane >> 4) * 8) * 2;
  for (int it = 0; it < n_tiles; it++) {
    cp_async_wait<0>();
    __syncthreads();                                                     // tile it is there; everyone is through tile it - 1
    if (it + 1 < n_tiles) fetch(it + 1);
    const uint32_t kt = ks0 + (uint32_t)(it & 1) * buf, vt = kt + PARTS * kpart;
    float s[4][4];
#pragma unroll
    for (int n = 0; n < 4; n++)
#pragma unroll
      for (int i = 0; i < 4; i++) s[n][i] = 0.f;
    const uint32_t kaddr = kt + (uint32_t)(((lane & 7) + (lane >> 4) * 8) * pq + ((lane >> 3) & 1) * 8) * 2;
    for (int k = 0; k < Dp; k += 16) {
      uint32_t a[PARTS][4];
#pragma unroll
      for (int i = 0; i < PARTS; i++) ldmatrix_x4_at(a[i], qa + i * qpart + k * 2);
#pragma unroll
      for (int np = 0; np < 2; np++) {
        uint32_t b0[PARTS][2], b1[PARTS][2];
#pragma unroll
        for (int i = 0; i < PARTS; i++) {
          uint32_t r[4];
          ldmatrix_x4_at(r, kaddr + i * kpart + (uint32_t)(np * 16 * pq + k) * 2);
          b0[i][0] = r[0]; b0[i][1] = r[1]; b1[i][0] = r[2]; b1[i][1] = r[3];
        }
        mma_parts<PARTS>(s[2 * np], a, b0);
        mma_parts<PARTS>(s[2 * np + 1], a, b1);
      }
    }
    // mask and softmax: rows row_lo (entries 0, 1) and row_lo + 8 (entries 2, 3); keys n * 8 + (lane & 3) * 2 + {0, 1}
    const int key0 = tile_key(it);
    float mx[2] = {-1e30f, -1e30f};
#pragma unroll
    for (int n = 0; n < 4; n++)
#pragma unroll
      for (int i = 0; i < 4; i++) {
        const int t = row_lo + (i >> 1) * 8, pos = P.pos0 + t, v = key0 + n * 8 + (lane & 3) * 2 + (i & 1), p = v < P.nk ? v : P.first + v - P.nk;
        const bool ok = v < P.Lk && p <= pos && (p < P.mods.keep || p >= first_lo[i >> 1]);
        s[n][i] = ok ? mod_score(P.mods, s[n][i] * P.scale, pos - p, h, P.H) : -INFINITY;
        mx[i >> 1] = fmaxf(mx[i >> 1], s[n][i]);
      }
    float c[2];
#pragma unroll
    for (int r = 0; r < 2; r++) {
      mx[r] = fmaxf(mx[r], __shfl_xor_sync(0xffffffffu, mx[r], 1));
      mx[r] = fmaxf(mx[r], __shfl_xor_sync(0xffffffffu, mx[r], 2));
      const float m_new = fmaxf(m[r], mx[r]);
      c[r] = expf(m[r] - m_new);
      m[r] = m_new;
    }
    float sum[2] = {0.f, 0.f};
#pragma unroll
    for (int n = 0; n < 4; n++)
#pragma unroll
      for (int i = 0; i < 4; i++) { s[n][i] = expf(s[n][i] - m[i >> 1]); sum[i >> 1] += s[n][i]; }   // (a key out of sight: e^-inf = 0)
#pragma unroll
    for (int r = 0; r < 2; r++) {
      sum[r] += __shfl_xor_sync(0xffffffffu, sum[r], 1);
      sum[r] += __shfl_xor_sync(0xffffffffu, sum[r], 2);
      l[r] = fmaf(l[r], c[r], sum[r]);
    }
#pragma unroll
    for (int n = 0; n < VN; n++) { o[n][0] *= c[0]; o[n][1] *= c[0]; o[n][2] *= c[1]; o[n][3] *= c[1]; }
    const uint32_t vaddr = vt + (uint32_t)(((lane & 7) + ((lane >> 3) & 1) * 8) * pvt + (lane >> 4) * 8) * 2;
#pragma unroll
    for (int kk = 0; kk < 2; kk++) {
      uint32_t a[PARTS][4];
#pragma unroll
      for (int q = 0; q < 4; q++) {   // fragment registers: {row, keys 0-7}, {row + 8, keys 0-7}, {row, keys 8-15}, {row + 8, keys 8-15}
        const int n = 2 * kk + (q >> 1), i0 = (q & 1) * 2;
        __nv_bfloat16 x0[PARTS], x1[PARTS];
        split_bf16<PARTS>(s[n][i0], x0);
        split_bf16<PARTS>(s[n][i0 + 1], x1);
#pragma unroll
        for (int i = 0; i < PARTS; i++) { __nv_bfloat162 pr; pr.x = x0[i]; pr.y = x1[i]; a[i][q] = *reinterpret_cast<const uint32_t*>(&pr); }
      }
#pragma unroll
      for (int n = 0; n < VN; n += 2) {
        uint32_t b0[PARTS][2], b1[PARTS][2];
#pragma unroll
        for (int i = 0; i < PARTS; i++) {
          uint32_t r[4];
          ldmatrix_x4_trans(r, vaddr + i * vpart + (uint32_t)(kk * 16 * pvt + n * 8) * 2);
          b0[i][0] = r[0]; b0[i][1] = r[1]; b1[i][0] = r[2]; b1[i][1] = r[3];
        }
        mma_parts<PARTS>(o[n], a, b0);
        mma_parts<PARTS>(o[n + 1], a, b1);
      }
    }
  }
#pragma unroll
  for (int r = 0; r < 2; r++) {
    const int t = row_lo + r * 8;
    if (t >= P.T) continue;
    float f = 1.f;
    if (P.mods.sink) {   // a key with a zero value vector
      const float sk = P.mods.sink[h], m_new = fmaxf(m[r], sk);
      f = expf(m[r] - m_new);
      l[r] = l[r] * f + expf(sk - m_new);
    }
    const float inv = f / l[r] * P.alpha;
#pragma unroll
    for (int n = 0; n < VN; n++)
#pragma unroll
      for (int i = 0; i < 2; i++) {
        const int c = v0 + n * 8 + (lane & 3) * 2 + i;
        if (c >= P.V) continue;
        const float gt = P.gate ? sigmoid_f(P.gate[(size_t)t * P.ld_gate + (P.gate_head ? (size_t)h : (size_t)h * P.V + c)]) : 1.f;
        P.out[(size_t)t * P.ld_out + (size_t)h * P.V + c] = o[n][r * 2 + i] * inv * gt;
      }
  }
}

}  // namespace hy
}  // namespace dsk

// dsk_linmma.cuh — the walk over the blocks of a portion (lin_scan's plain and mLSTM forms: o_j = G_j S0^T q_j + sum_i M_ji v_i, S <- G_end S0 + sum_j E_j k_j v_j^T) on tensor cores,
// in segments that run at once.
//
// Two warps have 16 value channels of a head, half of the key entries each, with their state in registers, transposed: S^T [16 channels][N / 2] as accumulators of mma.sync m16n8k16, which are the left operand of
// S^T q once they are split, without a shuffle.  Operands in three bf16 parts, six products, sums of 16 values joined in fp32 registers (mma_parts).  Four warps of a CTA stage the next
// block meanwhile: q scaled by G and k by E, split, M and v split.
// Segments: the state is linear in what came before, so that every segment but the last is first walked from zero for its end state alone (mode 0), and then all are walked
// from their true starts, which each works out from those (mode 1).
// Bound: the chain of a block (products of a sum wait for one another, then a barrier) and the issue slots of its warps: 204 products and 64 numbers into parts.  Counters, 64 heads of 64
// channels, 1024 tokens, two segments, walked for results: issue slots 44 % and tensor pipe 41 % of an SM's active cycles, DRAM 5 %.  FMAs of the whole state
// by every token, with their operands from shared memory, bound lin_scan: 2048 tokens, 64 heads of 64 channels and 128 entries 312 us, here 222 in two segments and 257 in one walk;
// 16 heads of 128 channels 186, 116 in four and 255 in one, where heads are few the segments are the gain; with the matrix memory's normaliser, a column in a third CTA a head, 188 and 152
// (three); 600 tokens, 16 heads of 64 channels and entries 46, 23.  Two blocks of loads ahead instead of one: the same.
// Error against 64 bits 1.7e-7 of the largest result, lin_scan's 2.8e-7.  lin_scan stays for other sizes and for short steps, where the two launches and the first split cost more.
// Values that are not finite: results that come out so are summed again from the numbers, as lin_scan sums them, and blocks with such keys or values update the state with FMAs.
#pragma once

#include "dsk_linattn.cuh"
#include "dsk_pattn.cuh"

namespace dsk {
namespace hy {

constexpr int kLmGroups = 4, kLmCh = 16 * kLmGroups, kLmStage = 4, kLmThreads = 32 * (2 * kLmGroups + kLmStage), kLmSegs = 8;   // channels of a CTA, threads, segments at most
template <int NT> struct LinMma {
  static constexpr int N = 8 * NT, NP = N + 8, VP = kLmCh + 8, MP = kLinBlk + 8;
  static constexpr int QB = kLinBlk * NP * 2, VB = kLinBlk * VP * 2, MB = kLinBlk * MP * 2;       // bytes of a part
  static constexpr int BUF = 3 * (2 * QB + VB + MB), SP = N / 2 + 4;
  static constexpr int SMEM = 2 * BUF + 2 * kLmGroups * 16 * SP * 4 + 2 * kLmGroups * 32 * 8 * 4;   // (two blocks, the state of rare second looks, halves of results)
};
struct LinMmaP {
  const float *q, *k, *v, *rec;
  float *state, *out, *nst, *den, *seg;   // seg: [slot][head][channel group][fragment][lane] initial state (slot 0) and end states of segments walked from zero; then [segment][head] decays
  int ldq, hs, rep, ldv, ldo, T, H, P, sn, sp, groups, nseg, per, mode;   // per: blocks of a segment
};
// floats of seg
__host__ __device__ inline size_t lin_mma_floats(int H, int groups, int N, int nseg) { return (size_t)nseg * H * groups * 16 * N + (size_t)nseg * H; }

// mma_parts<3, 2> of two left operands at once (a sum's products wait for one another: four sums are under way)
template <typename Load0, typename Load1>
__device__ __forceinline__ void mma_parts_twice(float (*acc)[4], const uint32_t (&a0)[3][4], const uint32_t (&a1)[3][4], Load0 load0, Load1 load1) {
  uint32_t b0[2][2], b1[2][2];
  float t[4][4];
  auto step = [&](int p) {
#pragma unroll
    for (int n = 0; n < 2; n++) {
      mma_bf16_16816(t[n], a0[p][0], a0[p][1], a0[p][2], a0[p][3], b0[n][0], b0[n][1]);
      mma_bf16_16816(t[2 + n], a1[p][0], a1[p][1], a1[p][2], a1[p][3], b1[n][0], b1[n][1]);
    }
  };
  load0(2, b0); load1(2, b1);
#pragma unroll
  for (int n = 0; n < 2; n++) { mma_bf16_first(t[n], a0[0], b0[n]); mma_bf16_first(t[2 + n], a1[0], b1[n]); }
  load0(1, b0); load1(1, b1);
  step(1); step(0);
  load0(0, b0); load1(0, b1);
  step(2); step(1); step(0);
#pragma unroll
  for (int n = 0; n < 2; n++)
#pragma unroll
    for (int i = 0; i < 4; i++) acc[n][i] += t[n][i] + t[2 + n][i];
}

template <int NT>
__global__ void __launch_bounds__(kLmThreads, 1) lin_mma(const LinMmaP P) {
  using L = LinMma<NT>;
  constexpr int N = L::N, C = kLinBlk;
  extern __shared__ __align__(16) unsigned char lm_raw[];
  __shared__ int bad[2];                                     // block whose keys or values do not go into parts
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, h = blockIdx.x, hk = h / P.rep, ch0 = (int)blockIdx.y * kLmCh, seg = blockIdx.z;
  const int nb = (P.T + C - 1) / C, b0 = seg * P.per, b1 = min(nb, b0 + P.per);
  const bool outputs = P.mode == 1;
  if (threadIdx.x < 2) bad[threadIdx.x] = -1;
  __syncthreads();                                           // (the staging warps mark the first block ahead of the barrier that all meet on)
  grid_enter();
  if (warp >= 2 * kLmGroups) {
    const int st = threadIdx.x - 64 * kLmGroups;
    constexpr int QU = NT / 4;
    struct Regs { float4 rq[QU], rk[QU], rv[2], rm; float sg[QU], se[QU]; } one, two;   // blocks of even and odd number: a block's loads are under way while the one ahead is split
    auto load = [&](int b, Regs& r) {
      const int t0 = b * C, nt = min(C, P.T - t0);
      const float* rc = P.rec + ((size_t)b * P.H + h) * kRecFloats;
      const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int u = 0; u < QU; u++) {
        const int e = st + 128 * u, j = e / (N / 4), c = (e - j * (N / 4)) * 4;
        const size_t at = (size_t)(t0 + j) * P.ldq + (size_t)hk * P.hs + c;
        r.rk[u] = j < nt ? *reinterpret_cast<const float4*>(P.k + at) : zero;
        r.se[u] = rc[kRecE + j];
        if (outputs) { r.rq[u] = j < nt ? *reinterpret_cast<const float4*>(P.q + at) : zero; r.sg[u] = rc[kRecG + j]; }
      }
#pragma unroll
      for (int u = 0; u < 2; u++) {
        const int e = st + 128 * u, j = e >> 4, c = ch0 + (e & 15) * 4;
        r.rv[u] = zero;
        if (j < nt && c < P.P) r.rv[u] = *reinterpret_cast<const float4*>(P.v + (size_t)(t0 + j) * P.ldv + (size_t)h * P.P + c);
        else if (j < nt && P.nst && c == P.P) r.rv[u].x = 1.f;
      }
      if (outputs && st < 64) r.rm = *reinterpret_cast<const float4*>(rc + kRecM + st * 4);
    };
    auto put = [&](unsigned char* dst, int part, const float4& x) {
      uint32_t a[3], b[3];
      split_pair<3>(x.x, x.y, a);
      split_pair<3>(x.z, x.w, b);
#pragma unroll
      for (int i = 0; i < 3; i++) *reinterpret_cast<uint2*>(dst + i * part) = make_uint2(a[i], b[i]);
    };
    auto fits = [](const float4& x) { return fabsf(x.x) <= 3e38f && fabsf(x.y) <= 3e38f && fabsf(x.z) <= 3e38f && fabsf(x.w) <= 3e38f; };
    auto store = [&](int b, const Regs& r) {
      unsigned char* buf = lm_raw + (b & 1) * L::BUF;
      bool ok = true;
#pragma unroll
      for (int u = 0; u < QU; u++) {
        const int e = st + 128 * u, j = e / (N / 4), c = (e - j * (N / 4)) * 4;
        const float4 x = make_float4(r.rk[u].x * r.se[u], r.rk[u].y * r.se[u], r.rk[u].z * r.se[u], r.rk[u].w * r.se[u]);
        ok = ok && fits(x);                                  // (E of a key may be e^40)
        put(buf + 3 * L::QB + (j * L::NP + c) * 2, L::QB, x);
        if (outputs) put(buf + (j * L::NP + c) * 2, L::QB, make_float4(r.rq[u].x * r.sg[u], r.rq[u].y * r.sg[u], r.rq[u].z * r.sg[u], r.rq[u].w * r.sg[u]));
      }
#pragma unroll
      for (int u = 0; u < 2; u++) {
        const int e = st + 128 * u, j = e >> 4, c = (e & 15) * 4;
        ok = ok && fits(r.rv[u]);
        put(buf + 6 * L::QB + (j * L::VP + c) * 2, L::VB, r.rv[u]);
      }
      if (outputs && st < 64) put(buf + 6 * L::QB + 3 * L::VB + ((st >> 2) * L::MP + (st & 3) * 4) * 2, L::MB, r.rm);
      if (!ok) bad[b & 1] = b;
    };
    if (b0 < b1) load(b0, one);
    if (b0 + 1 < b1) load(b0 + 1, two);
    if (b0 < b1) store(b0, one);
    __syncthreads();
    for (int b = b0; b < b1; b += 2) {
      if (b + 2 < b1) load(b + 2, one);
      if (b + 1 < b1) store(b + 1, two);
      __syncthreads();
      if (b + 1 >= b1) break;
      if (b + 3 < b1) load(b + 3, two);
      if (b + 2 < b1) store(b + 2, one);
      __syncthreads();
    }
    __syncthreads();                                         // (the last block's halves)
    return;
  }
  const int gw = warp % kLmGroups, half = warp / kLmGroups, n0 = half * (N / 2), grp = (int)blockIdx.y * kLmGroups + gw;
  const int c_lo = ch0 + gw * 16 + (lane >> 2);             // this lane's channels c_lo and c_lo + 8, state rows n0 + 8 t + 2 (lane & 3) + {0, 1}
  const bool live = grp < P.groups;
  constexpr int NH = NT / 2;
  float S[NH][4];
  const size_t frag = (size_t)NH * 4 * 32;
  auto slot = [&](int s) { return P.seg + ((((size_t)s * P.H + h) * P.groups + grp) * 2 + half) * frag + lane; };
  const float* decays = P.seg + (size_t)P.nseg * P.H * P.groups * 2 * frag;
  auto from_state = [&](int t, int i) {
    const int n = n0 + 8 * t + 2 * (lane & 3) + (i & 1), c = c_lo + (i >> 1) * 8;
    return c < P.P ? P.state[(size_t)h * N * P.P + (size_t)n * P.sn + (size_t)c * P.sp] : P.nst && c == P.P ? P.nst[(size_t)h * N + n] : 0.f;
  };
#pragma unroll
  for (int t = 0; t < NH; t++)
#pragma unroll
    for (int i = 0; i < 4; i++) {
      S[t][i] = 0.f;
      if (!live) continue;
      if (!outputs) { if (seg == 0) slot(0)[(t * 4 + i) * 32] = from_state(t, i); }         // (kept for the second walk: its last segment writes the state)
      else if (P.nseg == 1) S[t][i] = from_state(t, i);
      else S[t][i] = slot(0)[(t * 4 + i) * 32];
    }
  if (outputs && live)
    for (int s = 0; s < seg; s++) {
      const float g = decays[(size_t)s * P.H + h];
      const float* at = slot(s + 1);
#pragma unroll
      for (int t = 0; t < NH; t++)
#pragma unroll
        for (int i = 0; i < 4; i++) S[t][i] = fmaf(S[t][i], g, at[(t * 4 + i) * 32]);
    }
  float decay = 1.f;
  const uint32_t base = smem_u32(lm_raw);
  float* scratch = reinterpret_cast<float*>(lm_raw + 2 * L::BUF) + warp * 16 * L::SP;
  float* halves = reinterpret_cast<float*>(lm_raw + 2 * L::BUF) + 2 * kLmGroups * 16 * L::SP + gw * 32 * 8 + lane;   // [block & 1][group][8][32]
  float y[2][4];
  // a block's results, joined a block later (the barrier between them is there anyway): the first half's warp stores
  auto finish = [&](int b) {
    const int t0 = b * C, nt = min(C, P.T - t0);
#pragma unroll
    for (int u = 0; u < 2; u++)
#pragma unroll
      for (int i = 0; i < 4; i++) {
        const int j = u * 8 + 2 * (lane & 3) + (i & 1), c = c_lo + (i >> 1) * 8;
        const float r = y[u][i] + halves[(b & 1) * kLmGroups * 32 * 8 + (u * 4 + i) * 32];
        if (j < nt && c < P.P) P.out[(size_t)(t0 + j) * P.ldo + (size_t)h * P.P + c] = r;
        else if (j < nt && P.nst && c == P.P) P.den[(size_t)(t0 + j) * P.H + h] = r;
      }
  };
  __syncthreads();
  for (int b = b0; b < b1; b++) {
    if (live) {
      if (outputs && half == 0 && b > b0) finish(b - 1);
      const int t0 = b * C, nt = min(C, P.T - t0);
      const uint32_t buf = base + (b & 1) * L::BUF, vs = buf + 6 * L::QB, ms = vs + 3 * L::VB;
      const float* rc = P.rec + ((size_t)b * P.H + h) * kRecFloats;
      const float ge = rc[kRecEnd];
      uint32_t av[3][4];                                     // v^T
#pragma unroll
      for (int p = 0; p < 3; p++) ldmatrix_x4_trans(av[p], vs + p * L::VB + (uint32_t)(((lane & 7) + (lane >> 4) * 8) * L::VP + gw * 16 + ((lane >> 3) & 1) * 8) * 2);
      const uint32_t row = (lane & 7) + (lane >> 4) * 8, col = ((lane >> 3) & 1) * 8;         // rows of tokens 0 - 7 and 8 - 15, two groups of eight values
      if (outputs) {
#pragma unroll
        for (int u = 0; u < 2; u++)
#pragma unroll
          for (int i = 0; i < 4; i++) y[u][i] = 0.f;
        if (half) mma_parts<3, 2>(y, av, [&](int part, uint32_t (&bb)[2][2]) {
          uint32_t r[4];
          ldmatrix_x4_at(r, ms + part * L::MB + (row * L::MP + col) * 2);
          bb[0][0] = r[0]; bb[0][1] = r[1]; bb[1][0] = r[2]; bb[1][1] = r[3];
        });
#pragma unroll
        for (int ks = 0; ks < NH / 2; ks += 2) {
          uint32_t a[2][3][4];
#pragma unroll
          for (int w = 0; w < 2; w++)
#pragma unroll
            for (int i = 0; i < 4; i++) {
              uint32_t x[3];
              split_pair<3>(S[2 * (ks + w) + (i >> 1)][(i & 1) * 2], S[2 * (ks + w) + (i >> 1)][(i & 1) * 2 + 1], x);
#pragma unroll
              for (int p = 0; p < 3; p++) a[w][p][i] = x[p];
            }
          auto tokens = [&](int k) {
            return [=](int part, uint32_t (&bb)[2][2]) {
              uint32_t r[4];
              ldmatrix_x4_at(r, buf + part * L::QB + (row * L::NP + n0 + k * 16 + col) * 2);
              bb[0][0] = r[0]; bb[0][1] = r[1]; bb[1][0] = r[2]; bb[1][1] = r[3];
            };
          };
          mma_parts_twice(y, a[0], a[1], tokens(ks), tokens(ks + 1));
        }
        float any = 0.f;                                     // (stays 0 as long as every result is finite)
#pragma unroll
        for (int u = 0; u < 2; u++)
#pragma unroll
          for (int i = 0; i < 4; i++) any = fmaf(0.f, y[u][i], any);
        if (__any_sync(0xffffffffu, any != 0.f)) {           // again, from the numbers: the weights of later tokens are 0, and 0 x Inf is NaN
#pragma unroll
          for (int t = 0; t < NH; t++)
#pragma unroll
            for (int i = 0; i < 4; i++) scratch[((lane >> 2) + (i >> 1) * 8) * L::SP + 8 * t + 2 * (lane & 3) + (i & 1)] = S[t][i];
          __syncwarp();
#pragma unroll
          for (int u = 0; u < 2; u++)
#pragma unroll
            for (int i = 0; i < 4; i++) {
              const int j = u * 8 + 2 * (lane & 3) + (i & 1), c = c_lo + (i >> 1) * 8;
              if (j >= nt || c >= P.P + (P.nst ? 1 : 0)) continue;
              const float* qr = P.q + (size_t)(t0 + j) * P.ldq + (size_t)hk * P.hs;
              float s = 0.f;
#pragma unroll 1
              for (int n = 0; n < N / 2; n++) s = fmaf(qr[n0 + n], scratch[((lane >> 2) + (i >> 1) * 8) * L::SP + n], s);
              s *= rc[kRecG + j];
#pragma unroll 1
              for (int e = 0; half && e <= j; e++) s = fmaf(rc[kRecM + j * C + e], c < P.P ? P.v[(size_t)(t0 + e) * P.ldv + (size_t)h * P.P + c] : 1.f, s);
              y[u][i] = s;
            }
          __syncwarp();
        }
        if (half) {
#pragma unroll
          for (int u = 0; u < 2; u++)
#pragma unroll
            for (int i = 0; i < 4; i++) halves[(b & 1) * kLmGroups * 32 * 8 + (u * 4 + i) * 32] = y[u][i];
        }
      }
      decay *= ge;
#pragma unroll
      for (int t = 0; t < NH; t++)
#pragma unroll
        for (int i = 0; i < 4; i++) S[t][i] *= ge;
      if (bad[b & 1] != b) {
#pragma unroll
        for (int t = 0; t < NH; t += 4)
          mma_parts<3, 4>(S + t, av, [&](int part, uint32_t (&bb)[4][2]) {
#pragma unroll
            for (int w = 0; w < 2; w++) {
              uint32_t r[4];
              ldmatrix_x4_trans(r, buf + 3 * L::QB + part * L::QB + (uint32_t)(((lane & 7) + ((lane >> 3) & 1) * 8) * L::NP + n0 + (t + 2 * w + (lane >> 4)) * 8) * 2);
              bb[2 * w][0] = r[0]; bb[2 * w][1] = r[1]; bb[2 * w + 1][0] = r[2]; bb[2 * w + 1][1] = r[3];
            }
          });
      } else {
        for (int j = 0; j < nt; j++) {
          const float* kr = P.k + (size_t)(t0 + j) * P.ldq + (size_t)hk * P.hs;
          float x[2];
#pragma unroll
          for (int u = 0; u < 2; u++) {
            const int c = c_lo + u * 8;
            x[u] = rc[kRecE + j] * (c < P.P ? P.v[(size_t)(t0 + j) * P.ldv + (size_t)h * P.P + c] : P.nst && c == P.P ? 1.f : 0.f);
          }
#pragma unroll
          for (int t = 0; t < NH; t++)
#pragma unroll
            for (int i = 0; i < 4; i++) S[t][i] = fmaf(kr[n0 + 8 * t + 2 * (lane & 3) + (i & 1)], x[i >> 1], S[t][i]);
        }
      }
    }
    __syncthreads();
  }
  __syncthreads();
  if (!live) return;
  if (outputs && half == 0 && b0 < b1) finish(b1 - 1);
  if (!outputs) {
    float* at = slot(seg + 1);
#pragma unroll
    for (int t = 0; t < NH; t++)
#pragma unroll
      for (int i = 0; i < 4; i++) at[(t * 4 + i) * 32] = S[t][i];
    if (grp == 0 && half == 0 && lane == 0) const_cast<float*>(decays)[(size_t)seg * P.H + h] = decay;
  } else if (seg == P.nseg - 1) {
#pragma unroll
    for (int t = 0; t < NH; t++)
#pragma unroll
      for (int i = 0; i < 4; i++) {
        const int n = n0 + 8 * t + 2 * (lane & 3) + (i & 1), c = c_lo + (i >> 1) * 8;
        if (c < P.P) P.state[(size_t)h * N * P.P + (size_t)n * P.sn + (size_t)c * P.sp] = S[t][i];
        else if (P.nst && c == P.P) P.nst[(size_t)h * N + n] = S[t][i];
      }
  }
}

}  // namespace hy
}  // namespace dsk

// dsk_split.cuh — fp32 products of many rows (fp32 models; the score and value products of attention with mixed heads) on the 5th-generation tensor cores:
// C = A W^T, both operands split into three bf16 parts on their way into shared memory, six products per element, sums of 64 values joined in fp32 registers.
// Interface, row maps, expert tiles, batches and epilogues of GemmP.
//
// A CTA has 128 rows x 64 columns.  Sixteen warps read 64-deep slices of both operands as fp32 (four groups of four, half a slice each, the next one's numbers
// on their way while this one's are split), and put the parts into a ring of three stages (K-major rows of 128 bytes, swizzled).  One thread issues the products: a part of A
// against several parts of W in one instruction, as the parts of W are rows of one operand and the sums of different order columns of one accumulator:
//   [A0 W0 | A0 W1 | A0 W2],  [A1 W0 | A1 W1] on columns 64 ..,  A2 W0 on columns 128 ..    (kSplitHalves: A0 W0 of every second half slice on columns 192 ..)
// so that 24 KB per 16 values of depth come out of shared memory and not 36.  Four warps read a finished slice's 3 x 64 columns (two accumulators in TMEM: the
// next slice's products run meanwhile) and add them, smallest first, to what they hold in registers: a sum of n elements sees n / 64 roundings at its own size, and
// inside of 64 elements (32, where a product has few of them: kSplitHalves) the leading products are four (two) additions of the tensor core.
// A slice takes some 2000 cycles, its products 890 by themselves: the rest is splitting, for every column tile again, through L1 and the banks of shared memory (768 cycles for the operands of
// the products, 576 for the parts, 384 for the numbers on their way).  Counters, 600 x 4672 x 1024: L1's data pipe 60 % of an SM's active cycles, issue slots 43 %, tensor pipe 27 %, DRAM 3 %.  Measured, us, before (the same six products on mma.sync, two CTAs of 128 x 64 an SM) and now, rows x columns x
// depth: 600 x 4160 x 1024 139 and 72, 600 x 1024 x 2816 140 and 57, 45 x 1024 x 4096 203 and 27 (four CTAs share a tile's depth, 61 by one), 5 x 1024 x 1024 53 and 12, 1024 x 128 x
// 512 30 and 13; 64 x 100 x 36 8 and 9.  Error against 64 bits, normal operands, depth 1024 / 2816 / 4096: 1.5, 2.4, 2.9e-7 before, 1.0, 1.4, 1.6e-7 now; positive ones, depth 512 /
// 1000: 1.0 and 1.3e-7 before, 0.9 and 1.0e-7 now.  Tried: numbers past L1 (3 to 10 % longer), rows' addresses in registers (they spill), eight or twelve splitting warps (84 and 60
// instead of 55 us).
// The products that the three parts leave out are below an fp32 rounding.
#pragma once

#include "dsk_pattn.cuh"
#include "dsk_tc5.cuh"

namespace dsk {
namespace hy {

// The same sum as a chain of FMAs over the numbers themselves, for a result that is not finite: an infinite operand has no three parts (what is left
// of it is inf - inf), nor has a finite one that rounds to an infinity in bf16 (from 2^128 - 2^119).  Such operands make every result that they enter
// NaN, so that looking at the results is enough.  weights: A holds softmax weights, 0 for keys out of sight, which do not enter.
__device__ __noinline__ float plain_dot(const float* a, const float* w, int k_lo, int k_hi, bool weights) {
  float s = 0.f;
  for (int k = k_lo; k < k_hi && !isnan(s); k++)
    if (!weights || a[k] != 0.f) s = fmaf(a[k], w[k], s);
  return s;
}

constexpr int kSplitN = 64, kSplitDepth = 64, kSplitStages = 3;
// Products of fewer slices than this have an accumulator of its own for the leading products of every half slice: where the slices are few, the tensor core's own, truncated, additions are
// a sum's largest errors.  Error against 64 bits of depths 64 / 128 / 256 / 384, the six products on mma.sync (additions of 16 values, joined in registers), whole slices, halves: normal
// operands 6.3, 7.4, 9.0, 10.4e-8; 6.9, 7.4, 8.1, 8.5; 5.1, 5.9, 7.0; positive ones 5.7, 6.1, 7.2, 8.8; 8.2, 8.1, 8.1, 8.5; 5.1, 5.3, 5.8.  Halves everywhere: an fp32 prompt of 600 tokens
// (depths of 1024 and 2816) 734 -> 766 us.
constexpr int kSplitHalves = 6;
constexpr int kSplitPartA = kTcRows * 128, kSplitPartW = kSplitN * 128;              // bytes of a part of a slice
constexpr int kSplitStage = 3 * (kSplitPartA + kSplitPartW);
constexpr int kSplitGroups = 4, kSplitWarps = 4 * kSplitGroups, kSplitThreads = (kSplitWarps + 4 + 4) * 32;   // splitting, summing, issuing (one of the last four warps)
__host__ __device__ constexpr int split_smem(int stages) { return 1024 + stages * kSplitStage + 128; }   // (+ alignment, + barriers)
static_assert(4 * 32 * 65 * 4 <= kSplitStage, "the summing warps turn their results in the ring");

// Four rows' quads as three quads of bf16 each (split_pair<3>'s parts), into rows 2048 bytes apart of three parts `part` bytes apart.  A step of all eight pairs comes before the
// next step of any: a pair's conversions wait for one another, those of eight pairs do not.
__device__ __forceinline__ void split_rows(const float4 (&x)[4], unsigned char* dst, int part) {
  float v[16];
#pragma unroll
  for (int i = 0; i < 4; i++) { v[4 * i] = x[i].x; v[4 * i + 1] = x[i].y; v[4 * i + 2] = x[i].z; v[4 * i + 3] = x[i].w; }
#pragma unroll
  for (int p = 0; p < 3; p++) {
    uint32_t o[8];
#pragma unroll
    for (int j = 0; j < 8; j++) {
      const __nv_bfloat162 b = __floats2bfloat162_rn(v[2 * j], v[2 * j + 1]);
      o[j] = *reinterpret_cast<const uint32_t*>(&b);
    }
#pragma unroll
    for (int i = 0; i < 4; i++) *reinterpret_cast<uint2*>(dst + p * part + i * 2048) = make_uint2(o[2 * i], o[2 * i + 1]);
    if (p < 2) {
#pragma unroll
      for (int j = 0; j < 8; j++)   // both differences in one instruction
        asm("{\n\t.reg .b64 v, h, m;\n\tmov.b64 v, {%0, %1};\n\tmov.b64 h, {%2, %3};\n\tmov.b64 m, {%4, %4};\n\tfma.rn.f32x2 v, h, m, v;\n\tmov.b64 {%0, %1}, v;\n\t}"
            : "+f"(v[2 * j]), "+f"(v[2 * j + 1]) : "r"(o[j] << 16), "r"(o[j] & 0xffff0000u), "f"(-1.f));
    }
  }
}
// A splitting warp's way through the half slices of its group: group g has half slices g, g + 4, ..  Eight lanes have the 32 values of a row, a load four rows: w + 4 q of every
// 16 (rows 4 apart are on different banks behind the swizzle, whose phase is one for all rows of a lane).  The numbers of a group's next half slice are asked for as soon as
// the registers of this one's are free: 48 KB a slice cross from L2 at some 64 bytes a clock, which is as long as the products of a slice take.
// VEC: rows on 16-byte boundaries with whole quads behind their last numbers; the others are read number by number when they are needed.
template <bool VEC>
__device__ __forceinline__ void split_walk(const float* const* rows, unsigned char* gbase, uint32_t full0, uint32_t empty0, int k_lo, int K, int nk, int nrows, int stages, int* err) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, r0 = (warp & 3) + 4 * (lane >> 3), kk = (lane & 7) * 4, n4 = (nrows + 63) / 64;   // (64 rows at a time)
  const float* const* row = rows + r0;
  float4 x[VEC ? 3 : 1][4];                                  // rows 0 - 63 and 64 - 127 of A, rows of W
  auto fetch = [&](int j, int k) {
    if (VEC && k >= K) return;
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const float* p = row[64 * j + 16 * i] + k;
      float4& v = x[VEC ? j : 0][i];
      if (VEC) v = *reinterpret_cast<const float4*>(p);
      else v = make_float4(k < K ? p[0] : 0.f, k + 1 < K ? p[1] : 0.f, k + 2 < K ? p[2] : 0.f, k + 3 < K ? p[3] : 0.f);
    }
  };
  int k = k_lo + (warp >> 2) * 32 + kk;
  if (VEC && (warp >> 2) < 2 * nk) {
    fetch(0, k);
    if (n4 > 1) fetch(1, k);
    fetch(2, k);
  }
  for (int u = warp >> 2; u < 2 * nk; u += kSplitGroups) {
    const int kb = u >> 1, s = kb % stages, kn = k + kSplitGroups * 32;
    const bool more = VEC && u + kSplitGroups < 2 * nk;
    if (VEC && k + 4 > K) {                                  // the end of the last slice
#pragma unroll
      for (int j = 0; j < 3; j++)
#pragma unroll
        for (int i = 0; i < 4; i++) {
          float4& v = x[VEC ? j : 0][i];
          v = make_float4(k < K ? v.x : 0.f, k + 1 < K ? v.y : 0.f, k + 2 < K ? v.z : 0.f, 0.f);
        }
    }
    if (!__all_sync(0xffffffffu, tc_wait(empty0 + 8 * s, ((kb / stages) & 1) ^ 1, err))) break;
    unsigned char* dst = gbase + s * kSplitStage + r0 * 128 + ((((u & 1) * 4 + (kk >> 3)) ^ (r0 & 7)) << 4) + (kk & 4) * 2;
    if (!VEC) fetch(0, k);
    split_rows(x[0], dst, kSplitPartA);
    if (more) fetch(0, kn);
    if (n4 > 1) {
      if (!VEC) fetch(1, k);
      split_rows(x[VEC ? 1 : 0], dst + 64 * 128, kSplitPartA);
      if (more) fetch(1, kn);
    }
    if (!VEC) fetch(2, k);
    split_rows(x[VEC ? 2 : 0], dst + 3 * kSplitPartA, kSplitPartW);
    if (more) fetch(2, kn);
    k = kn;
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncwarp();
    if (lane == 0) tc_arrive(full0 + 8 * s);
  }
}

__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire;" ::: "memory"); }
__device__ __forceinline__ float load_of_rank(uint32_t addr, int rank) {   // shared memory of a CTA of the cluster
  uint32_t at;
  float v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"(addr), "r"(rank));
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(at) : "memory");
  return v;
}

// SHARES: a cluster of S CTAs shares a tile's depth; each joins the sums of 128 / S rows, in the order of the shares (a form of its own: on one for both the splitting warps
// spill, and products that take no shares ran 10 % longer).
template <int EPI, bool SHARES>
__global__ void __launch_bounds__(kSplitThreads, 1) gemm_split(const GemmP P, int stages, int S_, int* err) {
  const int S = SHARES ? S_ : 1;
  constexpr bool DUAL = epi_dual(EPI);
  constexpr int BN = DUAL ? kSplitN / 2 : kSplitN;                                  // output columns (DUAL: rows 0 - 31 of a slice of W, 32 - 63 of W2)
  extern __shared__ unsigned char sp_raw[];
  __shared__ int rowsC[kTcRows];
  __shared__ const float* rows[kTcRows + kSplitN];           // of A and of W; those out of the product are another row of theirs, no result reads them
  __shared__ uint32_t tmem_slot;
  const int share = SHARES ? (int)blockIdx.x % S : 0, n0 = (int)blockIdx.x / S * BN;
  if (P.band == BAND_COLS) {                                 // a tile that no query of its rows sees
    const int i0 = P.band_pos + (int)blockIdx.y * kTcRows, lo = max(0, mask_first(P.band_mask, P.band_window, i0) - P.band_first);
    if (n0 >= i0 + min(kTcRows, P.M - (int)blockIdx.y * kTcRows) - P.band_first || (n0 + BN <= lo && n0 >= P.band_keep)) { grid_enter(); return; }
  }
  const uint32_t base = (smem_u32(sp_raw) + 1023u) & ~1023u;
  unsigned char* gbase = sp_raw + (base - smem_u32(sp_raw));
  const uint32_t full0 = base + stages * kSplitStage, empty0 = full0 + 8 * kSplitStages, done0 = empty0 + 8 * kSplitStages, drained0 = done0 + 16, flushed0 = drained0 + 16;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < stages; s++) { mbar_init(full0 + 8 * s, 8); mbar_init(empty0 + 8 * s, 1); }
    for (int b = 0; b < 2; b++) { mbar_init(done0 + 8 * b, 1); mbar_init(drained0 + 8 * b, 4); }
    mbar_init(flushed0, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == kSplitWarps + 4) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)), "r"(512u) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  grid_enter();                                              // barriers and TMEM are set up under the kernel ahead
  long long aoff = (long long)blockIdx.z * P.sA, woff = (long long)((int)blockIdx.z / P.z_wdiv) * P.sW, coff = (long long)blockIdx.z * P.sC;
  int row0, nrows;
  if (P.tiles) {
    if ((int)blockIdx.y < *P.n_tiles) {
      const int4 t = P.tiles[blockIdx.y];
      woff = (long long)t.x * P.sW;
      row0 = t.y;
      nrows = t.z;
    } else row0 = nrows = 0;
  } else {
    row0 = blockIdx.y * kTcRows;
    nrows = min(kTcRows, P.M - row0);
  }
  const float* __restrict__ A = P.A + aoff;
  const float* __restrict__ W = reinterpret_cast<const float*>(P.W) + woff;
  const float* __restrict__ W2 = reinterpret_cast<const float*>(P.W2) + woff;      // (DUAL)
  if (threadIdx.x < kTcRows) {
    const int r = threadIdx.x, i = row0 + (r < nrows ? r : 0);
    rows[r] = A + (nrows > 0 ? (size_t)(P.a_map ? P.a_map[i] / P.a_div : i) * P.lda : 0);
    rowsC[r] = r < nrows ? (P.c_map ? P.c_map[i] : i) : -1;
  } else if (threadIdx.x < kTcRows + kSplitN) {
    const int r = threadIdx.x - kTcRows, n = min(n0 + (DUAL ? r & 31 : r), P.N - 1);
    rows[threadIdx.x] = (DUAL && r >= 32 ? W2 : W) + (size_t)n * P.ldw;
  }
  auto al = [](const float* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; };
  const bool vec = P.lda % 4 == 0 && P.ldw % 4 == 0 && al(A) && al(W) && (!DUAL || al(W2)) && P.sA % 4 == 0 && P.sW % 4 == 0 && P.ldw >= P.K && P.lda >= P.K;   // rows take 16-byte loads (K may end inside the last)
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = tmem_slot;
  int k_lo = 0, k_hi = P.K;
  if (P.band == BAND_DEPTH) {
    const int i0 = P.band_pos + row0, lo = max(0, mask_first(P.band_mask, P.band_window, i0) - P.band_first);
    k_lo = P.band_keep ? 0 : lo / kSplitDepth * kSplitDepth;
    k_hi = min(P.K, i0 + nrows - P.band_first);
  }
  const int all = nrows > 0 ? (k_hi - k_lo + kSplitDepth - 1) / kSplitDepth : 0, per = (all + S - 1) / S;   // slices of the tile, of a share
  const int nk = max(0, min(per, all - share * per)), k_from = k_lo + share * per * kSplitDepth;
  const bool halves = all < kSplitHalves;
  if (warp < kSplitWarps) {
    if (vec) split_walk<true>(rows, gbase, full0, empty0, k_from, P.K, nk, nrows, stages, err);
    else split_walk<false>(rows, gbase, full0, empty0, k_from, P.K, nk, nrows, stages, err);
    if (SHARES) { cluster_arrive(); cluster_wait(); cluster_arrive(); cluster_wait(); }
  } else if (warp >= kSplitWarps + 4) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 32;");
    if (warp == kSplitWarps + 4 && tc_elect()) {
      // fp32 accumulate, bf16 x bf16, both K-major; 192, 128 and 64 columns
      const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(kTcRows / 16) << 24);
      int s = 0;
      uint32_t turn = 0;
      for (int kb = 0; kb < nk; kb++) {
        const int buf = kb & 1;
        if (!tc_wait(drained0 + 8 * buf, ((kb >> 1) & 1) ^ 1, err) || !tc_wait(full0 + 8 * s, turn, err)) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t a = base + (uint32_t)s * kSplitStage, d = tmem + buf * 256;
        const uint64_t d0 = tc_desc(a), d1 = tc_desc(a + kSplitPartA), d2 = tc_desc(a + 2 * kSplitPartA), dw = tc_desc(a + 3 * kSplitPartA);
#pragma unroll
        for (int k = 0; k < kSplitDepth / 16; k++) {
          if (k < kSplitDepth / 32 || !halves) tc_mma(d, d0 + 2 * k, dw + 2 * k, idesc | (3u * kSplitN / 8 << 17), k > 0);
          else {                                             // the second half's leading products by themselves
            tc_mma(d + 3 * kSplitN, d0 + 2 * k, dw + 2 * k, idesc | (1u * kSplitN / 8 << 17), k > kSplitDepth / 32);
            tc_mma(d + kSplitN, d0 + 2 * k, dw + (kSplitPartW >> 4) + 2 * k, idesc | (2u * kSplitN / 8 << 17), true);
          }
          tc_mma(d + kSplitN, d1 + 2 * k, dw + 2 * k, idesc | (2u * kSplitN / 8 << 17), true);
          tc_mma(d + 2 * kSplitN, d2 + 2 * k, dw + 2 * k, idesc | (1u * kSplitN / 8 << 17), true);
        }
        tc_commit(empty0 + 8 * s);
        tc_commit(done0 + 8 * buf);
        if (++s == stages) { s = 0; turn ^= 1; }
      }
      tc_commit(flushed0);                                   // no product is under way when TMEM is given back
      tc_wait(flushed0, 0, err);
    }
    __syncwarp();
    if (SHARES) { cluster_arrive(); cluster_wait(); cluster_arrive(); cluster_wait(); }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 120;");    // (with the others' 4 x 80 and 32: 472 of the 480 that the CTA has)
    const int quad = warp & 3;                               // a warp reads the TMEM lanes of its place in a group of four
    float acc[kSplitN];
#pragma unroll
    for (int c = 0; c < kSplitN; c++) acc[c] = 0.f;
    bool ok = true;
    for (int kb = 0; kb < nk; kb++) {
      const int buf = kb & 1;
      ok = __all_sync(0xffffffffu, tc_wait(done0 + 8 * buf, (kb >> 1) & 1, err));
      if (!ok) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t from = tmem + ((uint32_t)(quad * 32) << 16) + buf * 256;
#pragma unroll
      for (int c0 = 0; c0 < kSplitN; c0 += 16) {
        uint32_t t0[16], t1[16], t2[16];
        tc_load16(from + kSplitN + c0, t1);
        tc_load16(from + 2 * kSplitN + c0, t2);
        tc_load16(from + c0, t0);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
        for (int c = 0; c < 16; c++) acc[c0 + c] += __uint_as_float(t0[c]) + (__uint_as_float(t1[c]) + __uint_as_float(t2[c]));
        if (halves) {
          tc_load16(from + 3 * kSplitN + c0, t0);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
          for (int c = 0; c < 16; c++) acc[c0 + c] += __uint_as_float(t0[c]);
        }
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) tc_arrive(drained0 + 8 * buf);
    }
    // results, turned so that a warp stores along rows (the ring is free: all products are through it)
    float* turn = reinterpret_cast<float*>(gbase);           // [row][65]
    auto again = [&](int row, int c) { return plain_dot(rows[row], rows[kTcRows + c], k_lo, k_hi, P.band == BAND_DEPTH); };
    auto store = [&](int row, float v, float v2) {
      const int cr = rowsC[row], n = n0 + lane;
      if (cr < 0) return;
      float* crow = P.C + coff + (size_t)cr * P.ldc;
      if (n < P.N) gemm_epilogue<float, EPI>(P, crow, cr, n, v, v2);
      if (!DUAL && n + 32 < P.N) gemm_epilogue<float, EPI>(P, crow, cr, n + 32, v2, 0.f);
    };
    if constexpr (!SHARES) {
      const int row = quad * 32 + lane, count = min(32, nrows - quad * 32);
      float any = 0.f;                                       // (stays 0 as long as every sum is finite)
#pragma unroll
      for (int c = 0; c < kSplitN; c++) { any = fmaf(0.f, acc[c], any); turn[row * 65 + c] = acc[c]; }
      if (any != 0.f && row < nrows) {
#pragma unroll 1
        for (int c = 0; c < kSplitN; c++) if (!isfinite(turn[row * 65 + c])) turn[row * 65 + c] = again(row, c);
      }
      __syncwarp();
      if (ok)
        for (int i0 = 0; i0 < count; i0 += 8) {              // (eight rows' values ahead of their stores, which may not pass one another)
          float v[8][2];
#pragma unroll
          for (int i = 0; i < 8; i++) { v[i][0] = turn[(quad * 32 + i0 + i) * 65 + lane]; v[i][1] = turn[(quad * 32 + i0 + i) * 65 + 32 + lane]; }
#pragma unroll
          for (int i = 0; i < 8; i++) store(quad * 32 + i0 + i, v[i][0], v[i][1]);
        }
    } else {
#pragma unroll
      for (int c = 0; c < kSplitN; c++) turn[(quad * 32 + lane) * 65 + c] = acc[c];
      cluster_arrive();
      cluster_wait();
      const int mine = kTcRows / S / 4, from = share * (kTcRows / S) + quad * mine;   // this warp's rows, two at a time
      if (ok)
#pragma unroll 1
        for (int i = 0; i < min(mine, nrows - from); i += 2) {
          float v[2][2] = {{0.f, 0.f}, {0.f, 0.f}};
          const uint32_t at = base + (uint32_t)((from + i) * 65 + lane) * 4;
#pragma unroll
          for (int q = 0; q < 8; q++)
            if (q < S) {
#pragma unroll
              for (int u = 0; u < 2; u++) { v[u][0] += load_of_rank(at + u * 260, q); v[u][1] += load_of_rank(at + u * 260 + 128, q); }
            }
          if (__any_sync(0xffffffffu, !isfinite(v[0][0] + v[0][1] + v[1][0] + v[1][1]))) {   // (a sum of finite ones may be infinite too: looked at one by one)
#pragma unroll
            for (int u = 0; u < 2; u++) {
              if (!isfinite(v[u][0])) v[u][0] = again(from + i + u, lane);
              if (!isfinite(v[u][1])) v[u][1] = again(from + i + u, 32 + lane);
            }
          }
          store(from + i, v[0][0], v[0][1]);
          store(from + i + 1, v[1][0], v[1][1]);
        }
      cluster_arrive();                                      // (no CTA leaves while another reads its sums)
      cluster_wait();
    }
  }
  __syncthreads();
  if (warp == kSplitWarps + 4) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u));
  }
}

}  // namespace hy
}  // namespace dsk

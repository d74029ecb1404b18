// dsk_pattn5.cuh — softmax attention of portions on the 5th-generation tensor cores, for heads of 64 to 192 entries (a rotated part counted) whatever the number of queries; where the query
// blocks leave SMs idle, the keys are cut into shares that latent_swa_merge joins.  pattn has the other heads: smaller ones would be half padding, larger ones do not fit.
//
// A CTA has 128 query rows of a head and walks their visible keys in tiles of 32.  Operands in PARTS bf16 parts as in pattn.  Keys and values come by TMA from what pattn_pack
// made; products:
//   scores: the parts of a tile's keys are rows of one operand, [Q0 K0 | Q0 K1 | Q0 K2], [Q1 K0 | Q1 K1] and Q2 K0 on columns of one accumulator, as in gemm_split; the leading products
//   of every 32 to 64 entries of depth have an accumulator of their own, so that a score is a sum of few long-rounded pieces joined in registers;
//   values: the weights' parts are the operand in TMEM, written there by the softmax; the six pairs of a tile add up smallest first, and a tile's 32 keys leave TMEM before the next one's.
// Eight warps have the softmax (two threads a row), four the output rows in registers (scaled and added to tile by tile).  Two accumulators for scores: a tile's products run under
// the softmax of the one ahead.  Copies of keys and of values, products for scores and for values have a thread each: with one thread for all products a tile took 3950 to 5900
// cycles, of which it waited 1000 for barriers in turn.
// Bound: a tile's narrow tensor core instructions, which take longer than they are counted (2300 cycles at 128 entries and 3000 at 192 by themselves; 3250 and 4300 here), one behind the other with
// the softmax (2000, what binds at a part).  Counters, 1024 queries of 16 heads, 128 + 128 entries, all keys, three parts: on the busiest SM the tensor pipe is active for 52 % of its
// cycles and fed for 60 %; issue slots 40 %, L1 28 %, DRAM 2 %.  512 threads have 128 registers each at launch, and no more:
// 44 bytes (two blocks of value columns) or 20 to 24 (one) are spilled, with 1.2 or 0.6 KB of loads in the code.
// Measured, us, pattn and this: 2048 queries, 16 heads, 128 + 128 entries, window 1024, capped 433 and 148; 192 + 128 entries, all keys 576 and 183; 777 queries, 64 + 64
// entries, window 512 99 and 42; 300 queries 54 and 25; 64 queries 19 and 15; one part, 2048 queries, 128 + 128, window 1024 108 and 91.  Error against 64 bits 0.77 to 1.06 times
// pattn's over 64, 80, 96, 128, 160 and 192 entries, normal operands, biased ones, positive values and scores three and nine times as large (64 entries in one accumulator, and not in two of 32:
// up to 1.3 times; 80 in accumulators of 64 and 16, and not of 48 and 32: up to 1.11; 128 in three instead of two: 1.04 instead of 1.06, and 82 -> 91 us).
#pragma once

#include "dsk_pattn.cuh"
#include "dsk_tc5.cuh"

namespace dsk {
namespace hy {

constexpr int kP5Rows = 128, kP5Keys = 32, kP5Threads = 512, kP5MaxChunks = 3, kP5MaxK = 8;
constexpr int kP5Tile = kP5Keys * 128;                       // bytes of 32 rows of 64 entries
__host__ __device__ inline int p5_smem(int parts, int chunks, int vb, int kst, int vst) {
  return 1024 + parts * chunks * kP5Rows * 128 + kst * parts * kP5Tile + vst * parts * vb * kP5Tile + 9 * kP5Rows * 4 + 384;
}

__device__ __forceinline__ void tma_box(uint32_t dst, const CUtensorMap* map, int x, int y, int z, uint32_t bar) {
  asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
               ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(x), "r"(y), "r"(z) : "memory");
}
// operand whose rows are the depth: 64 columns to a swizzled 128-byte row, groups of eight rows 1024 bytes apart, the next 64 columns kP5Tile behind
__device__ __forceinline__ uint64_t tc_desc_mn(uint32_t addr) {
  return (uint64_t)((addr & 0x3FFFFu) >> 4) | ((uint64_t)(kP5Tile >> 4) << 16) | (64ull << 32) | (1ull << 46) | (2ull << 61);
}
__device__ __forceinline__ void tc_mma_ta(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, bool add) {   // A in TMEM
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
               ::"r"(d), "r"(a), "l"(b), "r"(idesc), "r"((uint32_t)add) : "memory");
}
__device__ __forceinline__ void tc_store8(uint32_t addr, const uint32_t (&r)[8]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};"
               ::"r"(addr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]) : "memory");
}

// VB: 64-column blocks of values in a CTA (blockIdx.z picks the columns); kst, vst: in shared memory, pieces of 64 entries of a tile's keys and tiles of values
template <int PARTS, int VB>
__global__ void __launch_bounds__(kP5Threads, 1) pattn5(const __grid_constant__ PattnP P, const __grid_constant__ CUtensorMap mapK, const __grid_constant__ CUtensorMap mapV, int kst,
                                                        int vst, int* err) {
  extern __shared__ unsigned char p5_raw[];
  __shared__ uint32_t tmem_slot;
  const uint32_t base = (smem_u32(p5_raw) + 1023u) & ~1023u;
  unsigned char* gbase = p5_raw + (base - smem_u32(p5_raw));
  const int nch = (P.Dp + 63) / 64, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t kbytes = PARTS * kP5Tile, vbytes = PARTS * VB * kP5Tile;
  const uint32_t q0s = base, ks = q0s + PARTS * nch * kP5Rows * 128, vs = ks + kst * kbytes, cs = vs + vst * vbytes, bars = cs + 9 * kP5Rows * 4;
  float* corr = reinterpret_cast<float*>(gbase + (cs - base));          // [2][128] factors of a tile, [2][128] sums and [128] maxima at the end, ..
  float* half_max = corr + 5 * kP5Rows;                                 // .. [2][2 halves][128] of a tile (who writes the next but one has met, on the next one, the thread that reads this)
  const uint32_t kfull = bars, kempty = bars + 64, vfull = bars + 128, vempty = bars + 144, sfull = bars + 160, sempty = bars + 176, cfull = bars + 192, met = bars + 208, pfull = bars + 272,
                 pdone = bars + 280, ofull = bars + 288, oempty = bars + 296, lfull = bars + 304, flushed = bars + 312;   // (and 8 bytes behind)
  if (threadIdx.x == 0) {
    for (int i = 0; i < kst; i++) { mbar_init(kfull + 8 * i, 1); mbar_init(kempty + 8 * i, 1); }
    for (int i = 0; i < 2; i++) { mbar_init(vfull + 8 * i, 1); mbar_init(vempty + 8 * i, 1); mbar_init(sfull + 8 * i, 1); mbar_init(sempty + 8 * i, 8); mbar_init(cfull + 8 * i, 4); }
    for (int i = 0; i < 8; i++) mbar_init(met + 8 * i, 2);
    mbar_init(pfull, 8); mbar_init(pdone, 1); mbar_init(ofull, 1); mbar_init(oempty, 4); mbar_init(lfull, 8); mbar_init(flushed, 1); mbar_init(flushed + 8, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 12) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)), "r"(512u) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  const int qb = (int)gridDim.y - 1 - (int)blockIdx.y, q0 = qb * kP5Rows;   // late queries, which see most keys, first for every head
  const int zc = (int)gridDim.z / P.NS, share = (int)blockIdx.z / zc;       // (NS > 1: shares of the keys, joined by latent_swa_merge)
  const int h = blockIdx.x, g = h / (P.H / P.G), v0 = ((int)blockIdx.z - share * zc) * VB * 64;
  const KeyTiles tiles = key_tiles(P, q0, kP5Rows, kP5Keys, share, P.NS);
  const int n = max(0, tiles.end - tiles.begin);
  grid_enter();
  {   // query rows in parts: [part][64 entries][row], four entries a thread
    const int per = nch * 16;
    const bool vec = P.D % 4 == 0 && P.ldq % 4 == 0 && (reinterpret_cast<uintptr_t>(P.q) & 15) == 0;
    for (int e = threadIdx.x; e < kP5Rows * per; e += kP5Threads) {
      const int r = e / per, c = (e - r * per) * 4;
      const float* src = P.q + (size_t)(q0 + r) * P.ldq + (size_t)h * P.D + c;
      float x[4] = {0.f, 0.f, 0.f, 0.f};
      if (q0 + r < P.T) {
        if (vec && c + 4 <= P.D) { const float4 v = *reinterpret_cast<const float4*>(src); x[0] = v.x; x[1] = v.y; x[2] = v.z; x[3] = v.w; }
        else
#pragma unroll
          for (int u = 0; u < 4; u++) if (c + u < P.D) x[u] = src[u];
      }
      __nv_bfloat16 s[4][PARTS];
#pragma unroll
      for (int u = 0; u < 4; u++) split_bf16<PARTS>(x[u], s[u]);
#pragma unroll
      for (int i = 0; i < PARTS; i++) {
        __nv_bfloat162 lo, hi;
        lo.x = s[0][i]; lo.y = s[1][i]; hi.x = s[2][i]; hi.y = s[3][i];
        *reinterpret_cast<uint2*>(gbase + (size_t)(i * nch + (c >> 6)) * kP5Rows * 128 + r * 128 + (((((c & 63) >> 3) ^ (r & 7)) << 4) | ((c & 4) * 2))) =
            make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
      }
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = tmem_slot;
  // columns: scores [2][main of the first entries | two of lower order | mains of the other entries], weights' parts, values.  As many mains as pieces of 64 entries, two at least, of
  // equal depth (three parts)
  const int all_steps = (P.Dp + 15) / 16, mains = PARTS == 3 ? max(nch, 2) : nch, per_main = PARTS == 3 ? (all_steps + mains - 1) / mains : 4, s_cols = (PARTS == 3 ? mains + 2 : mains) * kP5Keys;
  const uint32_t p_at = tmem + 320, o_at = tmem + 384;
  if (warp >= 12) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 40;");
    // four threads, so that none of them waits for what another one is to bring: products for scores, copies of keys, products for values, copies of values
    const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(kP5Rows / 16) << 24);   // fp32 accumulate, bf16 x bf16
    if (warp == 12 && tc_elect()) {
      constexpr uint32_t n1 = (uint32_t)(kP5Keys / 8) << 17;                // 32 columns
      int at = 0;
      uint32_t turn = 0;
      bool alive = true;
      for (int i = 0; i < n && alive; i++) {
        if (!tc_wait(sempty + 8 * (i & 1), ((i >> 1) & 1) ^ 1, err)) break;
        const uint32_t d = tmem + (i & 1) * s_cols;
        int main = 0, nth = 0;
        for (int c = 0; c < nch; c++) {
          alive = tc_wait(kfull + 8 * at, turn, err);
          if (!alive) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint64_t k0 = tc_desc(ks + at * kbytes), a0 = tc_desc(q0s + c * kP5Rows * 128), a1 = tc_desc(q0s + (nch + c) * kP5Rows * 128),
                         a2 = tc_desc(q0s + (2 * nch + c) * kP5Rows * 128);
          const int steps = min(4, all_steps - c * 4);
          for (int k = 0; k < steps; k++) {
            if (PARTS == 1) tc_mma(d + c * kP5Keys, a0 + 2 * k, k0 + 2 * k, idesc | n1, k > 0);
            else {
              const bool add = nth > 0;                                     // main: the accumulator of this step's leading products, of which it is the nth
              if (main == 0) tc_mma(d, a0 + 2 * k, k0 + 2 * k, idesc | 3 * n1, add);
              else {
                tc_mma(d + (2 + main) * kP5Keys, a0 + 2 * k, k0 + 2 * k, idesc | n1, add);
                tc_mma(d + kP5Keys, a0 + 2 * k, k0 + (kP5Tile >> 4) + 2 * k, idesc | 2 * n1, true);
              }
              tc_mma(d + kP5Keys, a1 + 2 * k, k0 + 2 * k, idesc | 2 * n1, true);
              tc_mma(d + 2 * kP5Keys, a2 + 2 * k, k0 + 2 * k, idesc | n1, true);
              if (++nth == per_main) { nth = 0; main++; }
            }
          }
          tc_commit(kempty + 8 * at);
          if (++at == kst) { at = 0; turn ^= 1; }
        }
        if (alive) tc_commit(sfull + 8 * (i & 1));
      }
      tc_commit(flushed);                                    // no product is under way when TMEM is given back
      tc_wait(flushed, 0, err);
    } else if (warp == 13 && tc_elect()) {
      int nk = 0, at = 0;
      uint32_t turn = 1;
      bool alive = true;
      for (int i = 0; i < n && alive; i++) {
        const int key0 = tile_key(tiles, tiles.begin + i, kP5Keys);
        for (int c = 0; c < nch; c++) {
          alive = tc_wait(kempty + 8 * at, turn, err);
          if (!alive) break;
          mbar_expect_tx(kfull + 8 * at, kbytes);
          for (int p = 0; p < PARTS; p++) tma_box(ks + at * kbytes + p * kP5Tile, &mapK, c * 64, key0, p * P.G + g, kfull + 8 * at);
          nk++;
          if (++at == kst) { at = 0; turn ^= 1; }
        }
      }
      // no copy of this CTA is under way when it leaves, also where a wait gave up
      for (int k = max(0, nk - kst); k < nk; k++) tc_wait(kfull + 8 * (k % kst), (k / kst) & 1, err);
    } else if (warp == 14 && tc_elect()) {
      const uint32_t pdesc = idesc | (1u << 16) | ((uint32_t)(VB * 8) << 17);   // values: rows are the depth
      int at = 0;
      uint32_t turn = 0;
      for (int i = 0; i < n; i++) {
        if (!tc_wait(vfull + 8 * at, turn, err) || !tc_wait(oempty, (i & 1) ^ 1, err) || !tc_wait(pfull, i & 1, err)) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint64_t b = tc_desc_mn(vs + at * vbytes);
        auto pair = [&](int pp, int vp, bool first) {
#pragma unroll
          for (int k = 0; k < kP5Keys / 16; k++) tc_mma_ta(o_at, p_at + pp * 16 + k * 8, b + vp * (VB * kP5Tile >> 4) + k * 128, pdesc, !first || k > 0);
        };
        if (PARTS == 1) pair(0, 0, true);
        else { pair(2, 0, true); pair(1, 1, false); pair(0, 2, false); pair(1, 0, false); pair(0, 1, false); pair(0, 0, false); }
        tc_commit(pdone);
        tc_commit(ofull);
        tc_commit(vempty + 8 * at);
        if (++at == vst) { at = 0; turn ^= 1; }
      }
      tc_commit(flushed + 8);
      tc_wait(flushed + 8, 0, err);
    } else if (warp == 15 && tc_elect()) {
      int i = 0, at = 0;
      uint32_t turn = 1;
      for (; i < n; i++) {
        if (!tc_wait(vempty + 8 * at, turn, err)) break;
        const int key0 = tile_key(tiles, tiles.begin + i, kP5Keys);
        mbar_expect_tx(vfull + 8 * at, vbytes);
        for (int p = 0; p < PARTS; p++)
          for (int b = 0; b < VB; b++) tma_box(vs + at * vbytes + (p * VB + b) * kP5Tile, &mapV, v0 + b * 64, key0, p * P.G + g, vfull + 8 * at);
        if (++at == vst) { at = 0; turn ^= 1; }
      }
      for (int k = max(0, i - vst); k < i; k++) tc_wait(vfull + 8 * (k % vst), (k / vst) & 1, err);
    }
    __syncwarp();
  } else if (warp < 8) {
    // softmax: two threads have a row, 16 keys of a tile each
    constexpr int NK = kP5Keys / 2;
    const int quad = warp & 3, half = warp >> 2, row = quad * 32 + lane, pos = P.pos0 + q0 + row, first_lo = mask_first(P.mask, P.span, pos);
    const int w_pos = P.pos0 + q0 + quad * 32, w_lo = mask_first(P.mask, P.span, w_pos + 31);   // a tile whose keys every row of the warp sees needs no mask
    const uint32_t lanes = (uint32_t)(quad * 32) << 16;
    const bool capped = P.mods.cap > 0.f;
    const float s_mul = capped ? P.scale / P.mods.cap : P.scale;
    float m = -1e30f, l = 0.f;
    for (int i = 0; i < n; i++) {
      if (!__all_sync(0xffffffffu, tc_wait(sfull + 8 * (i & 1), (i >> 1) & 1, err))) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      float s[NK];
      const uint32_t from = tmem + lanes + (i & 1) * s_cols + half * NK;
      {
        uint32_t a[NK], b[NK], c[NK], e[2][NK];
        tc_load16(from, a);
        if (PARTS == 3) { tc_load16(from + kP5Keys, b); tc_load16(from + 2 * kP5Keys, c); }
        if (mains > 1) tc_load16(from + (PARTS == 3 ? 3 : 1) * kP5Keys, e[0]);
        if (mains > 2) tc_load16(from + (PARTS == 3 ? 4 : 2) * kP5Keys, e[1]);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
        for (int k = 0; k < NK; k++) s[k] = PARTS == 3 ? __uint_as_float(a[k]) + (__uint_as_float(b[k]) + __uint_as_float(c[k])) : __uint_as_float(a[k]);
        if (mains > 1) {
#pragma unroll
          for (int k = 0; k < NK; k++) s[k] += __uint_as_float(e[0][k]);
        }
        if (mains > 2) {
#pragma unroll
          for (int k = 0; k < NK; k++) s[k] += __uint_as_float(e[1][k]);
        }
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) tc_arrive(sempty + 8 * (i & 1));
      // scale, cap, bias and mask
      const int key0 = tile_key(tiles, tiles.begin + i, kP5Keys);
#pragma unroll
      for (int k = 0; k < NK; k++) s[k] *= s_mul;
      if (capped) {
#pragma unroll
        for (int k = 0; k < NK; k++) s[k] = P.mods.cap * tanhf(s[k]);
      }
      const int p_lo = P.first + key0 - P.nk, p_hi = p_lo + kP5Keys - 1;     // positions of a tile behind the kept rows
      if (P.mods.rel || key0 < P.nk || p_hi > w_pos || p_lo < w_lo || key0 + kP5Keys > P.Lk) {
#pragma unroll
        for (int k = 0; k < NK; k++) {
          const int v = key0 + half * NK + k, p = v < P.nk ? v : P.first + v - P.nk;
          const bool ok = v < P.Lk && p <= pos && (p < P.mods.keep || p >= first_lo);
          if (ok && P.mods.rel) s[k] += P.mods.rel[(size_t)P.mods.bucket[min(pos - p, P.mods.rel_max)] * P.H + h];
          if (!ok) s[k] = -INFINITY;
        }
      }
      float mx = s[0], sum = 0.f;
#pragma unroll
      for (int k = 1; k < NK; k++) mx = fmaxf(mx, s[k]);
      half_max[((i & 1) * 2 + half) * kP5Rows + row] = mx;
      __syncwarp();
      if (lane == 0) tc_arrive(met + 8 * quad);
      if (!__all_sync(0xffffffffu, tc_wait(met + 8 * quad, i & 1, err))) break;
      const float m_new = fmaxf(m, fmaxf(mx, half_max[((i & 1) * 2 + (half ^ 1)) * kP5Rows + row])), c = expf(m - m_new);
      m = m_new;
#pragma unroll
      for (int k = 0; k < NK; k++) { s[k] = expf(s[k] - m); sum += s[k]; }   // (a key out of sight: e^-inf = 0)
      l = fmaf(l, c, sum);
      if (!__all_sync(0xffffffffu, tc_wait(pdone, (i & 1) ^ 1, err))) break;   // the tile ahead is through with the weights, and its factors are used
      if (half == 0) corr[(i & 1) * kP5Rows + row] = c;
      uint32_t x[PARTS][8];
#pragma unroll
      for (int j = 0; j < 8; j++) {
        uint32_t o[PARTS];
        split_pair<PARTS>(s[2 * j], s[2 * j + 1], o);
#pragma unroll
        for (int p = 0; p < PARTS; p++) x[p][j] = o[p];
      }
#pragma unroll
      for (int p = 0; p < PARTS; p++) tc_store8(p_at + lanes + p * 16 + half * 8, x[p]);
      asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) {
        if (half == 0) tc_arrive(cfull + 8 * (i & 1));
        tc_arrive(pfull);
      }
    }
    corr[(2 + half) * kP5Rows + row] = l;
    if (half == 0) corr[4 * kP5Rows + row] = m;
    __syncwarp();
    if (lane == 0) tc_arrive(lfull);
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 208;");    // (with the softmax's 2 x 128 and 40: 504 of the 512 that the CTA has)
    const int quad = warp & 3, row = quad * 32 + lane, t = q0 + row;
    const uint32_t lanes = (uint32_t)(quad * 32) << 16;
    float acc[VB * 64];
#pragma unroll
    for (int k = 0; k < VB * 64; k++) acc[k] = 0.f;
    bool ok = true;
    for (int i = 0; i < n; i++) {
      ok = __all_sync(0xffffffffu, tc_wait(cfull + 8 * (i & 1), (i >> 1) & 1, err) && tc_wait(ofull, i & 1, err));
      if (!ok) break;
      const float c = corr[(i & 1) * kP5Rows + row];
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
      for (int k0 = 0; k0 < VB * 64; k0 += 32) {
        uint32_t o[32];
        tc_load32(o_at + lanes + k0, o);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
        for (int k = 0; k < 32; k++) acc[k0 + k] = fmaf(acc[k0 + k], c, __uint_as_float(o[k]));
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) tc_arrive(oempty);
    }
    ok = __all_sync(0xffffffffu, tc_wait(lfull, 0, err)) && ok;
    float l = corr[2 * kP5Rows + row] + corr[3 * kP5Rows + row], m = corr[4 * kP5Rows + row], any = l;
#pragma unroll
    for (int k = 0; k < VB * 64; k++) any = fmaf(0.f, acc[k], any);
    uint32_t again = __ballot_sync(0xffffffffu, ok && t < P.T && !isfinite(any));   // rows of the warp whose result is not finite
    if (ok && t < P.T && isfinite(any)) {
      float f = 1.f;
      if (P.mods.sink && share == 0) {                       // a key with a zero value vector
        const float sk = P.mods.sink[h], m_new = fmaxf(m, sk);
        f = expf(m - m_new);
        l = l * f + expf(sk - m_new);
        m = m_new;
      }
      const bool joins = P.NS > 1;
      const float inv = joins ? f : f / l * P.alpha;
      float* pp = P.part + (joins ? (((size_t)t * P.H + h) * P.NS + share) * (P.V + 2) : 0);
      if (joins && v0 == 0) { pp[0] = m; pp[1] = l; }
      float* out = joins ? pp + 2 + v0 : P.out + (size_t)t * P.ld_out + (size_t)h * P.V + v0;
      const float* gate = P.gate && !joins ? P.gate + (size_t)t * P.ld_gate + (P.gate_head ? (size_t)h : (size_t)h * P.V + v0) : nullptr;
      auto al = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 31) == 0; };
      const bool wide = al(out) && (!gate || P.gate_head || al(gate));
      const float gh = gate && P.gate_head ? sigmoid_f(gate[0]) : 1.f;
#pragma unroll
      for (int k0 = 0; k0 < VB * 64; k0 += 8) {
        float v[8], gt[8];
#pragma unroll
        for (int k = 0; k < 8; k++) { v[k] = acc[k0 + k] * inv; gt[k] = gh; }
        if (wide && v0 + k0 + 8 <= P.V) {
          if (gate && !P.gate_head) {
            load8(gate + k0, gt);
#pragma unroll
            for (int k = 0; k < 8; k++) gt[k] = sigmoid_f(gt[k]);
          }
#pragma unroll
          for (int k = 0; k < 8; k++) v[k] *= gt[k];
          store8(out + k0, v);
        } else
#pragma unroll
          for (int k = 0; k < 8; k++) if (v0 + k0 + k < P.V) out[k0 + k] = v[k] * (gate && !P.gate_head ? sigmoid_f(gate[k0 + k]) : gh);
      }
    }
    for (; again; again &= again - 1) {
      const int tr = q0 + quad * 32 + __ffs(again) - 1;
      if (P.NS > 1) pattn_row<PARTS, VB * 8, kP5Keys, true>(P, tr, h, v0, tiles, share);
      else pattn_row<PARTS, VB * 8, kP5Keys, false>(P, tr, h, v0, tiles, share);
    }
  }
  __syncthreads();
  if (warp == 12) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u));
  }
}

}  // namespace hy
}  // namespace dsk

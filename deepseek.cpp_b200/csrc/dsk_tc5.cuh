// dsk_tc5.cuh — bf16 matrix products of portions on the 5th-generation tensor cores (layer-list models): C = A W^T with TMA-staged
// operands, tcgen05.mma into TMEM and the epilogues of dsk_hybrid.cuh.
//
// One CTA per SM walks output tiles of 128 rows x bn columns (bn = 32 .. 256, picked by the host for the grid it gives).  Warp 0 copies
// 64-deep slices of both operands into a ring of shared memory (128-byte swizzle), one thread of warp 1 issues the products, warps 2 - 9 (two a row
// block, every second block of 32 columns) read the finished accumulators (two in TMEM: a tile's epilogue runs under the next tile's products), turn them through shared
// memory, apply the epilogue and store 128 bytes of a row by eight lanes.
// The activations are rounded to bf16 (as gemm_mma rounds them while staging) and, in routed products, put into expert order by one
// pass ahead of the product (bf16_rows), or by the epilogue of the product that made them (TcP::C16): every column tile then reads half
// the bytes, by TMA, instead of gathering and converting fp32 rows again.
// Bound: large products by the tensor pipe (2048 x 8192 x 8192: 1325 TFLOP/s, a 64-deep slice 640 cycles); one-tile grids by what is not under the products
// (ring fill 1300 to 3000 cycles, the one epilogue); narrow tiles by the two issuing threads.  Those are elected lanes that count stages and parities:
// lanes picked by number, which divided by the number of stages, took 650 cycles a slice at any width, now 535 at 256 columns, 340 at 128, 285 at 64, 270 at 32
// (512 x 2048 x 2048: 21 -> 14.5 us, 45 x 1024 x 4096: 29 -> 17 us).
// Epilogues: a warp a row block whose lanes each stored their own row met 32 lines a store and hid no latency, and a value's branches (a division's, expm1's, the sign's) kept
// those of a lane from running next to one another.  Two warps, stores along rows, no branches (2048 x 2048 x 2048 with cold operands, launch and all, us): plain 26.6 -> 24.6,
// on top of C 32.8 -> 28.7, gate on C 57 -> 31; 512 x 8192 x 2048 xIELU 51 -> 37; 777 x 3072 x 1024 linear-recurrence gates 63 -> 31.
#pragma once

#include <cuda.h>   // CUtensorMap

#include "dsk_hybrid.cuh"

namespace dsk {
namespace hy {

constexpr int kTcRows = 128, kTcDepth = 64, kTcEpi = 8, kTcThreads = 64 + 32 * kTcEpi, kTcMaxStages = 10;   // kTcEpi: warps that finish tiles
constexpr int kTcRing = 192 * 1024;                                  // operand ring
constexpr int kTcTurn = kTcEpi * 32 * 32 * 4;                           // epilogue: a 32 x 32 block per warp
constexpr int kTcSmem = 1024 + kTcRing + kTcTurn + 256;              // (+ alignment, + barriers)
constexpr long long kTcWaitCycles = 1ll << 32;                       // how long a wait polls a barrier before it gives up (two seconds)

struct TcP {
  int bn, stages, n_mt, rows_per_expert;   // column tile, ring stages, row tiles (no tile list), weight rows between experts
  __nv_bfloat16* C16;                      // non-null: results go here as bf16, row = position in the product (no c_map), pitch ldc16
  int ldc16;
  int wide;                                // rows of C (C16) take 16-byte (8-byte) accesses at columns that are multiples of four
  int* err;                                // host-visible word: set when a wait gave up
};

__device__ __forceinline__ bool tc_poll(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
               : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
  return ok != 0;
}
__device__ __forceinline__ bool tc_wait(uint32_t bar, uint32_t parity, int* err) {
  if (tc_poll(bar, parity)) return true;
  const long long from = clock64();
  do {
    if (tc_poll(bar, parity)) return true;
  } while (clock64() - from < kTcWaitCycles);
  *reinterpret_cast<volatile int*>(err) = 1;
  return false;
}
// one lane of a whole warp
__device__ __forceinline__ bool tc_elect() {
  uint32_t p;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(p));
  return p != 0;
}
__device__ __forceinline__ void tc_arrive(uint32_t bar) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory"); }
__device__ __forceinline__ void tma_tile(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
  asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
               ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(x), "r"(y) : "memory");
}
// K-major operand in 128-byte swizzled rows (8-row groups 1024 bytes apart)
__device__ __forceinline__ uint64_t tc_desc(uint32_t addr) {
  return (uint64_t)((addr & 0x3FFFFu) >> 4) | (1ull << 16) | (64ull << 32) | (1ull << 46) | (2ull << 61);
}
__device__ __forceinline__ void tc_mma(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, bool add) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
               ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"((uint32_t)add) : "memory");
}
__device__ __forceinline__ void tc_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tc_load32(uint32_t addr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]),
        "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
        "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(addr));
}

__device__ __forceinline__ void tc_load16(uint32_t addr, uint32_t (&r)[16]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]),
                 "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
               : "r"(addr));
}

__device__ __forceinline__ void store8(float* p, const float* v) {   // 32 bytes
  asm volatile("st.global.v8.f32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(p), "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7]) : "memory");
}
__device__ __forceinline__ void load8(const float* p, float* v) {
  asm volatile("ld.global.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7]) : "l"(p) : "memory");
}

template <int EPI>
__global__ void __launch_bounds__(kTcThreads, 1) gemm_tc5(const GemmP P, const TcP T, const __grid_constant__ CUtensorMap mapA,
                                                          const __grid_constant__ CUtensorMap mapB, const __grid_constant__ CUtensorMap mapB2) {
  constexpr bool DUAL = epi_dual(EPI);
  extern __shared__ unsigned char tc_raw[];
  const uint32_t base = (smem_u32(tc_raw) + 1023u) & ~1023u;
  unsigned char* gbase = tc_raw + (base - smem_u32(tc_raw));
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t bars = base + kTcRing + kTcTurn;            // full[stages], empty[stages], done[2], drained[2], flushed, then the TMEM address
  const uint32_t full0 = bars, empty0 = bars + 8 * kTcMaxStages, done0 = bars + 16 * kTcMaxStages, drained0 = done0 + 16, flushed0 = done0 + 32;
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(gbase + kTcRing + kTcTurn + 16 * kTcMaxStages + 40);
  if (threadIdx.x == 0) {
    for (int s = 0; s < T.stages; s++) { mbar_init(full0 + 8 * s, 1); mbar_init(empty0 + 8 * s, 1); }
    for (int b = 0; b < 2; b++) { mbar_init(done0 + 8 * b, 1); mbar_init(drained0 + 8 * b, kTcEpi); }
    mbar_init(flushed0, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32((const void*)tmem_slot)), "r"(512u) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_slot;
  grid_enter();                                              // barriers and TMEM are set up under the kernel ahead
  const int n_mt = P.tiles ? *P.n_tiles : T.n_mt;
  const int cols = DUAL ? T.bn / 2 : T.bn;                   // output columns of a tile
  const int n_nt = (P.N + cols - 1) / cols, total = n_mt * n_nt, nk = (P.K + kTcDepth - 1) / kTcDepth;
  const uint32_t stage_bytes = (uint32_t)(kTcRows + T.bn) * kTcDepth * 2;
  // Row tiles first: neighbours share a slice of the weights.  Routed products have a matrix for every other row tile: columns first, so that the tiles of an
  // expert run at a time and its weights, and the rows that all columns read again, cross from HBM once.
  auto row_tile = [&](int tile) { return P.tiles ? tile / n_nt : tile % n_mt; };
  auto column = [&](int tile) { return (P.tiles ? tile % n_nt : tile / n_mt) * cols; };
  if (warp == 0) {
    if (tc_elect()) {
      int it = 0, s = 0;
      uint32_t turn = 1;                                     // parity that a stage's barrier has next
      bool alive = true;
      for (int tile = blockIdx.x; tile < total && alive; tile += gridDim.x) {
        const int mt = row_tile(tile), n0 = column(tile);
        int rowA = mt * kTcRows, rowB = n0;
        if (P.tiles) { const int4 t = P.tiles[mt]; rowA = t.y; rowB += t.x * T.rows_per_expert; }
        for (int kb = 0; kb < nk; kb++, it++) {
          if (!tc_wait(empty0 + 8 * s, turn, T.err)) { alive = false; break; }
          const uint32_t a = base + (uint32_t)s * stage_bytes, b = a + kTcRows * kTcDepth * 2, bar = full0 + 8 * s;
          mbar_expect_tx(bar, stage_bytes);
          tma_tile(a, &mapA, kb * kTcDepth, rowA, bar);
          tma_tile(b, &mapB, kb * kTcDepth, rowB, bar);
          if (DUAL) tma_tile(b + (uint32_t)cols * kTcDepth * 2, &mapB2, kb * kTcDepth, rowB, bar);
          if (++s == T.stages) { s = 0; turn ^= 1; }
        }
      }
      // no copy of this CTA is under way when it leaves, also where a wait gave up (else the products have waited for all of them already)
      for (int i = max(0, it - T.stages); i < it; i++) tc_wait(full0 + 8 * (i % T.stages), (i / T.stages) & 1, T.err);
    }
    __syncwarp();
  } else if (warp == 1) {
    if (tc_elect()) {
      // fp32 accumulate, bf16 x bf16, both K-major
      const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(T.bn / 8) << 17) | ((uint32_t)(kTcRows / 16) << 24);
      int s = 0, nth = 0;
      uint32_t turn = 0;
      bool alive = true;
      for (int tile = blockIdx.x; tile < total && alive; tile += gridDim.x, nth++) {
        const int buf = nth & 1;
        if (!tc_wait(drained0 + 8 * buf, ((nth >> 1) & 1) ^ 1, T.err)) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        for (int kb = 0; kb < nk; kb++) {
          if (!tc_wait(full0 + 8 * s, turn, T.err)) { alive = false; break; }
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint32_t a = base + (uint32_t)s * stage_bytes;
          const uint64_t da = tc_desc(a), db = tc_desc(a + kTcRows * kTcDepth * 2);
#pragma unroll
          for (int k = 0; k < kTcDepth / 16; k++) tc_mma(tmem + buf * 256, da + 2 * k, db + 2 * k, idesc, kb > 0 || k > 0);
          tc_commit(empty0 + 8 * s);
          if (++s == T.stages) { s = 0; turn ^= 1; }
        }
        if (alive) tc_commit(done0 + 8 * buf);
      }
      tc_commit(flushed0);                                   // nor a product, ahead of giving TMEM back
      tc_wait(flushed0, 0, T.err);
    }
    __syncwarp();
  } else {
    const int quad = warp & 3, first = ((warp - 2) >> 2) * 32;   // a warp reads the TMEM lanes of its place in a group of four, every second block of 32 columns
    float* turn = reinterpret_cast<float*>(gbase + kTcRing) + (warp - 2) * 32 * 32;
    int nth = 0;
    for (int tile = blockIdx.x; tile < total; tile += gridDim.x, nth++) {
      const int buf = nth & 1, mt = row_tile(tile), n0 = column(tile);
      int row0 = mt * kTcRows, nrows = min(kTcRows, P.M - row0);
      if (P.tiles) { const int4 t = P.tiles[mt]; row0 = t.y; nrows = t.z; }
      const int mine = min(32, nrows - quad * 32);            // rows of this warp
      // (lanes behind the last row have the first one's: epilogues look up what belongs to a row ahead of asking whether the row is stored)
      int cr_lane = row0 + (lane < mine ? quad * 32 + lane : 0);
      if (!T.C16 && P.c_map) cr_lane = P.c_map[cr_lane];
      // A lane has one row of the accumulator.  Blocks of 32 x 32 are turned through shared memory (16-byte pieces, piece j of row r at place j ^ (r & 7): no bank is met
      // twice), so that eight lanes hold 128 bytes of a row.  Epilogues on top of what C holds read it a block ahead (the first under the products).
      const int sub = lane >> 3, piece = lane & 7;           // this lane's rows 4 i + sub, columns 4 piece .. + 3 of a turned block
      int to[8];
#pragma unroll
      for (int i = 0; i < 8; i++) to[i] = __shfl_sync(0xffffffffu, cr_lane, 4 * i + sub);
      constexpr bool ON_C = EPI == HEPI_ADD || EPI == HEPI_SIGMUL;
      float4 held[ON_C ? 8 : 1];
      auto fetch_c = [&](int c0) {
        if constexpr (ON_C) {
          if (c0 < cols && T.wide && n0 + c0 + 32 <= P.N) {
#pragma unroll
            for (int i = 0; i < 8; i++)
              if (4 * i + sub < mine) held[i] = *reinterpret_cast<const float4*>(P.C + (size_t)to[i] * P.ldc + n0 + c0 + 4 * piece);
          }
        }
      };
      fetch_c(first);
      const bool ok = tc_wait(done0 + 8 * buf, (nth >> 1) & 1, T.err);   // (every lane polls: the loads below are warp-wide)
      if (!__all_sync(0xffffffffu, ok)) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      if (first >= cols && lane == 0) tc_arrive(drained0 + 8 * buf);
      for (int c0 = first; c0 < cols; c0 += 8 * kTcEpi) {
        uint32_t r[32];
        const uint32_t at = tmem + ((uint32_t)(quad * 32) << 16) + buf * 256 + c0;
        tc_load32(at, r);
        uint32_t r2[DUAL ? 32 : 1];
        if constexpr (DUAL) tc_load32(at + cols, r2);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        if (c0 + 8 * kTcEpi >= cols) {                             // the accumulator is read: the next tile but one may have it
          asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
          __syncwarp();
          if (lane == 0) tc_arrive(drained0 + 8 * buf);
        }
        float v[32];
#pragma unroll
        for (int c = 0; c < 32; c++) v[c] = __uint_as_float(r[c]);
        if constexpr (DUAL) {
#pragma unroll
          for (int c = 0; c < 32; c++) v[c] = dual_value<EPI, true>(P, v[c], __uint_as_float(r2[c]));
        }
#pragma unroll
        for (int j = 0; j < 8; j++) *reinterpret_cast<float4*>(turn + lane * 32 + (j ^ (lane & 7)) * 4) = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
        __syncwarp();
        if (T.wide && n0 + c0 + 32 <= P.N) {
          const int n = n0 + c0 + 4 * piece;
          float4 x[8];
#pragma unroll
          for (int i = 0; i < 8; i++) x[i] = *reinterpret_cast<const float4*>(turn + (4 * i + sub) * 32 + (piece ^ ((4 * i + sub) & 7)) * 4);
          if constexpr (!DUAL) {
#pragma unroll
            for (int i = 0; i < 8; i++) {
              const float4 old = ON_C ? held[ON_C ? i : 0] : make_float4(0.f, 0.f, 0.f, 0.f);
              x[i].x = final_value<__nv_bfloat16, EPI, true>(P, to[i], n, x[i].x, old.x);
              x[i].y = final_value<__nv_bfloat16, EPI, true>(P, to[i], n + 1, x[i].y, old.y);
              x[i].z = final_value<__nv_bfloat16, EPI, true>(P, to[i], n + 2, x[i].z, old.z);
              x[i].w = final_value<__nv_bfloat16, EPI, true>(P, to[i], n + 3, x[i].w, old.w);
            }
          }
          fetch_c(c0 + 8 * kTcEpi);
#pragma unroll
          for (int i = 0; i < 8; i++) {
            if (4 * i + sub >= mine) continue;
            if (T.C16) {
              const __nv_bfloat162 lo = __floats2bfloat162_rn(x[i].x, x[i].y), hi = __floats2bfloat162_rn(x[i].z, x[i].w);
              *reinterpret_cast<uint2*>(T.C16 + (size_t)to[i] * T.ldc16 + n) = make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
            } else {
              *reinterpret_cast<float4*>(P.C + (size_t)to[i] * P.ldc + n) = x[i];
            }
          }
        } else {
          const int n = n0 + c0 + lane;
#pragma unroll 4
          for (int i = 0; i < 32; i++) {
            const int cr = __shfl_sync(0xffffffffu, cr_lane, i);
            if (i < mine && n < P.N) {
              float* c = P.C + (size_t)cr * P.ldc + n;
              const float got = turn[i * 32 + ((lane >> 2) ^ (i & 7)) * 4 + (lane & 3)], old = ON_C ? *c : 0.f;
              const float x = DUAL ? got : final_value<__nv_bfloat16, EPI, true>(P, cr, n, got, old);
              if (T.C16) T.C16[(size_t)cr * T.ldc16 + n] = __float2bfloat16_rn(x);
              else *c = x;
            }
          }
        }
        __syncwarp();
      }
    }
  }
  __syncthreads();
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u));
  }
}

// out[i] = bf16(A[a_map ? a_map[i] / a_div : i]), K values each (K a multiple of 8), eight per thread
__global__ void __launch_bounds__(256) bf16_rows(const float* __restrict__ A, int lda, const int* __restrict__ a_map, int a_div, __nv_bfloat16* __restrict__ out,
                                                 int rows, int K, int vec) {
  grid_enter();
  const int per = K / 8;
  const long long n = (long long)rows * per;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const int row = (int)(i / per), k = (int)(i - (long long)row * per) * 8;
    const float* src = A + (size_t)(a_map ? a_map[row] / a_div : row) * lda + k;
    float v[8];
    if (vec) {
      const float4 lo = *reinterpret_cast<const float4*>(src), hi = *reinterpret_cast<const float4*>(src + 4);
      v[0] = lo.x; v[1] = lo.y; v[2] = lo.z; v[3] = lo.w; v[4] = hi.x; v[5] = hi.y; v[6] = hi.z; v[7] = hi.w;
    } else {
#pragma unroll
      for (int q = 0; q < 8; q++) v[q] = src[q];
    }
    uint4 o;
    uint32_t* w = reinterpret_cast<uint32_t*>(&o);
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const __nv_bfloat162 pr = __floats2bfloat162_rn(v[2 * q], v[2 * q + 1]);
      w[q] = *reinterpret_cast<const uint32_t*>(&pr);
    }
    *reinterpret_cast<uint4*>(out + (size_t)row * K + k) = o;
  }
}

// out[i] = in[a_map[i] / a_div], rows of K bf16 values (K a multiple of 8)
__global__ void __launch_bounds__(256) gather_rows16(const __nv_bfloat16* __restrict__ in, const int* __restrict__ a_map, int a_div, __nv_bfloat16* __restrict__ out, int rows, int K) {
  grid_enter();
  const int per = K / 8;
  const long long n = (long long)rows * per;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const int row = (int)(i / per), k = (int)(i - (long long)row * per);
    reinterpret_cast<uint4*>(out + (size_t)row * K)[k] = reinterpret_cast<const uint4*>(in + (size_t)(a_map[row] / a_div) * K)[k];
  }
}

}  // namespace hy
}  // namespace dsk

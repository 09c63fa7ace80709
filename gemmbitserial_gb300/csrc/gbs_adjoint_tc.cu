// gbs_adjoint_tc.cu -- the FP32 adjoint of the bit-serial GEMM on the
// 5th-generation tensor cores, with an exact bf16 split of dC.
//
// No reference counterpart (the reference has no backward pass).  With the
// forward res[n, m] = sum_k A[m, k] * B[n, k] and an FP32 upstream gradient
// dC in the result layout dC[n*M + m]:
//   dA[m, k] = sum_n dC[n, m] * B[n, k]      (M x K, row-major)
//   dB[n, k] = sum_m dC[n, m] * A[m, k]      (N x K, row-major)
// where A and B are the values the planes encode (gemmbitserial.hpp:313-333):
// sum_j s_j 2^j bit_j, s_j = -1 for a signed MSB plane; 2*bit - 1 for bipolar.
//
// Exactness of the operands: every value has at most 8 significant bits, so
// it is exact in bf16.  dC is split as dC = hi + mid + lo with hi = bf16(dC),
// mid = bf16(dC - hi), lo = bf16(dC - hi - mid); each residual is exact in
// fp32 and the three bf16 terms carry all 24 bits of the fp32 significand.
// Every product (8 x 8 significant bits) is exact in fp32.  The tensor core
// accumulates hi*V in one fp32 TMEM accumulator and (mid + lo)*V, 2^-8 of its
// size, in a second; the epilogue adds the two.  So the only rounding is the
// fp32 accumulation itself, done 16 products per MMA step.
//
// Both products are Out[r, k] = sum_s X[r, s] * V[s, k] with the operands left
// as they lie in memory: the three bf16 terms of dC as [3][N][M] (dB: r = n, s
// = m, a contraction-major X; dA: r = m, s = n, an X whose rows r are
// contiguous, which tcgen05 reads as an MN-major operand) and the operand
// values as [rows][K] (V, MN-major).  One pass over dC and the planes
// (adjoint_prepare) makes all of them; transposing dC and the values for a
// contraction-major form took two split passes and two transpositions, 30 us of
// a 174 us adjoint at 4096 x 2048 x 2048.
//
// GEMM kernel: one launch computes dA and dB.  Persistent SM pairs
// (cta_group::2, M = 256, N = 256) walk 256 x 256 tiles of both, the gradient
// with the longer contraction first, the other's tiles and parts of tiles given
// out so that the pairs finish together (deal_tiles).  64 values of s per stage in a 3-stage
// ring, 64 KB of each SM; the leader's TMA loads a stage for both (the three
// terms in one box), its MMA thread issues 12 tcgen05.mma.kind::f16 (K = 16) into
// the two accumulators (all 512 TMEM columns).  Eight epilogue warps add the
// accumulators into registers, release TMEM to the next tile's MMAs and store
// while these run.  Tensor-bound: 0.80 us a stage, its MMAs' own time (12 pair
// MMAs of 66-68 ns); a lone SM on 128 x 256 tiles moved 112 KB of shared memory per
// half stage and ran 0.98 us.  Stages of 32 values hold the same bytes in
// flight, but their 64-byte rows (64-byte swizzle) read slower than whole
// 128-byte ones: 0.93 us per 64 values of the contraction-major gradient.
// Every mbarrier wait is bounded.
#include <cuda_bf16.h>

#include <algorithm>
#include <atomic>
#include <cstdlib>
#include <cstring>

#include "gbs_internal.h"
#include "gbs_tc_common.cuh"

namespace gbs {
namespace {

constexpr int kAdjEpiWarps = 8;
constexpr int kAdjThreads = 64 + 32 * kAdjEpiWarps;
constexpr uint32_t kAdjScratchFloats = 32 * 33;  // per epilogue warp
constexpr int kAdjKs = 64;
constexpr int kAdjStages = 3;
constexpr uint32_t kAdjTermBytes = 128 * kAdjKs * 2;  // one term: 128 rows x kAdjKs bf16
constexpr uint32_t kAdjValBytes = 128 * kAdjKs * 2;   // this CTA's 128 of the tile's 256 value columns
constexpr uint32_t kAdjStageBytes = 3 * kAdjTermBytes + kAdjValBytes;

constexpr size_t adj_smem_bytes() {
  return 1024 + kAdjStages * kAdjStageBytes + kAdjEpiWarps * kAdjScratchFloats * 4 + 8 * (2 * kAdjStages + 3) + 16;
}
static_assert(adj_smem_bytes() <= 232448, "shared memory per CTA");

// One gradient: R x K row-major, tiles row block t / ctiles, column block t % ctiles.
struct AdjOut {
  float *out;
  uint32_t R, tiles, nstages;
  uint32_t idesc;
};

// Tiles of the two gradients dealt to the pairs (deal_tiles): gradient `first`
// round robin (pairs below `a` get one more than the rest), or, with fpieces
// above 1, in that many parts of its contraction, a part a pair; then a
// contiguous run of the other's tiles, sa or sb for a pair below `a` or not;
// the `rem` tiles left over go out in `pieces` parts, a part a pair from p0 on.
struct AdjDeal {
  uint32_t first, pairs, a, sa, sb, rem, pieces, p0, fpieces;
  uint32_t grid;  // pairs that have work
};

struct AdjTcArgs {
  AdjOut o[2];  // 0: dB (contraction-major X), 1: dA (row-contiguous X)
  uint32_t K, ctiles, vec;  // vec: K and both outputs allow 32-byte stores
  AdjDeal deal;
  // split tiles: [first gradient or other][pair][CTA][epilogue warp][128 columns][32 rows] sums of a part,
  // and whether they are there (zeroed by adjoint_prepare)
  float *part;
  uint32_t *flags;
};

// A tile, or part `piece` of `pieces` of its contraction, that a pair works on.
struct AdjTile {
  uint32_t grad, t, piece, pieces;
};

// The i-th of pair p; false when it has no i-th.
__host__ __device__ inline bool dealt_tile(const AdjDeal &d, uint32_t nfirst, uint32_t p, uint32_t i, AdjTile &w) {
  w.piece = 0;
  w.pieces = 1;
  w.grad = d.first;
  uint32_t mine;
  if (d.fpieces > 1) {
    mine = p < nfirst * d.fpieces ? 1 : 0;
    w.t = p / d.fpieces;
    if (i < mine) {
      w.piece = p % d.fpieces;
      w.pieces = d.fpieces;
      return true;
    }
  } else {
    mine = nfirst > p ? (nfirst - p - 1) / d.pairs + 1 : 0;
    w.t = p + i * d.pairs;
    if (i < mine) return true;
  }
  i -= mine;
  w.grad = 1 - d.first;
  const uint32_t per = p < d.a ? d.sa : d.sb;
  w.t = (p < d.a ? p * d.sa : d.a * d.sa + (p - d.a) * d.sb) + i;
  if (i < per) return true;
  const uint32_t x = p - d.p0;
  if (i > per || p < d.p0 || x >= d.rem * d.pieces) return false;
  w.t = d.a * d.sa + (d.pairs - d.a) * d.sb + x / d.pieces;
  w.piece = x % d.pieces;
  w.pieces = d.pieces;
  return true;
}

// Stages [lo, hi) of a tile's contraction that the piece covers.
__host__ __device__ inline void piece_stages(const AdjTile &w, uint32_t nstages, uint32_t &lo, uint32_t &hi) {
  lo = (uint32_t)((uint64_t)w.piece * nstages / w.pieces);
  hi = (uint32_t)((uint64_t)(w.piece + 1) * nstages / w.pieces);
}

__device__ __forceinline__ void mma_bf16_pair(uint32_t tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                              uint32_t acc) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(tmem),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(acc));
}
__device__ __forceinline__ void tma_load_3d_pair(uint32_t dst, const CUtensorMap *map, int x, int y, int z,
                                                 uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.cta_group::2 [%0], [%1, {%2, "
      "%3, %4}], [%5];" ::"r"(dst),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(z), "r"(bar)
      : "memory");
}
__device__ __forceinline__ void tma_load_4d_pair(uint32_t dst, const CUtensorMap *map, int x, int y, int z, int w,
                                                 uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.cta_group::2 [%0], [%1, {%2, "
      "%3, %4, %5}], [%6];" ::"r"(dst),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(z), "r"(w), "r"(bar)
      : "memory");
}
// MN-major operand, 128-byte swizzle: 64 values of the row (column) dimension
// contiguous, the kAdjKs contraction steps of a stage 128 bytes apart (groups of
// 8 1024 bytes apart), the next 64 values after all of them.
__device__ __forceinline__ uint64_t mn128_desc(uint32_t addr) {
  return (uint64_t)((addr & 0x3FFFFu) >> 4) | ((uint64_t)(kAdjKs * 128 >> 4) << 16) | ((uint64_t)(1024 >> 4) << 32) |
         ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&v)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
        "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
      : "r"(taddr));
}
// Waits for the thread's TMEM loads; the registers are operands, so no use of
// them is scheduled ahead of the wait.
__device__ __forceinline__ void tmem_wait_ld16(uint32_t (&v)[16], uint32_t (&w)[16]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(v[0]), "+r"(v[1]), "+r"(v[2]), "+r"(v[3]), "+r"(v[4]), "+r"(v[5]), "+r"(v[6]), "+r"(v[7]),
                 "+r"(v[8]), "+r"(v[9]), "+r"(v[10]), "+r"(v[11]), "+r"(v[12]), "+r"(v[13]), "+r"(v[14]), "+r"(v[15])
               :
               : "memory");
  asm volatile(""
               : "+r"(w[0]), "+r"(w[1]), "+r"(w[2]), "+r"(w[3]), "+r"(w[4]), "+r"(w[5]), "+r"(w[6]), "+r"(w[7]),
                 "+r"(w[8]), "+r"(w[9]), "+r"(w[10]), "+r"(w[11]), "+r"(w[12]), "+r"(w[13]), "+r"(w[14]), "+r"(w[15])
               :
               : "memory");
}

__global__ void __launch_bounds__(kAdjThreads, 1)
    adjoint_tc_kernel(const __grid_constant__ CUtensorMap tmXk, const __grid_constant__ CUtensorMap tmXmn,
                      const __grid_constant__ CUtensorMap tmVa, const __grid_constant__ CUtensorMap tmVb,
                      const __grid_constant__ AdjTcArgs a, uint32_t *err) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t *smem = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t peer = cluster_rank();  // rank 0 leads
  float *scratch = reinterpret_cast<float *>(smem + kAdjStages * kAdjStageBytes);
  uint64_t *bars = reinterpret_cast<uint64_t *>(scratch + kAdjEpiWarps * kAdjScratchFloats);
  const uint32_t full = smem_u32(bars), empty = full + 8 * kAdjStages, acc_full = empty + 8 * kAdjStages;
  const uint32_t acc_empty = acc_full + 8, mma_done = acc_empty + 8;
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(bars + 2 * kAdjStages + 3);
  volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);
  const uint32_t pid = blockIdx.x >> 1, nfirst = a.o[a.deal.first].tiles;
  griddep_launch_dependents();

  if (tid == 0) {
    for (int i = 0; i < kAdjStages; i++) {
      mbar_init(full + 8 * i, 1);
      mbar_init(empty + 8 * i, 1);
    }
    mbar_init(acc_full, 1);
    mbar_init(acc_empty, 2 * kAdjEpiWarps);  // the epilogue warps of both CTAs
    mbar_init(mma_done, 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(tmem_slot)));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;");
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
  asm volatile("tcgen05.fence::after_thread_sync;");
  const uint32_t tmem = *tmem_slot;  // columns [0, 256): hi accumulator; [256, 512): mid + lo
  griddep_wait();  // operands and gradients belong to earlier kernels until here

  if (warp == 0) {
    if (lane == 0 && peer == 0) {
      uint32_t g = 0, k_lo, k_hi;
      AdjTile w;
      bool stop = false;
      for (uint32_t i = 0; !stop && dealt_tile(a.deal, nfirst, pid, i, w); i++) {
        const uint32_t r0 = w.t / a.ctiles * 256u, k0 = w.t % a.ctiles * 256u;
        piece_stages(w, a.o[w.grad].nstages, k_lo, k_hi);
        for (uint32_t k = k_lo; k < k_hi; k++, g++) {
          const uint32_t s = g % kAdjStages, use = g / kAdjStages;
          if (use > 0 && !mbar_wait_err(empty + 8 * s, (use - 1) & 1, abort_flag, err)) {
            stop = true;
            break;
          }
          const uint32_t fb = map_to_rank(full + 8 * s, 0);
          mbar_expect_tx(full + 8 * s, 2 * kAdjStageBytes);
          const uint32_t dst = smem_u32(smem + s * kAdjStageBytes);
          const int sk = (int)(k * kAdjKs);
#pragma unroll
          for (uint32_t h = 0; h < 2; h++) {  // the leader's halves, then the peer's
            const uint32_t d = h ? map_to_rank(dst, 1) : dst;
            if (w.grad == 0) tma_load_3d_pair(d, &tmXk, sk, (int)(r0 + 128 * h), 0, fb);
            else tma_load_4d_pair(d, &tmXmn, 0, sk, (int)(r0 / 64 + 2 * h), 0, fb);
            tma_load_3d_pair(d + 3 * kAdjTermBytes, w.grad == 0 ? &tmVa : &tmVb, 0, sk, (int)(k0 / 64 + 2 * h), fb);
          }
        }
      }
      if (*abort_flag)  // wait (bounded) for the loads the barriers still expect
        for (uint32_t q = (g > (uint32_t)kAdjStages ? g - kAdjStages : 0); q < g; q++)
          mbar_drain_err(full + 8 * (q % kAdjStages), (q / kAdjStages) & 1, err);
    }
  } else if (warp == 1) {
    if (lane == 0 && peer == 0) {
      bool ok = true;
      uint32_t g = 0, k_lo, k_hi;
      AdjTile w;
      for (uint32_t i = 0; ok && dealt_tile(a.deal, nfirst, pid, i, w); i++) {
        if (i > 0 && !mbar_wait_err(acc_empty, (i - 1) & 1, abort_flag, err)) {
          ok = false;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;");
        const uint32_t idesc = a.o[w.grad].idesc;
        piece_stages(w, a.o[w.grad].nstages, k_lo, k_hi);
        for (uint32_t k = k_lo; k < k_hi; k++, g++) {
          const uint32_t s = g % kAdjStages;
          if (!mbar_wait_err(full + 8 * s, (g / kAdjStages) & 1, abort_flag, err)) {
            ok = false;
            break;
          }
          asm volatile("tcgen05.fence::after_thread_sync;");
          const uint32_t base = smem_u32(smem + s * kAdjStageBytes), vb = base + 3 * kAdjTermBytes;
#pragma unroll
          for (int kk = 0; kk < kAdjKs / 16; kk++) {  // K = 16 per MMA
            const uint64_t bd = mn128_desc(vb + kk * 2048);
            const uint32_t more = k != k_lo || kk != 0;
            uint64_t x[3];
#pragma unroll
            for (int j = 0; j < 3; j++)
              x[j] = w.grad == 0 ? sw128_desc(base + j * kAdjTermBytes + kk * 32)
                               : mn128_desc(base + j * kAdjTermBytes + kk * 2048);
            mma_bf16_pair(tmem, x[0], bd, idesc, more);
            mma_bf16_pair(tmem + 256, x[1], bd, idesc, more);
            mma_bf16_pair(tmem + 256, x[2], bd, idesc, 1u);
          }
          mma_commit_pair(empty + 8 * s, 3);
        }
        if (ok) mma_commit_pair(acc_full, 3);
      }
      if (!ok) {  // issued MMAs finish before TMEM is freed
        asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(mma_done)
                     : "memory");
        mbar_drain_err(mma_done, 0, err);
      }
    }
  } else {
    // a warp takes 32 rows (its TMEM lanes) x 128 columns of the tile
    const int q = warp & 3;
    const uint32_t half = (uint32_t)(warp - 2) >> 2;
    float *sc = scratch + (warp - 2) * kAdjScratchFloats;  // [32 rows][33]
    const uint32_t taddr = tmem + ((uint32_t)(q * 32) << 16) + 128 * half;
    // this warp's slot of the partial sums: pair p's of the same CTA and warp are 2 * kAdjEpiWarps slots apart
    const uint32_t slot0 = (pid * 2 + peer) * kAdjEpiWarps + (warp - 2), kind_slots = a.deal.pairs * 2 * kAdjEpiWarps;
    AdjTile w;
    for (uint32_t i = 0; dealt_tile(a.deal, nfirst, pid, i, w); i++) {
      if (!__all_sync(0xffffffffu, mbar_wait_err(acc_full, i & 1, abort_flag, err))) break;
      asm volatile("tcgen05.fence::after_thread_sync;");
      float o[128];
#pragma unroll
      for (int c = 0; c < 128; c += 16) {
        uint32_t hi[16], lo[16];
        tmem_ld16(taddr + c, hi);
        tmem_ld16(taddr + 256 + c, lo);
        tmem_wait_ld16(hi, lo);
#pragma unroll
        for (int j = 0; j < 16; j++) o[c + j] = __uint_as_float(hi[j]) + __uint_as_float(lo[j]);
      }
      asm volatile("tcgen05.fence::before_thread_sync;");
      __syncwarp();
      if (lane == 0) {  // the accumulators may take the next tile
        if (peer == 0) {
          mbar_arrive(acc_empty);
        } else {
          const uint32_t rb = map_to_rank(acc_empty, 0);
          asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(rb) : "memory");
        }
      }
      if (w.pieces > 1) {
        // A split tile: the pairs of its first parts leave their sums, the last part's pair adds them in
        // order.  It waits only for pairs before its own, each of which leaves its sums without waiting.
        const uint32_t slot = slot0 + (w.grad == a.deal.first ? 0 : kind_slots);
        if (w.piece + 1 < w.pieces) {
          float *dst = a.part + (uint64_t)slot * 4096 + lane;
#pragma unroll
          for (int c = 0; c < 128; c++) dst[32 * c] = o[c];
          __threadfence();
          __syncwarp();
          if (lane == 0)
            asm volatile("st.release.gpu.global.u32 [%0], 1;" ::"l"(a.flags + slot) : "memory");
          continue;
        }
        bool ok = true;
        for (uint32_t h = w.pieces - 1; h > 0 && ok; h--) {
          const uint32_t from = slot - h * 2 * kAdjEpiWarps;
          uint32_t seen = 0;
          for (uint32_t it = 0; it < kTcWaitLimit && !seen; it++) {
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(a.flags + from) : "memory");
            if (!seen) {
              if (*abort_flag) break;
              __nanosleep(64);
            }
          }
          ok = __all_sync(0xffffffffu, seen != 0);
          if (!ok) break;
          const float *src = a.part + (uint64_t)from * 4096 + lane;
#pragma unroll
          for (int c = 0; c < 128; c++) o[c] += __ldcg(src + 32 * c);
        }
        if (!ok) {
          *abort_flag = 1;
          if (lane == 0) atomicOr(err, 1u);
          break;
        }
      }
      const uint32_t row0 = w.t / a.ctiles * 256u + 128u * peer + q * 32, col0 = w.t % a.ctiles * 256u + 128 * half;
      const uint32_t R = a.o[w.grad].R;
      if (a.vec) {  // K % 8 == 0: each lane writes its row, 32 bytes at a time
        if (row0 + lane < R) {
          float *p = a.o[w.grad].out + (uint64_t)(row0 + lane) * a.K + col0;
#pragma unroll
          for (int c = 0; c < 128; c += 8)
            if (col0 + c < a.K)
              asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(p + c), "f"(o[c]), "f"(o[c + 1]),
                           "f"(o[c + 2]), "f"(o[c + 3]), "f"(o[c + 4]), "f"(o[c + 5]), "f"(o[c + 6]), "f"(o[c + 7])
                           : "memory");
        }
      } else {  // through shared memory: the lanes write 32 consecutive columns of a row
#pragma unroll
        for (int c = 0; c < 128; c += 32) {
          __syncwarp();
#pragma unroll
          for (int j = 0; j < 32; j++) sc[lane * 33 + j] = o[c + j];
          __syncwarp();
          if (col0 + c + lane < a.K) {
            float *p = a.o[w.grad].out + (uint64_t)row0 * a.K + col0 + c + lane;
#pragma unroll 4
            for (int r = 0; r < 32; r++)
              if (row0 + r < R) p[(uint64_t)r * a.K] = sc[r * 33 + lane];
          }
        }
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;");
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, 512;" ::"r"(tmem));
  }
}

// ------------------------------------------------------------ pre-pass
__device__ __forceinline__ void split3(float x, __nv_bfloat16 &h, __nv_bfloat16 &m, __nv_bfloat16 &l) {
  h = __float2bfloat16_rn(x);
  const float r1 = x - __bfloat162float(h);
  m = __float2bfloat16_rn(r1);
  l = __float2bfloat16_rn(r1 - __bfloat162float(m));
}

__device__ __forceinline__ uint32_t bf16_bits(__nv_bfloat16 x) { return (uint32_t)__bfloat16_as_ushort(x); }

// One operand's values, [rows][pitch] bf16.
struct AdjValues {
  const uint64_t *planes;
  __nv_bfloat16 *out;
  uint64_t plane_words, wpr, pitch;
  uint32_t rows, chunks;  // chunks: 16-column pieces per row
  int nbits, neg_msb;
  uint32_t blocks;  // blocks of the launch that work on it (0: already valid)
  // at most 4 bits: low and high bytes of the bf16 value of every code, 4 per word (four bytes off 16, the prepare
  // pass of a 500 x 777 x 333 step took 2 us more)
  alignas(16) uint32_t lo[4], hi[4];
};

struct AdjPrepare {
  const float *dC;
  __nv_bfloat16 *split;  // [3][N][pM]
  uint64_t pM, term;     // row pitch, elements per term
  uint32_t N, M, chunks, blocks;  // chunks: 8-value pieces per row
  AdjValues v[2];
  uint32_t *flags;  // the GEMM's split-tile flags, zeroed here
  uint32_t nflags;
};

// idx -> (row, piece) of rows of `per` pieces.
__device__ __forceinline__ void piece_of(uint64_t idx, uint32_t per, uint32_t &row, uint32_t &piece) {
  if (idx <= 0xFFFFFFFFull) {
    row = (uint32_t)idx / per;
    piece = (uint32_t)idx - row * per;
  } else {
    row = (uint32_t)(idx / per);
    piece = (uint32_t)(idx - (uint64_t)row * per);
  }
}

// dC into its three terms (8 values a thread, 16 bytes of each term) and both
// operands' planes into bf16 values (16 a thread), in one launch: block ranges.
// 34 MB in, 50 + 25 MB out at 4096 x 2048 x 2048 in 13.8 us, neither HBM (33 %: what it
// writes stays in the L2) nor the SMs (42 %) busy: a warp has one piece's loads in flight.
__global__ void __launch_bounds__(256) adjoint_prepare(const __grid_constant__ AdjPrepare a) {
  griddep_launch_dependents();
  griddep_wait();  // dC, the planes and the workspace belong to earlier kernels until here
  uint32_t b = blockIdx.x;
  if (b == 0)
    for (uint32_t i = threadIdx.x; i < a.nflags; i += 256) a.flags[i] = 0u;
  if (b < a.blocks) {
    const uint64_t idx = (uint64_t)b * 256 + threadIdx.x;
    uint32_t n, c;
    piece_of(idx, a.chunks, n, c);
    if (n >= a.N) return;
    const uint32_t m0 = 8 * c;
    const float *src = a.dC + (uint64_t)n * a.M + m0;
    float x[8];
    if ((a.M & 3) == 0 && m0 + 8 <= a.M) {
      const float4 u = reinterpret_cast<const float4 *>(src)[0], v = reinterpret_cast<const float4 *>(src)[1];
      x[0] = u.x; x[1] = u.y; x[2] = u.z; x[3] = u.w;
      x[4] = v.x; x[5] = v.y; x[6] = v.z; x[7] = v.w;
    } else {
#pragma unroll
      for (int j = 0; j < 8; j++) x[j] = m0 + j < a.M ? src[j] : 0.f;
    }
    uint32_t w[3][4];
#pragma unroll
    for (int j = 0; j < 4; j++) {
      __nv_bfloat16 h0, m0_, l0, h1, m1, l1;
      split3(x[2 * j], h0, m0_, l0);
      split3(x[2 * j + 1], h1, m1, l1);
      w[0][j] = bf16_bits(h0) | (bf16_bits(h1) << 16);
      w[1][j] = bf16_bits(m0_) | (bf16_bits(m1) << 16);
      w[2][j] = bf16_bits(l0) | (bf16_bits(l1) << 16);
    }
    __nv_bfloat16 *dst = a.split + (uint64_t)n * a.pM + m0;  // pM is a multiple of 64: whole pieces
#pragma unroll
    for (int j = 0; j < 3; j++)
      *reinterpret_cast<uint4 *>(dst + j * a.term) = make_uint4(w[j][0], w[j][1], w[j][2], w[j][3]);
    return;
  }
  b -= a.blocks;
  const bool second = b >= a.v[0].blocks;
  const AdjValues &o = a.v[second ? 1 : 0];
  if (second) b -= a.v[0].blocks;
  const uint64_t idx = (uint64_t)b * 256 + threadIdx.x;
  uint32_t r, c;
  piece_of(idx, o.chunks, r, c);
  if (r >= o.rows) return;
  const uint16_t *src = reinterpret_cast<const uint16_t *>(o.planes + (uint64_t)r * o.wpr) + c;
  uint32_t w[8];
  if (o.nbits <= 4) {
    // the plane bits of 4 columns spread to the low bits of 4 nibbles, the planes or-ed into 4 codes, which
    // select their bf16 bytes by byte permutes (adding 16 floats per plane bit by bit took 8 us of integer
    // instructions at 4096 x 2048 and 2048 x 2048)
    uint32_t p[4] = {0u, 0u, 0u, 0u};
#pragma unroll
    for (int i = 0; i < 4; i++)
      if (i < o.nbits) p[i] = src[(uint64_t)i * o.plane_words * 4];
#pragma unroll
    for (int j = 0; j < 4; j++) {
      uint32_t sel = 0u;
#pragma unroll
      for (int i = 0; i < 4; i++) {
        uint32_t x = (p[i] >> (4 * j)) & 15u;
        x = (x | (x << 6)) & 0x0303u;
        sel |= ((x | (x << 3)) & 0x1111u) << i;
      }
      uint32_t lo = __byte_perm(o.lo[0], o.lo[1], sel & 0x7777u), hi = __byte_perm(o.hi[0], o.hi[1], sel & 0x7777u);
      if (o.nbits == 4) {  // codes of 8 and more take the tables' second half
        uint32_t m;  // 0xFF in byte i when code i has bit 3: prmt replicating the sign bits
        asm("prmt.b32 %0, %1, %2, 0xD9C8;" : "=r"(m) : "r"(sel << 4), "r"(sel));
        lo = (lo & ~m) | (__byte_perm(o.lo[2], o.lo[3], sel & 0x7777u) & m);
        hi = (hi & ~m) | (__byte_perm(o.hi[2], o.hi[3], sel & 0x7777u) & m);
      }
      w[2 * j] = __byte_perm(lo, hi, 0x5140u);
      w[2 * j + 1] = __byte_perm(lo, hi, 0x7362u);
    }
  } else {  // bit j of plane i adds +-2^i
    float v[16];
#pragma unroll
    for (int j = 0; j < 16; j++) v[j] = 0.f;
    for (int i = 0; i < o.nbits; i++) {
      const uint32_t bits = src[(uint64_t)i * o.plane_words * 4];
      const float f = i == o.neg_msb ? -(float)(1 << i) : (float)(1 << i);
#pragma unroll
      for (int j = 0; j < 16; j++) v[j] += ((bits >> j) & 1u) ? f : 0.f;
    }
#pragma unroll
    for (int j = 0; j < 8; j++)
      w[j] = bf16_bits(__float2bfloat16_rn(v[2 * j])) | (bf16_bits(__float2bfloat16_rn(v[2 * j + 1])) << 16);
  }
  asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(o.out + (uint64_t)r * o.pitch + 16 * c),
               "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]), "r"(w[4]), "r"(w[5]), "r"(w[6]), "r"(w[7])
               : "memory");
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                  const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn adj_encode_fn() {
  static std::atomic<EncodeTiledFn> fn{nullptr};  // racing first calls store the same value
  EncodeTiledFn f = fn.load(std::memory_order_relaxed);
  if (!f) {
    void *p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess) {
      f = (EncodeTiledFn)p;
      fn.store(f, std::memory_order_relaxed);
    } else {
      cudaGetLastError();
    }
  }
  return f;
}

bool bf16_map(CUtensorMap *map, const void *base, int rank, const cuuint64_t *dims, const cuuint64_t *strides,
              const cuuint32_t *box, CUtensorMapSwizzle swizzle) {
  EncodeTiledFn fn = adj_encode_fn();
  if (!fn) return false;
  const cuuint32_t estr[4] = {1, 1, 1, 1};
  return fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, (cuuint32_t)rank, (void *)base, dims, strides, box, estr,
            CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Operand values [rows][pitch] as [pitch / 64][rows][64]: a box is kAdjKs rows of 128 columns, MN-major.
bool values_map(CUtensorMap *map, const void *base, uint64_t rows, uint64_t pitch) {
  const cuuint64_t dims[3] = {64, rows, pitch / 64}, strides[2] = {pitch * 2, 128};
  const cuuint32_t box[3] = {64, (cuuint32_t)kAdjKs, 2};
  return bf16_map(map, base, 3, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B);
}

uint64_t pitch64(uint64_t x) { return (x + 63) / 64 * 64; }

}  // namespace

// Workspace of a context's tensor-core adjoint: the three terms of dC and both
// operands' values, with their tensor maps.  Row pitches are multiples of 64
// values, so a box of an MN-major map never leaves its row's pitch; columns past
// the matrix are unwritten there and reach only outputs that are not stored.
struct AdjPlan {
  __nv_bfloat16 *ws = nullptr;
  __nv_bfloat16 *split = nullptr;  // [3][N][pM]
  __nv_bfloat16 *val[2] = {};      // lhs values [M][pK], rhs values [N][pK]
  CUtensorMap xk, xmn, va, vb;
  float *part = nullptr;      // split tiles' sums and flags (AdjTcArgs), behind the operands, when a deal splits
  uint32_t *flags = nullptr;
  uint32_t nflags = 0;
  AdjDeal deal[4];            // by the wanted gradients: bit 0 dB, bit 1 dA
};

void adj_plan_free(AdjPlan *p) {
  if (!p) return;
  if (p->ws) cudaFree(p->ws);
  delete p;
}

bool adjoint_tc_available() { return adj_encode_fn() != nullptr; }

namespace {

// SM pairs the adjoint kernel can hold at once, cached per device.
int adj_max_pairs() {
  static std::atomic<int> cache[64];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
  int v = cache[dev].load(std::memory_order_relaxed);
  if (v == 0) {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.gridDim = dim3(2);
    cfg.blockDim = dim3(kAdjThreads);
    cfg.dynamicSmemBytes = adj_smem_bytes();
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int n = 0;
    cudaError_t e = cudaFuncSetAttribute(adjoint_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)adj_smem_bytes());
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveClusters(&n, adjoint_tc_kernel, &cfg);
    if (e != cudaSuccess || n < 1) {
      cudaGetLastError();
      return 0;
    }
    v = n;
    cache[dev].store(v, std::memory_order_relaxed);
  }
  return v;
}

// Deals nfirst tiles of cfirst stages round robin over the pairs, then nother
// tiles of cother stages in whole rounds over the pairs with the least work so
// far; the tiles left over, fewer than those pairs, are split in parts of at
// least kMinPiece stages.  4096 x 2048 x 2048: 64 tiles of 64 stages and 128 of
// 32 over 76 pairs; whole tiles only would end with 28 pairs a tile (26 us)
// behind the rest, halves of those 28 end half a tile behind.  Few long tiles (a
// large batch against a small layer) are split too, in as many parts as end soonest.
// A part costs its sums' way through L2, about 3 us: kMinPiece stages of 0.8 us keep
// it worth while.  A tile takes about 4 us, kTileStages stages, for its stores however short
// its contraction: counted by their stages alone, the 256 one-stage tiles of dA at 4096
// x 4096 x 1 all went to the 12 pairs that dB's long ones had left idle (109 us, 69 so;
// 4096 x 4096 x 64 86 and 45).
constexpr uint32_t kMinPiece = 6, kMaxPieces = 8, kTileStages = 5, kPieceStages = 4;

// The deal with the first gradient's tiles in fpieces parts, and the stages until it ends.
AdjDeal deal_parts(uint32_t first, uint64_t nfirst, uint64_t cfirst, uint64_t nother, uint64_t cother, uint32_t pairs,
                   uint32_t fpieces, uint64_t &span) {
  AdjDeal d;
  memset(&d, 0, sizeof(d));
  d.first = first;
  d.pairs = pairs;
  d.pieces = 1;
  d.fpieces = fpieces;
  const bool split = fpieces > 1;
  d.a = (uint32_t)(split ? nfirst * fpieces : nfirst % pairs);
  const uint64_t tfirst = std::max<uint64_t>(cfirst, kTileStages), tother = std::max<uint64_t>(cother, kTileStages);
  const uint64_t size[2] = {d.a, pairs - d.a};
  uint64_t load[2] = {split ? (cfirst + fpieces - 1) / fpieces + kPieceStages : (nfirst / pairs + 1) * tfirst,
                      split ? 0 : nfirst / pairs * tfirst};
  uint64_t s[2] = {0, 0}, takers = pairs;
  int g = 0;
  while (nother) {
    // (the last few whole tiles, where both are equal, to the pairs that had no long ones)
    const bool all = !size[0] || !size[1] ||
                     (load[0] == load[1] && (nother > size[1] || cother >= 2 * kMinPiece));
    g = load[0] < load[1] ? 0 : 1;
    takers = all ? pairs : size[g];
    d.p0 = all || g == 0 ? 0 : d.a;
    if (nother < takers) break;
    for (int i = 0; i < 2; i++)
      if (all || i == g) {
        s[i]++;
        load[i] += tother;
      }
    nother -= takers;
  }
  d.sa = (uint32_t)s[0];
  d.sb = (uint32_t)s[1];
  d.rem = (uint32_t)nother;
  if (nother) {
    d.pieces = (uint32_t)std::max<uint64_t>(
        1, std::min<uint64_t>(std::min<uint64_t>(kMaxPieces, takers / nother), cother / kMinPiece));
    load[g] += d.pieces > 1 ? (cother + d.pieces - 1) / d.pieces + kPieceStages : tother;
  }
  span = std::max(size[0] ? load[0] : 0, size[1] ? load[1] : 0);
  return d;
}

AdjDeal deal_tiles(uint32_t first, uint64_t nfirst, uint64_t cfirst, uint64_t nother, uint64_t cother,
                   uint32_t pairs) {
  uint64_t best = 0, span = 0;
  AdjDeal d = deal_parts(first, nfirst, cfirst, nother, cother, pairs, 1, best);
  for (uint32_t f = 2; nfirst && f <= kMaxPieces && nfirst * f <= pairs && cfirst / f >= kMinPiece; f++) {
    const AdjDeal e = deal_parts(first, nfirst, cfirst, nother, cother, pairs, f, span);
    if (10 * span < 9 * best) {  // parts of long tiles, unless a tenth is all they save
      best = span;
      d = e;
    }
  }
  AdjTile w;
  for (d.grid = pairs; d.grid > 1 && !dealt_tile(d, (uint32_t)(d.fpieces > 1 || nfirst < pairs ? nfirst : pairs),
                                                 d.grid - 1, 0, w);)
    d.grid--;
  return d;
}

uint32_t adj_stages(uint64_t S) { return (uint32_t)((S + kAdjKs - 1) / kAdjKs); }
uint32_t adj_tiles(uint64_t R, uint64_t K) { return (uint32_t)(((R + 255) / 256) * ((K + 255) / 256)); }

int build_plan(gbs_ctx *c) {
  const uint64_t M = c->lhs.nrows, N = c->rhs.nrows, K = c->lhs.ncols;
  const uint64_t pM = pitch64(M), pK = pitch64(K), term = N * pM;
  AdjPlan *p = new AdjPlan();
  const int max_pairs = adj_max_pairs();
  if (!max_pairs) {
    adj_plan_free(p);
    return fail(GBS_ECUDA, "gbs_adjoint: the SM-pair kernel does not fit this device");
  }
  uint32_t split_pairs = 0;
  for (uint32_t want = 1; want < 4; want++) {
    const uint32_t n[2] = {(want & 1) ? adj_tiles(N, K) : 0, (want & 2) ? adj_tiles(M, K) : 0};
    const uint32_t cost[2] = {adj_stages(M), adj_stages(N)};
    const uint32_t pairs = (uint32_t)std::min<uint64_t>(
        (uint64_t)max_pairs, std::max<uint64_t>((uint64_t)n[0] + n[1], 1) * kMaxPieces);
    // the gradient with the longer contraction first; a lone one is dealt as the other, which may split
    const uint32_t first = !n[0] ? 0 : !n[1] ? 1 : cost[0] >= cost[1] ? 0 : 1;
    p->deal[want] = deal_tiles(first, n[first], cost[first], n[1 - first], cost[1 - first], pairs);
    if (p->deal[want].pieces > 1 || p->deal[want].fpieces > 1) split_pairs = std::max(split_pairs, pairs);
  }
  p->nflags = 2 * split_pairs * 2 * kAdjEpiWarps;
  // One allocation: operands (every array starts on a 128-byte boundary: the pitches are multiples of 64 values),
  // then the split tiles' sums and flags
  const size_t bytes = ((3 * term + (M + N) * pK) * sizeof(__nv_bfloat16) + 255) / 256 * 256;
  const size_t sums = (size_t)p->nflags * 4096 * sizeof(float);
  if (dev_alloc((void **)&p->ws, bytes + sums + p->nflags * sizeof(uint32_t)) != cudaSuccess) {
    cudaGetLastError();
    delete p;
    return fail(GBS_ENOMEM, "gbs_adjoint: workspace allocation failed");
  }
  if (split_pairs) {
    p->part = reinterpret_cast<float *>(reinterpret_cast<uint8_t *>(p->ws) + bytes);
    p->flags = reinterpret_cast<uint32_t *>(reinterpret_cast<uint8_t *>(p->part) + sums);
  }
  p->split = p->ws;
  p->val[0] = p->ws + 3 * term;
  p->val[1] = p->val[0] + M * pK;
  // dB: rows n, contraction m (contiguous); the true M and N bound the boxes, past them reads are 0
  const cuuint64_t dk[3] = {M, N, 3}, sk[2] = {pM * 2, term * 2};
  const cuuint32_t bk[3] = {(cuuint32_t)kAdjKs, 128, 3};
  // dA: rows m (contiguous, 64 at a time), contraction n
  const cuuint64_t dmn[4] = {64, N, pM / 64, 3}, smn[3] = {pM * 2, 128, term * 2};
  const cuuint32_t bmn[4] = {64, (cuuint32_t)kAdjKs, 2, 3};
  if (!bf16_map(&p->xk, p->split, 3, dk, sk, bk, CU_TENSOR_MAP_SWIZZLE_128B) ||
      !bf16_map(&p->xmn, p->split, 4, dmn, smn, bmn, CU_TENSOR_MAP_SWIZZLE_128B) ||
      !values_map(&p->va, p->val[0], M, pK) || !values_map(&p->vb, p->val[1], N, pK)) {
    adj_plan_free(p);
    return fail(GBS_EUNSUPPORTED, "gbs_adjoint: tensor map encoding failed");
  }
  c->adj = p;
  return GBS_OK;
}

AdjValues values_job(const Mat &op, __nv_bfloat16 *out, bool wanted) {
  AdjValues v;
  memset(&v, 0, sizeof(v));
  v.planes = op.planes;
  v.out = out;
  v.plane_words = op.nrows_a * op.wpr();
  v.wpr = op.wpr();
  v.pitch = pitch64(op.ncols);
  v.rows = (uint32_t)op.nrows;
  v.chunks = (uint32_t)((op.ncols + 15) / 16);
  v.nbits = (int)op.nbits;
  v.neg_msb = (op.issigned && !op.bipolar()) ? (int)op.nbits - 1 : -1;
  for (int code = 0; code < 16 && op.nbits <= 4; code++) {  // bf16 of small integers: the high half of the float
    int x = op.bipolar() ? ((code & 1) ? 1 : -1) : 0;
    for (int i = 0; i < v.nbits && !op.bipolar(); i++)
      if ((code >> i) & 1) x += i == v.neg_msb ? -(1 << i) : 1 << i;
    const float f = (float)x;
    uint32_t bits;
    memcpy(&bits, &f, 4);
    v.lo[code >> 2] |= ((bits >> 16) & 0xFFu) << (8 * (code & 3));
    v.hi[code >> 2] |= (bits >> 24) << (8 * (code & 3));
  }
  v.blocks = wanted ? (uint32_t)(((uint64_t)v.rows * v.chunks + 255) / 256) : 0;
  return v;
}

}  // namespace

// dA = dC . B and dB = dC^T . A on the tensor cores (either output may be null).
int adjoint_tc(gbs_ctx *c, const float *dC, float *dA, float *dB, cudaStream_t s) {
  const uint64_t M = c->lhs.nrows, N = c->rhs.nrows, K = c->lhs.ncols;
  if (M * K + N * K == 0) return GBS_OK;
  if (M == 0 || N == 0) {  // an empty contraction: zero gradients
    cudaError_t e = cudaSuccess;
    if (dA && M && K) e = cudaMemsetAsync(dA, 0, M * K * 4, s);
    if (e == cudaSuccess && dB && N && K) e = cudaMemsetAsync(dB, 0, N * K * 4, s);
    return e == cudaSuccess ? GBS_OK : cuda_fail(e, "gbs_adjoint: memset");
  }
  if (!dA && !dB) return GBS_OK;
  if (!c->adj) {
    const int rc = build_plan(c);
    if (rc != GBS_OK) return rc;
  }
  AdjPlan &p = *c->adj;
  // dB contracts over m with A's values, dA over n with B's
  const bool want[2] = {dB != nullptr, dA != nullptr};
  AdjPrepare pr;
  memset(&pr, 0, sizeof(pr));
  pr.dC = dC;
  pr.split = p.split;
  pr.pM = pitch64(M);
  pr.term = N * pr.pM;
  pr.N = (uint32_t)N;
  pr.M = (uint32_t)M;
  pr.chunks = (uint32_t)((M + 7) / 8);
  pr.blocks = (uint32_t)((N * pr.chunks + 255) / 256);
  pr.v[0] = values_job(c->lhs, p.val[0], want[0] && !c->vt_valid[0]);
  pr.v[1] = values_job(c->rhs, p.val[1], want[1] && !c->vt_valid[1]);
  pr.flags = p.flags;
  pr.nflags = p.nflags;
  cudaError_t e = launch_pdl(adjoint_prepare, pr.blocks + pr.v[0].blocks + pr.v[1].blocks, 256, 0, s, pr);
  count_launch();
  if (e != cudaSuccess) return cuda_fail(e, "gbs_adjoint: split kernel");
  for (int side = 0; side < 2; side++)
    if (want[side]) c->vt_valid[side] = true;

  AdjTcArgs a;
  memset(&a, 0, sizeof(a));
  a.K = (uint32_t)K;
  a.ctiles = (uint32_t)((K + 255) / 256);
  a.vec = K % 8 == 0 && ((uintptr_t)dA | (uintptr_t)dB) % 32 == 0;
  for (int g = 0; g < 2; g++) {
    AdjOut &o = a.o[g];
    const uint64_t R = g ? M : N, S = g ? N : M;
    o.out = g ? dA : dB;
    o.R = (uint32_t)R;
    o.tiles = want[g] ? adj_tiles(R, K) : 0;
    o.nstages = adj_stages(S);
    // kind::f16: D fp32, A and B bf16, M = 256, N = 256; B MN-major, A MN-major for dA
    o.idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)g << 15) | (1u << 16) | ((256u >> 3) << 17) |
              ((256u >> 4) << 24);
  }
  a.deal = p.deal[(dB ? 1 : 0) | (dA ? 2 : 0)];
  a.part = p.part;
  a.flags = p.flags;
  uint32_t *err = tc_error_ptr();
  if (!err) return fail(GBS_ECUDA, "gbs_adjoint: no error word");
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.gridDim = dim3(2 * a.deal.grid);
  cfg.blockDim = dim3(kAdjThreads);
  cfg.dynamicSmemBytes = adj_smem_bytes();
  cfg.stream = s;
  cfg.attrs = attr;
  cfg.numAttrs = pdl_for(s) ? 2 : 1;
  e = cudaLaunchKernelEx(&cfg, adjoint_tc_kernel, p.xk, p.xmn, p.va, p.vb, a, err);
  count_launch();
  return e == cudaSuccess ? GBS_OK : cuda_fail(e, "gbs_adjoint: GEMM kernel");
}

}  // namespace gbs

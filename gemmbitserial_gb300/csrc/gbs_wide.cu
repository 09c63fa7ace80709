// gbs_wide.cu -- the tensor-core digit pipe for operands of 5 to 8 bits.
//
// An operand of w > 4 bits does not fit one e4m3 digit exactly, so it is
// split by planes into a low part (planes [0, lo), unsigned, lo = w - hi) and
// a high part (planes [lo, w), signed when the operand is, hi = max(2, w - 4)
// bits: never a lone signed plane, which would read as bipolar).  Each part
// holds at most 4 significant bits, so
//   A.B = sum_{pa, pb} 2^(lo_A pa + lo_B pb) (A_pa . B_pb)
// the plane-weight identity of gemmBitSerial_generic_usingBinary
// (arch-generic.hpp:179-192) grouped by part instead of by single plane.
//
// Fused form (M, N >= 256): one SM-pair kernel runs every part product.  A
// stage loads each part tile once and multiplies every (lhs part, rhs part)
// of it into two fp32 accumulators, X and Y (all 512 TMEM columns).  e4m3
// holds a part times a power of two just as exactly, so scaled parts let
// several products share an accumulator.  With l = min(lo_A, lo_B), on the
// side whose lo is l the low part is stored times 2^-l, on the other the high part
// times 2^lo; then for two wide operands (say lo_A = l)
//   X = ah.(2^lo_B bh) + ah.bl + (2^-l al).(2^lo_B bh),  Y = (2^-l al).bl
//   A.B = 2^l X + 2^l Y
// and for one wide operand X = ah.b, Y = al.b, A.B = 2^lo X + Y (parts
// unscaled).  X and Y are exact while K times the largest |term| sum stays
// below 2^24 (X in units of 1, Y in units of 2^-l); longer K splits in two or
// four over as many times the CTAs, whose int32 partial results the combine kernel
// adds.  8 x 8 bits at 2048 x 4096 x 2048: four part GEMMs and their
// combination took 87 us and re-read both operands twice.
//
// Separate form (a side under 256 rows, K beyond the splits, forced
// variants): every part product is an ordinary digit GEMM on a sub-context
// whose planes alias the parent's, exact while K * max|a part| * max|b part| <
// 2^24, and one combine kernel sums the shifted partial results.  All sums are
// 32-bit wrap-around arithmetic, as the reference's int32 accumulators.
#include <algorithm>
#include <cstring>

#include "gbs_internal.h"
#include "gbs_tc_common.cuh"

namespace gbs {

struct WidePlan {
  int parts[2] = {1, 1};    // parts per side (1 or 2)
  int lo_bits[2] = {0, 0};  // bits of a side's low part (the high part's weight is 2^lo_bits)
  // Each form has its own [side][part] digit matrices (a captured graph of one
  // must not find the other's): the fused form's match the planes while the
  // context's digits_valid says so, the separate form's while its packed_valid
  // does (a wide context has no packed matrices of its own).
  uint8_t *sep[2][2] = {{nullptr, nullptr}, {nullptr, nullptr}};
  gbs_ctx *sub[2][2] = {{nullptr, nullptr}, {nullptr, nullptr}};  // [lhs part][rhs part], separate form
  int fused_splits = 0;  // K splits of the fused kernel, 0: the separate form only
  uint8_t *digits[2][2] = {{nullptr, nullptr}, {nullptr, nullptr}};
  int scale[2][2] = {{0, 0}, {0, 0}};  // power of two of the fused form's digits
  CUtensorMap maps[2][2];   // [side][part] digit maps, boxes of 128 rows
  int32_t *partial = nullptr;  // fused_splits results when it splits
};

namespace {

int hi_bits(int w) { return w > 4 ? std::max(2, w - 4) : 0; }

// Part `part` of operand m (part 0 is the whole operand when it has <= 4 bits).
Mat part_of(const Mat &m, int part) {
  const int w = (int)m.nbits, hi = hi_bits(w), lo = w - hi;
  Mat p = m;
  if (w <= 4) return p;
  if (part == 0) {
    p.nbits = (uint64_t)lo;
    p.issigned = 0;
  } else {
    p.nbits = (uint64_t)hi;
    p.planes = m.planes + (uint64_t)lo * m.nrows_a * m.wpr();
  }
  return p;
}

uint64_t part_max_abs(const Mat &m) {
  if (m.bipolar()) return 1;
  return m.issigned ? (1ull << (m.nbits - 1)) : ((1ull << m.nbits) - 1);
}

// out[i] = sum_k in_k[i] << shift_k (mod 2^32), 4 elements per thread
__global__ void __launch_bounds__(256) combine_kernel(int32_t *__restrict__ out, const int32_t *__restrict__ in0,
                                                      const int32_t *__restrict__ in1, const int32_t *__restrict__ in2,
                                                      const int32_t *__restrict__ in3, int nin, uint32_t sh1,
                                                      uint32_t sh2, uint32_t sh3, uint64_t n) {
  griddep_launch_dependents();
  griddep_wait();
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t q = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; q < (n + 3) / 4; q += stride) {
    const uint64_t i0 = 4 * q;
    if (i0 + 4 <= n) {
      uint4 a = *reinterpret_cast<const uint4 *>(in0 + i0);
      auto add = [&](const int32_t *in, uint32_t sh) {
        const uint4 b = *reinterpret_cast<const uint4 *>(in + i0);
        a.x += b.x << sh;
        a.y += b.y << sh;
        a.z += b.z << sh;
        a.w += b.w << sh;
      };
      if (nin > 1) add(in1, sh1);
      if (nin > 2) add(in2, sh2);
      if (nin > 3) add(in3, sh3);
      *reinterpret_cast<uint4 *>(out + i0) = a;
    } else {
      for (uint64_t i = i0; i < n; i++) {
        uint32_t v = (uint32_t)in0[i];
        if (nin > 1) v += (uint32_t)in1[i] << sh1;
        if (nin > 2) v += (uint32_t)in2[i] << sh2;
        if (nin > 3) v += (uint32_t)in3[i] << sh3;
        out[i] = (int32_t)v;
      }
    }
  }
}

constexpr int kWideThreads = 192;
constexpr uint32_t kWideTile = 128 * 128;  // 128 rows x 128 digits of one part

constexpr int wide_stages(int parts) { return (int)((227 * 1024 - 1024 - 256) / (parts * kWideTile)); }
constexpr size_t wide_smem(int parts) {
  return 1024 + (size_t)wide_stages(parts) * parts * kWideTile + 8 * (2 * wide_stages(parts) + 2) + 16;
}

struct WideArgs {
  int32_t *C;          // result, or the first of the splits' partial results
  uint64_t M, N, cstride;  // cstride: elements from one split's results to the next (16-byte aligned)
  uint32_t nstages;    // K stages of 128 digits
  uint32_t splits;
  uint32_t idesc;
  uint32_t xshift;     // result = (X << xshift) + Y * yscale
  float yscale;
};

// 256 x 256 tiles on SM pairs (tcgen05.mma.cta_group::2, M = 256, N = 256),
// every part product of the tile: the leader's TMA loads PA + PB part tiles a
// stage for both CTAs, its MMA thread issues PA * PB products of 4 K steps, X in
// TMEM columns [0, 256), Y in [256, 512).  Tensor-bound: a stage's 16 pair MMAs
// (8 x 8 bits) take 1.15 us against the 0.54 us of its 64 KB per SM -- each
// tile is read by two products, so the shared-memory traffic that holds the one-product
// kernel to 0.75 of the MMA rate is halved.  blockIdx.z is the K split.
// Every wait is bounded, with the SM-pair kernel's abort path.
template <int PA, int PB>
__global__ void __launch_bounds__(kWideThreads, 1)
    gemm_wide_pair_kernel(const __grid_constant__ CUtensorMap tmA0, const __grid_constant__ CUtensorMap tmA1,
                          const __grid_constant__ CUtensorMap tmB0, const __grid_constant__ CUtensorMap tmB1,
                          WideArgs a, uint32_t *err) {
  constexpr int kStages = wide_stages(PA + PB);
  constexpr uint32_t kStageBytes = (PA + PB) * kWideTile;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t *smem = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t peer = cluster_rank();  // the pair's leader is rank 0
  uint64_t *bars = reinterpret_cast<uint64_t *>(smem + kStages * kStageBytes);
  const uint32_t full = smem_u32(bars), empty = full + 8 * kStages, acc_full = empty + 8 * kStages;
  const uint32_t mma_done = acc_full + 8;
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(bars + 2 * kStages + 2);
  volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);
  const uint32_t m0 = (blockIdx.x >> 1) * 256, n0 = blockIdx.y * 256;
  const uint32_t k_lo = (uint32_t)((uint64_t)blockIdx.z * a.nstages / a.splits);
  const uint32_t nk = (uint32_t)((uint64_t)(blockIdx.z + 1) * a.nstages / a.splits) - k_lo;
  griddep_launch_dependents();
  if (tid == 0) {
    for (int i = 0; i < kStages; i++) {
      mbar_init(full + 8 * i, 1);
      mbar_init(empty + 8 * i, 1);
    }
    mbar_init(acc_full, 1);
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
  const uint32_t tmem = *tmem_slot;
  griddep_wait();  // operands and result belong to the previous kernels until here

  if (warp == 0) {
    if (lane == 0 && peer == 0) {
      uint32_t issued = 0;
      for (uint32_t k = 0; k < nk; k++) {
        const uint32_t s = k % kStages, use = k / kStages;
        if (use > 0 && !mbar_wait_err(empty + 8 * s, (use - 1) & 1, abort_flag, err)) break;
        const uint32_t fb = map_to_rank(full + 8 * s, 0);
        mbar_expect_tx(full + 8 * s, 2 * kStageBytes);
        const uint32_t dst = smem_u32(smem + s * kStageBytes);
        const int kc = (int)(k_lo + k);
#pragma unroll
        for (uint32_t p = 0; p < 2; p++) {  // the leader's own tiles, then the peer's
          uint32_t d = p ? map_to_rank(dst, 1) : dst;
          tma_load_digits_pair(d, &tmA0, kc, m0 + 128 * p, fb);
          d += kWideTile;
          if (PA == 2) {
            tma_load_digits_pair(d, &tmA1, kc, m0 + 128 * p, fb);
            d += kWideTile;
          }
          tma_load_digits_pair(d, &tmB0, kc, n0 + 128 * p, fb);
          d += kWideTile;
          if (PB == 2) tma_load_digits_pair(d, &tmB1, kc, n0 + 128 * p, fb);
        }
        issued = k + 1;
      }
      if (*abort_flag)  // wait (bounded) for the loads the barriers still expect, in the peer's memory too
        for (uint32_t k = (issued > (uint32_t)kStages ? issued - kStages : 0); k < issued; k++)
          mbar_drain_err(full + 8 * (k % kStages), (k / kStages) & 1, err);
    }
  } else if (warp == 1) {
    if (lane == 0 && peer == 0) {
      bool ok = true;
      for (uint32_t k = 0; k < nk; k++) {
        const uint32_t s = k % kStages;
        if (!mbar_wait_err(full + 8 * s, (k / kStages) & 1, abort_flag, err)) {
          ok = false;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;");
        const uint32_t base = smem_u32(smem + s * kStageBytes);
        const uint32_t A0 = base, A1 = base + kWideTile, B0 = base + PA * kWideTile, B1 = B0 + kWideTile;
#pragma unroll
        for (int kk = 0; kk < 4; kk++) {
          const uint32_t more = (k | kk) != 0, o = kk * 32;
          if (PA == 2 && PB == 2) {
            mma_f8_pair(tmem, sw128_desc(A1 + o), sw128_desc(B1 + o), a.idesc, more);
            mma_f8_pair(tmem, sw128_desc(A1 + o), sw128_desc(B0 + o), a.idesc, 1u);
            mma_f8_pair(tmem, sw128_desc(A0 + o), sw128_desc(B1 + o), a.idesc, 1u);
          } else if (PA == 2) {
            mma_f8_pair(tmem, sw128_desc(A1 + o), sw128_desc(B0 + o), a.idesc, more);
          } else {
            mma_f8_pair(tmem, sw128_desc(A0 + o), sw128_desc(B1 + o), a.idesc, more);
          }
          mma_f8_pair(tmem + 256, sw128_desc(A0 + o), sw128_desc(B0 + o), a.idesc, more);
        }
        mma_commit_pair(empty + 8 * s, 3);
      }
      if (ok) {
        mma_commit_pair(acc_full, 3);
      } else {  // issued MMAs finish before TMEM is freed
        asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(mma_done)
                     : "memory");
        mbar_drain_err(mma_done, 0, err);
      }
    }
  } else if (__all_sync(0xffffffffu, mbar_wait_err(acc_full, 0, abort_flag, err))) {
    asm volatile("tcgen05.fence::after_thread_sync;");
    const int q = warp & 3;
    const uint64_t gm = m0 + 128 * peer + q * 32 + lane;
    const uint32_t taddr = tmem + ((uint32_t)(q * 32) << 16);
    int32_t *C = a.C + (uint64_t)blockIdx.z * a.cstride;
#pragma unroll 1
    for (uint32_t col = 0; col < 256; col += 64) {
      uint32_t x[2][32], y[2][32];
#pragma unroll
      for (int i = 0; i < 2; i++) {
        tmem_ld32(taddr + col + 32 * i, x[i]);
        tmem_ld32(taddr + 256 + col + 32 * i, y[i]);
      }
      tmem_wait_ld(x[0]);
      tmem_after_wait(x[1]);
      tmem_after_wait(y[0]);
      tmem_after_wait(y[1]);
#pragma unroll
      for (int i = 0; i < 2; i++) {
        int32_t o[32];
#pragma unroll
        for (int j = 0; j < 32; j++)
          o[j] = (int32_t)(((uint32_t)__float2int_rn(__uint_as_float(x[i][j])) << a.xshift) +
                           (uint32_t)__float2int_rn(__uint_as_float(y[i][j]) * a.yscale));
        store_result_cols<32>(C, a.M, a.N, gm, n0 + col + 32 * i, o);
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

// K splits of the fused kernel, or 0 when it does not take the context.  Every
// split's X and Y must stay exact; of the splits that do, the least estimated
// time: a stage costs 0.29 us a product and a wave 7 us of setup, first load
// and epilogue, a split result its partials' traffic at ~6 TB/s and 3 us of
// launch (one 256 x 256 tile to a pair of SMs, 76 pairs).
int fused_splits(const gbs_ctx *c, const WidePlan &p) {
  const Mat &A = c->lhs, &B = c->rhs;
  if (A.nrows < 256 || B.nrows < 256) return 0;
  const bool two = p.parts[0] == 2 && p.parts[1] == 2;
  double bound;  // largest |X| or |Y| (in its units) per element of K
  if (two) {
    const int l = std::min(p.lo_bits[0], p.lo_bits[1]), s = p.lo_bits[0] == l ? 0 : 1;
    const Mat &P = s ? B : A, &Q = s ? A : B;  // P: the side whose lo is l
    const double ph = (double)part_max_abs(part_of(P, 1)), pl = (double)part_max_abs(part_of(P, 0));
    const double qh = (double)part_max_abs(part_of(Q, 1)), ql = (double)part_max_abs(part_of(Q, 0));
    const double u = (double)(1u << p.lo_bits[1 - s]);
    bound = std::max(u * ph * qh + ph * ql + u / (double)(1u << l) * pl * qh, pl * ql);
  } else {
    const Mat &W = p.parts[0] == 2 ? A : B, &R = p.parts[0] == 2 ? B : A;
    bound = (double)part_max_abs(R) *
            (double)std::max(part_max_abs(part_of(W, 0)), part_max_abs(part_of(W, 1)));
  }
  const uint64_t stages = A.dcols / 128, tiles = ((A.nrows + 255) / 256) * ((B.nrows + 255) / 256);
  if (tiles > 65535ull * 128 || (B.nrows + 255) / 256 > 65535) return 0;
  const double stage_us = 0.29 * p.parts[0] * p.parts[1], mn = (double)A.nrows * (double)B.nrows;
  int best = 0;
  double best_us = 0.0;
  for (int s : {1, 2, 4}) {
    const uint64_t chunk = (stages + s - 1) / s;
    if ((uint64_t)s > stages || (double)std::min<uint64_t>(chunk * 128, A.ncols) * bound >= 16777216.0) continue;
    const double waves = (double)((tiles * s + 75) / 76);
    const double us = waves * ((double)chunk * stage_us + 7.0) + (s > 1 ? 3.0 + (s + 1) * 4.0 * mn / 6e6 : 0.0);
    if (!best || us < best_us) {
      best = s;
      best_us = us;
    }
  }
  return best;
}

// Digit matrices of part `part` of a side: from unscaled to the fused kernel's scaled table.
void scale_table(uint32_t (&tab)[4], int power) {
  for (uint32_t &w : tab) {
    uint32_t r = 0;
    for (int i = 0; i < 4; i++) {
      const uint32_t b = (w >> (8 * i)) & 0xFFu;  // sign, exponent << 3, mantissa: a power of two moves the exponent
      r |= ((b & 0x7Fu) ? (uint32_t)((int)b + 8 * power) & 0xFFu : 0u) << (8 * i);
    }
    w = r;
  }
}

cudaError_t alloc_parts(const gbs_ctx *c, const WidePlan &p, uint8_t *(&digits)[2][2]) {
  // (both sides' buffers at once, which the two imports may write on different streams: zeroed before returning;
  // one allocation, whose start is the lhs's first part)
  if (digits[0][0]) return cudaSuccess;
  size_t bytes[2], total = 0;
  for (int side = 0; side < 2; side++) {
    const Mat &m = side ? c->rhs : c->lhs;
    bytes[side] = std::max<size_t>(m.drows * m.dcols, 256);
    total += p.parts[side] * bytes[side];
  }
  uint8_t *at = nullptr;
  if (alloc_zeroed((void **)&at, total, nullptr) != cudaSuccess) {
    cudaGetLastError();
    return cudaErrorMemoryAllocation;
  }
  for (int side = 0; side < 2; side++)
    for (int k = 0; k < p.parts[side]; k++, at += bytes[side]) digits[side][k] = at;
  return cudaSuccess;
}

// The plan of a wide context, with the fused form's digit buffers and maps where it applies; built on first use.
int build_plan(gbs_ctx *c) {
  WidePlan *p = new WidePlan();
  const Mat *side_m[2] = {&c->lhs, &c->rhs};
  for (int side = 0; side < 2; side++) {
    const int w = (int)side_m[side]->nbits;
    p->parts[side] = w > 4 ? 2 : 1;
    p->lo_bits[side] = w - hi_bits(w);
  }
  p->fused_splits = fused_splits(c, *p);
  if (p->parts[0] == 2 && p->parts[1] == 2) {
    const int l = std::min(p->lo_bits[0], p->lo_bits[1]), s = p->lo_bits[0] == l ? 0 : 1;
    p->scale[s][0] = -l;
    p->scale[1 - s][1] = p->lo_bits[1 - s];
  }
  if (p->fused_splits && alloc_parts(c, *p, p->digits) != cudaSuccess) {
    wide_plan_free(p);
    return fail(GBS_ENOMEM, "gbs_gemm: digit matrices of the wide-operand parts could not be allocated");
  }
  for (int side = 0; side < 2 && p->fused_splits; side++)
    for (int k = 0; k < p->parts[side]; k++)
      if (!tc_map_u8(&p->maps[side][k], p->digits[side][k], side_m[side]->dcols, side_m[side]->drows, 128))
        p->fused_splits = 0;
  c->wide = p;
  return GBS_OK;
}

// The separate form's digit buffers and sub-contexts, built when it first runs.
int build_subs(gbs_ctx *c) {
  WidePlan *p = c->wide;
  if (alloc_parts(c, *p, p->sep) != cudaSuccess)
    return fail(GBS_ENOMEM, "gbs_gemm: digit matrices of the wide-operand parts could not be allocated");
  for (int pa = 0; pa < p->parts[0]; pa++)
    for (int pb = 0; pb < p->parts[1]; pb++) {
      if (p->sub[pa][pb]) continue;
      int32_t *res = nullptr;
      if (dev_alloc((void **)&res, std::max<size_t>(c->lhs.nrows * c->rhs.nrows * 4, 16)) != cudaSuccess) {
        cudaGetLastError();
        return fail(GBS_ENOMEM, "gbs_gemm: partial results of the wide-operand parts could not be allocated");
      }
      gbs_ctx *s = new gbs_ctx();
      p->sub[pa][pb] = s;
      s->device = c->device;
      s->lhs = part_of(c->lhs, pa);
      s->rhs = part_of(c->rhs, pb);
      s->lhs.imported = s->rhs.imported = true;
      s->pipe = GBS_PIPE_TC;
      s->digits[0] = p->sep[0][pa];
      s->digits[1] = p->sep[1][pb];
      s->res = res;
    }
  return GBS_OK;
}

template <int PA, int PB>
cudaError_t launch_fused(const gbs_ctx *c, const WidePlan &p, const WideArgs &a, cudaStream_t s) {
  uint32_t *err = tc_error_ptr();
  if (!err) return cudaErrorInvalidSymbol;
  auto kern = gemm_wide_pair_kernel<PA, PB>;
  cudaError_t e =
      cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)wide_smem(PA + PB));
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.gridDim = dim3((unsigned)(2 * ((a.M + 255) / 256)), (unsigned)((a.N + 255) / 256), a.splits);
  cfg.blockDim = dim3(kWideThreads);
  cfg.dynamicSmemBytes = wide_smem(PA + PB);
  cfg.stream = s;
  cfg.attrs = attr;
  cfg.numAttrs = pdl_for(s) ? 2 : 1;
  e = cudaLaunchKernelEx(&cfg, kern, p.maps[0][0], p.maps[0][PA - 1], p.maps[1][0], p.maps[1][PB - 1], a, err);
  count_launch();
  return e != cudaSuccess ? e : cudaGetLastError();
}

// The digit matrices of one form, rebuilt from the planes where they are older.
cudaError_t expand_parts(gbs_ctx *c, const WidePlan &p, bool fused, cudaStream_t s) {
  bool(&valid)[2] = fused ? c->digits_valid : c->packed_valid;
  for (int side = 0; side < 2; side++) {
    if (valid[side]) continue;
    for (int k = 0; k < p.parts[side]; k++) {
      ExpandJob job = make_expand_job(part_of(side ? c->rhs : c->lhs, k), (fused ? p.digits : p.sep)[side][k]);
      if (fused) scale_table(job.tab, p.scale[side][k]);
      cudaError_t e = launch_expand(job, s);
      if (e != cudaSuccess) return e;
    }
    if (!fused)  // the parts' own packed matrices (one-problem plans) are stale too
      for (auto &row : p.sub)
        for (gbs_ctx *sub : row)
          if (sub) {
            sub->packed_valid[side] = false;
            release_split_workspace(sub, s);
          }
    valid[side] = true;
  }
  return cudaSuccess;
}

cudaError_t launch_combine(gbs_ctx *c, const int32_t *const (&parts)[4], int n, const uint32_t (&shift)[4],
                           cudaStream_t s) {
  const uint64_t total = c->lhs.nrows * c->rhs.nrows;
  const uint64_t threads = (total + 3) / 4;
  const unsigned blocks = (unsigned)std::min<uint64_t>((threads + 255) / 256, 152 * 32);
  const cudaError_t e = launch_pdl(combine_kernel, blocks, 256, 0, s, result_ptr(c), parts[0], parts[1], parts[2],
                                   parts[3], n, shift[1], shift[2], shift[3], total);
  count_launch();
  return e != cudaSuccess ? e : cudaGetLastError();
}

}  // namespace

bool tc_wide(const gbs_ctx *c) {
  const Mat &A = c->lhs, &B = c->rhs;
  if (A.nbits <= 4 && B.nbits <= 4) return false;
  if (A.nbits > 8 || B.nbits > 8 || A.nrows == 0 || B.nrows == 0 || A.ncols == 0 || !tc_encoder_available())
    return false;
  uint64_t ma = 0, mb = 0;
  for (int k = 0; k < (A.nbits > 4 ? 2 : 1); k++) ma = std::max(ma, part_max_abs(part_of(A, k)));
  for (int k = 0; k < (B.nbits > 4 ? 2 : 1); k++) mb = std::max(mb, part_max_abs(part_of(B, k)));
  return (double)A.ncols * (double)ma * (double)mb < 16777216.0 && A.drows * A.nbits < (1ull << 31) &&
         B.drows * B.nbits < (1ull << 31);
}

void wide_plan_free(WidePlan *p) {
  if (!p) return;
  for (auto &row : p->sub)
    for (gbs_ctx *s : row) {
      if (!s) continue;
      if (s->res) cudaFree(s->res);
      if (s->plan1) {
        tcg_plan_free(s->plan1);
        delete s->plan1;
      }
      small_plan_free(s->small);
      if (s->sk_ws) cudaFree(s->sk_ws);
      if (s->split_owned) cudaFree(s->split_owned);
      if (s->sk_flags) cudaFree(s->sk_flags);
      for (uint8_t *pk : s->packed)
        if (pk) cudaFree(pk);
      delete s;  // its planes alias the parent's, its digit matrices are the plan's
    }
  for (uint8_t *d : {p->digits[0][0], p->sep[0][0]})  // each form's one allocation
    if (d) cudaFree(d);
  if (p->partial) cudaFree(p->partial);
  delete p;
}

bool wide_digit_target(gbs_ctx *c, int side, DigitTarget &t, cudaStream_t s) {
  if (c->lhs.nrows < 256 || c->rhs.nrows < 256 || c->variant >= 0) return false;  // the separate form expands
  if (!c->wide) {
    cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;  // no allocation into a capture
    if (cudaStreamIsCapturing(s, &st) != cudaSuccess || st != cudaStreamCaptureStatusNone) {
      cudaGetLastError();
      return false;
    }
    if (build_plan(c) != GBS_OK) return false;
  }
  WidePlan &p = *c->wide;
  if (!p.fused_splits) return false;
  const Mat &m = side ? c->rhs : c->lhs;
  t.lo = p.digits[side][0];
  t.lo_bits = p.parts[side] == 2 ? p.lo_bits[side] : (int)m.nbits;
  tc_digit_table(part_of(m, 0), t.tab_lo);
  scale_table(t.tab_lo, p.scale[side][0]);
  if (p.parts[side] == 2) {
    t.hi = p.digits[side][1];
    tc_digit_table(part_of(m, 1), t.tab_hi);
    scale_table(t.tab_hi, p.scale[side][1]);
  }
  return true;
}

cudaError_t launch_gemm_wide(gbs_ctx *c, cudaStream_t s, int variant) {
  if (!c->wide && build_plan(c) != GBS_OK) return cudaErrorMemoryAllocation;
  WidePlan &p = *c->wide;
  const bool fused = p.fused_splits && variant < 0;
  if (!fused && build_subs(c) != GBS_OK) return cudaErrorMemoryAllocation;
  cudaError_t e = expand_parts(c, p, fused, s);
  if (e != cudaSuccess) return e;
  const int32_t *parts[4] = {nullptr, nullptr, nullptr, nullptr};
  uint32_t shift[4] = {0, 0, 0, 0};
  int n = 0;
  if (fused) {
    WideArgs a;
    a.M = c->lhs.nrows;
    a.N = c->rhs.nrows;
    a.nstages = (uint32_t)(c->lhs.dcols / 128);
    a.splits = (uint32_t)p.fused_splits;
    a.idesc = (1u << 4) | ((uint32_t)(256 >> 3) << 17) | ((uint32_t)(256 >> 4) << 24);
    const bool two = p.parts[0] == 2 && p.parts[1] == 2;
    a.xshift = (uint32_t)(two ? std::min(p.lo_bits[0], p.lo_bits[1]) : p.lo_bits[p.parts[0] == 2 ? 0 : 1]);
    a.yscale = two ? (float)(1u << a.xshift) : 1.f;
    a.cstride = (a.M * a.N + 3) / 4 * 4;
    if (a.splits > 1 && !p.partial) {
      if (dev_alloc((void **)&p.partial, (size_t)a.splits * a.cstride * 4) != cudaSuccess) {
        cudaGetLastError();
        return cudaErrorMemoryAllocation;
      }
    }
    a.C = a.splits > 1 ? p.partial : result_ptr(c);
    if (two) e = launch_fused<2, 2>(c, p, a, s);
    else if (p.parts[0] == 2) e = launch_fused<2, 1>(c, p, a, s);
    else e = launch_fused<1, 2>(c, p, a, s);
    if (e != cudaSuccess || a.splits == 1) return e;
    for (; n < (int)a.splits; n++) parts[n] = p.partial + (uint64_t)n * a.cstride;
    return launch_combine(c, parts, n, shift, s);
  }
  for (int pa = 0; pa < p.parts[0]; pa++)
    for (int pb = 0; pb < p.parts[1]; pb++) {
      gbs_ctx *sub = p.sub[pa][pb];
      sub->variant = variant;
      sub->digits_valid[0] = sub->digits_valid[1] = true;
      sub->out = nullptr;
      e = launch_gemm_tc_hbm(sub, s, variant);
      if (e != cudaSuccess) return e;
      parts[n] = sub->res;
      shift[n] = (uint32_t)(p.lo_bits[0] * pa + p.lo_bits[1] * pb);
      n++;
    }
  // the unshifted part product first: shift[0] is 0 by construction
  return launch_combine(c, parts, n, shift, s);
}

}  // namespace gbs

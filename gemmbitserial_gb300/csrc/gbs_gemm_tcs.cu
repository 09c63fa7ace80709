// gbs_gemm_tcs.cu -- tensor-core GEMM of one context with a side under 256 rows.
//
// Replaces gemmBitSerial for such a context (arch-generic.hpp:331-345) on the
// e4m3 digit matrices of both operands: one MMA over digits sums every plane
// pair with its weight, exact while K * max|a| * max|b| < 2^24.
//
// The persistent kernel over a problem table (gbs_gemm_tcg.cu) gives such a
// context one tile per 128 rows of its larger side, as wide as the smaller
// side: 3 of 152 SMs for 384 x 2304 x 169, each streaming 18 stages of 38 KB.
// Here the tiles are as narrow as it pays (MMA N = bn, 16 to 256) and K is
// split over the CTAs of a cluster, chosen by an estimate of the critical
// path (plan below); the maps and the problem are launch parameters, so no
// table is read before the first load.
//   warp 0     lane 0: TMA, 128 x 128 digits of the larger side and bn x 128 of
//              the smaller per stage, into a ring of as many stages as fit
//   warp 1     TMEM allocation; lane 0 issues 4 tcgen05.mma (M = 128, N = bn,
//              K = 32) per stage
//   warps 2-5  epilogue; with K split, the CTAs leave their fp32 partial tiles in
//              the drained ring and each sums its share of the columns over
//              distributed shared memory (integers below 2^24: exact)
// Every mbarrier wait is bounded; on timeout the CTA sets a bit in the error
// word, stops issuing, drains what it issued and frees TMEM.
#include <algorithm>
#include <cmath>
#include <cstring>

#include "gbs_internal.h"
#include "gbs_tc_common.cuh"

namespace gbs {

struct SmallPlan {
  CUtensorMap ma, mb;
  uint32_t bn, splits, swap, rt, ct;
};

namespace {

constexpr int kSmThreads = 192;
constexpr uint32_t kSmABytes = 128 * 128;
constexpr size_t kSmSmemCap = 200 * 1024;
constexpr int kSmStagesMax = 8;

struct SmallArgs {
  int32_t *C;
  uint32_t M, N, nk, bn, splits, swap, ct, stages, idesc, cols;  // cols: TMEM columns allocated
};

constexpr size_t small_smem(uint32_t bn, int stages) {
  return 1024 + (size_t)stages * (kSmABytes + bn * 128) + 8 * (2 * stages + 2) + 16;
}
int small_stages(uint32_t bn) {
  int s = kSmStagesMax;
  while (s > 2 && small_smem(bn, s) > kSmSmemCap) s--;
  return s;
}

// 16 accumulator columns of one row of MMA-A as result elements.
__device__ __forceinline__ void store16(const SmallArgs &a, const float (&v)[16], uint32_t row, uint32_t c0) {
  int32_t o[16];
#pragma unroll
  for (int i = 0; i < 16; i++) o[i] = __float2int_rn(v[i]);
  if (!a.swap) {  // row = m, column = n: the lanes write 32 consecutive m of one n
    store_result_cols<16>(a.C, a.M, a.N, row, c0, o);
  } else if (row < a.N) {  // row = n, column = m: each lane writes a run of its result row
    int32_t *dst = a.C + (uint64_t)row * a.M + c0;
    if ((a.M & 3u) == 0) {
#pragma unroll
      for (int i = 0; i < 16; i += 4)
        if (c0 + i < a.M) *reinterpret_cast<int4 *>(dst + i) = make_int4(o[i], o[i + 1], o[i + 2], o[i + 3]);
    } else {
#pragma unroll
      for (int i = 0; i < 16; i++)
        if (c0 + i < a.M) dst[i] = o[i];
    }
  }
}

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&v)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
        "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(v[0]), "+r"(v[1]), "+r"(v[2]), "+r"(v[3]), "+r"(v[4]), "+r"(v[5]), "+r"(v[6]), "+r"(v[7]),
                 "+r"(v[8]), "+r"(v[9]), "+r"(v[10]), "+r"(v[11]), "+r"(v[12]), "+r"(v[13]), "+r"(v[14]), "+r"(v[15])
               :
               : "memory");
}

// CTA `split` of a cluster of a.splits computes stages [split, split + 1) *
// nk / splits of tile blockIdx.x / splits.
__global__ void __launch_bounds__(kSmThreads, 1)
    gemm_tcs_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                    const __grid_constant__ SmallArgs a, uint32_t *err) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t *smem = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t stages = a.stages, slot = kSmABytes + a.bn * 128u;
  uint64_t *bars = reinterpret_cast<uint64_t *>(smem + stages * slot);
  const uint32_t full = smem_u32(bars), empty = full + 8 * stages, acc_full = empty + 8 * stages;
  const uint32_t mma_done = acc_full + 8;
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(bars + 2 * stages + 2);
  volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);
  const uint32_t split = blockIdx.x % a.splits, tile = blockIdx.x / a.splits;
  const uint32_t r0 = tile / a.ct * 128u, c0 = tile % a.ct * a.bn;
  const uint32_t k_lo = split * a.nk / a.splits, nk = (split + 1) * a.nk / a.splits - k_lo;
  griddep_launch_dependents();
  if (tid == 0) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&tmA)) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&tmB)) : "memory");
    for (uint32_t i = 0; i < stages; i++) {
      mbar_init(full + 8 * i, 1);
      mbar_init(empty + 8 * i, 1);
    }
    mbar_init(acc_full, 1);
    mbar_init(mma_done, 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"(a.cols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;");
  const uint32_t tmem = *tmem_slot;
  griddep_wait();  // operands and result belong to earlier kernels until here

  bool done = false;  // epilogue warps: the accumulator is complete
  const int q = warp & 3;
  const uint32_t taddr = tmem + ((uint32_t)(q * 32) << 16);
  float4 *part = reinterpret_cast<float4 *>(smem) + q * 32 + lane;  // partial tile [bn / 4][128 rows][4 columns]
  if (warp == 0) {
    uint32_t k = 0;
    for (; k < nk; k++) {
      const uint32_t s = k % stages, use = k / stages;
      if (use > 0 && !__all_sync(0xffffffffu, mbar_wait_err(empty + 8 * s, (use - 1) & 1, abort_flag, err))) break;
      if (elect_one()) {
        mbar_expect_tx(full + 8 * s, slot);
        const uint32_t dst = smem_u32(smem + s * slot);
        tma_load_digits(dst, &tmA, (int)(k_lo + k), r0, full + 8 * s);
        tma_load_digits(dst + kSmABytes, &tmB, (int)(k_lo + k), c0, full + 8 * s);
      }
      __syncwarp();
    }
    if (lane == 0 && *abort_flag)
      for (uint32_t i = (k > stages ? k - stages : 0); i < k; i++)
        mbar_drain_err(full + 8 * (i % stages), (i / stages) & 1, err);
  } else if (warp == 1) {
    bool ok = true;
    for (uint32_t k = 0; k < nk; k++) {
      const uint32_t s = k % stages;
      if (!__all_sync(0xffffffffu, mbar_wait_err(full + 8 * s, (k / stages) & 1, abort_flag, err))) {
        ok = false;
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;");
      const uint32_t base = smem_u32(smem + s * slot);
      if (elect_one()) {
#pragma unroll
        for (int kk = 0; kk < 4; kk++)
          mma_f8(tmem, sw128_desc(base + kk * 32), sw128_desc(base + kSmABytes + kk * 32), a.idesc, (k | kk) != 0);
        mma_commit(empty + 8 * s);
      }
      __syncwarp();
    }
    if (ok) {
      if (elect_one()) mma_commit(acc_full);
      __syncwarp();
    } else {  // issued MMAs finish before TMEM is freed
      if (elect_one()) mma_commit(mma_done);
      __syncwarp();
      mbar_drain_err(mma_done, 0, err);
    }
  } else {
    done = __all_sync(0xffffffffu, mbar_wait_err(acc_full, 0, abort_flag, err));
    if (done) {
      asm volatile("tcgen05.fence::after_thread_sync;");
#pragma unroll 1
      for (uint32_t col = 0; col < a.bn; col += 16) {
        uint32_t v[16];
        tmem_ld16(taddr + col, v);
        float f[16];
#pragma unroll
        for (int i = 0; i < 16; i++) f[i] = __uint_as_float(v[i]);
        if (a.splits == 1) {
          store16(a, f, r0 + q * 32 + lane, c0 + col);
        } else {
#pragma unroll
          for (int i = 0; i < 16; i += 4)
            part[((col + i) >> 2) * 128] = make_float4(f[i], f[i + 1], f[i + 2], f[i + 3]);
        }
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(a.cols));
  }
  if (a.splits > 1) {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    if (done) {
      // this CTA's share of the column quads, over every CTA's partial tile
      const uint32_t quads = a.bn / 4, q_lo = split * quads / a.splits, q_hi = (split + 1) * quads / a.splits;
      const uint32_t row = r0 + q * 32 + lane;
      for (uint32_t i = q_lo; i < q_hi; i++) {
        float4 sum = part[i * 128];
        for (uint32_t j = 1; j < a.splits; j++) {
          const uint32_t from = split + j < a.splits ? split + j : split + j - a.splits;
          const float4 o = cluster_ptr(static_cast<const float4 *>(part), from)[i * 128];
          sum.x += o.x;
          sum.y += o.y;
          sum.z += o.z;
          sum.w += o.w;
        }
        const int32_t o[4] = {__float2int_rn(sum.x), __float2int_rn(sum.y), __float2int_rn(sum.z),
                              __float2int_rn(sum.w)};
        const uint32_t c = c0 + 4 * i;
        if (!a.swap) {
          store_result_cols<4>(a.C, a.M, a.N, row, c, o);
        } else if (row < a.N) {
          int32_t *dst = a.C + (uint64_t)row * a.M + c;
          if ((a.M & 3u) == 0) {
            if (c < a.M) *reinterpret_cast<int4 *>(dst) = make_int4(o[0], o[1], o[2], o[3]);
          } else {
#pragma unroll
            for (int x = 0; x < 4; x++)
              if (c + x < a.M) dst[x] = o[x];
          }
        }
      }
    }
    // no CTA leaves while another still reads its partial tile
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
  }
}

// Tile width and K split with the least estimated time: a stage costs the
// longer of its bytes at ~105 GB/s into one SM and its four MMAs (~37 ns each up
// to N = 128, 68 ns at 256); a wave of CTAs 2.5 us of setup, first load and
// stores; a split 1.5 us of cluster barriers and its remote reads at ~15 GB/s.
void choose_tiles(uint64_t large, uint64_t small, uint32_t nk, uint32_t &bn, uint32_t &splits) {
  double best = 0.0;
  bn = 0;
  const uint32_t whole = (uint32_t)std::min<uint64_t>(256, (small + 15) / 16 * 16);
  for (uint32_t w : {whole, 128u, 64u, 32u, 16u}) {  // the others divide 256, the rows' padding
    if (w > whole || (w == whole && bn)) continue;
    for (uint32_t s : {1u, 2u, 4u, 8u}) {
      if (s > 1 && (nk / s < 4 || w < 4 * s)) break;
      const double tiles = std::ceil((double)large / 128) * std::ceil((double)small / w);
      const double mma = w <= 128 ? 37.0 : 37.0 + (w - 128) * (31.0 / 128);
      const double stage = std::max((16384.0 + 128.0 * w) / 105.0, 4 * mma);
      const double waves = std::ceil(tiles * s / 152.0);
      const double ns = waves * (std::ceil((double)nk / s) * stage + 2500.0) +
                        (s > 1 ? 1500.0 + 512.0 * w * (s - 1) / s / 15.0 : 0.0);
      if (!bn || ns < best) {
        best = ns;
        bn = w;
        splits = s;
      }
    }
  }
}

}  // namespace

void small_plan_free(SmallPlan *p) { delete p; }

// The GEMM of a context whose digit matrices are built and current.
cudaError_t launch_gemm_tcs(gbs_ctx *c, cudaStream_t s) {
  const Mat &L = c->lhs, &R = c->rhs;
  if (!c->small) {
    SmallPlan *p = new SmallPlan();
    p->swap = L.nrows < R.nrows ? 1u : 0u;  // the larger side is the MMA's 128-row operand
    const Mat &A = p->swap ? R : L, &B = p->swap ? L : R;
    choose_tiles(A.nrows, B.nrows, (uint32_t)((L.ncols + 127) / 128), p->bn, p->splits);
    p->rt = (uint32_t)((A.nrows + 127) / 128);
    p->ct = (uint32_t)((B.nrows + p->bn - 1) / p->bn);
    if (!tc_map_u8(&p->ma, c->digits[p->swap ? 1 : 0], A.dcols, A.drows, 128) ||
        !tc_map_u8(&p->mb, c->digits[p->swap ? 0 : 1], B.dcols, B.drows, p->bn)) {
      delete p;
      return cudaErrorInvalidValue;
    }
    c->small = p;
  }
  const SmallPlan &p = *c->small;
  SmallArgs a;
  a.C = result_ptr(c);
  a.M = (uint32_t)L.nrows;
  a.N = (uint32_t)R.nrows;
  a.nk = (uint32_t)((L.ncols + 127) / 128);
  a.bn = p.bn;
  a.splits = p.splits;
  a.swap = p.swap;
  a.ct = p.ct;
  a.stages = (uint32_t)small_stages(p.bn);
  a.idesc = (1u << 4) | ((p.bn >> 3) << 17) | ((128u >> 4) << 24);
  for (a.cols = 32; a.cols < p.bn;) a.cols *= 2;
  uint32_t *err = tc_error_ptr();
  if (!err) return cudaErrorInvalidSymbol;
  const size_t smem = small_smem(p.bn, (int)a.stages);
  cudaError_t e = cudaFuncSetAttribute(gemm_tcs_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmSmemCap);
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = p.splits;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.gridDim = dim3(p.rt * p.ct * p.splits);
  cfg.blockDim = dim3(kSmThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cfg.attrs = attr;
  cfg.numAttrs = pdl_for(s) ? 2 : 1;
  e = cudaLaunchKernelEx(&cfg, gemm_tcs_kernel, p.ma, p.mb, a, err);
  count_launch();
  return e != cudaSuccess ? e : cudaGetLastError();
}

}  // namespace gbs

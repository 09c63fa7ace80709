// gbs_gemm_tcs.cu -- tensor-core GEMM of one context with a side under 256 rows.
//
// Replaces gemmBitSerial for such a context (arch-generic.hpp:331-345) on the
// e4m3 digit matrices of both operands: one MMA over digits sums every plane
// pair with its weight, exact while K * max|a| * max|b| < 2^24.
//
// The persistent kernel over a problem table (gbs_gemm_tcg.cu) gives such a
// context one tile per 128 rows of its larger side, as wide as the smaller
// side: 3 of 152 SMs for 384 x 2304 x 169, each streaming 18 stages of 38 KB.
// Here the tiles are as narrow as it pays (MMA N = bn, 16 to 256), either side
// gives the MMA's 128 rows, and K is split over the CTAs of a cluster, chosen by an
// estimate of the critical path (choose_tiles); the maps and the problem are launch
// parameters, so no table is read before the first load.  Where the tiles take
// several waves, or a long K its narrow stages, the persistent kernel is the faster
// one and runs the context (small_persistent).
//   warp 0     TMA, 128 x 128 digits of the side that gives the rows and bn x 128 of
//              the other per stage, into a ring of as many stages as fit
//   warp 1     TMEM allocation; 4 tcgen05.mma (M = 128, N = bn, K = 32) per stage
//   warps 2-5  epilogue; with K split, the CTAs leave their fp32 partial tiles in
//              the drained ring and each sums its share of the columns over
//              distributed shared memory (integers below 2^24: exact)
// Warps 0 and 1 issue from an elected lane.
// Every mbarrier wait is bounded; on timeout the CTA sets a bit in the error
// word, stops issuing, drains what it issued and frees TMEM.
#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstring>

#include "gbs_internal.h"
#include "gbs_tc_common.cuh"

namespace gbs {

struct SmallPlan {
  CUtensorMap ma, mb;
  bool maps = false;
  uint32_t bn, splits, swap, rt, ct;
  bool persistent = false;  // the persistent kernel is estimated faster
  TcgForm form;
};

namespace {

constexpr int kSmThreads = 192;
constexpr uint32_t kSmABytes = 128 * 128;
constexpr size_t kSmSmemCap = 200 * 1024;
constexpr int kSmStagesMax = 8;

struct SmallArgs {
  int32_t *C;
  uint32_t M, N, nk, bn, splits, swap, rt, ct, stages, idesc, cols;  // cols: TMEM columns allocated
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
  // neighbouring tiles share the rows or columns of the side with more of them
  const bool byrow = a.rt <= a.ct;
  const uint32_t r0 = (byrow ? tile % a.rt : tile / a.ct) * 128u, c0 = (byrow ? tile / a.rt : tile % a.ct) * a.bn;
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

// CTAs of a cluster of `splits` that the GPU holds at once, one to an SM, cached per device.
double cluster_ctas(uint32_t splits) {
  static std::atomic<int> cache[64][4];
  const int i = splits == 1 ? 0 : splits == 2 ? 1 : splits == 4 ? 2 : 3;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 1.0;
  int v = cache[dev][i].load(std::memory_order_relaxed);
  if (v == 0) {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = splits;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.gridDim = dim3(splits);
    cfg.blockDim = dim3(kSmThreads);
    cfg.dynamicSmemBytes = kSmSmemCap;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int n = 0;
    cudaError_t e = cudaFuncSetAttribute(gemm_tcs_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmSmemCap);
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveClusters(&n, gemm_tcs_kernel, &cfg);
    if (e != cudaSuccess || n < 1) {
      cudaGetLastError();
      return 1.0;
    }
    v = n * (int)splits;
    cache[dev][i].store(v, std::memory_order_relaxed);
  }
  return v;
}

// Which side gives the MMA's 128 rows, the tile width and the K split with the least
// estimated time, and whether the persistent kernel, with a table of the context's
// tiles, beats it.  In ns, fitted to both kernels' times over 9 to 255 x 64 to 8192 x
// 300 to 100000 and the same transposed: a stage costs its bytes at 105 GB/s into one
// SM and no less than 345 here, 115 GB/s and 300 there (205 up to 64 columns, where two
// chunks share a stage).  A wave of CTAs here adds 1700 and its stores: 16 a column where the
// tile's rows are lhs rows (the lanes write consecutive elements of the result), 22
// where they are rhs rows and the result's rows are 16-byte aligned, 73 where they are
// not; a split, of one wave at most, 2900 of cluster barriers and its remote reads at 15
// GB/s.  There a tile is stored while the next is multiplied, in 1600 + 10.7 a column,
// or 1400 + 27 staged for rhs rows, 2400 at least, and the first takes 1900 more, 4000
// with others after it.  A larger lhs gives the rows itself: the result's rows are then
// long, and rhs rows of a tile far apart.
// With the larger side's rows and this kernel in every case 255 x 256 x 100000 took 126
// us (35 so), 128 x 1024 x 100000 46 (32), 20000 x 8192 x 255 94 (60), 255 x 64 x 10000
// 22.5 (6.4).
void choose_tiles(const gbs_ctx *c, SmallPlan &p) {
  const uint64_t M = c->lhs.nrows, N = c->rhs.nrows;
  const double nk = (double)((c->lhs.ncols + 127) / 128), sms = cluster_ctas(1);
  double best = 0.0, other = 0.0;
  p.bn = p.form.bn = 0;
  auto bytes = [](double w) { return 16384.0 + 128.0 * w; };
  for (uint32_t swap = 0; swap < (M < N ? 2u : 1u); swap++) {
    const uint64_t rows = swap ? N : M, cols = swap ? M : N;
    const double rt = std::ceil((double)rows / 128);
    const uint32_t whole = (uint32_t)std::min<uint64_t>(256, (cols + 15) / 16 * 16);
    for (uint32_t w : {whole, 128u, 64u, 32u, 16u}) {  // the others divide 256, the rows' padding
      if (w > whole) continue;
      const double ct = std::ceil((double)cols / w), used = std::min<double>(w, (double)cols);
      const double store = used * (!swap ? 16.0 : (M & 3) == 0 ? 22.0 : 73.0);
      for (uint32_t s : {1u, 2u, 4u, 8u}) {
        if (s > 1 && (nk / s < 4 || w < 4 * s || rt * ct * s > cluster_ctas(s))) break;
        const double waves = std::ceil(rt * ct * s / sms);
        const double ns = waves * (std::ceil(nk / s) * std::max(345.0, bytes(w) / 105.0) + 1700.0 + store / s) +
                          (s > 1 ? 2900.0 + 512.0 * w * (s - 1) / s / 15.0 : 0.0);
        if (!p.bn || ns < best) {
          best = ns;
          p.bn = w;
          p.splits = s;
          p.swap = swap;
        }
      }
      const double mul = nk * std::max(w <= 64 ? 205.0 : 300.0, bytes(w) / 115.0);
      const double epi = std::max(2400.0, swap ? 1400.0 + 27.0 * used : 1600.0 + 10.7 * used);
      const double rounds = std::ceil(rt * ct / sms);
      const double ns = (rounds > 1.0 ? 4000.0 : 1900.0) + (rounds - 1.0) * std::max(mul, epi) + mul + epi;
      if (!p.form.bn || ns < other) {
        other = ns;
        p.form.bn = w;
        p.form.swap = swap;
      }
    }
  }
  p.rt = (uint32_t)(((p.swap ? N : M) + 127) / 128);
  p.ct = (uint32_t)(((p.swap ? M : N) + p.bn - 1) / p.bn);
  p.persistent = other < 0.95 * best;
}

// The context's tiles, chosen on first use.
SmallPlan &small_plan(gbs_ctx *c) {
  if (!c->small) {
    c->small = new SmallPlan();
    choose_tiles(c, *c->small);
  }
  return *c->small;
}

}  // namespace

void small_plan_free(SmallPlan *p) { delete p; }

const TcgForm *small_persistent(gbs_ctx *c) {
  const SmallPlan &p = small_plan(c);
  return p.persistent ? &p.form : nullptr;
}

// The GEMM of a context whose digit matrices are built and current.
cudaError_t launch_gemm_tcs(gbs_ctx *c, cudaStream_t s) {
  const Mat &L = c->lhs, &R = c->rhs;
  SmallPlan &p = small_plan(c);
  if (!p.maps) {
    const Mat &A = p.swap ? R : L, &B = p.swap ? L : R;
    if (!tc_map_u8(&p.ma, c->digits[p.swap ? 1 : 0], A.dcols, A.drows, 128) ||
        !tc_map_u8(&p.mb, c->digits[p.swap ? 0 : 1], B.dcols, B.drows, p.bn))
      return cudaErrorInvalidValue;
    p.maps = true;
  }
  SmallArgs a;
  a.C = result_ptr(c);
  a.M = (uint32_t)L.nrows;
  a.N = (uint32_t)R.nrows;
  a.nk = (uint32_t)((L.ncols + 127) / 128);
  a.bn = p.bn;
  a.splits = p.splits;
  a.swap = p.swap;
  a.rt = p.rt;
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

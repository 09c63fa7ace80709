// gbs_gemm_tcp.cu -- SM-pair digit GEMM with K split, partial tiles summed through L2.
//
// Replaces gemmBitSerial (arch-generic.hpp:331-345) for contexts of M, N >= 256
// whose 256 x 256 tiles are too few for the GPU: every tile is computed by
// `splits` SM pairs (tcgen05.mma.cta_group::2, M = 256, N = 256, e4m3 digits, exact
// below 2^24), each over its share of the K stages.
//
// Splitting inside a cluster (gbs_gemm_tc.cu) needs all of a tile's pairs in one
// GPC: clusters of 8 CTAs with a full ring do not fit 16 times, so 256 x 9216 x
// 4096 ran 256 x 128 tiles split in two -- 36 stages a pair at the cost of
// 256-wide ones (a pair MMA of N = 128 takes as long as one of N = 256).  Here the
// pairs of a tile are independent: each leaves its partial columns in a
// workspace (L2), and for every share of the columns the pair that arrives last
// adds the others' to its own, still in TMEM, and stores the result.  Nobody
// depends on anybody's progress, so any number of contexts' GEMMs may run at once;
// but a pair looks at its own share for 2 us before leaving that too, so pairs in
// step each sum their own.  (A fence, a counter and a look per share, one after
// the other, cost 2.7 us more.)
//
// The workspace is the context's, so two such GEMMs of one context must not
// overlap: one stream at a time owns it (ensure_split_workspace), and a GEMM on
// another stream, or recorded into a graph, splits inside clusters instead, which
// keeps nothing outside the launch.
#include <algorithm>
#include <cstring>

#include "gbs_internal.h"
#include "gbs_tc_common.cuh"

namespace gbs {
namespace {

constexpr int kSpThreads = 192;
constexpr int kSpStages = 7;
constexpr uint32_t kSpLooks = 24;  // at its own share before leaving it: about 2 us
constexpr uint32_t kSpHalf = 128 * 128;  // 128 rows x 128 digits
constexpr uint32_t kSpStageBytes = 2 * kSpHalf;
constexpr size_t kSpSmem = 1024 + kSpStages * kSpStageBytes + 8 * (2 * kSpStages + 2) + 16;
static_assert(kSpSmem <= 227 * 1024, "shared memory per CTA");

struct SplitArgs {
  int32_t *C;
  uint64_t M, N;
  uint32_t nstages, idesc;
  float4 *ws;          // [tile][split][CTA][warp][64 column quads][32 rows]
  uint32_t *arrived;   // [tile][CTA][warp][share]: pairs that have left or hold their columns; 0 between launches
  uint32_t wait_limit; // test hook: the pairs of split 0 load nothing and wait this many rounds (0: normal launches)
};

template <int SPLITS>
__global__ void __launch_bounds__(kSpThreads, 1)
    gemm_tc_pair_split_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                              const __grid_constant__ SplitArgs a, uint32_t *err) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t *smem = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t peer = cluster_rank();  // rank 0 leads
  uint64_t *bars = reinterpret_cast<uint64_t *>(smem + kSpStages * kSpStageBytes);
  const uint32_t full = smem_u32(bars), empty = full + 8 * kSpStages, acc_full = empty + 8 * kSpStages;
  const uint32_t mma_done = acc_full + 8;
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(bars + 2 * kSpStages + 2);
  volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);
  const uint32_t m0 = (blockIdx.x >> 1) * 256, n0 = blockIdx.y * 256, split = blockIdx.z;
  const uint32_t k_lo = split * a.nstages / SPLITS, nk = (split + 1) * a.nstages / SPLITS - k_lo;
  const bool idle = a.wait_limit != 0 && split == 0;  // of the test hook
  griddep_launch_dependents();
  if (tid == 0) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&tmA)) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&tmB)) : "memory");
    for (int i = 0; i < kSpStages; i++) {
      mbar_init(full + 8 * i, 1);
      mbar_init(empty + 8 * i, 1);
    }
    mbar_init(acc_full, 1);
    mbar_init(mma_done, 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (tid == 64 && peer == 0) {  // the first stages towards L2 while setup runs (as in the SM-pair kernel)
    const uint32_t pre = nk < 3u ? nk : 3u;
    for (uint32_t k = 0; k < pre; k++)
#pragma unroll
      for (uint32_t h = 0; h < 2; h++) {
        tma_prefetch_digits(&tmA, (int)(k_lo + k), m0 + 128 * h);
        tma_prefetch_digits(&tmB, (int)(k_lo + k), n0 + 128 * h);
      }
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], 256;" ::"r"(smem_u32(tmem_slot)));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;");
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
  asm volatile("tcgen05.fence::after_thread_sync;");
  const uint32_t tmem = *tmem_slot;
  griddep_wait();  // operands, result and workspace belong to earlier kernels until here

  if (warp == 0) {
    if (peer == 0 && !idle) {  // the leader's TMA: both CTAs' halves of every stage
      uint32_t k = 0;
      for (; k < nk; k++) {
        const uint32_t s = k % kSpStages, use = k / kSpStages;
        if (use > 0 && !__all_sync(0xffffffffu, mbar_wait_err(empty + 8 * s, (use - 1) & 1, abort_flag, err))) break;
        if (elect_one()) {
          const uint32_t fb = map_to_rank(full + 8 * s, 0);
          mbar_expect_tx(full + 8 * s, 2 * kSpStageBytes);
          const uint32_t dst = smem_u32(smem + s * kSpStageBytes);
#pragma unroll
          for (uint32_t h = 0; h < 2; h++) {
            const uint32_t d = h ? map_to_rank(dst, 1) : dst;
            tma_load_digits_pair(d, &tmA, (int)(k_lo + k), m0 + 128 * h, fb);
            tma_load_digits_pair(d + kSpHalf, &tmB, (int)(k_lo + k), n0 + 128 * h, fb);
          }
        }
        __syncwarp();
      }
      if (lane == 0 && *abort_flag)  // wait (bounded) for the loads the barriers still expect, in the peer's memory too
        for (uint32_t i = (k > (uint32_t)kSpStages ? k - kSpStages : 0); i < k; i++)
          mbar_drain_err(full + 8 * (i % kSpStages), (i / kSpStages) & 1, err);
    }
  } else if (warp == 1) {
    if (peer == 0) {
      bool ok = !idle || __all_sync(0xffffffffu, mbar_wait_rounds_err(full, 0, abort_flag, err, a.wait_limit));
      for (uint32_t k = 0; k < nk && ok; k++) {
        const uint32_t s = k % kSpStages;
        if (!__all_sync(0xffffffffu, mbar_wait_err(full + 8 * s, (k / kSpStages) & 1, abort_flag, err))) {
          ok = false;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;");
        const uint32_t base = smem_u32(smem + s * kSpStageBytes);
        if (elect_one()) {
#pragma unroll
          for (int kk = 0; kk < 4; kk++)
            mma_f8_pair(tmem, sw128_desc(base + kk * 32), sw128_desc(base + kSpHalf + kk * 32), a.idesc, (k | kk) != 0);
          mma_commit_pair(empty + 8 * s, 3);
        }
        __syncwarp();
      }
      if (ok) {
        if (elect_one()) mma_commit_pair(acc_full, 3);
        __syncwarp();
      } else {  // issued MMAs finish before TMEM is freed
        if (elect_one()) mma_commit_done(mma_done);
        __syncwarp();
        mbar_drain_err(mma_done, 0, err);
      }
    }
  } else {
    // A pair whose wait gave up counts in all the same, with nothing left or stored: the counters end at 0, and only
    // this launch's results, which the error word disowns, are wrong.
    const bool done = __all_sync(0xffffffffu, idle ? mbar_wait_rounds_err(acc_full, 0, abort_flag, err, a.wait_limit)
                                                   : mbar_wait_err(acc_full, 0, abort_flag, err));
    asm volatile("tcgen05.fence::after_thread_sync;");
    constexpr uint32_t kShare = 256 / SPLITS;  // columns of a share
    constexpr int kBatch = SPLITS - 1 < 3 ? SPLITS - 1 : 3;  // others' columns in flight
    const uint32_t q = warp & 3, taddr = tmem + ((q * 32) << 16);
    const uint64_t gm = m0 + 128 * peer + q * 32 + lane;
    const uint32_t tile = (blockIdx.x >> 1) * gridDim.y + blockIdx.y;
    // this warp's slots: split s's columns at ws + s * stride
    const uint64_t stride = 2 * 4 * 2048;
    float4 *ws = a.ws + ((uint64_t)tile * SPLITS * 8 + peer * 4 + q) * 2048 + lane;
    uint32_t *arrived = a.arrived + ((tile * 2 + peer) * 4 + q) * SPLITS;
    auto leave = [&](uint32_t share) {  // this pair's columns of a share into the workspace
#pragma unroll 1
      for (uint32_t c = share * kShare; c < (share + 1) * kShare; c += 32) {
        uint32_t v[32];
        tmem_ld32(taddr + c, v);
        tmem_wait_ld(v);
#pragma unroll
        for (int i = 0; i < 32; i += 4)
          ws[split * stride + ((c + i) >> 2) * 32] =
              make_float4(__uint_as_float(v[i]), __uint_as_float(v[i + 1]), __uint_as_float(v[i + 2]),
                          __uint_as_float(v[i + 3]));
      }
    };
#pragma unroll 1
    for (uint32_t j = 1; j < SPLITS && done; j++) leave((split + j) % SPLITS);
    __threadfence();
    __syncwarp();
    // lane l counts this pair in for share l, all shares but its own at once
    uint32_t count = 0;
    if (lane < SPLITS && lane != split) count = atomicAdd(arrived + lane, 1u);
    // its own share: the others arrive within a us of each other as a rule, so look a few times before
    // leaving that too (whoever counts in last then sums it)
    if (lane == split)
      for (uint32_t it = 0; it < kSpLooks; it++) {
        count = *reinterpret_cast<volatile uint32_t *>(arrived + lane);
        if (count == SPLITS - 1) break;
        __nanosleep(50);
      }
    __syncwarp();
    if (__shfl_sync(0xffffffffu, count, split) != SPLITS - 1) {
      if (done) leave(split);
      __threadfence();
      __syncwarp();
      if (lane == split) count = atomicAdd(arrived + lane, 1u);
    }
    // the shares it is the last of: the others' columns are in the workspace, its own in TMEM
    uint32_t mine = __ballot_sync(0xffffffffu, lane < SPLITS && count == SPLITS - 1);
    __threadfence();
    while (mine) {
      const uint32_t share = __ffs(mine) - 1;
      mine &= mine - 1;
      if (lane == 0) arrived[share] = 0u;  // ready for the next launch
      if (!done) continue;
#pragma unroll 1
      for (uint32_t c = share * kShare; c < (share + 1) * kShare; c += 32) {
        float4 r[kBatch][8];  // the others' loads first
        auto load = [&](uint32_t s0) {
#pragma unroll
          for (int b = 0; b < kBatch; b++)
#pragma unroll
            for (int i = 0; i < 8; i++)
              r[b][i] = s0 + b < SPLITS ? __ldcg(ws + ((split + s0 + b) % SPLITS) * stride + ((c >> 2) + i) * 32)
                                        : make_float4(0.f, 0.f, 0.f, 0.f);
        };
        load(1);
        float acc[32];
        {
          uint32_t v[32];
          tmem_ld32(taddr + c, v);
          tmem_wait_ld(v);
#pragma unroll
          for (int i = 0; i < 32; i++) acc[i] = __uint_as_float(v[i]);
        }
#pragma unroll 1
        for (uint32_t s0 = 1;;) {
#pragma unroll
          for (int b = 0; b < kBatch; b++)
#pragma unroll
            for (int i = 0; i < 8; i++) {
              acc[4 * i] += r[b][i].x;
              acc[4 * i + 1] += r[b][i].y;
              acc[4 * i + 2] += r[b][i].z;
              acc[4 * i + 3] += r[b][i].w;
            }
          s0 += kBatch;
          if (s0 >= SPLITS) break;
          load(s0);
        }
        int32_t o[32];
#pragma unroll
        for (int i = 0; i < 32; i++) o[i] = __float2int_rn(acc[i]);
        store_result_cols<32>(a.C, a.M, a.N, gm, n0 + c, o);
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;");
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, 256;" ::"r"(tmem));
  }
}

uint64_t split_tiles(const gbs_ctx *c) { return ((c->lhs.nrows + 255) / 256) * ((c->rhs.nrows + 255) / 256); }
size_t split_counter_bytes(const gbs_ctx *c, uint32_t splits) {
  return (split_tiles(c) * 8 * splits * sizeof(uint32_t) + 255) / 256 * 256;
}

template <int SPLITS>
cudaError_t launch(const CUtensorMap &ma, const CUtensorMap &mb, const SplitArgs &a, cudaStream_t s) {
  uint32_t *err = tc_error_ptr();
  if (!err) return cudaErrorInvalidSymbol;
  cudaError_t e = cudaFuncSetAttribute(gemm_tc_pair_split_kernel<SPLITS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)kSpSmem);
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.gridDim = dim3((unsigned)(2 * ((a.M + 255) / 256)), (unsigned)((a.N + 255) / 256), SPLITS);
  cfg.blockDim = dim3(kSpThreads);
  cfg.dynamicSmemBytes = kSpSmem;
  cfg.stream = s;
  cfg.attrs = attr;
  cfg.numAttrs = pdl_for(s) ? 2 : 1;
  e = cudaLaunchKernelEx(&cfg, gemm_tc_pair_split_kernel<SPLITS>, ma, mb, a, err);
  count_launch();
  return e != cudaSuccess ? e : cudaGetLastError();
}

}  // namespace

// K split of a GEMM of `tiles` 256 x 256 tiles and nstages K stages on `pairs`
// SM pairs, 1 unless it beats other_us, the estimate of the kernel it would
// replace, by 8 %: 0.33 us a stage, 8 us of launch, exchange and stores and 0.12 us
// a split.  Measured back to back (us, workspaces hot / rotating over four
// contexts; in-cluster split in parentheses): 256 x 9216 x 4096 in 4 14.4 / 16.9
// (18.9 / 19.2), 256 x 4608 x 4096 11.8 / 13.1 (12.5 / 12.8), 256 x 2304 x 4096
// 10.6 / 11.1 (9.4 / 9.3); 512 x 16384 x 1024 in 8 14.0 / 15.5 (28.2 / 28.5).
uint32_t pair_gather_splits(uint64_t tiles, uint32_t nstages, uint64_t pairs, double other_us) {
  uint32_t best = 1;
  for (uint32_t s : {2u, 4u, 8u}) {
    if (tiles * s > pairs || nstages / s < 4) break;
    const double us = 0.33 * ((nstages + s - 1) / s) + 8.0 + 0.12 * s;
    if (us * (best == 1 ? 1.08 : 1.0) < other_us) {
      other_us = us;
      best = s;
    }
  }
  return best;
}

// Bytes of a context's workspace, the arrival counters first; 0 where the rule does
// not split its K.  It is laid out behind the first digit matrix the context
// allocates: an allocation of its own cost the context's first GEMM 45 us.
size_t split_workspace_bytes(const gbs_ctx *c) {
  const uint32_t splits = pair_gather_choice(c);
  return splits > 1 ? split_counter_bytes(c, splits) + split_tiles(c) * splits * 8 * 2048 * sizeof(float4) : 0;
}
size_t split_workspace_zeroed(const gbs_ctx *c) { return split_counter_bytes(c, pair_gather_choice(c)); }
void set_split_workspace(gbs_ctx *c, void *p) {
  c->split_counters = static_cast<uint32_t *>(p);
  c->split_ws = static_cast<uint8_t *>(p) + split_counter_bytes(c, pair_gather_choice(c));
}

static bool in_capture(cudaStream_t s) {
  cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(s, &st) == cudaSuccess && st == cudaStreamCaptureStatusNone) return false;
  cudaGetLastError();
  return true;
}

// The context's workspace for a GEMM on s; false where it has none, or where a
// GEMM that may still run holds it.  Launches of one stream follow each other, so
// the stream that first takes the workspace keeps it (by its id: a handle may be
// another stream's later) until an import gives it back.  A graph replays on any
// stream, so none is recorded with it.  A context whose digits are another's (a
// part of a wide operand's) gets an allocation of its own here.
bool ensure_split_workspace(gbs_ctx *c, uint32_t splits, cudaStream_t s) {
  unsigned long long id = 0;
  if (in_capture(s)) return false;
  if (cudaStreamGetId(s, &id) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  if (c->split_taken && c->split_stream != id) return false;
  c->split_taken = true;
  c->split_stream = id;
  if (c->split_ws) return true;  // a context keeps its shape, and the rule its choice
  void *p = nullptr;             // the zeroing below is queued before the GEMM that counts
  cudaError_t e = dev_alloc(&p, split_workspace_bytes(c));
  if (e == cudaSuccess) e = cudaMemsetAsync(p, 0, split_counter_bytes(c, splits), s);
  if (e != cudaSuccess) {
    cudaGetLastError();
    if (p) cudaFree(p);
    return false;
  }
  c->split_owned = p;
  set_split_workspace(c, p);
  return true;
}

// An import on s: it overwrites what the context's earlier GEMMs read, so it is
// ordered after them, and the GEMMs of what it imports after it.  Their stream may
// be another.
void release_split_workspace(gbs_ctx *c, cudaStream_t s) {
  if (c->split_taken && !in_capture(s)) c->split_taken = false;
}

cudaError_t launch_pair_gather(gbs_ctx *c, const void *map_a, const void *map_b, uint32_t splits, cudaStream_t s) {
  SplitArgs a;
  a.C = result_ptr(c);
  a.M = c->lhs.nrows;
  a.N = c->rhs.nrows;
  a.nstages = (uint32_t)(c->lhs.dcols / 128);
  a.idesc = (1u << 4) | ((256u >> 3) << 17) | ((256u >> 4) << 24);
  a.ws = static_cast<float4 *>(c->split_ws);
  a.arrived = c->split_counters;
  a.wait_limit = c->debug_wait_limit;
  const CUtensorMap &ma = *reinterpret_cast<const CUtensorMap *>(map_a);
  const CUtensorMap &mb = *reinterpret_cast<const CUtensorMap *>(map_b);
  if (splits == 8) return launch<8>(ma, mb, a, s);
  if (splits == 4) return launch<4>(ma, mb, a, s);
  return launch<2>(ma, mb, a, s);
}

}  // namespace gbs

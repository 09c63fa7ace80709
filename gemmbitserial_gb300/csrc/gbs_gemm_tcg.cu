// gbs_gemm_tcg.cu -- persistent tensor-core GEMM over a table of problems,
// and the planes -> e4m3 digit expansion that feeds it.
//
// The reference evaluates a list of GEMMs as a host loop of gemmBitSerial
// calls (benchmark.cpp:192-206); each call is AND + popcount over every plane
// pair weighted by +-2^(i+j) (arch-generic.hpp:179-192), with the bipolar
// corrections of arch-generic.hpp:45-71.  Here every operand of a problem is
// first expanded to an e4m3 "digit" matrix whose byte is the element's whole
// few-bit value (bipolar: +-1; columns past K and rows past nrows: 0), so one
// fp8 tcgen05.mma over digits covers all plane pairs and all corrections at
// once.  Products and partial sums are integers, exact in the fp32 TMEM
// accumulator while K * max|a| * max|b| < 2^24 (the eligibility rule), so
// the int32 result is bit-exact.
//
// Kernel: one CTA per SM walks its share of a cost-sorted tile table (snake
// order, no atomics).  A tile is 128 rows of the MMA-A operand x bn rows of
// the MMA-B operand; per problem the larger side is MMA-A ("swap" when that
// is the rhs), so a problem with few lhs rows uses an MMA N as small as 16
// instead of padding M to 128.  A plan of one context's own GEMM may give MMA-A to the
// smaller lhs (TcgForm): its rows are consecutive in the result.
//
// Large groups read HBM once per element of the larger sides, so a "packed" plan
// holds those that allow it as 4-bit floats (packed_offset): the TMA unpacks them
// on the way into shared memory and the MMA takes them as they land there (e2m1
// against the other side's e4m3), so nothing is decoded by threads.
//
//   warp 0     TMA producer -- A box 128 x 128 values and B box
//              bn x 128 bytes, 128-byte swizzle, one or two of each a stage,
//              into a 4-slot ring that runs across tile boundaries
//   warp 1     allocates all 512 TMEM columns (two 256-column accumulators);
//              issues 4 or 8 tcgen05.mma (K = 32) per stage and commits the
//              accumulator of each tile
//   warps 2-5  epilogue of tile j while the MMAs of tile j+1 run: tcgen05.ld
//              32 lanes x 32 columns, fp32 -> int32, stores into res[n*M + m]
//
// Warps 0 and 1 walk the stages whole and issue from an elected lane: from lane 0
// of a diverged warp an MMA took 47-76 ns to issue, so even the narrowest stage
// took 0.27 us; elected, eight MMAs of N = 16 take 34 ns each, of 256 66 (the
// rate of the tensor cores).  The 397 tensor-core problems of the 512-problem mix:
// 589 us on digits, 448 packed (2.3 GB of operands, 350 us at the copy rate); a
// kernel whose warps decoded 4-bit codes into digits took 579.
// Every mbarrier wait is bounded; on timeout the CTA sets a bit in the
// caller's error word, stops issuing, drains what it issued and frees TMEM.
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <vector>

#include "gbs_internal.h"
#include "gbs_tc_common.cuh"

namespace gbs {
namespace {

constexpr uint32_t kTgStages = 4;
constexpr uint32_t kTgABytes = 128 * 128;  // MMA-A chunk: 128 rows x 128 digits (packed values in 16-byte groups)
// A stage is one 128-column chunk of MMA-A and up to 256 rows of MMA-B, or two
// chunks of each where MMA-B has at most kTgTwoRows rows: as many bytes, and half
// as many barriers for the MMAs of narrow tiles to wait on.
constexpr uint32_t kTgSlotBytes = kTgABytes + 256 * 128;
constexpr uint32_t kTgTwoRows = 64;
static_assert(2 * (kTgABytes + kTgTwoRows * 128) <= kTgSlotBytes, "two chunks must fit a slot");
constexpr int kTgThreads = 192;
constexpr uint32_t kTgAccCols = 256;
constexpr uint32_t kTgBarBytes = 128;
static_assert(8 * (2 * kTgStages + 5) + 8 <= kTgBarBytes, "barriers, TMEM address, abort flag");
constexpr size_t tcg_smem_bytes() { return 1024 + kTgStages * kTgSlotBytes + kTgBarBytes + 4 * 32 * 33 * 4; }

// Tile j of CTA b among G CTAs: rounds of G consecutive table entries, every
// other round walked backwards, so each CTA's share of a cost-sorted table
// sums to nearly the same cost.
__device__ __forceinline__ uint32_t snake_tile(uint32_t j, uint32_t b, uint32_t G) {
  return j * G + ((j & 1u) ? G - 1u - b : b);
}

__device__ __forceinline__ bool tile_ok(const TcgTile &t, const TcgProblem &P, uint32_t nprob) {
  return t.p < nprob && P.bn >= 16 && P.bn <= 256 && (P.bn & 15u) == 0 && P.nk > 0 &&
         (t.r + 1) * 128u <= P.a_rows && (t.c + 1) * P.bn <= P.b_rows && P.a_bytes <= kTgABytes;
}

// 32 rows (n) from row0 x up to 32 columns (m) from c0 of a swapped tile, staged as
// [32][33]: the warp walks the block flat, so what a result row has of it is
// written by neighbouring lanes.  With each lane on a row of its own a store
// touched 32 sectors, and the epilogue took a fifth of a large group's time.
__device__ __forceinline__ void store_staged(const TcgProblem &P, uint32_t row0, uint32_t c0, uint32_t left,
                                             const int32_t *stage, int lane) {
  if (row0 >= P.N || c0 >= P.M) return;
  const uint32_t nc = min(32u, min(left, P.M - c0)), nr = min(32u, P.N - row0);
  int32_t *dst = P.C + (uint64_t)row0 * P.M + c0;
  if (nc == 32) {
#pragma unroll 8
    for (uint32_t r = 0; r < nr; r++) dst[(uint64_t)r * P.M + lane] = stage[r * 33 + lane];
    return;
  }
  const uint32_t magic = 65536u / nc + 1;  // e / nc for e < 1024, nc < 32
#pragma unroll 4
  for (uint32_t e = lane; e < nr * nc; e += 32) {
    const uint32_t r = (e * magic) >> 16, c = e - r * nc;
    dst[(uint64_t)r * P.M + c] = stage[r * 33 + c];
  }
}

// The tiles of one CTA in turn, each with its problem.  The entry of the next tile
// is asked for when a tile begins and its problem once the tile is under way, so
// neither load's latency stands between two tiles.
struct TileWalk {
  const TcgProblem *probs;
  const TcgTile *tiles;
  uint32_t ntiles, nprob, G, b;
  uint32_t j;
  bool live, ok, next_live;  // a tile is there; it can be run
  TcgTile tl, ntl;
  TcgProblem P, nP;

  __device__ __forceinline__ void fetch_entry(uint32_t at) {
    const uint32_t t = snake_tile(at, b, G);
    next_live = t < ntiles;
    if (next_live) ntl = tiles[t];
  }
  __device__ __forceinline__ void fetch_problem() {
    if (next_live && ntl.p < nprob) nP = probs[ntl.p];
  }
  __device__ __forceinline__ void advance() {  // to the fetched tile
    live = next_live;
    tl = ntl;
    P = nP;
    ok = live && tl.p < nprob && tile_ok(tl, P, nprob);
    j++;
    fetch_entry(j);
  }
  __device__ __forceinline__ void start() {
    j = 0;
    fetch_entry(0);
    fetch_problem();
    advance();
  }
};

__global__ void __launch_bounds__(kTgThreads, 1)
    gemm_tcg_kernel(const TcgProblem *__restrict__ probs, const CUtensorMap *__restrict__ maps,
                    const TcgTile *__restrict__ tiles, uint32_t ntiles, uint32_t nprob, uint32_t *err,
                    int32_t *out0) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t *smem = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  uint64_t *bars = reinterpret_cast<uint64_t *>(smem + kTgStages * kTgSlotBytes);
  const uint32_t full = smem_u32(bars), empty = full + 8 * kTgStages, acc_full = empty + 8 * kTgStages;
  const uint32_t acc_empty = acc_full + 16, mma_done = acc_empty + 16;
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(bars + 2 * kTgStages + 5);
  volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);
  TileWalk w{probs, tiles, ntiles, nprob, gridDim.x, blockIdx.x};
  griddep_launch_dependents();

  if (tid == 0) {
    for (uint32_t i = 0; i < kTgStages; i++) {
      mbar_init(full + 8 * i, 1);
      mbar_init(empty + 8 * i, 1);
    }
    for (int i = 0; i < 2; i++) {
      mbar_init(acc_full + 8 * i, 1);
      mbar_init(acc_empty + 8 * i, 4);  // one arrival per epilogue warp
    }
    mbar_init(mma_done, 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "n"(2 * kTgAccCols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;");
  const uint32_t tmem = *tmem_slot;
  griddep_wait();  // operands and results belong to earlier kernels until here

  if (warp == 0) {
    uint32_t it = 0;  // stage loads issued
    bool stop = false;
    // the maps were written by a host copy: order them for the tensor-map proxy
    auto acquire_maps = [&](uint32_t p) {
      const CUtensorMap *m = maps + 2 * p;
      asm volatile("fence.proxy.tensormap::generic.acquire.gpu [%0], 128;" ::"l"(m) : "memory");
      asm volatile("fence.proxy.tensormap::generic.acquire.gpu [%0], 128;" ::"l"(m + 1) : "memory");
      asm volatile("prefetch.tensormap [%0];" ::"l"(m) : "memory");
      asm volatile("prefetch.tensormap [%0];" ::"l"(m + 1) : "memory");
    };
    w.start();
    if (w.ok) acquire_maps(w.tl.p);
    for (; w.live && !stop; w.advance()) {
      if (!w.ok) {
        w.fetch_problem();
        if (w.next_live && w.ntl.p < nprob) acquire_maps(w.ntl.p);
        continue;
      }
      const CUtensorMap *ma = maps + 2 * w.tl.p, *mb = ma + 1;
      const uint32_t kb = w.P.bn <= kTgTwoRows ? 2u : 1u, nk = w.P.nk, bn = w.P.bn, bytes = w.P.a_bytes + bn * 128u;
      const uint32_t arow = w.tl.r * 128, brow = w.tl.c * bn;
      for (uint32_t k = 0; k < nk; k += kb, it++) {
        const uint32_t s = it % kTgStages, use = it / kTgStages;
        if (use > 0 && !__all_sync(~0u, mbar_wait_err(empty + 8 * s, (use - 1) & 1, abort_flag, err))) {
          stop = true;
          break;
        }
        if (elect_one()) {
          const bool two = kb == 2 && k + 1 < nk;
          mbar_expect_tx(full + 8 * s, two ? 2 * bytes : bytes);
          const uint32_t dst = smem_u32(smem + s * kTgSlotBytes), dstb = dst + kb * kTgABytes;
          tma_load_digits(dst, ma, (int)k, arow, full + 8 * s);
          tma_load_digits(dstb, mb, (int)k, brow, full + 8 * s);
          if (two) {
            tma_load_digits(dst + kTgABytes, ma, (int)k + 1, arow, full + 8 * s);
            tma_load_digits(dstb + bn * 128u, mb, (int)k + 1, brow, full + 8 * s);
          }
        }
        __syncwarp();
        if (k == 0) {  // the first stage is on its way: the next tile's problem and maps
          w.fetch_problem();
          if (w.next_live && w.ntl.p < nprob) acquire_maps(w.ntl.p);
        }
      }
    }
    if (lane == 0 && *abort_flag)
      for (uint32_t q = (it > kTgStages ? it - kTgStages : 0); q < it; q++)
        mbar_drain_err(full + 8 * (q % kTgStages), (q / kTgStages) & 1, err);
  } else if (warp == 1) {
    uint32_t it = 0, jt = 0;  // stages consumed, tiles accumulated
    bool ok = true;
    for (w.start(); w.live && ok; w.advance()) {
      if (!w.ok) {
        w.fetch_problem();
        continue;
      }
      const uint32_t a = jt & 1, use = jt >> 1;
      if (use > 0 && !__all_sync(~0u, mbar_wait_err(acc_empty + 8 * a, (use - 1) & 1, abort_flag, err))) {
        ok = false;
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;");
      const uint32_t d = tmem + a * kTgAccCols;
      const uint32_t kb = w.P.bn <= kTgTwoRows ? 2u : 1u, nk = w.P.nk, bn = w.P.bn, idesc = w.P.idesc;
      for (uint32_t k = 0; k < nk; k += kb, it++) {
        const uint32_t s = it % kTgStages;
        if (!__all_sync(~0u, mbar_wait_err(full + 8 * s, (it / kTgStages) & 1, abort_flag, err))) {
          ok = false;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;");
        const uint32_t base = smem_u32(smem + s * kTgSlotBytes);
        const uint64_t da = sw128_desc(base), db = sw128_desc(base + kb * kTgABytes);
        if (elect_one()) {
#pragma unroll
          for (int kk = 0; kk < 4; kk++)  // the address field counts 16 bytes
            mma_f8(d, da + 2 * kk, db + 2 * kk, idesc, (k | kk) != 0);
          if (kb == 2 && k + 1 < nk) {
            const uint64_t da1 = da + kTgABytes / 16, db1 = db + bn * 8;
#pragma unroll
            for (int kk = 0; kk < 4; kk++) mma_f8(d, da1 + 2 * kk, db1 + 2 * kk, idesc, 1);
          }
          mma_commit(empty + 8 * s);
        }
        __syncwarp();
        if (k == 0) w.fetch_problem();
      }
      if (!ok) break;
      if (elect_one()) mma_commit(acc_full + 8 * a);
      __syncwarp();
      jt++;
    }
    if (!ok) {  // issued MMAs finish before TMEM is freed
      if (elect_one()) mma_commit(mma_done);
      __syncwarp();
      mbar_drain_err(mma_done, 0, err);
    }
  } else {
    const int q = warp & 3;  // TMEM lanes 32q .. 32q+31 belong to this warp
    int32_t *stage = reinterpret_cast<int32_t *>(smem + kTgStages * kTgSlotBytes + kTgBarBytes) + (warp - 2) * 32 * 33;
    uint32_t jt = 0;
    for (w.start(); w.live; w.advance()) {
      w.fetch_problem();
      const TcgTile tl = w.tl;
      TcgProblem P = w.P;
      if (!w.ok) {
        if (warp == 2 && lane == 0) atomicOr(err, 4u);
        continue;
      }
      if (out0 && tl.p == 0) P.C = out0;  // the caller's result buffer for problem 0
      const uint32_t a = jt & 1, use = jt >> 1;
      if (!__all_sync(0xffffffffu, mbar_wait_err(acc_full + 8 * a, use & 1, abort_flag, err))) break;
      asm volatile("tcgen05.fence::after_thread_sync;");
      const uint32_t row0 = tl.r * 128u + (uint32_t)(q * 32);
      const uint32_t taddr = tmem + a * kTgAccCols + ((uint32_t)(q * 32) << 16);
#pragma unroll 1
      for (uint32_t col = 0; col < P.bn; col += 32) {
        uint32_t v[32];
        tmem_ld32(taddr + col, v);
        tmem_wait_ld(v);
        const uint32_t c0 = tl.c * P.bn + col;
        if (!P.swap) {  // row = m, column = n: lanes write 32 consecutive m of one n
          int32_t o[2][16];
#pragma unroll
          for (int i = 0; i < 32; i++) o[i >> 4][i & 15] = __float2int_rn(__uint_as_float(v[i]) * P.scale);
          store_result_cols<16>(P.C, P.M, P.N, row0 + lane, c0, o[0]);
          if (col + 16 < P.bn) store_result_cols<16>(P.C, P.M, P.N, row0 + lane, c0 + 16, o[1]);
        } else {  // row = n, column = m
          __syncwarp();
#pragma unroll
          for (int i = 0; i < 32; i++) stage[lane * 33 + i] = __float2int_rn(__uint_as_float(v[i]) * P.scale);
          __syncwarp();
          store_staged(P, row0, c0, P.bn - col, stage, lane);
        }
      }
      asm volatile("tcgen05.fence::before_thread_sync;");
      __syncwarp();
      if (lane == 0) mbar_arrive(acc_empty + 8 * a);
      jt++;
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(2 * kTgAccCols));
  }
}

// ------------------------------------------------------------ digit expansion
// One thread writes 16 digits (one 16-byte store) of one row; chunks entirely
// past K are skipped, as are rows past nrows: the buffer is zeroed when it is
// allocated and those bytes never change.
template <int CNT>
__device__ __forceinline__ void expand_chunk(const ExpandJob &j, uint32_t r, uint32_t col0) {
  const uint64_t w = col0 >> 6;
  const int sh = (int)(col0 & 63);
  uint32_t pw[4] = {0u, 0u, 0u, 0u};
#pragma unroll
  for (int p = 0; p < CNT; p++) pw[p] = (uint32_t)(j.planes[(p * j.nrows_a + r) * j.wpr + w] >> (sh & 32));
  const uint32_t tab[4] = {j.tab[0], j.tab[1], j.tab[2], j.tab[3]};
  uint32_t q[4];
#pragma unroll
  for (int n = 0; n < 4; n++) {
    const int s4 = (sh & 16) + 4 * n;
    if (CNT == 1) {
      const uint32_t sp = decode4<1>(pw, s4, tab);
      q[n] = sp * ((tab[0] >> 8) & 0xFFu) + (sp ^ 0x01010101u) * (tab[0] & 0xFFu);
    } else {
      q[n] = decode4<CNT>(pw, s4, tab);
    }
    const uint32_t c0 = col0 + 4 * n;
    if (c0 + 4 > j.K) q[n] &= c0 >= j.K ? 0u : (0xFFFFFFFFu >> (8 * (4 - (j.K - c0))));
  }
  *reinterpret_cast<uint4 *>(j.digits + digit_offset(r, col0, j.dcols)) = make_uint4(q[0], q[1], q[2], q[3]);
}

// One thread writes 32 values of one row of a packed matrix: the codes of 4
// columns as bytes (plane p's 4 bits spread to bit p of each byte), packed.
template <int CNT>
__device__ __forceinline__ void expand_packed_chunk(const ExpandJob &j, uint32_t r, uint32_t col0) {
  const uint64_t w = col0 >> 6;
  const int sh = (int)(col0 & 63);
  uint32_t pw[CNT];
#pragma unroll
  for (int p = 0; p < CNT; p++) pw[p] = (uint32_t)(j.planes[(p * j.nrows_a + r) * j.wpr + w] >> sh);
  uint32_t c[8];
#pragma unroll
  for (int i = 0; i < 8; i++) {  // columns 4i .. 4i + 3
    c[i] = 0;
#pragma unroll
    for (int p = 0; p < CNT; p++) c[i] |= (bfe4(pw[p], 4 * i) * (0x00204081u << p)) & (0x01010101u << p);
  }
  store_packed32(j.digits, r, col0, j.dcols, CNT, (int)j.pform, c);
}

__device__ __forceinline__ void expand_thread(const ExpandJob &j, uint64_t local) {
  if (local >= (uint64_t)j.nrows * j.chunks) return;  // padding threads of the job
  uint32_t r, col0;
  if (local < 0xFFFFFFFFull) {  // 32-bit division in the common case
    r = (uint32_t)local / j.chunks;
    col0 = ((uint32_t)local - r * j.chunks) * 16u;
  } else {
    r = (uint32_t)(local / j.chunks);
    col0 = (uint32_t)(local % j.chunks) * 16u;
  }
  if (j.pform) {
    col0 *= 2;  // 32 values per thread
    switch (j.nbits) {
      case 1: expand_packed_chunk<1>(j, r, col0); break;
      case 2: expand_packed_chunk<2>(j, r, col0); break;
      default: expand_packed_chunk<3>(j, r, col0); break;
    }
    return;
  }
  switch (j.nbits) {
    case 1: expand_chunk<1>(j, r, col0); break;
    case 2: expand_chunk<2>(j, r, col0); break;
    case 3: expand_chunk<3>(j, r, col0); break;
    default: expand_chunk<4>(j, r, col0); break;
  }
}

__global__ void __launch_bounds__(256) expand_one_kernel(const ExpandJob job) {
  griddep_launch_dependents();
  griddep_wait();
  expand_thread(job, (uint64_t)blockIdx.x * blockDim.x + threadIdx.x);
}

// Every job's thread range is a multiple of 256, so all threads of a block
// belong to one job and the job search below is uniform within the block.
__global__ void __launch_bounds__(256) expand_grouped_kernel(const ExpandJob *__restrict__ jobs, int njobs,
                                                             uint64_t total) {
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total;
       i += (uint64_t)gridDim.x * blockDim.x) {
    int lo = 0, hi = njobs - 1;  // last job with thread0 <= i
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (jobs[mid].thread0 <= i) lo = mid;
      else hi = mid - 1;
    }
    const ExpandJob &j = jobs[lo];
    expand_thread(j, i - j.thread0);
  }
}

template <typename T>
cudaError_t upload(T **dst, const T *src, size_t n) {
  cudaError_t e = dev_alloc((void **)dst, std::max<size_t>(n, 1) * sizeof(T));
  if (e != cudaSuccess || n == 0) return e;
  return cudaMemcpy(*dst, src, n * sizeof(T), cudaMemcpyHostToDevice);
}

int sm_count() {
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return sms > 0 ? sms : 1;
}

}  // namespace

ExpandJob make_expand_job(const Mat &m, uint8_t *digits) {
  ExpandJob j;
  memset(&j, 0, sizeof(j));
  j.planes = m.planes;
  j.digits = digits;
  j.nrows_a = m.nrows_a;
  j.wpr = m.wpr();
  j.dcols = m.dcols;
  j.nrows = (uint32_t)m.nrows;
  j.K = (uint32_t)m.ncols;
  j.chunks = (uint32_t)((m.ncols + 15) / 16);
  j.nbits = (uint32_t)m.nbits;
  tc_digit_table(m, j.tab);
  return j;
}

ExpandJob make_packed_job(const Mat &m, uint8_t *packed) {
  ExpandJob j = make_expand_job(m, packed);
  j.pform = (uint32_t)m.packed_form();
  j.chunks = (uint32_t)((m.ncols + 31) / 32);
  return j;
}

cudaError_t launch_expand(const ExpandJob &job, cudaStream_t s) {
  const uint64_t threads = (uint64_t)job.nrows * job.chunks;
  if (threads == 0) return cudaSuccess;
  const cudaError_t e = launch_pdl(expand_one_kernel, (unsigned)((threads + 255) / 256), 256, 0, s, job);
  count_launch();
  return e != cudaSuccess ? e : cudaGetLastError();
}

// Allocates a zeroed buffer (and `more` bytes behind it, as they come).  With a
// stream (order) the zeroing is queued there, before whatever that stream does with
// the buffer next; into a capture, where it would be recorded instead, and without a
// stream it is done before returning, on a stream of its own: neither the device nor
// the default stream can be waited for while some stream is captured.  The thread's
// capture mode is relaxed meanwhile: an allocation is part of no capture and
// disturbs none.
// (Waiting for the device on each buffer was most of a new context's first call.)
cudaError_t alloc_zeroed(void **p, size_t bytes, const cudaStream_t *order, size_t more) {
  cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
  cudaError_t e = cudaThreadExchangeStreamCaptureMode(&mode);
  if (e != cudaSuccess) return e;
  e = dev_alloc(p, bytes + more);
  const bool allocated = e == cudaSuccess;
  cudaStreamCaptureStatus st = cudaStreamCaptureStatusActive;
  if (order && cudaStreamIsCapturing(*order, &st) != cudaSuccess) cudaGetLastError();
  if (allocated && order && st == cudaStreamCaptureStatusNone) {
    e = cudaMemsetAsync(*p, 0, bytes, *order);
  } else if (allocated) {
    cudaStream_t own = nullptr;
    e = cudaStreamCreateWithFlags(&own, cudaStreamNonBlocking);
    if (e == cudaSuccess) e = cudaMemsetAsync(*p, 0, bytes, own);
    if (e == cudaSuccess) e = cudaStreamSynchronize(own);
    if (own) cudaStreamDestroy(own);
  }
  cudaThreadExchangeStreamCaptureMode(&mode);
  if (allocated && e != cudaSuccess) {
    cudaFree(*p);
    *p = nullptr;
  }
  return e;
}

// Digit matrix [drows][dcols] of one side, allocated zeroed on first use
// (order: alloc_zeroed); the first of a context's two also holds the workspace of
// its K-split GEMM, where it will run one (not for a group's plan, without order).
cudaError_t ensure_digit_buffer(gbs_ctx *c, int side, const cudaStream_t *order) {
  if (c->digits[side]) return cudaSuccess;
  const Mat &m = side ? c->rhs : c->lhs;
  const size_t digits = std::max<size_t>(m.drows * m.dcols, 16);
  const size_t ws = order && !c->split_ws ? split_workspace_bytes(c) : 0, zeroed = ws ? split_workspace_zeroed(c) : 0;
  cudaError_t e = alloc_zeroed((void **)&c->digits[side], digits + zeroed, order, ws - zeroed);
  if (e == cudaSuccess && ws) {
    set_split_workspace(c, c->digits[side] + digits);
  } else if (e != cudaSuccess && ws) {
    cudaGetLastError();
    e = alloc_zeroed((void **)&c->digits[side], digits, order);
  }
  c->digit_maps_ready = false;
  c->digit_map_b64_ready = false;
  c->plan1_ready = false;
  c->digits_valid[side] = false;
  return e;
}

// Packed matrix of one side, allocated zeroed on first use.
cudaError_t ensure_packed_buffer(gbs_ctx *c, int side, const cudaStream_t *order) {
  if (c->packed[side]) return cudaSuccess;
  const Mat &m = side ? c->rhs : c->lhs;
  cudaError_t e = alloc_zeroed((void **)&c->packed[side],
                               std::max<size_t>(m.drows * m.dcols / 2, 16), order);
  c->plan1_ready = false;
  c->packed_valid[side] = false;
  return e;
}

// The digit kernel is exact when every partial sum stays below 2^24 in fp32
// and each operand's values fit e4m3 exactly (at most 4 bits).
bool tcg_eligible(const gbs_ctx *c) { return tc_exact(c, GBS_PIPE_TC); }

// Digits cost about one HBM byte per element of the larger operand; the
// CUDA-core popcount kernel costs 2 * min(M, N) * wA * wB bit operations per
// such element at ~1/45 of the HBM byte rate.  Below ~10 the latter is cheaper.
bool tcg_preferred(const gbs_ctx *c) {
  const uint64_t mn = std::min(c->lhs.nrows, c->rhs.nrows);
  return mn * c->lhs.nbits * c->rhs.nbits >= 10;
}

void tcg_plan_free(TcgPlan *p) {
  if (p->d_probs) cudaFree(p->d_probs);
  if (p->d_maps) cudaFree(p->d_maps);
  if (p->d_tiles) cudaFree(p->d_tiles);
  if (p->d_jobs) cudaFree(p->d_jobs);
  *p = TcgPlan();
}

// GBS_TCG_NIBBLES in the environment when a plan is built: 0 makes it a digit
// plan, 1 a packed one; unset, the estimate below chooses for groups, and single
// contexts run on the digits their imports write.  Returns 0, 1 or -1 (choose).
int tcg_packed_mode() {
  const char *v = getenv("GBS_TCG_NIBBLES");
  if (v && v[0] == '0') return 0;
  if (v && v[0] == '1') return 1;
  return -1;
}

namespace {

// Whether a plan runs faster with its problems' larger sides packed, by an
// estimate of its critical path: a chunk's boxes enter an SM at 105 bytes/ns (the
// unpacked side of the TMA, so packing does not help there) while its four MMAs
// take 0.15-0.27 us, and all tiles together stream their operands at 6 TB/s.
// Packing pays where HBM sets the pace.  Measured on the tensor cores alone,
// digits / packed: 4 problems of the 512-problem mix 15.3 / 15.4 us, 16 of them
// 34.8 / 23.8, 64 103 / 78, all 397 589 / 448; one of 16 x 8192 x 20000 40 / 28,
// of 128 x 4096 x 20000 28.1 / 27.5, of 256 x 9216 x 4096 19.9 / 20.1.
bool plan_prefers_packed(gbs_ctx *const *ctxs, int n) {
  const double sms = (double)std::max(1, sm_count());
  double tiles[2] = {0, 0}, work[2] = {0, 0}, longest[2] = {0, 0}, hbm[2] = {0, 0};
  auto mma_ns = [](double bn) { return bn <= 128 ? 37.0 : 37.0 + (bn - 128) * (31.0 / 128); };
  for (int i = 0; i < n; i++) {
    const Mat &L = ctxs[i]->lhs, &R = ctxs[i]->rhs;
    const Mat &A = L.nrows < R.nrows ? R : L;
    const double small = (double)std::min(L.nrows, R.nrows), large = (double)A.nrows;
    const double nk = (double)((L.ncols + 127) / 128), K = nk * 128;
    if (small == 0 || nk == 0) continue;
    for (int k = 0; k < 2; k++) {
      const double bn = std::min(256.0, std::ceil(small / 16) * 16);
      const double nt = std::ceil(large / 128) * std::ceil(small / bn);
      const double t = nk * std::max((128 * 128 + bn * 128) / 105.0, 4 * mma_ns(bn));  // ns
      tiles[k] += nt;
      work[k] += nt * t;
      longest[k] = std::max(longest[k], t);
      hbm[k] += large * K * (k && A.packable() ? 0.5 : 1.0) + small * K + 4 * small * large;
    }
  }
  double est[2];
  for (int k = 0; k < 2; k++)
    est[k] = std::max({tiles[k] > 0 ? work[k] / std::min(tiles[k], sms) : 0.0, longest[k], hbm[k] / 6000.0});
  return est[1] < 0.95 * est[0];
}

}  // namespace

// MMA N (tile width over the smaller side) of every problem of a plan:
// the whole smaller side up to 256 rows; while the plan's tiles leave SMs idle,
// the problem with the longest tiles gets narrower ones (a power of two: the
// padded rows are whole multiples).  CaffeNet's five GEMMs had 38 tiles, the
// longest 27 stages of 38 KB.
static std::vector<uint32_t> tile_widths(gbs_ctx *const *ctxs, int n) {
  const uint64_t sms = (uint64_t)std::max(1, sm_count());
  std::vector<uint32_t> bn(n);
  auto stage_ns = [](double w) {
    return std::max((16384.0 + 128.0 * w) / 105.0, 4 * (w <= 128 ? 37.0 : 37.0 + (w - 128) * (31.0 / 128)));
  };
  auto rows = [&](int i, bool large) {
    const uint64_t a = ctxs[i]->lhs.nrows, b = ctxs[i]->rhs.nrows;
    return large ? std::max(a, b) : std::min(a, b);
  };
  auto ntiles = [&](int i, uint32_t w) { return (rows(i, true) + 127) / 128 * ((rows(i, false) + w - 1) / w); };
  auto tile_ns = [&](int i) { return (double)((ctxs[i]->lhs.ncols + 127) / 128) * stage_ns(bn[i]); };
  uint64_t total = 0;
  for (int i = 0; i < n; i++) {
    bn[i] = (uint32_t)std::min<uint64_t>(256, std::max<uint64_t>(16, (rows(i, false) + 15) / 16 * 16));
    total += ntiles(i, bn[i]);
  }
  while (total < sms) {
    int worst = 0;
    for (int i = 1; i < n; i++)
      if (tile_ns(i) > tile_ns(worst)) worst = i;
    uint32_t next = 128;
    while (next >= bn[worst]) next /= 2;
    if (next < 16 || total - ntiles(worst, bn[worst]) + ntiles(worst, next) > sms) break;
    total += ntiles(worst, next) - ntiles(worst, bn[worst]);
    bn[worst] = next;
  }
  return bn;
}

// The plan of some contexts; `form` gives the tiles of a one-problem plan on digits.
int tcg_plan_build(TcgPlan *plan, gbs_ctx *const *ctxs, int n, const TcgForm *form) {
  tcg_plan_free(plan);
  const int mode = tcg_packed_mode();
  const bool packed = form ? false : mode < 0 ? plan_prefers_packed(ctxs, n) : mode == 1;
  plan->packed = packed;
  std::vector<TcgProblem> probs;
  std::vector<CUtensorMap> maps;
  std::vector<TcgTile> tiles;
  std::vector<uint64_t> cost;
  std::vector<ExpandJob> jobs;
  uint64_t threads = 0;
  const std::vector<uint32_t> widths = tile_widths(ctxs, n);
  for (int i = 0; i < n; i++) {
    gbs_ctx *c = ctxs[i];
    const Mat &L = c->lhs, &R = c->rhs;
    TcgProblem P;
    memset(&P, 0, sizeof(P));
    P.C = c->res;
    P.M = (uint32_t)L.nrows;
    P.N = (uint32_t)R.nrows;
    const uint32_t large = L.nrows < R.nrows ? 1u : 0u;
    P.swap = form ? form->swap : large;          // the larger side is MMA-A, unless the form says otherwise
    const int sa = P.swap ? 1 : 0, sb = 1 - sa;  // sides of MMA-A and MMA-B
    const bool pa = packed && (sa ? R : L).packable();
    const uint8_t sides = pa ? (uint8_t)((4u << sa) | (1u << sb)) : (uint8_t)3;
    for (int side = 0; side < 2; side++) {
      cudaError_t e = cudaSuccess;
      if ((sides >> side) & 1) e = ensure_digit_buffer(c, side);
      if (e == cudaSuccess && ((sides >> (2 + side)) & 1)) e = ensure_packed_buffer(c, side);
      if (e != cudaSuccess) {
        cudaGetLastError();
        return fail(GBS_ENOMEM, "tensor-core plan: digit or packed matrix allocation failed");
      }
    }
    plan->ctxs.push_back(c);
    plan->sides.push_back(sides);
    const Mat &MA = sa ? R : L, &MB = sb ? R : L;
    P.a_rows = (uint32_t)MA.drows;
    P.b_rows = (uint32_t)MB.drows;
    P.nk = (uint32_t)((L.ncols + 127) / 128);
    CUtensorMap m2[2];
    P.bn = form ? form->bn : widths[i];
    P.idesc = (1u << 4) | ((P.bn >> 3) << 17) | ((128u >> 4) << 24);  // fp32 += e4m3 x e4m3
    P.a_bytes = kTgABytes;
    P.scale = 1.f;
    bool ok = tc_map_u8(&m2[1], c->digits[sb], MB.dcols, MB.drows, P.bn);
    if (pa) {
      P.idesc |= 5u << 7;  // MMA-A: e2m1
      P.a_bytes = kTgABytes / 2;
      P.scale = 2.f;
      ok = ok && tc_map_packed(&m2[0], c->packed[sa], MA.dcols, MA.drows);
    } else {
      ok = ok && tc_map_u8(&m2[0], c->digits[sa], MA.dcols, MA.drows, 128);
    }
    if (!ok) return fail(GBS_EUNSUPPORTED, "tensor-core plan: tensor map encoding failed");
    const uint32_t rt = (uint32_t)((MA.nrows + 127) / 128), ct = (uint32_t)((MB.nrows + P.bn - 1) / P.bn);
    maps.push_back(m2[0]);
    maps.push_back(m2[1]);
    for (uint32_t t = 0; t < rt * ct; t++) {  // the tiles that share the larger side's rows in turn
      tiles.push_back(P.swap == large ? TcgTile{(uint32_t)probs.size(), t / ct, t % ct, 0u}
                                      : TcgTile{(uint32_t)probs.size(), t % rt, t / rt, 0u});
      cost.push_back((uint64_t)P.nk * (128 + P.bn));
    }
    probs.push_back(P);
    for (int side = 0; side < 2; side++) {
      const Mat &m = side ? R : L;
      for (int kind = 0; kind < 2; kind++) {  // digits, packed values
        if (!((sides >> (2 * kind + side)) & 1)) continue;
        ExpandJob j = kind ? make_packed_job(m, c->packed[side]) : make_expand_job(m, c->digits[side]);
        j.thread0 = threads;
        threads += ((uint64_t)j.nrows * j.chunks + 255) / 256 * 256;
        if (j.nrows && j.chunks) jobs.push_back(j);
      }
    }
  }
  std::vector<size_t> order(tiles.size());
  for (size_t i = 0; i < order.size(); i++) order[i] = i;
  std::stable_sort(order.begin(), order.end(), [&](size_t a, size_t b) { return cost[a] > cost[b]; });
  std::vector<TcgTile> sorted(tiles.size());
  for (size_t i = 0; i < order.size(); i++) sorted[i] = tiles[order[i]];

  cudaError_t e = upload(&plan->d_probs, probs.data(), probs.size());
  if (e == cudaSuccess) e = upload((CUtensorMap **)&plan->d_maps, maps.data(), maps.size());
  if (e == cudaSuccess) e = upload(&plan->d_tiles, sorted.data(), sorted.size());
  if (e == cudaSuccess) e = upload(&plan->d_jobs, jobs.data(), jobs.size());
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(gemm_tcg_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)tcg_smem_bytes());
  if (e != cudaSuccess) {
    cudaGetLastError();
    tcg_plan_free(plan);
    return fail(GBS_ENOMEM, "tensor-core plan: table upload failed");
  }
  plan->nprob = (uint32_t)probs.size();
  plan->ntiles = (uint32_t)sorted.size();
  plan->njobs = (int)jobs.size();
  plan->expand_threads = threads;
  plan->grid = (int)std::min<uint64_t>(plan->ntiles, (uint64_t)sm_count());
  return GBS_OK;
}

cudaError_t tcg_expand(TcgPlan &plan, cudaStream_t s) {
  if (plan.njobs && plan.expand_threads) {
    const uint64_t blocks = std::min<uint64_t>((plan.expand_threads + 255) / 256, (uint64_t)sm_count() * 16);
    expand_grouped_kernel<<<(unsigned)blocks, 256, 0, s>>>(plan.d_jobs, plan.njobs, plan.expand_threads);
    count_launch();
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  for (size_t i = 0; i < plan.ctxs.size(); i++)
    for (int side = 0; side < 2; side++) {
      if ((plan.sides[i] >> side) & 1) plan.ctxs[i]->digits_valid[side] = true;
      if ((plan.sides[i] >> (2 + side)) & 1) plan.ctxs[i]->packed_valid[side] = true;
    }
  return cudaSuccess;
}

cudaError_t tcg_gemm(const TcgPlan &plan, uint32_t *err, cudaStream_t s, int32_t *out0) {
  if (!plan.ntiles) return cudaSuccess;
  const cudaError_t e = launch_pdl(gemm_tcg_kernel, plan.grid, kTgThreads, tcg_smem_bytes(), s, plan.d_probs,
                                   reinterpret_cast<const CUtensorMap *>(plan.d_maps), plan.d_tiles, plan.ntiles,
                                   plan.nprob, err, out0);
  count_launch();
  return e != cudaSuccess ? e : cudaGetLastError();
}

}  // namespace gbs

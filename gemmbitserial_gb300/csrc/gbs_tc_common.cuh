// gbs_tc_common.cuh -- device primitives shared by the tensor-core kernels:
// mbarriers with bounded waits, TMA tile loads, tcgen05 descriptors and MMA
// issue, and the bit-plane -> e4m3 digit decode.
#pragma once
#include <cuda.h>
#include <stdint.h>

namespace gbs {

// Iterations of mbarrier try_wait before a wait gives up (each try_wait may
// also suspend the thread for a short, hardware-chosen time).
constexpr uint32_t kTcWaitLimit = 1u << 20;

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred P;\n mbarrier.try_wait.parity.shared::cta.b64 P, [%1], %2;\n selp.b32 %0, 1, 0, P;\n}\n"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
// Bounded wait: true when the phase completed; false on abort or timeout.
// A timeout raises the CTA's abort flag and sets bit 0 of *err.  The number of
// rounds is kTcWaitLimit but for the test hooks'.
__device__ __forceinline__ bool mbar_wait_rounds_err(uint32_t bar, uint32_t parity, volatile int *abort_flag,
                                                     uint32_t *err, uint32_t rounds) {
  for (uint32_t it = 0; it < rounds; ++it) {
    if (mbar_try(bar, parity)) return true;
    if (*abort_flag) return false;
  }
  *abort_flag = 1;
  atomicOr(err, 1u);
  return false;
}
__device__ __forceinline__ bool mbar_wait_err(uint32_t bar, uint32_t parity, volatile int *abort_flag,
                                              uint32_t *err) {
  return mbar_wait_rounds_err(bar, parity, abort_flag, err, kTcWaitLimit);
}
// Bounded wait that ignores the abort flag: drains work this thread issued.
// A timeout sets bit 1 of *err.
__device__ __forceinline__ void mbar_drain_err(uint32_t bar, uint32_t parity, uint32_t *err) {
  for (uint32_t it = 0; it < kTcWaitLimit; ++it)
    if (mbar_try(bar, parity)) return;
  atomicOr(err, 2u);
}

// Programmatic dependent launch.  A kernel launched with the
// programmatic-stream-serialization attribute may start while the kernel
// before it in the stream is still running: it sets up (barriers, TMEM) and
// then calls griddep_wait(), which returns once the previous grids have
// completed and their memory is visible; nothing before it may read or write
// global memory.  griddep_launch_dependents() lets the next such kernel in
// the stream be scheduled as soon as every CTA of this one has issued it (its
// CTAs then take SMs as ours leave and wait likewise).
__device__ __forceinline__ void griddep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void griddep_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;"); }

__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap *map, int x, int y, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
          dst),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(bar)
      : "memory");
}

// Rows [row, row + box) (row a multiple of 16) x digits [128 k, 128 k + 128)
// of a digit matrix through its blocked 4-D map (tc_map_u8): the box lands
// in shared memory as box x 128 bytes, rows in order, 128-byte swizzled.
__device__ __forceinline__ void tma_load_digits(uint32_t dst, const CUtensorMap *map, int k, uint32_t row,
                                                uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], "
      "[%6];" ::"r"(dst),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(0), "r"(0), "r"(k), "r"((int)(row >> 4)), "r"(bar)
      : "memory");
}

// ---- SM pairs (cta_group::2) and TMEM loads
__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t map_to_rank(uint32_t smem_addr, uint32_t rank) {
  uint32_t d;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(d) : "r"(smem_addr), "r"(rank));
  return d;
}
// tma_load_digits for an SM pair: completes on `bar`, the leader CTA's barrier.
__device__ __forceinline__ void tma_load_digits_pair(uint32_t dst, const CUtensorMap *map, int k, uint32_t row,
                                                     uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.cta_group::2 [%0], [%1, {%2, "
      "%3, %4, %5}], [%6];" ::"r"(dst),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(0), "r"(0), "r"(k), "r"((int)(row >> 4)), "r"(bar)
      : "memory");
}
// L2 prefetch of the box tma_load_digits(_pair) would load (a hint: no data
// lands in shared memory and no barrier is signalled).
__device__ __forceinline__ void tma_prefetch_digits(const CUtensorMap *map, int k, uint32_t row) {
  asm volatile("cp.async.bulk.prefetch.tensor.4d.L2.global.tile [%0, {%1, %2, %3, %4}];" ::"l"(
                   reinterpret_cast<uint64_t>(map)),
               "r"(0), "r"(0), "r"(k), "r"((int)(row >> 4))
               : "memory");
}
__device__ __forceinline__ void mma_f8_pair(uint32_t tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                            uint32_t acc) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::2.kind::f8f6f4 [%0], %1, %2, %3, p;\n}\n" ::"r"(tmem),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(acc));
}
// arrives on `bar` in both CTAs of the pair whose ranks are the set bits of `mask`
__device__ __forceinline__ void mma_commit_pair(uint32_t bar, uint16_t mask) {
  asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar),
      "h"(mask)
      : "memory");
}
// Generic address of the same shared-memory location in CTA `rank` of the
// cluster: plain loads through it can be batched by the compiler.
template <typename T>
__device__ __forceinline__ const T *cluster_ptr(const T *p, uint32_t rank) {
  uint64_t d;
  asm("mapa.u64 %0, %1, %2;" : "=l"(d) : "l"(reinterpret_cast<uint64_t>(p)), "r"(rank));
  return reinterpret_cast<const T *>(d);
}

__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&v)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
      "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
        "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]),
        "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]),
        "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
      : "r"(taddr));
}
// Waits for this thread's TMEM loads; the registers they fill are operands,
// so no use of them can be scheduled before the wait.
__device__ __forceinline__ void tmem_wait_ld(uint32_t (&v)[32]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(v[0]), "+r"(v[1]), "+r"(v[2]), "+r"(v[3]), "+r"(v[4]), "+r"(v[5]), "+r"(v[6]), "+r"(v[7]),
                 "+r"(v[8]), "+r"(v[9]), "+r"(v[10]), "+r"(v[11]), "+r"(v[12]), "+r"(v[13]), "+r"(v[14]), "+r"(v[15]),
                 "+r"(v[16]), "+r"(v[17]), "+r"(v[18]), "+r"(v[19]), "+r"(v[20]), "+r"(v[21]), "+r"(v[22]),
                 "+r"(v[23]), "+r"(v[24]), "+r"(v[25]), "+r"(v[26]), "+r"(v[27]), "+r"(v[28]), "+r"(v[29]),
                 "+r"(v[30]), "+r"(v[31])
               :
               : "memory");
}
// Marks registers a TMEM load filled as produced after the tcgen05.wait::ld
// issued just before (volatile asm keeps its place in program order): for
// several loads in flight behind one wait.
__device__ __forceinline__ void tmem_after_wait(uint32_t (&v)[32]) {
  asm volatile(""
               : "+r"(v[0]), "+r"(v[1]), "+r"(v[2]), "+r"(v[3]), "+r"(v[4]), "+r"(v[5]), "+r"(v[6]), "+r"(v[7]),
                 "+r"(v[8]), "+r"(v[9]), "+r"(v[10]), "+r"(v[11]), "+r"(v[12]), "+r"(v[13]), "+r"(v[14]), "+r"(v[15]),
                 "+r"(v[16]), "+r"(v[17]), "+r"(v[18]), "+r"(v[19]), "+r"(v[20]), "+r"(v[21]), "+r"(v[22]),
                 "+r"(v[23]), "+r"(v[24]), "+r"(v[25]), "+r"(v[26]), "+r"(v[27]), "+r"(v[28]), "+r"(v[29]),
                 "+r"(v[30]), "+r"(v[31])
               :
               : "memory");
}
// NC consecutive result columns n0 .. n0+NC-1 of result row m (res[n*M + m];
// a warp's lanes on consecutive m): one base pointer and a fixed column
// stride, whole blocks without per-column predicates.  A 64-bit index and a
// predicate per element measured up to ~2.5x slower in a persistent kernel.
template <int NC>
__device__ __forceinline__ void store_result_cols(int32_t *C, uint64_t M, uint64_t N, uint64_t m, uint64_t n0,
                                                  const int32_t (&o)[NC]) {
  if (m >= M) return;
  int32_t *p = C + n0 * M + m;
  if (n0 + NC <= N) {
#pragma unroll
    for (int j = 0; j < NC; j++) p[(uint64_t)j * M] = o[j];
  } else {
#pragma unroll
    for (int j = 0; j < NC; j++)
      if (n0 + j < N) p[(uint64_t)j * M] = o[j];
  }
}

// Shared-memory matrix descriptor: K-major, 128-byte swizzle, 8-row groups 1024 bytes apart.
__device__ __forceinline__ uint64_t sw128_desc(uint32_t addr) {
  return (uint64_t)((addr & 0x3FFFFu) >> 4) | ((uint64_t)1 << 16) | ((uint64_t)(1024 >> 4) << 32) |
         ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}
__device__ __forceinline__ void mma_f8(uint32_t tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], %1, %2, %3, p;\n}\n" ::"r"(tmem),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(acc));
}
// One lane of a converged warp, always the same: true there.  Warps that load or
// multiply walk their stages whole and issue from this lane: issued by lane 0 of a
// diverged warp, a stage of four MMAs takes 0.27 us to issue, as long as the four
// take on 256 columns (0.264), elected 0.19.  The one-tile pair kernel on
// 2048 x 4096 x 2048 went from 0.287 us a stage to that rate, 17.9 -> 17.1 us.
__device__ __forceinline__ bool elect_one() {
  uint32_t one;
  asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xffffffff;\n selp.u32 %0, 1, 0, p;\n}\n" : "=r"(one));
  return one != 0;
}
__device__ __forceinline__ void mma_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar)
               : "memory");
}

// The pair's form on one barrier of this CTA: issued MMAs finish before TMEM is freed.
__device__ __forceinline__ void mma_commit_done(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

__device__ __forceinline__ uint32_t bfe4(uint32_t x, int sh) {
  uint32_t r;
  asm("bfe.u32 %0, %1, %2, 4;" : "=r"(r) : "r"(x), "r"(sh));
  return r;
}

// 32 columns of row r of a packed matrix, from their codes (a byte each in q,
// bits above nbits ignored): even and odd columns gathered by byte, then eight
// elements at a time, with multiply-adds where they save integer instructions,
// which run at half their rate.
__device__ __forceinline__ void store_packed32(uint8_t *base, uint32_t r, uint32_t col0, uint64_t dcols, int nbits,
                                               int form, const uint32_t (&q)[8]) {
  const uint32_t ones = (1u << nbits) - 1u, msk = 0x01010101u * ones;
  uint32_t o[4];
#pragma unroll
  for (int i = 0; i < 4; i++)
    o[i] = (__byte_perm(q[2 * i], q[2 * i + 1], 0x7531u) & msk) * 16u +
           (__byte_perm(q[2 * i], q[2 * i + 1], 0x6420u) & msk);
  if (form == 2) {  // two's complement: magnitude (x ^ ones) + 1 and the sign bit, 8
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const uint32_t neg = (o[i] >> (nbits - 1)) & 0x11111111u;
      o[i] = (o[i] ^ (neg * ones)) + neg * 9u;
    }
  } else if (form == 3) {  // 0: -1 (9), 1: +1
#pragma unroll
    for (int i = 0; i < 4; i++) o[i] = 0x99999999u - o[i] * 8u;
  }
  *reinterpret_cast<uint4 *>(base + packed_offset(r, col0, dcols)) = make_uint4(o[0], o[1], o[2], o[3]);
}

// e4m3 bytes of 4 consecutive columns of one tile row: codes from the tile's
// planes (bits at column offset `sh` of each plane's 32-bit word), then a
// byte-permute lookup in the tile's 16-entry table.  Plane p's nibble is
// spread straight to bit p of each byte (multiplier and mask shifted by p).
template <int CNT>
__device__ __forceinline__ uint32_t decode4(const uint32_t (&pw)[4], int sh, const uint32_t (&tab)[4]) {
  uint32_t c = 0;
#pragma unroll
  for (int p = 0; p < CNT; p++) c |= (bfe4(pw[p], sh) * (0x00204081u << p)) & (0x01010101u << p);
  if (CNT == 1) return c;  // caller maps 0/1 bytes itself
  const uint32_t t = c | (c >> 4);                        // byte 0 = c0 | c1<<4, byte 2 = c2 | c3<<4
  const uint32_t sel = __byte_perm(t, 0u, 0x0020u);        // nibbles c0 c1 c2 c3 in the low 16 bits
  if (CNT <= 3) return __byte_perm(tab[0], tab[1], sel);
  const uint32_t lo = __byte_perm(tab[0], tab[1], sel & 0x7777u);
  const uint32_t hi = __byte_perm(tab[2], tab[3], sel & 0x7777u);
  const uint32_t m = ((c >> 3) & 0x01010101u) * 0xFFu;     // codes 8..15 take the high table
  return (lo & ~m) | (hi & m);
}


}  // namespace gbs

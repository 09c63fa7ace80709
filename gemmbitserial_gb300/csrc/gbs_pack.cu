// gbs_pack.cu -- packing of regular integer matrices into bit planes, and the
// plane-reading helpers (row sums, export).
//
// Semantics follow BitSerialMatrix::importRegular<T> (gemmbitserial.hpp:213-245),
// its quantize step (:170-186) and the uint8_t overload (:249-275): element
// (r, c) of plane b is bit b of the element's code, where the code is
//   * the raw byte for uint8 input (no quantisation),
//   * 1 if x > 0 else 0 for bipolar matrices (1-bit signed),
//   * the low byte of x otherwise (two's complement for signed matrices; the
//     reference's "add 2^(w-1) twice" leaves the low w bits of x unchanged).
// Rows >= nrows and columns >= ncols are zero in every plane.
//
// Every import ends the same way: a lane holds the codes of one "chunk", 32
// consecutive columns of one row (byte j%4 of q[j/4]), and emits one 32-bit
// word per plane, 32 bytes of the digit matrix and 16 bytes of the packed
// matrix.  Chunks are numbered along the padded rows, so chunk c of a plane is
// its 32-bit word c: a warp's 32 chunks store 128 contiguous bytes per plane
// whatever the row length, and no lane idles on short rows.
#include <algorithm>
#include <cstring>
#include <type_traits>

#include "gbs_internal.h"
#include "gbs_tc_common.cuh"

namespace gbs {
namespace {

constexpr unsigned kFull = 0xffffffffu;

// ---------------------------------------------------------------- emission

// One 32-bit word per plane from the lane's 32 codes.  Four codes at a time:
// a mask leaves bit b of each byte and a dp4a weighs the bytes 1, 2, 4, 8 (the
// next word's 16 .. 128), so two dp4a gather eight codes into a byte (times
// 2^b): 21 instructions a plane, where gathering through a 64-bit multiply
// took about 45.
__device__ __forceinline__ void emit_planes32(int nbits, uint32_t *__restrict__ p32, uint64_t plane32, uint64_t idx,
                                              const uint32_t (&q)[8]) {
  for (int b = 0; b < nbits; b++) {
    const uint32_t m = 0x01010101u << b;
    uint32_t a[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
      a[i] = __dp4a(q[2 * i] & m, 0x08040201u, 0u);
      a[i] = __dp4a(q[2 * i + 1] & m, 0x80402010u, a[i]);
    }
    const uint32_t lo = (a[0] + (a[1] << 8)) >> b, hi = (a[2] + (a[3] << 8)) >> b;
    p32[(uint64_t)b * plane32 + idx] = __byte_perm(lo, hi, 0x5410u);
  }
}

// Byte permute by 4-bit selectors: bit 3 of one gives the sign bit of the byte it
// names, eight times.
__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t sel) {
  uint32_t r;
  asm("prmt.b32 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(sel));
  return r;
}

// e4m3 digits of 8 codes (bytes of q0 and q1, bits above nbits ignored) out of the
// 16-entry byte table tab.  The codes' low bits, gathered eight to a word, are the
// selectors of a byte permute.  Of 4-bit codes the permute of the low half of the
// table, all of it positive, leaves 0 where bit 3 is set, the permute of the high
// half without its signs by the inverted bit 3 leaves 0 elsewhere, and the signs, one
// for the half, follow bit 3.
__device__ __forceinline__ void digits8(uint32_t q0, uint32_t q1, int nbits, uint32_t msk, uint4 tab, uint32_t &d0,
                                        uint32_t &d1) {
  const uint32_t sel = (__byte_perm(q0, q1, 0x7531u) & msk) * 16u + (__byte_perm(q0, q1, 0x6420u) & msk);
  d0 = prmt(tab.x, tab.y, sel);
  d1 = prmt(tab.x, tab.y, sel >> 16);
  if (nbits > 3) {
    const uint32_t inv = sel ^ 0x88888888u, sign = tab.z & 0x80808080u;
    const uint32_t z = tab.z & 0x7F7F7F7Fu, w = tab.w & 0x7F7F7F7Fu;
    d0 |= prmt(z, w, inv) | (q0 * 16u & sign);
    d1 |= prmt(z, w, inv >> 16) | (q1 * 16u & sign);
  }
}

// The lane's 32 digits (0 past ncols) into the digit matrix (dcols columns,
// 16-row blocks: digit_offset) as one 32-byte store.  Digit rows past nrows
// and columns past the planes' padded width stay as allocated: zero.
__device__ __forceinline__ void write_digits32(uint8_t *__restrict__ digits, int nbits, uint32_t ncols, uint64_t dcols,
                                               uint4 tab, uint32_t r, uint32_t col0, const uint32_t (&q)[8]) {
  const uint32_t msk = 0x01010101u * ((1u << nbits) - 1u);
  uint32_t d[8];
#pragma unroll
  for (int i = 0; i < 8; i += 2) digits8(q[i], q[i + 1], nbits, msk, tab, d[i], d[i + 1]);
  if (col0 + 32 > ncols) {
#pragma unroll
    for (int i = 0; i < 8; i++) {
      const uint32_t c = col0 + 4 * i;
      if (c + 4 > ncols) d[i] &= c >= ncols ? 0u : (0xFFFFFFFFu >> (8 * (4 - (ncols - c))));
    }
  }
  asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(digits + digit_offset(r, col0, dcols)),
               "r"(d[0]), "r"(d[1]), "r"(d[2]), "r"(d[3]), "r"(d[4]), "r"(d[5]), "r"(d[6]), "r"(d[7])
               : "memory");
}

// Everything chunk cc of row r writes; idx is its number along the padded
// rows, derived says whether the row is one of the matrix's own (padding rows
// have no digits or packed values).
__device__ __forceinline__ void emit_chunk(const PackJob &J, uint64_t idx, uint32_t r, uint32_t cc, bool derived,
                                           const uint32_t (&q)[8]) {
  emit_planes32(J.nbits, reinterpret_cast<uint32_t *>(J.planes), J.nrows_a * J.cpr, idx, q);
  if (!derived) return;
  if (J.digits)
    write_digits32(J.digits, J.lo_bits, (uint32_t)J.ncols, J.dcols,
                   make_uint4(J.dtab[0], J.dtab[1], J.dtab[2], J.dtab[3]), r, cc * 32, q);
  if (J.digits_hi) {  // the planes past lo_bits of a wide operand
    uint32_t h[8];
#pragma unroll
    for (int i = 0; i < 8; i++) h[i] = q[i] >> J.lo_bits;  // bits of the next byte are masked off with the rest
    write_digits32(J.digits_hi, J.nbits - J.lo_bits, (uint32_t)J.ncols, J.dcols,
                   make_uint4(J.dtab_hi[0], J.dtab_hi[1], J.dtab_hi[2], J.dtab_hi[3]), r, cc * 32, h);
  }
  // columns past ncols hold whatever the codes there give: the tensor-core kernel
  // multiplies them by digits that are zero
  if (J.packed) store_packed32(J.packed, r, cc * 32, J.dcols, J.nbits, J.pform, q);
}

// ---------------------------------------------------------------- chunk numbering

// A unit is 32 chunks, a lane each.  The unit's first chunk is located once, in
// 64 bits: its row r, its chunk of the row cc, and how many rows from r on are
// the matrix's own (rows) and to be written (rows_a).  The lanes then work in
// 32 bits, integer arithmetic being at half the rate of the other instructions (the
// grouped import issues 0.69 instructions a cycle and scheduler; a single operand's is a
// wave or two that wait on memory): chunk i is dr rows
// further, t = cc + i divided by cpr through a multiply-high by magic = 2^32 /
// cpr + 1 (exact while t * cpr < 2^32, i < 32 (kMaxRun + 1)), or, for rows of
// 65000 chunks and more, 0 or 1.
struct UnitBase {
  uint64_t r;
  uint32_t cc, rows, rows_a;
};
struct Chunk {
  uint32_t dr, cc;
};

__device__ __forceinline__ UnitBase unit_base(const PackJob &J, uint64_t row0, uint64_t rend, uint64_t unit) {
  const uint64_t c = unit * 32;
  UnitBase b;
  if (c <= 0xFFFFFFFFull) {
    const uint32_t q = (uint32_t)c / J.cpr;
    b.r = row0 + q;
    b.cc = (uint32_t)c - q * J.cpr;
  } else {
    const uint64_t q = c / J.cpr;
    b.r = row0 + q;
    b.cc = (uint32_t)(c - q * J.cpr);
  }
  b.rows = J.nrows > b.r ? (uint32_t)min(J.nrows - b.r, (uint64_t)0x80000000u) : 0u;
  b.rows_a = rend > b.r ? (uint32_t)min(rend - b.r, (uint64_t)0x80000000u) : 0u;
  return b;
}

__device__ __forceinline__ Chunk unit_chunk(const UnitBase &b, uint32_t i, uint32_t cpr, uint32_t magic) {
  const uint32_t t = b.cc + i;
  Chunk c;
  c.dr = cpr < 65000u ? __umulhi(t, magic) : (t >= cpr ? 1u : 0u);
  c.cc = t - c.dr * cpr;
  return c;
}

// ---------------------------------------------------------------- 1-byte rows, 16-byte aligned

// The lane's chunk straight from memory: one 32-byte load (VEC 2: rows and
// source 32-byte aligned) or two of 16 bytes (VEC 1).  A warp's two strided
// 16-byte loads touch each sector twice; the single load touches it once.
template <int VEC>
__device__ __forceinline__ void load_bytes32(const PackJob &J, const UnitBase &b, const Chunk &c, uint32_t (&q)[8]) {
#pragma unroll
  for (int i = 0; i < 8; i++) q[i] = 0u;
  const uint32_t col0 = c.cc * 32, ncols = (uint32_t)J.ncols;
  if (c.dr >= b.rows || col0 >= ncols) return;
  const uint8_t *p = (const uint8_t *)J.src + (b.r + c.dr) * J.ncols + col0;
  if (VEC == 2) {  // ncols is a multiple of 32: the chunk is whole
    asm volatile("ld.global.L1::no_allocate.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(q[0]), "=r"(q[1]), "=r"(q[2]), "=r"(q[3]), "=r"(q[4]), "=r"(q[5]), "=r"(q[6]), "=r"(q[7])
                 : "l"(p));
  } else {  // a multiple of 16: the chunk may be half
    const uint4 v0 = reinterpret_cast<const uint4 *>(p)[0];
    q[0] = v0.x; q[1] = v0.y; q[2] = v0.z; q[3] = v0.w;
    if (col0 + 32 <= ncols) {
      const uint4 v1 = reinterpret_cast<const uint4 *>(p)[1];
      q[4] = v1.x; q[5] = v1.y; q[6] = v1.z; q[7] = v1.w;
    }
  }
}

__device__ __forceinline__ void codes_of_bytes(int dtype, int bipolar, uint32_t (&q)[8]) {
  if (bipolar && dtype == GBS_I8) {
#pragma unroll
    for (int i = 0; i < 8; i++)  // 1 where the signed byte is above 0: bits 0-6 not zero, bit 7 clear
      q[i] = ((((q[i] & 0x7F7F7F7Fu) + 0x7F7F7F7Fu) & ~q[i]) >> 7) & 0x01010101u;
  }
}

template <int VEC>
__global__ void __launch_bounds__(256) pack_bytes(const __grid_constant__ PackJob J, uint64_t row0, uint64_t rend,
                                                  uint64_t units) {
  griddep_launch_dependents();
  griddep_wait();  // source, planes and digits belong to earlier kernels until here
  const uint64_t u = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (u >= units) return;  // warp-uniform
  const uint32_t lane = threadIdx.x & 31;
  uint32_t q[8];
  const UnitBase b = unit_base(J, row0, rend, u);
  const Chunk c = unit_chunk(b, lane, J.cpr, J.magic);
  if (c.dr >= b.rows_a) return;
  load_bytes32<VEC>(J, b, c, q);
  codes_of_bytes(J.dtype, J.nbits == 1 && J.issigned, q);
  emit_chunk(J, row0 * J.cpr + u * 32 + lane, (uint32_t)b.r + c.dr, c.cc, c.dr < b.rows, q);
}

// ---------------------------------------------------------------- every other source

// Four consecutive elements of a row (or, column-major, of a column) held raw.
template <typename T>
struct alignas(4 * sizeof(T)) Raw4 {
  uint32_t w[sizeof(T)];
};

// Elements [e, e + n) of the source, n <= 4 of them wanted (0 in the place of
// the others).  ALIGNED: e and the source's address allow one vector load
// whenever n = 4.  Otherwise 4-byte elements load one by one (the lanes' four
// loads share their sectors), and 1- and 2-byte elements as the two aligned
// words around them, shifted together, where those words lie inside the
// source (total elements).
template <typename T, bool ALIGNED>
__device__ __forceinline__ Raw4<T> load4(const T *__restrict__ src, uint64_t e, uint32_t n, uint64_t total) {
  Raw4<T> x;
#pragma unroll
  for (int i = 0; i < (int)sizeof(T); i++) x.w[i] = 0u;
  if (n == 0) return x;
  const T *p = src + e;
  if (ALIGNED && n == 4) {
    if constexpr (sizeof(T) == 1) {
      x.w[0] = *reinterpret_cast<const uint32_t *>(p);
    } else if constexpr (sizeof(T) == 2) {
      const uint2 v = *reinterpret_cast<const uint2 *>(p);
      x.w[0] = v.x; x.w[1] = v.y;
    } else {
      const uint4 v = *reinterpret_cast<const uint4 *>(p);
      x.w[0] = v.x; x.w[1] = v.y; x.w[2] = v.z; x.w[3] = v.w;
    }
    return x;
  }
  if constexpr (sizeof(T) == 4) {
    const uint32_t *p32 = reinterpret_cast<const uint32_t *>(p);
#pragma unroll
    for (int i = 0; i < 4; i++)
      if ((uint32_t)i < n) x.w[i] = p32[i];
  } else {
    constexpr int W = (int)sizeof(T);  // words of four elements
    const uintptr_t a = (uintptr_t)p, first = a & ~(uintptr_t)3;
    const uint32_t off = (uint32_t)(a & 3);
    if (n == 4 && first >= (uintptr_t)src && first + 4 * (W + 1) <= (uintptr_t)(src + total)) {
      const uint32_t *p32 = reinterpret_cast<const uint32_t *>(first);
      uint32_t v[W + 1];
#pragma unroll
      for (int i = 0; i <= W; i++) v[i] = p32[i];
#pragma unroll
      for (int i = 0; i < W; i++) x.w[i] = __funnelshift_r(v[i], v[i + 1], 8 * off);
    } else {
#pragma unroll
      for (int i = 0; i < 4; i++)
        if ((uint32_t)i < n) {
          if constexpr (sizeof(T) == 1) x.w[0] |= (uint32_t)(uint8_t)p[i] << (8 * i);
          else x.w[i >> 1] |= (uint32_t)(uint16_t)p[i] << (16 * (i & 1));
        }
    }
  }
  return x;
}

template <typename T>
__device__ __forceinline__ T elem_of(const Raw4<T> &x, int i) {
  if constexpr (sizeof(T) == 1) return (T)(x.w[0] >> (8 * i));
  else if constexpr (sizeof(T) == 2) return (T)(x.w[i >> 1] >> (16 * (i & 1)));
  else if constexpr (std::is_same<T, float>::value) return __uint_as_float(x.w[i]);
  else return (T)x.w[i];
}

// The low byte of (int64)x.  The 32-bit conversion gives it, saturation
// included, but for 2^31 <= x < 2^63, whose low byte is 0 (a float that large
// is a multiple of 2^8) where the 32-bit conversion saturates to 0x7FFFFFFF.
__device__ __forceinline__ uint32_t low_byte(float x) {
  const uint32_t v = (uint32_t)__float2int_rz(x);
  return (x >= 2147483648.f && x < 9223372036854775808.f) ? 0u : (v & 0xffu);
}

// quantize<float> (gemmbitserial.hpp:170-186): bipolar maps x > 0 to 1; a
// negative x of a signed matrix becomes 2^(w-1) + (uint8_t)(x + 2^(w-1)), the
// sum taken in float; otherwise (uint8_t)x.  Float -> integer casts truncate
// toward zero, then keep the low byte.
__device__ __forceinline__ uint32_t code_of_f32(float x, int bipolar, int issigned, int nbits) {
  if (bipolar) return x > 0.f ? 1u : 0u;
  if (issigned && x < 0.f) {
    const int h = 1 << (nbits - 1);
    return ((uint32_t)h + low_byte(x + (float)h)) & 0xffu;
  }
  return low_byte(x);
}

__device__ __forceinline__ uint32_t pack4(uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  return __byte_perm(__byte_perm(a, b, 0x0040u), __byte_perm(c, d, 0x0040u), 0x5410u);
}

// Codes of importRegular<T> for four elements, one byte each.
template <typename T>
__device__ __forceinline__ uint32_t codes4(const Raw4<T> &x, int bipolar, int issigned, int nbits) {
  if constexpr (std::is_same<T, uint8_t>::value) {
    return x.w[0];  // the uint8_t overload keeps the raw byte, bipolar or not
  } else if constexpr (std::is_same<T, float>::value) {
    uint32_t c[4];
#pragma unroll
    for (int i = 0; i < 4; i++) c[i] = code_of_f32(__uint_as_float(x.w[i]), bipolar, issigned, nbits);
    return pack4(c[0], c[1], c[2], c[3]);
  } else if (bipolar) {
    if constexpr (sizeof(T) == 1) return __vcmpgts4(x.w[0], 0u) & 0x01010101u;
    return pack4(elem_of<T>(x, 0) > 0, elem_of<T>(x, 1) > 0, elem_of<T>(x, 2) > 0, elem_of<T>(x, 3) > 0);
  } else {
    if constexpr (sizeof(T) == 1) return x.w[0];
    else if constexpr (sizeof(T) == 2) return __byte_perm(x.w[0], x.w[1], 0x6420u);
    else return pack4(x.w[0], x.w[1], x.w[2], x.w[3]);
  }
}

// importRegularAndQuantize<T> (gemmbitserial.hpp:282-305): element x of row r
// becomes the index of the first threshold thr[t * nrows + r] with x <= thr
// (compared in T), or nthres when x exceeds them all; with no thresholds the
// element keeps its own value.  The low byte of that index is the code the
// planes store (the (uint8_t) cast of :298).  For float input without
// thresholds the float is truncated toward zero to an integer first.  Four
// elements are scanned together; `over` says which have exceeded every
// threshold so far.
template <typename T>
__device__ __forceinline__ uint32_t own_codes4(const Raw4<T> &x) {
  uint32_t c[4];
#pragma unroll
  for (int i = 0; i < 4; i++) {
    if constexpr (std::is_same<T, float>::value) c[i] = low_byte(elem_of<T>(x, i));
    else c[i] = (uint32_t)elem_of<T>(x, i) & 0xffu;
  }
  return pack4(c[0], c[1], c[2], c[3]);
}

// A value no x exceeds, in the place of thresholds past the last.
template <typename T>
__device__ __forceinline__ T no_threshold() {
  if constexpr (std::is_same<T, float>::value) return __int_as_float(0x7f800000);
  else if constexpr (sizeof(T) == 4) return (T)0x7fffffff;
  else if constexpr (sizeof(T) == 2) return (T)0x7fff;
  else return std::is_same<T, uint8_t>::value ? (T)0xff : (T)0x7f;
}

template <typename T>
using Shuffled = typename std::conditional<std::is_same<T, float>::value, float, int>::type;  // a type to shuffle

// At most 7 thresholds of a row, lane j of each 8 holding the j-th (past the
// last the fill value), and what a search of them reads: every code of the row
// costs LEVELS compares, the threshold of each picked by a shuffle of the
// element's own index.
template <typename T>
struct RowThresholds {
  Shuffled<T> tv, next, mid;
  bool sorted;
  __device__ __forceinline__ explicit RowThresholds(T t) {
    tv = (Shuffled<T>)t;
    next = __shfl_down_sync(kFull, tv, 1, 8);  // lane j: threshold j + 1
    mid = __shfl_sync(kFull, tv, 3, 8);
    sorted = __all_sync(kFull, (threadIdx.x & 7) == 7 || tv <= next);
  }
  template <int LEVELS>
  __device__ __forceinline__ void search(const Shuffled<T> (&v)[4], uint32_t (&n)[4]) const {
#pragma unroll
    for (int i = 0; i < 4; i++) n[i] = LEVELS >= 3 && !(v[i] <= mid) ? 4u : 0u;
    if (LEVELS >= 2) {
#pragma unroll
      for (int i = 0; i < 4; i++)
        if (!(v[i] <= __shfl_sync(kFull, next, n[i], 8))) n[i] += 2u;
    }
#pragma unroll
    for (int i = 0; i < 4; i++)
      if (!(v[i] <= __shfl_sync(kFull, tv, n[i], 8))) n[i] += 1u;
  }
  template <int LEVELS>
  __device__ __forceinline__ uint32_t codes4(const Raw4<T> &x, int nthres) const {
    Shuffled<T> v[4];
    uint32_t n[4];
#pragma unroll
    for (int i = 0; i < 4; i++) v[i] = (Shuffled<T>)elem_of<T>(x, i);
    search<LEVELS>(v, n);
#pragma unroll
    for (int i = 0; i < 4; i++)
      if (std::is_same<T, float>::value) n[i] = min(n[i], (uint32_t)nthres);  // a NaN exceeds the fill value too
    return pack4(n[0], n[1], n[2], n[3]);
  }
};

// Four columns of one row, the row's thresholds in the 8 lanes of its chunk
// (lane j holds threshold 8 k + j of block k, block 0 in t0; past the last the
// fill value): one load and shuffles, where a load per threshold (each a line
// of its own, waited for in turn) took 31 us for 2048 x 4096 int32 against 7
// thresholds.  A block that ascends, as the reference assumes, is searched:
// LEVELS compares an element (3 for up to 7 thresholds), the threshold of
// each picked by a shuffle of the element's own index (a scan of all 7 ran
// 22 us, bound by integer instructions).  A block that does not is scanned for
// its first crossing.  Elements past every threshold of a block of 8 go on to
// the next.  2048 x 4096 int32 against 7 thresholds: 58 us loading a column
// run per lane, 15 us now (33.5 MB in, 11.5 MB out: 6.6 us at the copy rate).  No unit is
// busy there, SM 37 %, DRAM 28 %: 80 registers and the staging leave 24 warps an SM,
// 2.25 waves of them, and those wait on memory.  (A NaN exceeds the fill value too: counts are cut to the
// thresholds there are.)  Every lane of the warp calls it.
template <typename T, int LEVELS>
__device__ __forceinline__ uint32_t row_threshold_codes4(const Raw4<T> &x, T t0, const T *__restrict__ thr, int nthres,
                                                         uint64_t rthr, uint64_t nrows, bool row, bool wanted) {
  using S = Shuffled<T>;
  constexpr int kLast = LEVELS == 4 ? 8 : (1 << LEVELS) - 1;  // thresholds of a block
  const int lane = threadIdx.x & 31, j = lane & 7;
  S v[4], tv = (S)t0;
  uint32_t c[4] = {0u, 0u, 0u, 0u};
#pragma unroll
  for (int i = 0; i < 4; i++) v[i] = (S)elem_of<T>(x, i);
  bool over[4] = {wanted, wanted, wanted, wanted};
  for (int k = 0;; k += 8) {
    const RowThresholds<T> block((T)tv);
    uint32_t n[4];
    if (block.sorted) {
      block.template search<(LEVELS < 3 ? LEVELS : 3)>(v, n);
      if (LEVELS == 4) {  // a block of 8: past 7 of them, the last is left (below 7 the answer stands)
#pragma unroll
        for (int i = 0; i < 4; i++)
          if (!(v[i] <= __shfl_sync(kFull, tv, n[i], 8))) n[i] += 1u;
      }
    } else {
      bool on[4] = {true, true, true, true};
#pragma unroll
      for (int i = 0; i < 4; i++) n[i] = 0u;
#pragma unroll
      for (int t = 0; t < kLast; t++) {
        const S th = __shfl_sync(kFull, tv, t, 8);
#pragma unroll
        for (int i = 0; i < 4; i++) {
          on[i] = on[i] && !(v[i] <= th);
          if (on[i]) n[i] += 1u;
        }
      }
    }
    const uint32_t have = (uint32_t)min(kLast, nthres - k);
#pragma unroll
    for (int i = 0; i < 4; i++) {
      if (std::is_same<T, float>::value) n[i] = min(n[i], have);
      if (LEVELS == 4) {
        if (over[i]) c[i] += n[i];
        over[i] = over[i] && n[i] == have;
      } else {
        c[i] = n[i];
      }
    }
    if (LEVELS < 4 || k + 8 >= nthres || !__any_sync(kFull, over[0] || over[1] || over[2] || over[3]))
      return pack4(c[0], c[1], c[2], c[3]);
    tv = (S)((k + 8 + j < nthres && row) ? thr[(uint64_t)(k + 8 + j) * nrows + rthr] : no_threshold<T>());
  }
}

// Row-major sources of any element type and alignment.  A warp loads the unit's
// 1024 columns four elements a lane, 8 lanes to a chunk, so that its loads
// are contiguous whatever the element size (a lane loading the 32 columns it
// packs strides 32 elements from its neighbour, and every load then touches
// 32 lines: 60 us for 2048 x 4096 floats); the codes, a word of four, change
// hands through shared memory.  All eight loads are in flight before the first is converted.
// Word j of chunk i lies at 8 i + (j ^ 4 (i / 4 & 1)): the 16-byte reads of
// whole chunks then meet no bank conflict.
template <typename T>
struct QuantStage {  // a threshold import's raw elements and first thresholds, per warp and load
  Raw4<T> raw[8][8][32];
  T thr[8][8][32];
};

template <typename T, bool QUANT, bool ALIGNED>
__device__ __forceinline__ void pack_staged_unit(const PackJob &J, const T *__restrict__ thr, int nthres,
                                                 uint64_t row0, uint64_t rend, uint64_t u, uint32_t *__restrict__ st,
                                                 QuantStage<T> *__restrict__ qs) {
  const uint32_t lane = threadIdx.x & 31, j = lane & 7, ncols = (uint32_t)J.ncols;
  const UnitBase b = unit_base(J, row0, rend, u);
  const uint64_t total = J.nrows * J.ncols, e0 = b.r * J.ncols;
  const int bip = J.nbits == 1 && J.issigned;
  Raw4<T> x[8];
  const uint32_t at = (lane >> 3) * 8;
  const auto put = [&](int s, uint32_t w) { st[32 * s + at + (j ^ ((s & 1) << 2))] = w; };
  if (ALIGNED && (!QUANT || (nthres > 0 && nthres < 8)) && b.rows && b.cc + 32 <= J.cpr &&
      (b.cc + 32) * 32 <= ncols) {
    // The whole unit lies in one row: element 128 s + 4 lane of it, one set of thresholds
    const Raw4<T> *p = reinterpret_cast<const Raw4<T> *>((const T *)J.src + e0 + b.cc * 32 + 4 * lane);
#pragma unroll
    for (int s = 0; s < 8; s++) x[s] = p[32 * s];
    if (QUANT) {
      const T t = (int)j < nthres ? thr[(uint64_t)j * J.nrows + b.r] : no_threshold<T>();
      auto search = [&](auto levels) {
        const RowThresholds<T> r(t);
        if (r.sorted) {
#pragma unroll
          for (int s = 0; s < 8; s++) put(s, r.template codes4<decltype(levels)::value>(x[s], nthres));
        } else {
#pragma unroll 1
          for (int s = 0; s < 8; s++) {
            Raw4<T> v = x[0];
#pragma unroll
            for (int i = 1; i < 8; i++) v = s == i ? x[i] : v;
            put(s, row_threshold_codes4<T, decltype(levels)::value>(v, t, thr, nthres, b.r, J.nrows, true, true));
          }
        }
      };
      if (nthres == 1) search(std::integral_constant<int, 1>{});
      else if (nthres <= 3) search(std::integral_constant<int, 2>{});
      else search(std::integral_constant<int, 3>{});
    } else {
#pragma unroll
      for (int s = 0; s < 8; s++) put(s, codes4<T>(x[s], bip, J.issigned, J.nbits));
    }
  } else {
    T t0[8];
    uint32_t part = 0u;  // nibble s: the elements of load s that exist
#pragma unroll
    for (int s = 0; s < 8; s++) {
      const Chunk c = unit_chunk(b, 4 * s + (lane >> 3), J.cpr, J.magic);
      const uint32_t col = c.cc * 32 + 4 * j;
      const bool row = c.dr < b.rows;
      const uint32_t n = (row && col < ncols) ? min(4u, ncols - col) : 0u;
      x[s] = load4<T, ALIGNED>((const T *)J.src, e0 + (uint64_t)c.dr * ncols + col, n, total);
      if (QUANT) {
        t0[s] = (row && (int)j < nthres) ? thr[(uint64_t)j * J.nrows + (uint32_t)b.r + c.dr] : no_threshold<T>();
        part |= n << (4 * s);
      }
    }
    if (QUANT) {
      // the raw elements and first thresholds go through shared memory (the lane's own
      // words), so that the search is a loop: unrolled over eight loads in registers
      // it stalled on instruction fetch
      Raw4<T> *rx = qs->raw[threadIdx.x >> 5][0] + lane;
      T *rt = qs->thr[threadIdx.x >> 5][0] + lane;
#pragma unroll
      for (int s = 0; s < 8; s++) {
        rx[32 * s] = x[s];
        rt[32 * s] = t0[s];
      }
      auto codes = [&](auto scan) {
#pragma unroll 1
        for (int s = 0; s < 8; s++) {
          const uint32_t n = (part >> (4 * s)) & 15u;
          uint32_t w = scan(rx[32 * s], rt[32 * s], s, n != 0u);
          if (n < 4) w &= (1u << (8 * n)) - 1u;  // the code of a 0 put past the row's end is no code
          put(s, w);
        }
      };
      auto search = [&](auto levels) {
        codes([&](const Raw4<T> &v, T t, int s, bool wanted) {
          uint32_t dr = 0u;
          if (decltype(levels)::value == 4) dr = unit_chunk(b, 4 * s + (lane >> 3), J.cpr, J.magic).dr;
          return row_threshold_codes4<T, decltype(levels)::value>(v, t, thr, nthres, b.r + dr, J.nrows, dr < b.rows,
                                                                  wanted);
        });
      };
      if (nthres == 0) codes([&](const Raw4<T> &v, T, int, bool) { return own_codes4<T>(v); });
      else if (nthres == 1) search(std::integral_constant<int, 1>{});
      else if (nthres <= 3) search(std::integral_constant<int, 2>{});
      else if (nthres <= 7) search(std::integral_constant<int, 3>{});
      else search(std::integral_constant<int, 4>{});
    } else {
#pragma unroll
      for (int s = 0; s < 8; s++)
        put(s, codes4<T>(x[s], bip, J.issigned, J.nbits));
    }
  }
  __syncwarp();
  const uint32_t sw = ((lane >> 2) & 1u) << 2;
  const uint4 v0 = *reinterpret_cast<const uint4 *>(st + lane * 8 + sw);
  const uint4 v1 = *reinterpret_cast<const uint4 *>(st + lane * 8 + (sw ^ 4u));
  const uint32_t q[8] = {v0.x, v0.y, v0.z, v0.w, v1.x, v1.y, v1.z, v1.w};
  const Chunk c = unit_chunk(b, lane, J.cpr, J.magic);
  if (c.dr < b.rows_a)
    emit_chunk(J, row0 * J.cpr + u * 32 + lane, (uint32_t)b.r + c.dr, c.cc, c.dr < b.rows, q);
  __syncwarp();  // the next unit writes the staging words again
}

template <typename T, bool QUANT, bool ALIGNED>
__global__ void __launch_bounds__(256) pack_staged(const __grid_constant__ PackJob J, const T *__restrict__ thr,
                                                   int nthres, uint64_t row0, uint64_t rend, uint64_t units) {
  __shared__ __align__(16) uint32_t st[8][256];
  __shared__ typename std::conditional<QUANT, QuantStage<T>, char>::type qs;
  griddep_launch_dependents();
  griddep_wait();  // source, planes and digits belong to earlier kernels until here
  const uint64_t u = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (u >= units) return;  // warp-uniform; no block-wide barrier follows
  pack_staged_unit<T, QUANT, ALIGNED>(J, thr, nthres, row0, rend, u, st[threadIdx.x >> 5],
                                      reinterpret_cast<QuantStage<T> *>(&qs));
}

// ---------------------------------------------------------------- column-major sources

// The reference's readColMajor: element (r, c) at c * nrows + r.  A block takes
// 64 rows x 256 columns: threads load four consecutive rows of a column (a
// vector load where ALIGNED allows), put the code word in shared memory, and
// then each takes one chunk.  (Loading a column's rows one byte at a time by a
// lane per column, each lane a whole column apart from the next, ran 15 us on
// 169 x 2304.)  256 columns make the plane stores whole 32-byte sectors; 512
// threads have the tile's loads in flight at once (128 threads in four
// batches: 11.7 us on 169 x 2304, whose 27 tiles leave most SMs idle).  Word g
// (rows 4g ..) of column c lies at 17 c + 4 (c / 32) + g: the warp's 8 chunks
// read 8 different banks.
constexpr int kCmRows = 64, kCmCols = 256, kCmThreads = 512;
constexpr int kCmWords = kCmCols * 17 + 4 * (kCmCols / 32);

template <typename T, bool ALIGNED>
__global__ void __launch_bounds__(kCmThreads) pack_colmajor(const __grid_constant__ PackJob J) {
  __shared__ uint32_t st[kCmWords];
  griddep_launch_dependents();
  griddep_wait();  // source, planes and digits belong to earlier kernels until here
  // neighbouring blocks take neighbouring rows of the same columns: their reads are contiguous
  const uint32_t rblocks = (uint32_t)((J.nrows_a + kCmRows - 1) / kCmRows);
  const uint64_t r0 = (uint64_t)(blockIdx.x % rblocks) * kCmRows, c0 = (uint64_t)(blockIdx.x / rblocks) * kCmCols;
  const uint32_t tid = threadIdx.x;
  const uint64_t total = J.nrows * J.ncols;
  const int bip = J.nbits == 1 && J.issigned;
  constexpr int kLoads = kCmCols * (kCmRows / 4) / kCmThreads;  // a thread's row quadruples, all in flight at once
  Raw4<T> x[kLoads];
#pragma unroll
  for (int i = 0; i < kLoads; i++) {
    const uint32_t t = i * kCmThreads + tid;
    const uint64_t c = c0 + (t >> 4), r = r0 + 4 * (t & 15);
    const uint32_t n = (c < J.ncols && r < J.nrows) ? (uint32_t)min((uint64_t)4, J.nrows - r) : 0u;
    x[i] = load4<T, ALIGNED>((const T *)J.src, c * J.nrows + r, n, total);
  }
#pragma unroll
  for (int i = 0; i < kLoads; i++) {
    const uint32_t t = i * kCmThreads + tid, col = t >> 4, g = t & 15;
    st[col * 17 + 4 * (col >> 5) + g] = codes4<T>(x[i], bip, J.issigned, J.nbits);
  }
  __syncthreads();
  // a thread per (row, chunk): lanes 0..7 of a row its 8 chunks, four rows of a quadruple a warp
  const uint32_t k = tid & 7, i = (tid >> 3) & 3, g = tid >> 5;
  const uint64_t cc = c0 / 32 + k, r = r0 + 4 * g + i;
  if (cc >= J.cpr || r >= J.nrows_a) return;
  const uint32_t *p = st + k * (32 * 17 + 4) + g;
  const uint32_t sel = i | ((i + 4) << 4);  // byte i of two words
  uint32_t q[8];
#pragma unroll
  for (int w = 0; w < 8; w++)
    q[w] = __byte_perm(__byte_perm(p[(4 * w) * 17], p[(4 * w + 1) * 17], sel),
                       __byte_perm(p[(4 * w + 2) * 17], p[(4 * w + 3) * 17], sel), 0x5410u);
  emit_chunk(J, r * J.cpr + cc, (uint32_t)r, (uint32_t)cc, r < J.nrows, q);
}

// Threshold imports: a warp takes 32 rows x 32 columns, a lane a row, so a column's
// loads are contiguous, all 32 are in flight at once, and each threshold of a row is
// read once for its 32 columns.  In the tiles above, each thread with the thresholds of
// four rows, one load after the other: 8192 x 8192 int32 against 3 thresholds 151 us, 92
// this way, 2048 x 4096 24 and 14, 1048576 x 1 (tiles mostly empty) 277 and 53,
// 1 x 1048576 132 and 42.
template <typename T>
__global__ void __launch_bounds__(256) pack_colmajor_quant(const __grid_constant__ PackJob J,
                                                          const T *__restrict__ thr, int nthres) {
  griddep_launch_dependents();
  griddep_wait();  // source, planes and digits belong to earlier kernels until here
  const uint64_t w = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint64_t r = w / J.cpr * 32 + (threadIdx.x & 31);
  const uint32_t cc = (uint32_t)(w % J.cpr);
  if (r >= J.nrows_a) return;  // no warp-wide step follows
  uint32_t q[8] = {0u, 0u, 0u, 0u, 0u, 0u, 0u, 0u};
  const uint64_t c0 = (uint64_t)cc * 32;
  if (r < J.nrows && c0 < J.ncols) {
    const uint32_t n = (uint32_t)min((uint64_t)32, J.ncols - c0);
    const T *src = (const T *)J.src + c0 * J.nrows + r;
    T x[32];
#pragma unroll
    for (int j = 0; j < 32; j++) x[j] = (uint32_t)j < n ? src[(uint64_t)j * J.nrows] : (T)0;
    if (nthres == 0) {
#pragma unroll
      for (int j = 0; j < 32; j++)
        q[j >> 2] |= (std::is_same<T, float>::value ? low_byte((float)x[j]) : (uint32_t)x[j] & 0xffu) << (8 * (j & 3));
    } else {
      uint32_t over = n == 32 ? kFull : (1u << n) - 1u;  // columns above every threshold so far
      for (int t = 0; t < nthres && over; t++) {
        const T th = thr[(uint64_t)t * J.nrows + r];
        uint32_t above = 0u;
#pragma unroll
        for (int g = 0; g < 32; g += 8)
          if (g < (int)n) {  // the last columns of a row, or its only ones, are few
#pragma unroll
            for (int j = g; j < g + 8; j++) above |= !(x[j] <= th) ? 1u << j : 0u;
          }
        over &= above;
#pragma unroll
        for (int i = 0; i < 8; i++)  // one more in the bytes of those columns (mod 256, as the reference's cast)
          if (4 * i < (int)n) q[i] = __vadd4(q[i], (((over >> (4 * i)) & 15u) * 0x00204081u) & 0x01010101u);
      }
    }
  }
  emit_chunk(J, r * J.cpr + cc, (uint32_t)r, cc, r < J.nrows, q);
}

// ---------------------------------------------------------------- grouped import

// The job owning run w (the last with warp0 <= w), found by the whole warp: 32
// jobs probed a step, so 1024 jobs take two dependent loads, not ten.
__device__ __forceinline__ int find_job(const PackJob *jobs, int njobs, uint64_t w, int lane) {
  int lo = 0, n = njobs;  // the answer is in [lo, lo + n)
  while (n > 1) {
    const int step = (n + 31) / 32;
    const int j = lo + lane * step;
    const unsigned m = __ballot_sync(kFull, j < lo + n && jobs[j].warp0 <= w);  // lane 0 is always set
    const int k = 31 - __clz(m);
    n = min(step, n - k * step);
    lo += k * step;
  }
  return lo;
}

// One launch packs every operand of a grouped GEMM whose rows are 1-byte and
// 16-byte aligned.  A run is `run` units of one job (pack_run_units); a warp takes
// runs in a grid stride and keeps kDepth units' loads in flight.
// Bound by integer instructions beside HBM on large groups: 8.1 GB of the
// 512-problem mix (1-byte sources in, planes and packed or digit matrices out) in
// 1.34 ms, 0.9 of the copy rate, 0.69 instructions a cycle and scheduler; one strided
// pair of 16-byte loads per lane, a unit to a row segment and a binary search per run
// took 2.17 ms.
constexpr int kMaxRun = 8;
constexpr int kDepth = 2;

// Jobs of a small group as a kernel parameter: no table to copy before the launch.
struct InlineJobs {
  PackJob jobs[kInlinePackJobs];
};
static_assert(sizeof(InlineJobs) <= 4000, "kernel parameters");

// Packs direct runs w0, w0 + nw, ... of the warp; sj is the warp's shared-memory copy of its job.
__device__ __forceinline__ void pack_direct_runs(const PackJob *jobs, int njobs, uint64_t w0, uint64_t nw,
                                                 uint64_t runs, uint32_t run, PackJob &J) {
  const int lane = threadIdx.x & 31;
  for (uint64_t w = w0; w < runs; w += nw) {
    const int j = find_job(jobs, njobs, w, lane);
    static_assert(sizeof(PackJob) % 8 == 0 && sizeof(PackJob) / 8 <= 32, "one word a lane");
    __syncwarp();
    if (lane < (int)(sizeof(PackJob) / 8))
      reinterpret_cast<uint64_t *>(&J)[lane] = reinterpret_cast<const uint64_t *>(jobs + j)[lane];
    __syncwarp();
    const uint64_t u0 = (w - J.warp0) * run;
    const UnitBase b = unit_base(J, 0, J.nrows_a, u0);
    const int bip = J.nbits == 1 && J.issigned;
#pragma unroll 1
    for (uint32_t u = 0; u < run; u += kDepth) {
      Chunk c[kDepth];
      uint32_t q[kDepth][8];
#pragma unroll
      for (uint32_t d = 0; d < kDepth; d++) {
        if (u + d >= run) break;
        c[d] = unit_chunk(b, 32 * (u + d) + lane, J.cpr, J.magic);
        if (J.vec == 2) load_bytes32<2>(J, b, c[d], q[d]);
        else load_bytes32<1>(J, b, c[d], q[d]);
      }
#pragma unroll
      for (uint32_t d = 0; d < kDepth; d++) {
        if (u + d >= run) break;
        codes_of_bytes(J.dtype, bip, q[d]);
        if (c[d].dr < b.rows_a)
          emit_chunk(J, (u0 + u + d) * 32 + lane, (uint32_t)b.r + c[d].dr, c[d].cc, c[d].dr < b.rows, q[d]);
      }
    }
  }
}

__global__ void __launch_bounds__(256, 4) pack_grouped(const PackJob *__restrict__ jobs, int njobs, uint64_t runs,
                                                       uint32_t run) {
  __shared__ PackJob sj[8];  // each warp's job: its fields stay out of the registers
  griddep_launch_dependents();
  griddep_wait();  // sources, planes and digits belong to earlier kernels until here
  pack_direct_runs(jobs, njobs, ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5,
                   ((uint64_t)gridDim.x * blockDim.x) >> 5, runs, run, sj[threadIdx.x >> 5]);
}

// The same for the other operands (wider elements, unaligned rows).
template <typename T>
__device__ __forceinline__ void pack_staged_run(const PackJob &J, uint64_t u0, uint32_t run, uint32_t *st) {
  const uint64_t units = min((uint64_t)run, (J.nrows_a * J.cpr + 31) / 32 - u0);
#pragma unroll 1
  for (uint64_t u = u0; u < u0 + units; u++) {
    if (J.vec) pack_staged_unit<T, false, true>(J, nullptr, 0, 0, J.nrows_a, u, st, nullptr);
    else pack_staged_unit<T, false, false>(J, nullptr, 0, 0, J.nrows_a, u, st, nullptr);
  }
}

__device__ __forceinline__ void pack_staged_runs(const PackJob *jobs, int njobs, uint64_t w0, uint64_t nw,
                                                 uint64_t runs, uint32_t run, uint32_t *my) {
  const int lane = threadIdx.x & 31;
  for (uint64_t w = w0; w < runs; w += nw) {
    const PackJob &J = jobs[find_job(jobs, njobs, w, lane)];
    const uint64_t u0 = (w - J.warp0) * run;
    switch (J.dtype) {
      case GBS_I8: pack_staged_run<int8_t>(J, u0, run, my); break;
      case GBS_U8: pack_staged_run<uint8_t>(J, u0, run, my); break;
      case GBS_I16: pack_staged_run<int16_t>(J, u0, run, my); break;
      case GBS_I32: pack_staged_run<int32_t>(J, u0, run, my); break;
      default: pack_staged_run<float>(J, u0, run, my); break;
    }
  }
}

// Both kinds of jobs in one launch: the first `sblocks` blocks take the staged
// ones, which wait longer per unit, the others the direct ones.  CaffeNet's
// two kinds one after the other took 20 + 17 us.
struct PackRuns {
  int n;  // jobs of the kind
  uint32_t run;
  uint64_t runs;
};

__device__ __forceinline__ void pack_both(const PackJob *jobs, PackRuns direct, PackRuns staged, uint32_t sblocks) {
  union Shared {
    PackJob sj[8];
    uint32_t st[8][256];
  };
  __shared__ __align__(16) unsigned char raw[sizeof(Shared)];
  Shared &sh = *reinterpret_cast<Shared *>(raw);
  griddep_launch_dependents();
  griddep_wait();  // sources, planes and digits belong to earlier kernels until here
  const uint32_t warp = threadIdx.x >> 5;
  if (blockIdx.x < sblocks)
    pack_staged_runs(jobs + direct.n, staged.n, (uint64_t)blockIdx.x * 8 + warp, (uint64_t)sblocks * 8, staged.runs,
                     staged.run, sh.st[warp]);
  else
    pack_direct_runs(jobs, direct.n, (uint64_t)(blockIdx.x - sblocks) * 8 + warp,
                     (uint64_t)(gridDim.x - sblocks) * 8, direct.runs, direct.run, sh.sj[warp]);
}

__global__ void __launch_bounds__(256, 4) pack_grouped_both(const PackJob *__restrict__ jobs, PackRuns direct,
                                                            PackRuns staged, uint32_t sblocks) {
  pack_both(jobs, direct, staged, sblocks);
}
__global__ void __launch_bounds__(256, 4) pack_grouped_inline(const __grid_constant__ InlineJobs t, PackRuns direct,
                                                              PackRuns staged, uint32_t sblocks) {
  pack_both(t.jobs, direct, staged, sblocks);
}

// sumRows (arch-generic.hpp:6-37) of row r by one warp.  uint32 arithmetic
// reproduces the reference's int32 wrap-around.
__device__ __forceinline__ int32_t row_sum(const uint64_t *__restrict__ planes, int nbits, int issigned,
                                           uint64_t ncols, uint64_t nrows_a, uint64_t wpr, uint64_t r, int lane) {
  const bool bip = nbits == 1 && issigned;
  uint32_t acc = 0;
  for (int b = 0; b < nbits; b++) {
    const uint64_t *row = planes + (uint64_t)b * nrows_a * wpr + r * wpr;
    uint32_t cnt = 0;
    for (uint64_t w = lane; w < wpr; w += 32) cnt += __popcll(row[w]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) cnt += __shfl_xor_sync(kFull, cnt, o);
    cnt <<= b;
    if (issigned && !bip && b == nbits - 1) cnt = 0u - cnt;
    acc += cnt;
  }
  if (bip) acc = 2u * acc - (uint32_t)ncols;
  return (int32_t)acc;
}

__global__ void __launch_bounds__(256) rowsum_kernel(const uint64_t *__restrict__ planes, int nbits, int issigned,
                                                     uint64_t nrows, uint64_t ncols, uint64_t nrows_a,
                                                     uint64_t wpr, int32_t *__restrict__ dst) {
  griddep_launch_dependents();
  griddep_wait();  // source, planes and digits belong to earlier kernels until here
  const uint64_t r = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (r >= nrows) return;
  const int32_t v = row_sum(planes, nbits, issigned, ncols, nrows_a, wpr, r, lane);
  if (lane == 0) dst[r] = v;
}

// Grouped row sums: one warp per row over every job (warp0 counts rows).
__global__ void __launch_bounds__(256) rowsum_grouped(const PackJob *__restrict__ jobs, int njobs, uint64_t total) {
  griddep_launch_dependents();
  griddep_wait();  // source, planes and digits belong to earlier kernels until here
  const uint64_t nw = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  const int lane = threadIdx.x & 31;
  for (uint64_t w = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; w < total; w += nw) {
    const PackJob &J = jobs[find_job(jobs, njobs, w, lane)];
    const uint64_t r = w - J.warp0;
    const int32_t v = row_sum(J.planes, J.nbits, J.issigned, J.ncols, J.nrows_a, J.wpr, r, lane);
    if (lane == 0) J.rowsum[r] = v;
  }
}

// exportRegular (gemmbitserial.hpp:313-333): one thread per element.
__global__ void __launch_bounds__(256) export_kernel(const uint64_t *__restrict__ planes, int nbits, int issigned,
                                                     uint64_t nrows, uint64_t ncols, uint64_t nrows_a,
                                                     uint64_t wpr, int32_t *__restrict__ dst) {
  const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nrows * ncols) return;
  const uint64_t r = i / ncols, c = i % ncols;
  const bool bip = nbits == 1 && issigned;
  int32_t v = 0;
  for (int b = 0; b < nbits; b++) {
    uint64_t bit = (planes[(uint64_t)b * nrows_a * wpr + r * wpr + (c >> 6)] >> (c & 63)) & 1u;
    if (bip) v = bit ? 1 : -1;
    else if (bit) v += (issigned && b == nbits - 1) ? -(1 << b) : (1 << b);
  }
  dst[i] = v;
}

inline unsigned blocks_for(uint64_t threads, unsigned per_block) {
  return (unsigned)((threads + per_block - 1) / per_block);
}

}  // namespace

PackJob make_pack_job(const Mat &m, const void *src, int dtype, const DigitTarget *digits, uint8_t *packed) {
  PackJob j;
  memset(&j, 0, sizeof(j));
  j.src = src;
  j.planes = m.planes;
  j.packed = packed;
  j.pform = m.packed_form();
  j.nrows = m.nrows;
  j.ncols = m.ncols;
  j.nrows_a = m.nrows_a;
  j.wpr = m.wpr();
  j.dcols = m.dcols;
  j.nbits = (int)m.nbits;
  j.issigned = m.issigned;
  j.dtype = dtype;
  j.cpr = (uint32_t)(m.ncols_a / 32);
  j.magic = j.cpr ? (uint32_t)((1ull << 32) / j.cpr) + 1u : 0u;
  if (digits) {
    j.digits = digits->lo;
    j.digits_hi = digits->hi;
    j.lo_bits = digits->lo_bits;
    for (int i = 0; i < 4; i++) {
      j.dtab[i] = digits->tab_lo[i];
      j.dtab_hi[i] = digits->tab_hi[i];
    }
  }
  return j;
}

// 2 / 1: 1-byte rows, 32- / 16-byte aligned, packed by a load per lane; 0:
// the staged kernels.
static int bytes_vec(const Mat &m, const void *src, int dtype) {
  if (dtype != GBS_I8 && dtype != GBS_U8) return 0;
  const uintptr_t a = (uintptr_t)src | (uintptr_t)m.ncols;
  return a % 32 == 0 ? 2 : (a % 16 == 0 ? 1 : 0);
}

// Four consecutive elements can be one vector load: `run` (columns, or rows
// column-major) and the source's address allow it.
static bool aligned4(const void *src, int dtype, uint64_t run) {
  const uintptr_t size = (dtype == GBS_I16) ? 2 : (dtype == GBS_I32 || dtype == GBS_F32) ? 4 : 1;
  return run % 4 == 0 && (uintptr_t)src % (4 * size) == 0;
}

bool pack_job_direct(PackJob &j, const Mat &m) {
  j.vec = bytes_vec(m, j.src, j.dtype);
  if (j.vec) return true;
  j.vec = aligned4(j.src, j.dtype, m.ncols) ? 1 : 0;
  return false;
}

uint64_t pack_job_units(const PackJob &j) { return (j.nrows_a * j.cpr + 31) / 32; }

// Units per run of a grouped import of `units` units: two runs for each of 32
// warps on 152 SMs, whole pairs of units up to kMaxRun; finding a run's job and
// first row costs as much as two units.  CaffeNet's 61 K units take 19.7 us in runs
// of 8, 21.8 in runs of 3, and 23.8 in runs of 14, one to a warp.
uint32_t pack_run_units(uint64_t units) {
  const uint64_t each = (units + 152 * 64 - 1) / (152 * 64);
  return (uint32_t)(each <= 1 ? 1 : std::min<uint64_t>(kMaxRun, (each + kDepth - 1) / kDepth * kDepth));
}

namespace {

// Calls f with the source's element type and whether four elements load as one vector.
template <typename F>
void with_source(int dtype, bool aligned, F f) {
  auto go = [&](auto t) {
    if (aligned) f(t, std::true_type{});
    else f(t, std::false_type{});
  };
  switch (dtype) {
    case GBS_I8: go(int8_t{}); break;
    case GBS_U8: go(uint8_t{}); break;
    case GBS_I16: go(int16_t{}); break;
    case GBS_I32: go(int32_t{}); break;
    default: go(float{}); break;
  }
}

cudaError_t run_staged(const PackJob &j, const void *thr, int nthres, bool quant, bool aligned, uint64_t r0,
                       uint64_t r1, cudaStream_t s) {
  const uint64_t units = ((r1 - r0) * j.cpr + 31) / 32;
  cudaError_t e = cudaSuccess;
  with_source(j.dtype, aligned, [&](auto t, auto al) {
    using T = decltype(t);
    constexpr bool A = decltype(al)::value;
    const auto kern = quant ? pack_staged<T, true, A> : pack_staged<T, false, A>;
    e = launch_pdl(kern, blocks_for(units * 32, 256), 256, 0, s, j, (const T *)thr, nthres, r0, r1, units);
  });
  count_launch();
  return e != cudaSuccess ? e : cudaGetLastError();
}

cudaError_t run_colmajor(const PackJob &j, cudaStream_t s) {
  const uint64_t blocks = ((j.nrows_a + kCmRows - 1) / kCmRows) * ((j.wpr * 64 + kCmCols - 1) / kCmCols);
  if (blocks > 0x7FFFFFFFull) return cudaErrorInvalidConfiguration;
  cudaError_t e = cudaSuccess;
  with_source(j.dtype, aligned4(j.src, j.dtype, j.nrows), [&](auto t, auto al) {
    e = launch_pdl(pack_colmajor<decltype(t), decltype(al)::value>, (unsigned)blocks, kCmThreads, 0, s, j);
  });
  count_launch();
  return e != cudaSuccess ? e : cudaGetLastError();
}

cudaError_t run_colmajor_quant(const PackJob &j, const void *thr, int nthres, cudaStream_t s) {
  const uint64_t blocks = ((j.nrows_a + 31) / 32 * j.cpr + 7) / 8;
  if (blocks > 0x7FFFFFFFull) return cudaErrorInvalidConfiguration;
  cudaError_t e = cudaSuccess;
  with_source(j.dtype, false, [&](auto t, auto) {
    using T = decltype(t);
    e = launch_pdl(pack_colmajor_quant<T>, (unsigned)blocks, 256, 0, s, j, (const T *)thr, nthres);
  });
  count_launch();
  return e != cudaSuccess ? e : cudaGetLastError();
}

}  // namespace

cudaError_t launch_pack_rows(const Mat &m, const void *src, int dtype, uint64_t r0, uint64_t r1,
                             const DigitTarget *digits, cudaStream_t s) {
  if (m.nrows_a == 0 || m.wpr() == 0 || r1 <= r0) return cudaSuccess;
  PackJob j = make_pack_job(m, src, dtype, digits, nullptr);
  if (!pack_job_direct(j, m)) return run_staged(j, nullptr, 0, false, j.vec != 0, r0, r1, s);
  const uint64_t units = ((r1 - r0) * j.cpr + 31) / 32;
  const cudaError_t e =
      launch_pdl(j.vec == 2 ? pack_bytes<2> : pack_bytes<1>, blocks_for(units * 32, 256), 256, 0, s, j, r0, r1, units);
  count_launch();
  return e != cudaSuccess ? e : cudaGetLastError();
}

cudaError_t launch_pack_quantize(const Mat &m, const void *src, const void *thr, int nthres, int dtype,
                                 int col_major, const DigitTarget *digits, cudaStream_t s) {
  if (m.nrows_a == 0 || m.wpr() == 0) return cudaSuccess;
  const PackJob j = make_pack_job(m, src, dtype, digits, nullptr);
  if (col_major) return run_colmajor_quant(j, thr, nthres, s);
  return run_staged(j, thr, nthres, true, aligned4(src, dtype, m.ncols), 0, m.nrows_a, s);
}

cudaError_t launch_pack(const Mat &m, const void *src, int dtype, int col_major, const DigitTarget *digits,
                        cudaStream_t s) {
  if (m.nrows_a == 0 || m.wpr() == 0) return cudaSuccess;
  if (!col_major) return launch_pack_rows(m, src, dtype, 0, m.nrows_a, digits, s);
  return run_colmajor(make_pack_job(m, src, dtype, digits, nullptr), s);
}

cudaError_t launch_pack_grouped(const PackJob *host, const PackJob *jobs, const int (&n)[2], const uint64_t (&runs)[2],
                                const uint32_t (&run)[2], cudaStream_t s) {
  if (runs[0] + runs[1] == 0) return cudaSuccess;
  const PackRuns direct{n[0], run[0], runs[0]}, staged{n[1], run[1], runs[1]};
  const unsigned db = (unsigned)std::min<uint64_t>((runs[0] + 7) / 8, 152 * 64);
  const unsigned sb = (unsigned)std::min<uint64_t>((runs[1] + 7) / 8, 152 * 16);
  cudaError_t e;
  if (host) {
    InlineJobs t;
    memset(&t, 0, sizeof(t));
    memcpy(t.jobs, host, (size_t)(n[0] + n[1]) * sizeof(PackJob));
    e = launch_pdl(pack_grouped_inline, sb + db, 256, 0, s, t, direct, staged, sb);
  } else if (runs[1]) {
    e = launch_pdl(pack_grouped_both, sb + db, 256, 0, s, jobs, direct, staged, sb);
  } else {
    e = launch_pdl(pack_grouped, db, 256, 0, s, jobs, n[0], runs[0], run[0]);
  }
  count_launch();
  return e != cudaSuccess ? e : cudaGetLastError();
}

cudaError_t launch_rowsum_grouped(const PackJob *jobs, int njobs, uint64_t total_warps, cudaStream_t s) {
  if (total_warps == 0 || njobs == 0) return cudaSuccess;
  const uint64_t blocks = (total_warps + 7) / 8;
  const cudaError_t e =
      launch_pdl(rowsum_grouped, (unsigned)std::min<uint64_t>(blocks, 152 * 64), 256, 0, s, jobs, njobs, total_warps);
  count_launch();
  return e != cudaSuccess ? e : cudaGetLastError();
}

cudaError_t launch_rowsum(const Mat &m, int32_t *dst, cudaStream_t s) {
  if (m.nrows == 0) return cudaSuccess;
  const cudaError_t e = launch_pdl(rowsum_kernel, blocks_for(m.nrows * 32, 256), 256, 0, s, m.planes, (int)m.nbits,
                                   m.issigned, m.nrows, m.ncols, m.nrows_a, m.wpr(), dst);
  count_launch();
  return e != cudaSuccess ? e : cudaGetLastError();
}

cudaError_t launch_export(const Mat &m, int32_t *dst, cudaStream_t s) {
  if (m.nrows * m.ncols == 0) return cudaSuccess;
  export_kernel<<<blocks_for(m.nrows * m.ncols, 256), 256, 0, s>>>(m.planes, (int)m.nbits, m.issigned, m.nrows,
                                                                   m.ncols, m.nrows_a, m.wpr(), dst);
  count_launch();
  return cudaGetLastError();
}

}  // namespace gbs

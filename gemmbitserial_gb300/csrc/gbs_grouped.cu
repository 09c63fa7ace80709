// gbs_grouped.cu -- many independent bit-serial GEMMs in one persistent launch.
//
// The reference runs a list of GEMMs as a host loop of gemmBitSerial calls
// over a vector of contexts (benchmark.cpp:192-206, 217-219).  A group does the
// same work with
//   * one grouped pack launch for every operand (optional),
//   * one grouped row-sum launch when some problem is bipolar x regular,
//   * one persistent GEMM launch whose CTAs drain a device tile queue (an
//     atomic counter over a tile table sorted by decreasing cost),
// and can capture that sequence once into a CUDA graph for replay.  Each
// problem keeps its own context, so results land in each context's res.
//
// Problems go to one of two persistent kernels: the tensor-core kernel over
// e4m3 digit matrices (gbs_gemm_tcg.cu) where it is exact and cheaper, the
// CUDA-core popcount kernel otherwise.  GBS_GROUP_PIPE=popc or =tc in the
// environment forces one kernel (tc: wherever it is exact).  The grouped import
// writes the digit and packed matrices with the planes; where the planes came another
// way, one grouped expansion launch rebuilds them before the GEMM.
#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <string>
#include <vector>

#include "gbs_internal.h"

// Pack jobs of a grouped import on the device: those of the direct kernel, then those of the staged one.
struct PackTable {
  std::vector<gbs::PackJob> host;  // at most kInlinePackJobs of them go with the launch
  bool with_launch = false;
  gbs::PackJob *jobs = nullptr;    // the others' device table
  size_t capacity = 0;
  gbs::PackJob *recorded = nullptr;  // the table of an import recorded into a caller's capture
  int n[2] = {0, 0};
  uint64_t runs[2] = {0, 0};
  uint32_t run[2] = {1, 1};  // units per run
};

struct gbs_group {
  int device = 0;
  std::vector<gbs_ctx *> ctxs;
  gbs::GroupProblem *d_probs = nullptr;
  gbs::GroupTile *d_tiles = nullptr;
  uint32_t ntiles = 0;
  // [0] tile counter, [1] popcount-kernel error bits, [2] tensor-core error bits, [3] finished CTAs of the
  // popcount kernel, whose last one zeroes [0] and [3] for the next launch
  uint32_t *d_scratch = nullptr;
  uint32_t skinny = 1;  // outputs per warp of a skinny tile
  gbs::PackJob *d_rs_jobs = nullptr;
  int nrs = 0;
  uint64_t rs_warps = 0;
  PackTable imports, captured;  // of gbs_group_import, and of the captured graph (which keeps reading it)
  std::vector<gbs::PackJob *> foreign;  // tables of imports recorded into a caller's own capture
  cudaEvent_t packed = nullptr;  // after the last pack that read imports.jobs: that table may be written again
  bool packed_set = false;       // it has been recorded, which no capture ever does
  size_t smem = 0;
  int grid = 0;
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t exec = nullptr;
  bool graph_packs = false;  // the captured graph imports
  gbs::TcgPlan tc;  // problems on the tensor-core kernel
  std::vector<char> is_tc;  // per problem: on the tensor-core kernel
  // with both kernel types, the popcount kernel runs on a stream forked from
  // the caller's (and joined back), so the two share the SMs
  cudaStream_t side = nullptr;
  cudaEvent_t fork = nullptr, join = nullptr;
  uint64_t launches_per_replay = 0;
  uint32_t popc_tiles = 0;
};

namespace gbs {
namespace {

// Largest dynamic shared memory per CTA that still lets two CTAs share an SM.
constexpr size_t kGroupSmemCap = 113 * 1024;

bool device_ptr(const void *p) {
  cudaPointerAttributes a;
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return a.type == cudaMemoryTypeDevice || a.type == cudaMemoryTypeManaged;
}

void free_group(gbs_group *g) {
  tcg_plan_free(&g->tc);
  if (g->fork) cudaEventDestroy(g->fork);
  if (g->join) cudaEventDestroy(g->join);
  if (g->side) cudaStreamDestroy(g->side);
  if (g->exec) cudaGraphExecDestroy(g->exec);
  if (g->graph) cudaGraphDestroy(g->graph);
  if (g->d_probs) cudaFree(g->d_probs);
  if (g->d_tiles) cudaFree(g->d_tiles);
  if (g->d_scratch) cudaFree(g->d_scratch);
  if (g->d_rs_jobs) cudaFree(g->d_rs_jobs);
  if (g->imports.jobs) cudaFree(g->imports.jobs);
  if (g->captured.jobs) cudaFree(g->captured.jobs);
  for (gbs::PackJob *t : g->foreign) cudaFree(t);
  if (g->packed) cudaEventDestroy(g->packed);
  delete g;
}

template <typename T>
cudaError_t upload(T **dst, const std::vector<T> &v) {
  cudaError_t e = dev_alloc((void **)dst, v.size() * sizeof(T));
  if (e != cudaSuccess) return e;
  if (v.empty()) return cudaSuccess;
  return cudaMemcpy(*dst, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice);
}

// Builds the pack-job table for (lhs_srcs[p], rhs_srcs[p]) of every problem and
// copies it to the device in the order of stream s: after the last pack that
// read it, before the next.  (Allocating and copying it anew on each import
// freed the old one, which waited for the whole device: 25 us of a CaffeNet
// import.)
int build_pack_jobs(gbs_group *g, PackTable &tab, const void *const *lhs, const void *const *rhs, const int *dtypes,
                    cudaStream_t s) {
  std::vector<PackJob> jobs[2];  // direct, staged
  uint64_t units[2] = {0, 0};
  size_t ti = 0;  // index among the tensor-core problems
  for (size_t p = 0; p < g->ctxs.size(); p++) {
    const uint8_t digit_sides = g->is_tc[p] ? g->tc.sides[ti++] : 0;
    for (int side = 0; side < 2; side++) {
      const void *src = side ? rhs[p] : lhs[p];
      const int dt = dtypes ? dtypes[2 * p + side] : GBS_I8;
      if (dt < GBS_I8 || dt > GBS_F32) return fail(GBS_EINVAL, "gbs_group: unknown dtype");
      const Mat &m = side ? g->ctxs[p]->rhs : g->ctxs[p]->lhs;
      if (m.nrows_a == 0 || m.wpr() == 0) continue;
      if (m.nrows && m.ncols && (!src || !device_ptr(src)))
        return fail(GBS_EINVAL, "gbs_group: sources must be device pointers (problem " + std::to_string(p) + ")");
      DigitTarget digits;
      uint8_t *packed = nullptr;
      if ((digit_sides >> side) & 1) {  // tensor-core problem: the import writes the digit matrices it reads
        digits.lo = g->ctxs[p]->digits[side];
        digits.lo_bits = (int)m.nbits;
        tc_digit_table(m, digits.tab_lo);
      }
      if ((digit_sides >> (2 + side)) & 1) packed = g->ctxs[p]->packed[side];  // ... and packed matrices
      PackJob j = make_pack_job(m, src, dt, &digits, packed);
      const int kind = pack_job_direct(j, m) ? 0 : 1;
      units[kind] += pack_job_units(j);
      jobs[kind].push_back(j);
    }
  }
  for (int k = 0; k < 2; k++) {
    const uint32_t run = pack_run_units(units[k]);
    uint64_t runs = 0;
    for (PackJob &j : jobs[k]) {
      j.warp0 = runs;
      runs += (pack_job_units(j) + run - 1) / run;
    }
    tab.n[k] = (int)jobs[k].size();
    tab.runs[k] = runs;
    tab.run[k] = run;
  }
  jobs[0].insert(jobs[0].end(), jobs[1].begin(), jobs[1].end());
  tab.host.swap(jobs[0]);
  tab.with_launch = false;
  const size_t bytes = tab.host.size() * sizeof(PackJob);
  cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
  cudaError_t e = cudaStreamIsCapturing(s, &st);
  if (e == cudaSuccess && st != cudaStreamCaptureStatusNone) {
    // recorded into the caller's capture, where its mode allows allocating: a table that stays as it is
    gbs::PackJob *t = nullptr;
    e = upload(&t, tab.host);
    if (e == cudaSuccess) {
      g->foreign.push_back(t);
      tab.recorded = t;
    }
  } else if (e == cudaSuccess && tab.host.size() <= (size_t)kInlinePackJobs) {
    tab.with_launch = true;
    tab.recorded = nullptr;
  } else if (e == cudaSuccess) {
    if (tab.capacity < bytes) {
      if (tab.jobs) cudaFree(tab.jobs);  // waits for the device: nothing reads the old table any more
      tab.jobs = nullptr;
      tab.capacity = 0;
      e = dev_alloc((void **)&tab.jobs, bytes);
      if (e == cudaSuccess) tab.capacity = bytes;
    } else if (g->packed_set) {
      e = cudaStreamWaitEvent(s, g->packed, 0);
    }
    if (e == cudaSuccess) e = cudaMemcpyAsync(tab.jobs, tab.host.data(), bytes, cudaMemcpyHostToDevice, s);
    tab.recorded = nullptr;
  }
  if (e != cudaSuccess) {
    cudaGetLastError();
    tab.runs[0] = tab.runs[1] = 0;
    return fail(GBS_ENOMEM, "gbs_group: pack table upload failed");
  }
  return GBS_OK;
}

cudaError_t enqueue_pack(const PackTable &tab, cudaStream_t s) {
  return launch_pack_grouped(tab.with_launch ? tab.host.data() : nullptr, tab.recorded ? tab.recorded : tab.jobs, tab.n,
                             tab.runs, tab.run, s);
}

cudaError_t enqueue_popc(gbs_group *g, cudaStream_t s) {
  cudaError_t e = cudaSuccess;
  if (g->nrs) e = launch_rowsum_grouped(g->d_rs_jobs, g->nrs, g->rs_warps, s);
  if (e == cudaSuccess)
    e = launch_gemm_popc_grouped(g->d_probs, (int)g->ctxs.size(), g->d_tiles, g->popc_tiles, g->d_scratch,
                                 g->d_scratch + 3, g->d_scratch + 1, g->skinny, g->smem, g->grid, s);
  return e;
}

// With both kernel types, the tensor-core kernel follows on the caller's stream
// and the popcount kernel forks off: it starts a few us later, once the
// tensor-core CTAs have their SMs, and its CTAs take the room they leave (placed
// first, two of its CTAs fill an SM's registers).
cudaError_t enqueue_gemm(gbs_group *g, cudaStream_t s) {
  if (!g->popc_tiles) return tcg_gemm(g->tc, g->d_scratch + 2, s);
  if (!g->tc.ntiles) return enqueue_popc(g, s);
  cudaError_t e = cudaEventRecord(g->fork, s);
  if (e == cudaSuccess) e = tcg_gemm(g->tc, g->d_scratch + 2, s);
  if (e == cudaSuccess) e = cudaStreamWaitEvent(g->side, g->fork, 0);
  if (e == cudaSuccess) e = enqueue_popc(g, g->side);
  if (e == cudaSuccess) e = cudaEventRecord(g->join, g->side);
  if (e == cudaSuccess) e = cudaStreamWaitEvent(s, g->join, 0);
  return e;
}

// True when a digit or packed matrix some tensor-core problem reads is older than its planes.
bool digits_stale(const gbs_group *g) {
  for (size_t i = 0; i < g->tc.ctxs.size(); i++)
    for (int side = 0; side < 2; side++) {
      if (((g->tc.sides[i] >> side) & 1) && !g->tc.ctxs[i]->digits_valid[side]) return true;
      if (((g->tc.sides[i] >> (2 + side)) & 1) && !g->tc.ctxs[i]->packed_valid[side]) return true;
    }
  return false;
}

// After a grouped pack: the digit and packed matrices it wrote match the new
// planes, any other of the group's contexts is stale.
void mark_packed_digits(const gbs_group *g) {
  for (gbs_ctx *c : g->ctxs)
    for (int side = 0; side < 2; side++) c->digits_valid[side] = c->packed_valid[side] = false;
  for (size_t i = 0; i < g->tc.ctxs.size(); i++)
    for (int side = 0; side < 2; side++) {
      g->tc.ctxs[i]->digits_valid[side] = ((g->tc.sides[i] >> side) & 1) != 0;
      g->tc.ctxs[i]->packed_valid[side] = ((g->tc.sides[i] >> (2 + side)) & 1) != 0;
    }
}

// 0 = per-problem choice, 1 = popcount kernel only, 2 = tensor-core kernel wherever exact.
int group_pipe_mode() {
  const char *v = getenv("GBS_GROUP_PIPE");
  if (!v) return 0;
  if (!strcmp(v, "popc")) return 1;
  if (!strcmp(v, "tc")) return 2;
  return 0;
}

}  // namespace
}  // namespace gbs

using namespace gbs;

extern "C" {

int gbs_group_create(gbs_ctx *const *ctxs, int count, gbs_group **out) {
  if (!out) return fail(GBS_EINVAL, "gbs_group_create: out is NULL");
  *out = nullptr;
  if (count < 0 || (count > 0 && !ctxs)) return fail(GBS_EINVAL, "gbs_group_create: bad context list");
  gbs_group *g = new gbs_group();
  if (cudaGetDevice(&g->device) != cudaSuccess) {
    delete g;
    return cuda_fail(cudaGetLastError(), "gbs_group_create: no device");
  }
  std::vector<GroupProblem> probs;
  std::vector<GroupTile> tiles;
  std::vector<uint64_t> cost;
  std::vector<PackJob> rs;
  uint64_t rs_warps = 0;
  size_t smem = 16;
  const int mode = group_pipe_mode();
  std::vector<gbs_ctx *> tc_ctxs;
  std::vector<uint32_t> skinny_probs;
  uint64_t skinny_outputs = 0;
  for (int p = 0; p < count; p++) {
    gbs_ctx *c = ctxs[p];
    if (!c) {
      delete g;
      return fail(GBS_EINVAL, "gbs_group_create: context " + std::to_string(p) + " is NULL");
    }
    if (c->device != g->device) {
      delete g;
      return fail(GBS_EINVAL, "gbs_group_create: contexts must live on the current device");
    }
    g->ctxs.push_back(c);
    g->is_tc.push_back(mode != 1 && tcg_eligible(c) && (mode == 2 || tcg_preferred(c)) ? 1 : 0);
    if (g->is_tc.back()) {
      tc_ctxs.push_back(c);
      GroupProblem none;  // keeps the popcount table indexed by problem
      memset(&none, 0, sizeof(none));
      probs.push_back(none);
      continue;
    }
    Epilogue e;
    make_epilogue(c, e, c->rowsum);
    GroupProblem P;
    memset(&P, 0, sizeof(P));
    P.A = c->lhs.planes;
    P.B = c->rhs.planes;
    P.C = c->res;
    P.ra = e.ra;
    P.rb = e.rb;
    P.M = c->lhs.nrows;
    P.N = c->rhs.nrows;
    P.wpr = c->lhs.wpr();
    P.a_plane = c->lhs.nrows_a * P.wpr;
    P.b_plane = c->rhs.nrows_a * P.wpr;
    P.a_rows = c->lhs.nrows_a;
    P.b_rows = c->rhs.nrows_a;
    P.wa = (int)c->lhs.nbits;
    P.wb = (int)c->rhs.nbits;
    P.use_xor = e.use_xor;
    P.neg_i = e.neg_i;
    P.neg_j = e.neg_j;
    P.shift = e.shift;
    P.c0 = e.c0;
    // the skinny class, outputs of a warp each, where every BM x BN class would
    // leave most of its tile empty: fewer than 16 rhs rows (the classes' BN is
    // 64 or more), or a tiny output of more than 16 lhs rows; at most 16 lhs
    // rows take the rows class below (a warp per output waits on memory once
    // per output, a rows tile once per 128-byte step of 256 outputs)
    const bool rows_fit = P.M <= (uint64_t)kRowsMaxM && popc_rows_smem(P.wa, kRowsKC) <= kGroupSmemCap;
    if (P.N < 16 || (P.M * P.N <= 4096 && !rows_fit)) {
      P.cls = kSkinnyCls;
      probs.push_back(P);
      skinny_probs.push_back((uint32_t)p);
      skinny_outputs += P.M * P.N;
    } else if (rows_fit) {
      // at most 16 lhs rows: the rows class, one rhs row per thread (no popcounts on padding rows)
      P.cls = kRowsCls;
      smem = std::max(smem, popc_rows_smem(P.wa, kRowsKC));
      probs.push_back(P);
      const uint64_t bnr = (uint64_t)rows_tile_n(P.M), nt = (P.N + bnr - 1) / bnr;
      for (uint64_t j = 0; j < nt; j++) {
        tiles.push_back(GroupTile{(uint32_t)p, 0u, (uint32_t)j, (uint32_t)kRowsCls});
        cost.push_back((uint64_t)P.wa * P.wb * P.wpr);
      }
    } else {
      P.cls = popc_tile_class(P.M, P.wa, P.wb, kGroupSmemCap);
      smem = std::max(smem, popc_stage_smem(P.cls, P.wa, P.wb, kGroupKC));
      probs.push_back(P);
      const uint64_t bm = tile_bm(P.cls), bn = tile_bn(P.cls);
      const uint64_t mt = (P.M + bm - 1) / bm, nt = (P.N + bn - 1) / bn;
      for (uint64_t i = 0; i < mt; i++)
        for (uint64_t j = 0; j < nt; j++) {
          tiles.push_back(GroupTile{(uint32_t)p, (uint32_t)i, (uint32_t)j, (uint32_t)P.cls});
          cost.push_back((uint64_t)P.wa * P.wb * P.wpr);
        }
    }
    if (e.ra || e.rb) {  // bipolar x regular: row sums of the regular operand
      const Mat &reg = c->lhs.bipolar() ? c->rhs : c->lhs;
      PackJob j;
      memset(&j, 0, sizeof(j));
      j.planes = reg.planes;
      j.rowsum = c->rowsum;
      j.nrows = reg.nrows;
      j.ncols = reg.ncols;
      j.nrows_a = reg.nrows_a;
      j.wpr = reg.wpr();
      j.nbits = (int)reg.nbits;
      j.issigned = reg.issigned;
      j.warp0 = rs_warps;
      rs_warps += reg.nrows;
      if (reg.nrows) rs.push_back(j);
    }
  }
  // Skinny tiles: one output per warp until they fill the GPU (8 warps a CTA, 2
  // CTAs on each of 152 SMs), then up to 4: a warp's outputs share a trip to the queue
  g->skinny = (uint32_t)std::max<uint64_t>(1, std::min<uint64_t>(4, skinny_outputs / (8 * 2 * 152)));
  for (uint32_t p : skinny_probs) {
    const GroupProblem &P = probs[p];
    const uint64_t per = 8 * g->skinny, nt = (P.M * P.N + per - 1) / per;
    for (uint64_t i = 0; i < nt; i++) {
      tiles.push_back(GroupTile{p, (uint32_t)i, 0u, (uint32_t)kSkinnyCls});
      cost.push_back(std::max<uint64_t>(1, (uint64_t)g->skinny * P.wa * P.wb * P.wpr / 512));
    }
  }
  // Longest tiles first: the queue then balances like LPT scheduling.
  std::vector<size_t> order(tiles.size());
  for (size_t i = 0; i < order.size(); i++) order[i] = i;
  std::stable_sort(order.begin(), order.end(), [&](size_t a, size_t b) { return cost[a] > cost[b]; });
  std::vector<GroupTile> sorted(tiles.size());
  for (size_t i = 0; i < order.size(); i++) sorted[i] = tiles[order[i]];

  if (!tc_ctxs.empty()) {
    const int rc = tcg_plan_build(&g->tc, tc_ctxs.data(), (int)tc_ctxs.size());
    if (rc != GBS_OK) {
      free_group(g);
      return rc;
    }
  }
  cudaError_t e = upload(&g->d_probs, probs);
  if (e == cudaSuccess) e = upload(&g->d_tiles, sorted);
  if (e == cudaSuccess) e = upload(&g->d_rs_jobs, rs);
  if (e == cudaSuccess) e = dev_alloc((void **)&g->d_scratch, 4 * sizeof(uint32_t));
  if (e == cudaSuccess) e = cudaMemset(g->d_scratch, 0, 4 * sizeof(uint32_t));
  if (e == cudaSuccess) e = prepare_gemm_popc_grouped(smem);
  if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&g->side, cudaStreamNonBlocking);
  if (e == cudaSuccess) e = cudaEventCreateWithFlags(&g->fork, cudaEventDisableTiming);
  if (e == cudaSuccess) e = cudaEventCreateWithFlags(&g->join, cudaEventDisableTiming);
  if (e == cudaSuccess) e = cudaEventCreateWithFlags(&g->packed, cudaEventDisableTiming);
  if (e != cudaSuccess) {
    cudaGetLastError();
    free_group(g);
    return fail(GBS_ENOMEM, "gbs_group_create: device allocation or upload failed");
  }
  g->popc_tiles = (uint32_t)sorted.size();
  g->ntiles = g->popc_tiles + g->tc.ntiles;
  g->nrs = (int)rs.size();
  g->rs_warps = rs_warps;
  g->smem = smem;
  int sms = 0;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, g->device);
  g->grid = std::max(1, std::min<int>((int)g->popc_tiles, sms * grouped_blocks_per_sm(smem)));
  *out = g;
  return GBS_OK;
}

int gbs_group_free(gbs_group *g) {
  if (!g) return GBS_OK;
  cudaDeviceSynchronize();
  free_group(g);
  return GBS_OK;
}

int gbs_group_import(gbs_group *g, const void *const *lhs_srcs, const void *const *rhs_srcs, const int *dtypes,
                     void *stream) {
  if (!g || !lhs_srcs || !rhs_srcs) return fail(GBS_EINVAL, "gbs_group_import: NULL argument");
  int rc = build_pack_jobs(g, g->imports, lhs_srcs, rhs_srcs, dtypes, (cudaStream_t)stream);
  if (rc != GBS_OK) return rc;
  cudaError_t e = enqueue_pack(g->imports, (cudaStream_t)stream);
  if (e == cudaSuccess && !g->imports.with_launch && !g->imports.recorded) {
    e = cudaEventRecord(g->packed, (cudaStream_t)stream);
    g->packed_set = e == cudaSuccess;
  }
  if (e != cudaSuccess) return cuda_fail(e, "gbs_group_import: pack kernel");
  for (gbs_ctx *c : g->ctxs) {
    c->lhs.imported = c->rhs.imported = true;
    c->vt_valid[0] = c->vt_valid[1] = false;
  }
  mark_packed_digits(g);
  return GBS_OK;
}

int gbs_group_gemm(gbs_group *g, void *stream) {
  if (!g) return fail(GBS_EINVAL, "gbs_group_gemm: group is NULL");
  for (gbs_ctx *c : g->ctxs)
    if (!c->lhs.imported || !c->rhs.imported) return fail(GBS_ESTATE, "gbs_group_gemm: import every operand first");
  cudaError_t e = cudaSuccess;
  if (digits_stale(g)) e = tcg_expand(g->tc, (cudaStream_t)stream);
  if (e == cudaSuccess) e = enqueue_gemm(g, (cudaStream_t)stream);
  if (e == cudaSuccess)
    for (gbs_ctx *c : g->ctxs) c->res_stale = false;
  return e == cudaSuccess ? GBS_OK : cuda_fail(e, "gbs_group_gemm");
}

int gbs_group_capture(gbs_group *g, const void *const *lhs_srcs, const void *const *rhs_srcs, const int *dtypes,
                      void *stream) {
  if (!g) return fail(GBS_EINVAL, "gbs_group_capture: group is NULL");
  if (!stream)  // CUDA cannot capture the legacy default stream
    return fail(GBS_EINVAL, "gbs_group_capture: capture needs a created stream, not the legacy default stream");
  const bool with_pack = lhs_srcs && rhs_srcs;
  // a stream under capture cannot begin another, and waiting for it below would end the caller's
  cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
  cudaError_t ce = cudaStreamIsCapturing((cudaStream_t)stream, &st);
  if (ce == cudaSuccess && st != cudaStreamCaptureStatusNone) ce = cudaErrorIllegalState;
  if (ce != cudaSuccess) return cuda_fail(ce, "gbs_group_capture: the stream is being captured");
  if (with_pack) {
    // a graph captured before may still run and read its table; the new table is there before any replay
    cudaError_t se = g->captured.jobs ? cudaDeviceSynchronize() : cudaSuccess;
    if (se != cudaSuccess) return cuda_fail(se, "gbs_group_capture: device sync");
    int rc = build_pack_jobs(g, g->captured, lhs_srcs, rhs_srcs, dtypes, (cudaStream_t)stream);
    if (rc != GBS_OK) return rc;
    se = cudaStreamSynchronize((cudaStream_t)stream);
    if (se != cudaSuccess) return cuda_fail(se, "gbs_group_capture: pack table upload");
  } else {
    for (gbs_ctx *c : g->ctxs)
      if (!c->lhs.imported || !c->rhs.imported)
        return fail(GBS_ESTATE, "gbs_group_capture: without sources, import every operand first");
  }
  if (g->exec) cudaGraphExecDestroy(g->exec);
  if (g->graph) cudaGraphDestroy(g->graph);
  g->exec = nullptr;
  g->graph = nullptr;
  cudaStream_t s = (cudaStream_t)stream;
  if (!with_pack && digits_stale(g)) {  // the graph then holds the GEMMs only
    cudaError_t xe = tcg_expand(g->tc, s);
    if (xe != cudaSuccess) return cuda_fail(xe, "gbs_group_capture: digit expansion");
  }
  cudaError_t e = cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal);
  if (e != cudaSuccess) return cuda_fail(e, "gbs_group_capture: begin capture");
  cudaError_t ke = cudaSuccess;
  if (with_pack) ke = enqueue_pack(g->captured, s);
  if (ke == cudaSuccess) ke = enqueue_gemm(g, s);
  e = cudaStreamEndCapture(s, &g->graph);
  if (ke != cudaSuccess) return cuda_fail(ke, "gbs_group_capture: enqueue");
  if (e != cudaSuccess) return cuda_fail(e, "gbs_group_capture: end capture");
  e = cudaGraphInstantiate(&g->exec, g->graph, 0);
  if (e != cudaSuccess) return cuda_fail(e, "gbs_group_capture: instantiate");
  g->launches_per_replay = (with_pack && !g->captured.host.empty() ? 1 : 0) +
                           (g->popc_tiles ? 1 + (g->nrs ? 1 : 0) : 0) + (g->tc.ntiles ? 1 : 0);
  g->graph_packs = with_pack;
  if (with_pack) {
    for (gbs_ctx *c : g->ctxs) c->lhs.imported = c->rhs.imported = true;
    mark_packed_digits(g);  // each replay packs them
  }
  return GBS_OK;
}

int gbs_group_replay(gbs_group *g, void *stream) {
  if (!g || !g->exec) return fail(GBS_ESTATE, "gbs_group_replay: capture the group first");
  cudaError_t e = cudaGraphLaunch(g->exec, (cudaStream_t)stream);
  if (e != cudaSuccess) return cuda_fail(e, "gbs_group_replay");
  if (g->graph_packs) {  // the replay packs new planes: cached adjoint operands and other derived copies are stale
    for (gbs_ctx *c : g->ctxs) c->vt_valid[0] = c->vt_valid[1] = false;
    mark_packed_digits(g);
  }
  for (gbs_ctx *c : g->ctxs) c->res_stale = false;
  count_launch(g->launches_per_replay);
  return GBS_OK;
}

int gbs_group_status(gbs_group *g, void *stream) {
  if (!g) return fail(GBS_EINVAL, "gbs_group_status: group is NULL");
  uint32_t err[2] = {0, 0};
  cudaError_t e = cudaMemcpyAsync(err, g->d_scratch + 1, sizeof(err), cudaMemcpyDeviceToHost, (cudaStream_t)stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize((cudaStream_t)stream);
  if (e != cudaSuccess) return cuda_fail(e, "gbs_group_status");
  if (err[0]) return fail(GBS_EINVAL, "gbs_group_status: the grouped kernel rejected tile descriptors (bits " +
                                          std::to_string(err[0]) + ")");
  if (err[1] & 4u) return fail(GBS_EINVAL, "gbs_group_status: the tensor-core kernel rejected tile descriptors");
  if (err[1]) return fail(GBS_ECUDA, "gbs_group_status: a tensor-core pipeline wait timed out (bits " +
                                         std::to_string(err[1]) + ")");
  return GBS_OK;
}

int gbs_group_stats(const gbs_group *g, uint64_t *ntiles, uint64_t *smem_bytes, uint64_t *grid) {
  if (!g) return fail(GBS_EINVAL, "gbs_group_stats: group is NULL");
  if (ntiles) *ntiles = g->ntiles;
  if (smem_bytes) *smem_bytes = g->smem;
  if (grid) *grid = (uint64_t)g->grid;
  return GBS_OK;
}

int gbs_group_split(const gbs_group *g, uint64_t *popc_problems, uint64_t *tc_problems, uint64_t *tc_tiles) {
  if (!g) return fail(GBS_EINVAL, "gbs_group_split: group is NULL");
  if (popc_problems) *popc_problems = g->ctxs.size() - g->tc.ctxs.size();
  if (tc_problems) *tc_problems = g->tc.ctxs.size();
  if (tc_tiles) *tc_tiles = g->tc.ntiles;
  return GBS_OK;
}

int gbs_debug_group_tc_kernel(const gbs_group *g) {
  if (!g) return -fail(GBS_EINVAL, "gbs_debug_group_tc_kernel: group is NULL");  // negative: not a kernel code
  if (!g->tc.ntiles) return 0;
  return g->tc.packed ? 2 : 1;
}

int gbs_debug_group_poison_tile(gbs_group *g, uint32_t tile) {
  if (!g || tile >= g->ntiles) return fail(GBS_EINVAL, "gbs_debug_group_poison_tile: bad tile");
  cudaError_t e;
  if (tile < g->popc_tiles) {
    GroupTile bad{0xffffffffu, 0u, 0u, 0u};
    e = cudaMemcpy(g->d_tiles + tile, &bad, sizeof(bad), cudaMemcpyHostToDevice);
  } else {
    TcgTile bad{0xffffffffu, 0u, 0u, 0u};
    e = cudaMemcpy(g->tc.d_tiles + (tile - g->popc_tiles), &bad, sizeof(bad), cudaMemcpyHostToDevice);
  }
  return e == cudaSuccess ? GBS_OK : cuda_fail(e, "gbs_debug_group_poison_tile");
}

}  // extern "C"

// dd_host.cu — C-ABI implementation: contexts, launches, batches, graphs.
//
// The reference crosses the host/device boundary once per driver call:
// cudaMalloc + cudaMemset of the bins, one launch per device, a D2H copy and a
// host sum, then cudaDeviceReset (src/an_coding.cu:320-421).  Here a context
// keeps its device buffers resident across calls, one launch serves any number
// of instances, and the only per-call traffic is the job table (H2D) and the
// raw bins (D2H), both through pinned host buffers on the context's stream.
#include <cuda_runtime.h>

#include <algorithm>
#include <chrono>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <string>
#include <vector>

#include "../../include/codrel_b200.h"
#include "dd_carry.h"
#include "dd_device.cuh"
#include "dd_host.h"
#include "dd_kernels.h"
#include "dd_mma.h"

struct dd_context {
  int device = 0;
  cudaStream_t stream = nullptr;
  bool own_stream = false;
  int num_sms = 0;
  // device state
  // one buffer, so that a launch clears it with one memset and reads it back with one
  // copy: control words, the launch's bins (kMaxBins a slot), then the carry path's
  // sums (2 x kMaxBins a job)
  unsigned long long* d_mem = nullptr;
  unsigned long long* d_bins = nullptr;  // bin_slots x kMaxBins
  uint32_t bin_slots = 0;
  unsigned long long* d_ctl = nullptr;   // [0] popc work counter, [1] MMA work counter, [2] status, [3..15] diagnostics
  dd::Job* d_jobs = nullptr;
  uint32_t job_cap = 0;
  void* d_stage = nullptr;               // carry path: staged histograms of one block
  size_t stage_cap = 0;
  // pinned host mirrors
  unsigned long long* h_mem = nullptr;   // control words, bins
  unsigned long long* h_bins = nullptr;
  unsigned long long* h_ctl = nullptr;
  dd::Job* h_jobs = nullptr;
  cudaEvent_t ev0 = nullptr, ev1 = nullptr;
  // resident popc CTAs per SM by bin increment, job kind, bins and column table (0: not asked yet)
  int occupancy[2][4][dd::kMaxBins + 1][2] = {};
  // tuning
  int hist_mode = dd::HIST_RED;
  int tuned = 0;
  bool tune_due = false;  // a call asked for the autotuner: it runs before the first launch that reads its verdict
  uint32_t mma_epilogue = DD_MMA_EPILOGUE_AUTO;         // requested (dd_set_mma_epilogue)
  uint32_t mma_tuned_epilogue = DD_MMA_EPILOGUE_PAIRED;  // the autotuner's verdict for AUTO
  unsigned long long mma_timeout_ns = 2000000000ull;  // bound of every device-side wait
  // batch graph cache
  cudaGraphExec_t gexec = nullptr;
  std::vector<dd::Job> gjobs;  // job table the cached graph was built for
  int ggrid[2] = {0, 0};
  size_t gsmem[2] = {0, 0};
  int ghist_mode = 0;                  // popc bin-increment form the graph launches
  unsigned long long gtimeout_ns = 0;  // device-side wait bound baked into the graph
};

namespace dd {

constexpr int kCtlWords = 16;
static thread_local std::string t_last_error;
void set_error(const std::string& msg) { t_last_error = msg; }

static int cuda_fail(cudaError_t e, const char* what) {
  set_error(std::string(what) + ": " + cudaGetErrorString(e));
  return DD_ERR_CUDA;
}

#define DD_CUDA(call)                                   \
  do {                                                  \
    cudaError_t e_ = (call);                            \
    if (e_ != cudaSuccess) return cuda_fail(e_, #call); \
  } while (0)

// The cached launch graph's copy nodes and kernel arguments point at these
// buffers, so it is dropped whenever one of them is reallocated (no graph is in
// flight here: every launch is synchronised before its call returns).
static void drop_graph(dd_context* ctx) {
  if (ctx->gexec) cudaGraphExecDestroy(ctx->gexec);
  ctx->gexec = nullptr;
  ctx->gjobs.clear();
}

static int ensure_capacity(dd_context* ctx, uint32_t slots, uint32_t njobs) {
  DD_CUDA(cudaSetDevice(ctx->device));
  if (slots > ctx->bin_slots || njobs > ctx->job_cap) drop_graph(ctx);
  if (slots > ctx->bin_slots) {
    if (ctx->d_mem) cudaFree(ctx->d_mem);
    if (ctx->h_mem) cudaFreeHost(ctx->h_mem);
    ctx->d_mem = ctx->d_ctl = ctx->d_bins = nullptr;
    ctx->h_mem = ctx->h_ctl = ctx->h_bins = nullptr;
    ctx->bin_slots = 0;
    const uint32_t cap = std::max<uint32_t>(slots, 64);
    cudaError_t e = cudaMalloc(&ctx->d_mem, (kCtlWords + (size_t)cap * 3 * kMaxBins) * sizeof(unsigned long long));
    if (e != cudaSuccess) { set_error("bins: cudaMalloc failed"); return DD_ERR_OUT_OF_MEMORY; }
    DD_CUDA(cudaMallocHost(&ctx->h_mem, (kCtlWords + (size_t)cap * kMaxBins) * sizeof(unsigned long long)));
    ctx->d_ctl = ctx->d_mem;
    ctx->d_bins = ctx->d_mem + kCtlWords;
    ctx->h_ctl = ctx->h_mem;
    ctx->h_bins = ctx->h_mem + kCtlWords;
    ctx->bin_slots = cap;
  }
  if (njobs > ctx->job_cap) {
    if (ctx->d_jobs) cudaFree(ctx->d_jobs);
    if (ctx->h_jobs) cudaFreeHost(ctx->h_jobs);
    ctx->d_jobs = nullptr;
    ctx->h_jobs = nullptr;
    ctx->job_cap = 0;
    const uint32_t cap = std::max<uint32_t>(njobs, 64);
    cudaError_t e = cudaMalloc(&ctx->d_jobs, (size_t)cap * sizeof(Job));
    if (e != cudaSuccess) { set_error("jobs: cudaMalloc failed"); return DD_ERR_OUT_OF_MEMORY; }
    DD_CUDA(cudaMallocHost(&ctx->h_jobs, (size_t)cap * sizeof(Job)));
    ctx->job_cap = cap;
  }
  return DD_OK;
}

// Staging memory of the carry path, kept by the context and grown on demand; false
// when the device has no room for it (its jobs then take the pair kernels).
static bool ensure_stage(dd_context* ctx, size_t bytes) {
  if (bytes <= ctx->stage_cap) return true;
  void* mem = nullptr;
  if (cudaMalloc(&mem, bytes) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  drop_graph(ctx);
  if (ctx->d_stage) cudaFree(ctx->d_stage);
  ctx->d_stage = mem;
  ctx->stage_cap = bytes;
  return true;
}

enum Route : uint32_t { ROUTE_POPC = 0, ROUTE_MMA = 1, ROUTE_CARRY = 2, ROUTE_ROWS = 3 };

struct LaunchPlan {
  LaunchArgs pargs;          // popc kernel: table entries [0, npopc)
  int pgrid = 0, pkind = kMixedKinds;
  size_t psmem = 0;
  uint32_t npopc = 0;
  MmaArgs margs;             // MMA kernel: table entries [npopc, npopc + nmma)
  int mgrid = 0;
  size_t msmem = 0;
  uint32_t nmma = 0;
  std::vector<CarryPlan> carry;  // residue pairs, exhaustive: the table entries after those
  std::vector<RowsPlan> rows;    // residue pairs, 1-D grids: the last table entries
  uint32_t nslots = 0;       // bin slots (one per request, in request order)
};

// Epilogue of the context's tcgen05 launches.
static uint32_t mma_epilogue_of(const dd_context* ctx) {
  return ctx->mma_epilogue == DD_MMA_EPILOGUE_AUTO ? ctx->mma_tuned_epilogue : ctx->mma_epilogue;
}

// Under AUTO, jobs below these many distance evaluations stay on the popc kernel: the
// tcgen05 kernel's fixed cost per launch (TMEM allocation, clearing and folding its
// ~180 KB table) outweighs its rate there, and a triangle's diagonal strips weigh more
// on it.  Exhaustive, one instance: k = 15, 5.4e8 pairs, popc 0.144 ms, tcgen05 0.117 ms;
// k = 14 0.049 and 0.061 ms.  2-D grids, whose lattice columns the popc kernel computes
// one by one: 1.3e8 pairs (1000 x 134217) 0.164 and 0.080 ms.  In a launch of many
// instances the fixed cost is shared: 8 of k = 14 0.280 and 0.289 ms, 12 0.400 and 0.342,
// 16 0.53 and 0.41; 16 of k = 13 0.152 and 0.186 ms.
constexpr double kMmaMinTriangle = 536870912.0;  // 2^29
constexpr double kMmaMinRect = 134217728.0;      // 2^27
constexpr double kMmaMinShared = 67108864.0;     // 2^26, in a launch of
constexpr double kMmaMinTriangles = 1342177280.0;  // 1.25 x 2^30 or more in such jobs (triangles)
constexpr double kMmaMinRects = 1073741824.0;      // 2^30 (grids: 16 of k = 14, m = 4096 0.26 and 0.24 ms)
constexpr double kMmaAlways = 1073741824.0;      // 2^30

static double pairs_of(const Job& j) {
  return j.shape == SHAPE_TRIANGLE ? 0.5 * (double)j.rows * (double)j.rows : (double)j.rows * (double)j.cols;
}

// 1-D grids below kMmaAlways: their columns are codewords in sequence, which the popc
// kernel bins at its full rate where a tile has all of its 128 rows (a count of rows that
// is no multiple of 128 leaves one row tile on the checked loop, and the two loops
// together run slower), while the tcgen05 kernel writes an operand for every column tile
// whether 128 rows use it or 4096.  So the two costs, in microseconds of a launch, or of
// one more job of a launch that is shared (whose claims do not follow the columns): fixed,
// for each column tile, for each full tile, for each checked one.  The coefficients fit
// 450 measured shapes (k = 13 .. 24, m of 2^25.5 .. 2^30 / 2^k in whole and ragged tiles, A
// of 7, 11 and 16 bits); where the rule decides, its choice takes 1.005 times the faster
// kernel's time in the mean, and no longer than the popc kernel (A = 62307, popc and
// tcgen05: k = 20, m = 128 0.045 and 0.074 ms, m = 512 0.136 and 0.119; k = 17, m = 1024
// 0.044 and 0.047, m = 4096 0.136 and 0.088; k = 16, m = 2805 0.088 and 0.057; 16 jobs of
// k = 18, m = 256 0.26 and 0.36, of k = 14, m = 4096 0.26 and 0.24).
struct GridCost {
  double fixed, column, full, whole_warps, ragged;
};
constexpr GridCost kGridAlone{28.0, 0.035, 0.0145, 0.015, 0.030}, kGridShared{4.0, 0.045, 0.0135, 0.022, 0.042};

static bool progression_on_mma(const Job& j, bool shared) {
  const GridCost& c = shared ? kGridShared : kGridAlone;
  const double tiles = (double)j.col_tiles, full = (double)(j.rows / kWarpRows);
  const uint32_t rest = (uint32_t)(j.rows % kWarpRows);
  // the popc kernel starts anew where the columns' high word changes, every 2^32 / A of them
  // (k = 16, m = 2048: A of 28 bits 0.050 ms, 30 0.070, 32 0.144; tcgen05 0.047 to 0.052)
  const double starts = 1.0 + 5.0 * (double)j.A / 4294967296.0;
  double popc = shared ? 0.0 : 13.0, mma = c.fixed + tiles * (c.column + c.full * full);
  if (rest) {
    popc += tiles * (0.048 * starts * full + 0.066 + 0.013 * ((rest + 31) / 32));
    mma += tiles * (rest % 32 ? c.ragged : c.whole_warps);
  } else {
    popc += tiles * 0.0295 * starts * full;
  }
  return mma < popc;
}

// Whether a job that AUTO leaves to the pair kernels is one for the tcgen05 kernel where the
// autotuner prefers that.  launch_pairs: pairs of the launch's jobs that could share one
// (0: unknown).
static bool large_for_mma(const Job& j, double launch_pairs) {
  const bool triangle = j.shape == SHAPE_TRIANGLE, shared = launch_pairs >= (triangle ? kMmaMinTriangles : kMmaMinRects);
  const double pairs = pairs_of(j);
  if (pairs < (shared ? kMmaMinShared : triangle ? kMmaMinTriangle : kMmaMinRect)) return false;
  return pairs >= kMmaAlways || triangle || j.col_kind != COL_PROGRESSION || progression_on_mma(j, shared);
}

// Whether the pair kernel of a job depends on the autotuner's verdict.
static bool reads_verdict(const Job& j, uint32_t kernel, double launch_pairs = 0) {
  return kernel != DD_KERNEL_MMA && kernel != DD_KERNEL_POPC && mma_eligible(j) && large_for_mma(j, launch_pairs);
}

// Which pair kernel runs a job: explicit MMA or POPC requests are honoured where
// the job allows them; AUTO uses the context's measured preference for jobs
// large enough to amortise the tcgen05 kernel's launch.
static bool want_mma(const dd_context* ctx, const Job& j, uint32_t kernel, double launch_pairs = 0) {
  if (kernel == DD_KERNEL_MMA) return mma_eligible(j);
  return ctx->tuned == 2 && reads_verdict(j, kernel, launch_pairs);  // autotuner's verdict for AN exhaustive shapes
}

// The first large AUTO exhaustive request, and the first batch of 16, ask for the
// autotuner.  Residue routes do not read its verdict (a probe of 1.2 s before a call of 0.2 to
// 85 ms), so it runs before the first launch of the context that does.
static bool asks_for_tuning(const dd_request& q) {
  return q.kernel == DD_KERNEL_AUTO && q.code == DD_CODE_AN && q.mode == DD_MODE_EXHAUSTIVE && q.n >= 20;
}

// The jobs' routes: the carry path for each where it is asked for or wins and its
// staging memory is to be had, a pair kernel for the others.
static bool takes_carry(dd_context* ctx, const Job& j, uint32_t kernel, Route* route) {
  if (kernel != DD_KERNEL_CARRY && kernel != DD_KERNEL_AUTO) return false;
  const bool asked = kernel == DD_KERNEL_CARRY;
  if (carry_eligible(j) && (asked || carry_wins(j))) {
    std::vector<CarryPlan> p(1);
    carry_plan(j, p[0]);
    if (ensure_stage(ctx, carry_stage_bytes(p))) {
      *route = ROUTE_CARRY;
      return true;
    }
  }
  RowsPlan rp;
  if (rows_plan(j, ctx->num_sms, rp) && (asked || rows_win(j, rp))) {
    *route = ROUTE_ROWS;
    return true;
  }
  return false;
}
static int routes_of(dd_context* ctx, const std::vector<Job>& jobs, const dd_request* reqs, std::vector<Route>& routes) {
  routes.assign(jobs.size(), ROUTE_POPC);
  std::vector<bool> carry(jobs.size());
  double shared = 0;
  for (size_t i = 0; i < jobs.size(); ++i) {
    carry[i] = takes_carry(ctx, jobs[i], reqs[i].kernel, &routes[i]);
    if (!carry[i] && reqs[i].kernel != DD_KERNEL_POPC && mma_eligible(jobs[i]) && pairs_of(jobs[i]) >= kMmaMinShared)
      shared += pairs_of(jobs[i]);
  }
  for (size_t i = 0; i < jobs.size(); ++i) {
    if (carry[i]) continue;
    if (ctx->tune_due && !ctx->tuned && reads_verdict(jobs[i], reqs[i].kernel, shared)) {
      const int st = dd_autotune(ctx, nullptr);
      if (st != DD_OK) return st;
    }
    routes[i] = want_mma(ctx, jobs[i], reqs[i].kernel, shared) ? ROUTE_MMA : ROUTE_POPC;
  }
  return DD_OK;
}

// Orders the job table (popc jobs, MMA jobs, then the two kinds of carry jobs), assigns
// tile ranges and bin slots (slot = request index), and sizes both persistent grids.
static int plan_launch(dd_context* ctx, std::vector<Job>& jobs, const std::vector<Route>& routes,
                       LaunchPlan& lp, bool own_bins = true) {
  std::vector<Job> table;
  table.reserve(jobs.size());
  uint32_t of_route[4] = {0, 0, 0, 0};
  for (uint32_t route = 0; route < 4; ++route)
    for (size_t i = 0; i < jobs.size(); ++i) {
      if (routes[i] != route) continue;
      Job j = jobs[i];
      if (own_bins) j.bins = ctx->d_bins + i * kMaxBins;
      table.push_back(j);
      ++of_route[route];
    }
  lp.nslots = (uint32_t)jobs.size();
  uint64_t tp = 0, tm = 0;
  uint32_t maxb = 1, maxbm = 1;
  bool col_table = false;
  TileSpan span;
  lp.npopc = of_route[ROUTE_POPC];
  lp.nmma = of_route[ROUTE_MMA];
  lp.carry.resize(of_route[ROUTE_CARRY]);
  for (size_t c = 0; c < lp.carry.size(); ++c) carry_plan(table[lp.npopc + lp.nmma + c], lp.carry[c]);
  // room for several of them at once, where it is to be had (one fits: takes_carry)
  ensure_stage(ctx, carry_stage_bytes(lp.carry));
  const uint32_t pair_jobs = lp.npopc + lp.nmma;
  lp.rows.resize(of_route[ROUTE_ROWS]);
  for (size_t c = 0; c < lp.rows.size(); ++c) rows_plan(table[pair_jobs + lp.carry.size() + c], ctx->num_sms, lp.rows[c]);
  for (uint32_t k = 0; k < lp.npopc; ++k) {
    Job& j = table[k];
    j.tile_begin = tp;
    tp += j.tiles;
    maxb = std::max(maxb, j.nbins);
    span.add(j);
    lp.pkind = k == 0 || lp.pkind == (int)j.kind ? (int)j.kind : kMixedKinds;
    col_table |= (j.kind == JOB_PAIRS && j.col_kind == COL_HAMMING_EXT && !j.wide);
  }
  for (uint32_t k = lp.npopc; k < pair_jobs; ++k) {
    Job& j = table[k];
    j.tile_begin = tm;
    tm += j.tiles;
    maxbm = std::max(maxbm, j.nbins);
  }
  unsigned* status = reinterpret_cast<unsigned*>(ctx->d_ctl + 2);
  lp.pargs.jobs = ctx->d_jobs;
  lp.pargs.njobs = lp.npopc;
  lp.pargs.smem_bins = maxb;
  lp.pargs.total_tiles = tp;
  lp.pargs.counter = ctx->d_ctl;
  lp.pargs.status = status;
  lp.pargs.use_col_table = col_table ? 1u : 0u;
  lp.pargs.split_log = 0;
  if (lp.npopc && tp) {
    lp.psmem = hist_smem_bytes(maxb, col_table);
    int& occ = ctx->occupancy[ctx->hist_mode == HIST_RED][lp.pkind + 1][maxb][col_table];
    if (!occ) DD_CUDA(hist_occupancy(ctx->hist_mode, lp.pkind, lp.psmem, &occ));
    if (occ < 1) { set_error("kernel does not fit on an SM"); return DD_ERR_UNSUPPORTED; }
    lp.pargs.split_log = hist_split_log(tp, (uint64_t)ctx->num_sms * occ * kWarpsPerCta, span);
    const uint64_t want = ((tp << lp.pargs.split_log) + kWarpsPerCta - 1) / kWarpsPerCta;
    lp.pgrid = (int)std::min<uint64_t>((uint64_t)ctx->num_sms * occ, std::max<uint64_t>(want, 1));
  }
  lp.margs.jobs = ctx->d_jobs + lp.npopc;
  lp.margs.njobs = lp.nmma;
  // rows for every distance an operand can produce (<= L), flagged at flush when >= nbins
  uint32_t maxl = 0;
  for (uint32_t k = lp.npopc; k < pair_jobs; ++k) maxl = std::max(maxl, (uint32_t)mma_operand_bits(table[k]));
  lp.margs.hist_rows = std::max(maxbm, maxl + 1);
  lp.margs.total_tiles = tm;
  lp.margs.counter = ctx->d_ctl + 1;
  lp.margs.status = status;
  lp.margs.timeout_ns = ctx->mma_timeout_ns;
  lp.margs.packed = mma_epilogue_of(ctx) == DD_MMA_EPILOGUE_PAIRED ? 1u : 0u;
  lp.margs.pk_cells = 0;
  lp.margs.small_claim = 1;
  lp.margs.big_claims = 0;
  lp.margs.big_claim = 1;
  lp.margs.pad = 0;
  if (lp.nmma && tm) {
    if (lp.margs.packed) {
      // one joint table for the launch, sized for its largest S; each job's
      // window of d2 rows and its packing parameters follow from it
      uint32_t smax = 1;
      for (uint32_t k = lp.npopc; k < pair_jobs; ++k)
        smax = std::max(smax, (uint32_t)mma_max_distance(table[k]) + 1u);
      mma_pk_layout(smax, &lp.margs.pk_cells, &lp.margs.b_bufs);
      for (uint32_t k = lp.npopc; k < pair_jobs; ++k) mma_pack_setup(table[k], lp.margs.pk_cells);
    } else {
      lp.margs.b_bufs = mma_b_bufs(lp.margs.hist_rows);
    }
    lp.msmem = mma_smem_bytes(lp.margs.hist_rows, lp.margs.b_bufs, lp.margs.packed != 0, lp.margs.pk_cells);
    lp.mgrid = (int)std::min<uint64_t>((uint64_t)ctx->num_sms, tm);  // one CTA (one TMEM owner) per SM
    const Job& j = table[lp.npopc];
    const bool columns = lp.nmma == 1 && j.shape == SHAPE_RECT && j.cols % kTileCols == 0 && j.tiles == job_tiles(j);
    mma_claims(lp.margs, lp.mgrid, columns ? j.tiles / j.col_tiles : 0);
  }
  std::memcpy(ctx->h_jobs, table.data(), table.size() * sizeof(Job));
  return DD_OK;
}

// Enqueues: job table H2D, bins / counters / status reset, kernels (bracketed
// by events), bins + status D2H.
static int enqueue_launch(dd_context* ctx, const LaunchPlan& lp, bool capturing) {
  cudaStream_t s = ctx->stream;
  const uint32_t ncarry = (uint32_t)lp.carry.size(), nrows = (uint32_t)lp.rows.size();
  const uint32_t njobs = lp.npopc + lp.nmma + ncarry + nrows;
  DD_CUDA(cudaMemcpyAsync(ctx->d_jobs, ctx->h_jobs, njobs * sizeof(Job), cudaMemcpyHostToDevice, s));
  unsigned long long* acc = ctx->d_bins + (size_t)lp.nslots * kMaxBins;
  const size_t result_bytes = (kCtlWords + (size_t)lp.nslots * kMaxBins) * sizeof(unsigned long long);
  DD_CUDA(cudaMemsetAsync(ctx->d_mem, 0, result_bytes + (size_t)ncarry * 2 * kMaxBins * sizeof(unsigned long long), s));
  // Inside a stream capture the records must be external so that they become
  // event-record nodes of the graph (the kernel time is then measurable on
  // every replay); outside a capture the flag is not accepted.
  const unsigned evflags = capturing ? cudaEventRecordExternal : cudaEventRecordDefault;
  DD_CUDA(cudaEventRecordWithFlags(ctx->ev0, s, evflags));
  if (lp.pgrid) DD_CUDA(launch_hist(ctx->hist_mode, lp.pkind, lp.pargs, lp.pgrid, lp.psmem, s));
  if (lp.mgrid) DD_CUDA(launch_mma(lp.margs, lp.mgrid, lp.msmem, s));
  if (ncarry) DD_CUDA(launch_carry(lp.carry, ctx->num_sms, acc, ctx->d_stage, ctx->stage_cap, s));
  if (ncarry) DD_CUDA(launch_carry_finish(ctx->d_jobs + lp.npopc + lp.nmma, acc, ncarry, s));
  for (uint32_t c = 0; c < nrows; ++c) DD_CUDA(launch_rows(ctx->h_jobs[njobs - nrows + c], lp.rows[c], s));
  DD_CUDA(cudaEventRecordWithFlags(ctx->ev1, s, evflags));
  DD_CUDA(cudaMemcpyAsync(ctx->h_mem, ctx->d_mem, result_bytes, cudaMemcpyDeviceToHost, s));
  return DD_OK;
}

// Status word of the last launch (after the stream synchronised).
static int check_status(dd_context* ctx) {
  const unsigned st = (unsigned)ctx->h_ctl[2];
  if (st & 8u) {
    char buf[256];
    std::snprintf(buf, sizeof(buf), "self-check: shared access at %llu outside [%llu, %llu), tile %llu",
                  ctx->h_ctl[4], ctx->h_ctl[5], ctx->h_ctl[6], ctx->h_ctl[7]);
    set_error(buf);
    return DD_ERR_CUDA;
  }
  if (st & KSTATUS_TIMEOUT) { set_error("a device-side wait timed out"); return DD_ERR_TIMEOUT; }
  if (st & KSTATUS_BAD_DISTANCE) { set_error("kernel produced a distance outside the bins"); return DD_ERR_CUDA; }
  if (st & KSTATUS_BAD_JOB) { set_error("kernel saw a tile outside the job table"); return DD_ERR_CUDA; }
  return DD_OK;
}

// One launch over job sub-ranges whose bins live in caller-owned device
// memory (the server's resident slots): the bins are NOT reset, so successive
// rounds accumulate; only the control block is reset and read back.
int launch_round(dd_context* ctx, std::vector<Job>& jobs, const std::vector<uint32_t>& kernels, float* kernel_ms) {
  int st = ensure_capacity(ctx, 1, (uint32_t)jobs.size());
  if (st != DD_OK) return st;
  // tile sub-ranges are the pair kernels' work
  std::vector<Route> routes(jobs.size());
  for (size_t i = 0; i < jobs.size(); ++i) routes[i] = want_mma(ctx, jobs[i], kernels[i]) ? ROUTE_MMA : ROUTE_POPC;
  LaunchPlan lp;
  st = plan_launch(ctx, jobs, routes, lp, false);
  if (st != DD_OK) return st;
  cudaStream_t s = ctx->stream;
  const uint32_t njobs = lp.npopc + lp.nmma;
  DD_CUDA(cudaMemcpyAsync(ctx->d_jobs, ctx->h_jobs, njobs * sizeof(Job), cudaMemcpyHostToDevice, s));
  DD_CUDA(cudaMemsetAsync(ctx->d_ctl, 0, kCtlWords * sizeof(unsigned long long), s));
  DD_CUDA(cudaEventRecord(ctx->ev0, s));
  if (lp.pgrid) DD_CUDA(launch_hist(ctx->hist_mode, lp.pkind, lp.pargs, lp.pgrid, lp.psmem, s));
  if (lp.mgrid) DD_CUDA(launch_mma(lp.margs, lp.mgrid, lp.msmem, s));
  DD_CUDA(cudaEventRecord(ctx->ev1, s));
  DD_CUDA(cudaMemcpyAsync(ctx->h_ctl, ctx->d_ctl, kCtlWords * sizeof(unsigned long long), cudaMemcpyDeviceToHost, s));
  DD_CUDA(cudaStreamSynchronize(s));
  st = check_status(ctx);
  if (st != DD_OK) return st;
  if (kernel_ms) DD_CUDA(cudaEventElapsedTime(kernel_ms, ctx->ev0, ctx->ev1));
  return DD_OK;
}

bool uses_mma(const dd_context* ctx, const Job& j, uint32_t kernel) { return want_mma(ctx, j, kernel); }
uint32_t mma_epilogue_used(const dd_context* ctx) { return mma_epilogue_of(ctx); }
void* context_stream(const dd_context* ctx) { return (void*)ctx->stream; }
int context_device(const dd_context* ctx) { return ctx->device; }

static double now_ms() {
  using namespace std::chrono;
  return duration<double, std::milli>(steady_clock::now().time_since_epoch()).count();
}

static void fill_pairs(dd_result& r, u128 p) {
  r.pairs_lo = (uint64_t)p;
  r.pairs_hi = (uint64_t)(p >> 64);
}

}  // namespace dd

using namespace dd;

extern "C" {

const char* dd_version(void) { return "coding_reliability_b200 0.1 (sm_100a)"; }

const char* dd_status_string(int status) {
  switch (status) {
    case DD_OK: return "ok";
    case DD_ERR_INVALID_ARGUMENT: return "invalid argument";
    case DD_ERR_UNSUPPORTED: return "unsupported";
    case DD_ERR_CUDA: return "cuda error";
    case DD_ERR_NO_DEVICE: return "no device";
    case DD_ERR_OUT_OF_MEMORY: return "out of memory";
    case DD_ERR_BUSY: return "busy";
    case DD_ERR_TIMEOUT: return "timeout";
    case DD_ERR_NOT_FOUND: return "not found";
    case DD_ERR_CANCELLED: return "cancelled";
    default: return "unknown status";
  }
}

const char* dd_last_error(void) { return t_last_error.c_str(); }

int dd_device_count(void) {
  int n = 0;
  if (cudaGetDeviceCount(&n) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return n;
}

int dd_context_create(int device, void* stream, dd_context** out) {
  if (!out) { set_error("out is NULL"); return DD_ERR_INVALID_ARGUMENT; }
  *out = nullptr;
  int ndev = dd_device_count();
  if (ndev == 0) { set_error("no CUDA device"); return DD_ERR_NO_DEVICE; }
  if (device < 0 || device >= ndev) { set_error("device ordinal out of range"); return DD_ERR_INVALID_ARGUMENT; }
  dd_context* ctx = new dd_context();
  ctx->device = device;
  cudaError_t e = cudaSetDevice(device);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&ctx->num_sms, cudaDevAttrMultiProcessorCount, device);
  if (e == cudaSuccess) {
    // sm_100a code is arch-specific: it runs on compute capability 10.0 only
    int major = 0, minor = 0;
    cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, device);
    cudaDeviceGetAttribute(&minor, cudaDevAttrComputeCapabilityMinor, device);
    if (major != 10 || minor != 0) {
      delete ctx;
      set_error("this library is built for sm_100a (B200) only");
      return DD_ERR_NO_DEVICE;
    }
  }
  if (e == cudaSuccess) {
    if (stream) ctx->stream = (cudaStream_t)stream;
    else { e = cudaStreamCreateWithFlags(&ctx->stream, cudaStreamNonBlocking); ctx->own_stream = true; }
  }
  if (e == cudaSuccess) e = cudaEventCreate(&ctx->ev0);
  if (e == cudaSuccess) e = cudaEventCreate(&ctx->ev1);
  if (e != cudaSuccess) {
    set_error(std::string("context setup: ") + cudaGetErrorString(e));
    dd_context_destroy(ctx);
    return DD_ERR_CUDA;
  }
  int st = ensure_capacity(ctx, 64, 64);
  if (st != DD_OK) { dd_context_destroy(ctx); return st; }
  // Tuning override for measurements: CODREL_B200_HIST_MODE=red|ldst picks how
  // a lane bumps its shared-memory bin (default: red.shared.add).
  if (const char* m = std::getenv("CODREL_B200_HIST_MODE")) {
    if (std::strcmp(m, "ldst") == 0) ctx->hist_mode = HIST_LDST;
    else if (std::strcmp(m, "red") == 0) ctx->hist_mode = HIST_RED;
  }
  *out = ctx;
  return DD_OK;
}

int dd_context_destroy(dd_context* ctx) {
  if (!ctx) return DD_OK;
  cudaSetDevice(ctx->device);
  if (ctx->stream) cudaStreamSynchronize(ctx->stream);
  if (ctx->gexec) cudaGraphExecDestroy(ctx->gexec);
  if (ctx->d_mem) cudaFree(ctx->d_mem);
  if (ctx->d_jobs) cudaFree(ctx->d_jobs);
  if (ctx->d_stage) cudaFree(ctx->d_stage);
  if (ctx->h_mem) cudaFreeHost(ctx->h_mem);
  if (ctx->h_jobs) cudaFreeHost(ctx->h_jobs);
  if (ctx->ev0) cudaEventDestroy(ctx->ev0);
  if (ctx->ev1) cudaEventDestroy(ctx->ev1);
  if (ctx->own_stream && ctx->stream) cudaStreamDestroy(ctx->stream);
  delete ctx;
  return DD_OK;
}

int dd_request_shape(const dd_request* req, uint32_t* nbins, uint32_t* h, uint64_t* A_eff) {
  if (!req) { set_error("req is NULL"); return DD_ERR_INVALID_ARGUMENT; }
  Shape s;
  std::string err;
  int st = derive_shape(*req, s, err);
  if (st != DD_OK) { set_error(err); return st; }
  if (nbins) *nbins = s.nbins;
  if (h) *h = s.h;
  if (A_eff) *A_eff = s.A;
  return DD_OK;
}

int dd_request_plan(const dd_request* req, uint64_t* lattice, uint64_t* tiles, uint64_t* pairs_lo,
                    uint64_t* pairs_hi) {
  if (!req) { set_error("req is NULL"); return DD_ERR_INVALID_ARGUMENT; }
  Shape s;
  std::string err;
  int st = derive_shape(*req, s, err);
  if (st != DD_OK) { set_error(err); return st; }
  std::vector<Job> jobs;
  plan_jobs(s, *req, jobs);
  const u128 p = planned_pairs(s, *req);
  if (lattice) *lattice = s.lattice;
  if (tiles) *tiles = jobs[0].tiles;
  if (pairs_lo) *pairs_lo = (uint64_t)p;
  if (pairs_hi) *pairs_hi = (uint64_t)(p >> 64);
  return DD_OK;
}

int dd_postprocess(const dd_request* req, const uint64_t* raw, uint32_t nraw, dd_result* res) {
  if (!req || !raw || !res) { set_error("NULL argument"); return DD_ERR_INVALID_ARGUMENT; }
  Shape s;
  std::string err;
  int st = derive_shape(*req, s, err);
  if (st != DD_OK) { set_error(err); return st; }
  if (nraw < s.nbins) { set_error("raw histogram shorter than n+h+1"); return DD_ERR_INVALID_ARGUMENT; }
  std::memset(res, 0, sizeof(*res));
  postprocess(*req, s, raw, *res);
  res->user_tag = req->user_tag;
  res->status = DD_OK;
  return DD_OK;
}

void dd_philox4x32_10(const uint32_t ctr[4], const uint32_t key[2], uint32_t out[4]) {
  Philox4 o = philox4x32_10(ctr[0], ctr[1], ctr[2], ctr[3], key[0], key[1]);
  out[0] = o.x; out[1] = o.y; out[2] = o.z; out[3] = o.w;
}

}  // extern "C"

namespace dd {

// One launch for `count` requests: plan, (graph-)enqueue, synchronise, check
// the kernels' status word, post-process every request.
// `continued` (Monte Carlo continuation, one request): draw only the samples
// [continued->it_done, m) and add continued->raw_done to the device bins.
struct McContinuation {
  uint64_t it_done;
  const uint64_t* raw_done;
};

static int run_requests(dd_context* ctx, const dd_request* reqs, uint32_t count, dd_result* results,
                        bool use_graph, const McContinuation* continued = nullptr) {
  double t0 = now_ms();
  std::vector<Shape> shapes(count);
  std::vector<Job> jobs;
  jobs.reserve(count);
  for (uint32_t i = 0; i < count; ++i) {
    std::string err;
    int st = derive_shape(reqs[i], shapes[i], err);
    if (st != DD_OK) {
      set_error(count > 1 ? "request " + std::to_string(i) + ": " + err : err);
      return st;
    }
    plan_jobs(shapes[i], reqs[i], jobs);
  }
  if (continued) {
    Job& j = jobs[0];
    j.sample_begin = continued->it_done;
    j.tiles = job_tiles(j);
  }
  int st = ensure_capacity(ctx, count, count);
  if (st != DD_OK) return st;
  const double t_routes = now_ms();
  const bool tuned = ctx->tuned != 0;
  std::vector<Route> routes;
  st = routes_of(ctx, jobs, reqs, routes);
  if (st != DD_OK) return st;
  if (!tuned && ctx->tuned) t0 += now_ms() - t_routes;  // the autotuner's time is not the request's
  LaunchPlan lp;
  st = plan_launch(ctx, jobs, routes, lp);
  if (st != DD_OK) return st;
  cudaStream_t s = ctx->stream;
  if (use_graph) {
    const size_t nj = lp.npopc + lp.nmma + lp.carry.size() + lp.rows.size();
    const bool same = ctx->gexec && ctx->gjobs.size() == nj && ctx->ggrid[0] == lp.pgrid &&
                      ctx->ggrid[1] == lp.mgrid && ctx->gsmem[0] == lp.psmem && ctx->gsmem[1] == lp.msmem &&
                      ctx->ghist_mode == ctx->hist_mode && ctx->gtimeout_ns == lp.margs.timeout_ns &&
                      std::memcmp(ctx->gjobs.data(), ctx->h_jobs, nj * sizeof(Job)) == 0;
    if (!same) {
      drop_graph(ctx);
      cudaGraph_t g = nullptr;
      DD_CUDA(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
      st = enqueue_launch(ctx, lp, true);
      cudaError_t ce = cudaStreamEndCapture(s, &g);
      if (st != DD_OK) { if (g) cudaGraphDestroy(g); return st; }
      if (ce != cudaSuccess) return cuda_fail(ce, "cudaStreamEndCapture");
      ce = cudaGraphInstantiate(&ctx->gexec, g, 0);
      cudaGraphDestroy(g);
      if (ce != cudaSuccess) { ctx->gexec = nullptr; return cuda_fail(ce, "cudaGraphInstantiate"); }
      ctx->gjobs.assign(ctx->h_jobs, ctx->h_jobs + nj);
      ctx->ggrid[0] = lp.pgrid; ctx->ggrid[1] = lp.mgrid;
      ctx->gsmem[0] = lp.psmem; ctx->gsmem[1] = lp.msmem;
      ctx->ghist_mode = ctx->hist_mode;
      ctx->gtimeout_ns = lp.margs.timeout_ns;
    }
    DD_CUDA(cudaGraphLaunch(ctx->gexec, s));
  } else {
    st = enqueue_launch(ctx, lp, false);
    if (st != DD_OK) return st;
  }
  DD_CUDA(cudaStreamSynchronize(s));
  st = check_status(ctx);
  if (st != DD_OK) return st;
  float ms = 0;
  DD_CUDA(cudaEventElapsedTime(&ms, ctx->ev0, ctx->ev1));
  const double total = now_ms() - t0;
  std::vector<uint32_t> redo;
  for (uint32_t i = 0; i < count; ++i) {
    dd_result& r = results[i];
    std::memset(&r, 0, sizeof(r));
    uint64_t raw[kMaxBins];
    for (int b = 0; b < kMaxBins; ++b) raw[b] = ctx->h_bins[(size_t)i * kMaxBins + b];
    u128 pairs = planned_pairs(shapes[i], reqs[i]);
    if (continued) {
      for (uint32_t b = 0; b < shapes[i].nbins; ++b) raw[b] += continued->raw_done[b];
      pairs = (u128)(1ull << shapes[i].n) * (shapes[i].m - continued->it_done);
    }
    postprocess(reqs[i], shapes[i], raw, r);
    fill_pairs(r, pairs);
    r.kernel_used = routes[i] >= ROUTE_CARRY ? DD_KERNEL_CARRY : routes[i] == ROUTE_MMA ? DD_KERNEL_MMA : DD_KERNEL_POPC;
    r.mma_epilogue = r.kernel_used == DD_KERNEL_MMA ? mma_epilogue_of(ctx) : 0u;
    r.kernel_ms = ms;  // one launch: the whole batch's device time
    r.total_ms = total;
    r.user_tag = reqs[i].user_tag;
    r.status = DD_OK;
    if (routes[i] >= ROUTE_CARRY && !holds_all_pairs(raw, pairs)) redo.push_back(i);
  }
  return recount(reqs, results, redo,
                 [ctx](const dd_request& q, dd_result& r) { return run_requests(ctx, &q, 1, &r, false); });
}

}  // namespace dd

extern "C" {

int dd_autotune(dd_context* ctx, dd_tuning* out) {
  if (!ctx) { set_error("NULL argument"); return DD_ERR_INVALID_ARGUMENT; }
  dd_request q;
  std::memset(&q, 0, sizeof(q));
  q.code = DD_CODE_AN;
  q.mode = DD_MODE_EXHAUSTIVE;
  q.A = 65521;
  q.n = 20;  // large enough that every kernel reaches its steady state (0.1 s per run)
  const uint64_t pairs = (1ull << 20) * ((1ull << 20) - 1) / 2;
  auto best_ms = [&](uint32_t kernel, int mode, uint32_t epilogue, double* ms_out) -> int {
    const int saved_mode = ctx->hist_mode, saved_tuned = ctx->tuned;
    const uint32_t saved_epi = ctx->mma_epilogue;
    ctx->hist_mode = mode;
    ctx->tuned = 1;  // keep AUTO out of the way while probing
    ctx->mma_epilogue = epilogue;
    q.kernel = kernel;
    double best = 1e30;
    int st = DD_OK;
    for (int rep = 0; rep < 3 && st == DD_OK; ++rep) {
      dd_result r;
      st = run_requests(ctx, &q, 1, &r, false);
      if (st == DD_OK && rep > 0 && r.kernel_ms < best) best = r.kernel_ms;
    }
    ctx->hist_mode = saved_mode;
    ctx->tuned = saved_tuned;
    ctx->mma_epilogue = saved_epi;
    *ms_out = best;
    return st;
  };
  double red = 0, ldst = 0, mma = 0, paired = 0;
  int st = best_ms(DD_KERNEL_POPC, HIST_RED, DD_MMA_EPILOGUE_AUTO, &red);
  if (st == DD_OK) st = best_ms(DD_KERNEL_POPC, HIST_LDST, DD_MMA_EPILOGUE_AUTO, &ldst);
  if (st == DD_OK) st = best_ms(DD_KERNEL_MMA, ctx->hist_mode, DD_MMA_EPILOGUE_SINGLE, &mma);
  if (st == DD_OK) st = best_ms(DD_KERNEL_MMA, ctx->hist_mode, DD_MMA_EPILOGUE_PAIRED, &paired);
  if (st != DD_OK) return st;
  ctx->hist_mode = red <= ldst ? HIST_RED : HIST_LDST;
  ctx->mma_tuned_epilogue = paired <= mma ? DD_MMA_EPILOGUE_PAIRED : DD_MMA_EPILOGUE_SINGLE;
  ctx->tuned = std::min(mma, paired) < std::min(red, ldst) ? 2 : 1;
  if (out) {
    std::memset(out, 0, sizeof(*out));
    out->kernel = ctx->tuned == 2 ? DD_KERNEL_MMA : DD_KERNEL_POPC;
    out->hist_mode = (uint32_t)ctx->hist_mode;
    out->popc_red_pairs_per_s = pairs / (red * 1e-3);
    out->popc_ldst_pairs_per_s = pairs / (ldst * 1e-3);
    out->mma_pairs_per_s = pairs / (mma * 1e-3);
    out->mma_paired_pairs_per_s = pairs / (paired * 1e-3);
    out->mma_epilogue = ctx->mma_tuned_epilogue;
    out->probe_pairs = pairs;
  }
  return DD_OK;
}

int dd_histogram(dd_context* ctx, const dd_request* req, dd_result* res) {
  if (!ctx || !req || !res) { set_error("NULL argument"); return DD_ERR_INVALID_ARGUMENT; }
  if (asks_for_tuning(*req)) ctx->tune_due = true;
  return run_requests(ctx, req, 1, res, false);
}

int dd_batch_run(dd_context* ctx, const dd_request* reqs, uint32_t count, dd_result* results,
                 const dd_batch_options* opts) {
  if (!ctx || (!reqs && count) || (!results && count)) { set_error("NULL argument"); return DD_ERR_INVALID_ARGUMENT; }
  if (count == 0) return DD_OK;
  if (count >= 16 && (!opts || opts->kernel == DD_KERNEL_AUTO)) ctx->tune_due = true;
  if (opts && opts->kernel != DD_KERNEL_AUTO) {
    std::vector<dd_request> r(reqs, reqs + count);
    for (auto& q : r) q.kernel = opts->kernel;
    return run_requests(ctx, r.data(), count, results, opts->use_graph != 0);
  }
  return run_requests(ctx, reqs, count, results, opts && opts->use_graph);
}

int dd_mc_extend(dd_context* ctx, const dd_request* req, uint64_t it_done, const uint64_t* raw_done, dd_result* res) {
  if (!ctx || !req || !res || (it_done && !raw_done)) { set_error("NULL argument"); return DD_ERR_INVALID_ARGUMENT; }
  if (req->code != DD_CODE_AN || req->mode != DD_MODE_MONTE_CARLO) {
    set_error("dd_mc_extend: AN Monte Carlo requests only");
    return DD_ERR_UNSUPPORTED;
  }
  Shape s;
  std::string err;
  int st = derive_shape(*req, s, err);
  if (st != DD_OK) { set_error(err); return st; }
  if (it_done > s.m) {
    set_error("dd_mc_extend: more samples done than requested (after capping at 2^n)");
    return DD_ERR_INVALID_ARGUMENT;
  }
  if (it_done == s.m) {  // nothing left to draw: post-process what the caller has
    uint64_t raw[kMaxBins] = {0};
    for (uint32_t b = 0; b < s.nbins; ++b) raw[b] = raw_done[b];
    std::memset(res, 0, sizeof(*res));
    postprocess(*req, s, raw, *res);
    res->user_tag = req->user_tag;
    return DD_OK;
  }
  const McContinuation c{it_done, raw_done};
  return run_requests(ctx, req, 1, res, false, &c);
}

int dd_histogram_part(dd_context* ctx, const dd_request* req, uint64_t tile_begin, uint64_t tile_count,
                      uint64_t* raw, uint32_t nraw, double* kernel_ms) {
  if (!ctx || !req || !raw) { set_error("NULL argument"); return DD_ERR_INVALID_ARGUMENT; }
  if (kernel_ms) *kernel_ms = 0.0;
  Shape s;
  std::string err;
  int st = derive_shape(*req, s, err);
  if (st != DD_OK) { set_error(err); return st; }
  if (nraw < s.nbins) { set_error("raw histogram shorter than n+h+1"); return DD_ERR_INVALID_ARGUMENT; }
  std::vector<Job> jobs;
  plan_jobs(s, *req, jobs);
  Job& j = jobs[0];
  if (tile_begin > j.tiles || tile_count > j.tiles - tile_begin) {
    set_error("tile range outside the request's tile space (dd_request_plan gives its size)");
    return DD_ERR_INVALID_ARGUMENT;
  }
  if (tile_count == 0) return DD_OK;
  // the kernel choice follows dd_histogram's (the autotuner's verdict for AUTO)
  if (asks_for_tuning(*req)) ctx->tune_due = true;
  if (ctx->tune_due && !ctx->tuned && reads_verdict(j, req->kernel)) {
    st = dd_autotune(ctx, nullptr);
    if (st != DD_OK) return st;
  }
  st = ensure_capacity(ctx, 1, 1);
  if (st != DD_OK) return st;
  // the sub-range runs exactly as a query server round runs a query's share
  j.tile_offset = tile_begin;
  j.tiles = tile_count;
  j.bins = ctx->d_bins;
  DD_CUDA(cudaMemsetAsync(ctx->d_bins, 0, kMaxBins * sizeof(unsigned long long), ctx->stream));
  const std::vector<uint32_t> kernels{req->kernel};
  float ms = 0.0f;
  st = launch_round(ctx, jobs, kernels, &ms);
  if (st != DD_OK) return st;
  DD_CUDA(cudaMemcpyAsync(ctx->h_bins, ctx->d_bins, kMaxBins * sizeof(unsigned long long), cudaMemcpyDeviceToHost,
                          ctx->stream));
  DD_CUDA(cudaStreamSynchronize(ctx->stream));
  for (uint32_t b = 0; b < s.nbins; ++b) raw[b] += ctx->h_bins[b];
  if (kernel_ms) *kernel_ms = ms;
  return DD_OK;
}

int dd_histogram_plain(dd_context* ctx, const dd_request* req, dd_result* res) {
  if (!ctx || !req || !res) { set_error("NULL argument"); return DD_ERR_INVALID_ARGUMENT; }
  if (req->code != DD_CODE_AN || req->mode != DD_MODE_EXHAUSTIVE) {
    set_error("the plain baseline covers AN exhaustive requests only");
    return DD_ERR_UNSUPPORTED;
  }
  const double t0 = now_ms();
  Shape s;
  std::string err;
  int st = derive_shape(*req, s, err);
  if (st != DD_OK) { set_error(err); return st; }
  DD_CUDA(cudaSetDevice(ctx->device));
  // per call, as the reference's driver: allocate and clear the bins, launch
  // 128 CTAs per SM, copy the bins back, free them
  unsigned long long* bins = nullptr;
  DD_CUDA(cudaMalloc(&bins, s.nbins * sizeof(unsigned long long)));
  cudaError_t e = cudaMemsetAsync(bins, 0, s.nbins * sizeof(unsigned long long), ctx->stream);
  if (e == cudaSuccess) e = cudaEventRecord(ctx->ev0, ctx->stream);
  if (e == cudaSuccess) e = launch_plain(s.A, 1ull << s.n, s.nbins, bins, 128 * ctx->num_sms, ctx->stream);
  if (e == cudaSuccess) e = cudaEventRecord(ctx->ev1, ctx->stream);
  uint64_t raw[kMaxBins] = {0};
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(raw, bins, s.nbins * sizeof(unsigned long long), cudaMemcpyDeviceToHost, ctx->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
  float ms = 0;
  if (e == cudaSuccess) e = cudaEventElapsedTime(&ms, ctx->ev0, ctx->ev1);
  cudaFree(bins);
  if (e != cudaSuccess) return cuda_fail(e, "plain baseline");
  std::memset(res, 0, sizeof(*res));
  postprocess(*req, s, raw, *res);
  fill_pairs(*res, planned_pairs(s, *req));
  res->kernel_used = DD_KERNEL_POPC;
  res->kernel_ms = ms;
  res->user_tag = req->user_tag;
  res->total_ms = now_ms() - t0;
  return DD_OK;
}

int dd_measure_popc_peak(dd_context* ctx, double* popc_per_s) {
  if (!ctx || !popc_per_s) { set_error("NULL argument"); return DD_ERR_INVALID_ARGUMENT; }
  DD_CUDA(cudaSetDevice(ctx->device));
  uint32_t* sink = nullptr;
  const int grid = ctx->num_sms * 8;
  DD_CUDA(cudaMalloc(&sink, grid * sizeof(uint32_t)));
  const uint32_t iters = 4096;
  cudaError_t e = launch_popc_rate(iters / 8, grid, sink, ctx->stream);  // warm-up
  float best = 1e30f;
  for (int rep = 0; rep < 3 && e == cudaSuccess; ++rep) {
    e = cudaEventRecord(ctx->ev0, ctx->stream);
    if (e == cudaSuccess) e = launch_popc_rate(iters, grid, sink, ctx->stream);
    if (e == cudaSuccess) e = cudaEventRecord(ctx->ev1, ctx->stream);
    if (e == cudaSuccess) e = cudaEventSynchronize(ctx->ev1);
    float ms = 0;
    if (e == cudaSuccess) e = cudaEventElapsedTime(&ms, ctx->ev0, ctx->ev1);
    if (e == cudaSuccess && ms < best) best = ms;
  }
  cudaFree(sink);
  if (e != cudaSuccess) return cuda_fail(e, "popc probe");
  const double popcs = (double)grid * 256.0 * iters * 16.0 * 8.0;
  *popc_per_s = popcs / (best * 1e-3);
  return DD_OK;
}

int dd_set_mma_epilogue(dd_context* ctx, uint32_t epilogue) {
  if (!ctx) { set_error("NULL argument"); return DD_ERR_INVALID_ARGUMENT; }
  if (epilogue > DD_MMA_EPILOGUE_SINGLE) { set_error("unknown tcgen05 epilogue"); return DD_ERR_INVALID_ARGUMENT; }
  ctx->mma_epilogue = epilogue;
  return DD_OK;
}

int dd_set_wait_timeout(dd_context* ctx, uint64_t ns) {
  if (!ctx) { set_error("NULL argument"); return DD_ERR_INVALID_ARGUMENT; }
  ctx->mma_timeout_ns = ns ? ns : 2000000000ull;
  return DD_OK;
}

int dd_measure_red_sweep(dd_context* ctx, dd_red_probe* out, uint32_t cap, uint32_t* count) {
  if (!ctx || !out || !count) { set_error("NULL argument"); return DD_ERR_INVALID_ARGUMENT; }
  *count = 0;
  DD_CUDA(cudaSetDevice(ctx->device));
  uint32_t* sink = nullptr;
  const int grid = ctx->num_sms;
  DD_CUDA(cudaMalloc(&sink, grid * sizeof(uint32_t)));
  const uint32_t iters = 20000;
  cudaError_t e = cudaSuccess;
  for (int pattern = 0; pattern < 2 && e == cudaSuccess; ++pattern)
    for (int warps = 8; warps <= 32 && e == cudaSuccess; warps += 4) {
      const int threads = warps * 32;
      e = launch_red_rate(iters / 10, grid, threads, pattern, sink, ctx->stream);  // warm-up
      float best = 1e30f;
      for (int rep = 0; rep < 3 && e == cudaSuccess; ++rep) {
        e = cudaEventRecord(ctx->ev0, ctx->stream);
        if (e == cudaSuccess) e = launch_red_rate(iters, grid, threads, pattern, sink, ctx->stream);
        if (e == cudaSuccess) e = cudaEventRecord(ctx->ev1, ctx->stream);
        if (e == cudaSuccess) e = cudaEventSynchronize(ctx->ev1);
        float ms = 0;
        if (e == cudaSuccess) e = cudaEventElapsedTime(&ms, ctx->ev0, ctx->ev1);
        if (e == cudaSuccess && ms < best) best = ms;
      }
      if (e == cudaSuccess && *count < cap) {
        dd_red_probe& r = out[(*count)++];
        r.warps_per_sm = (uint32_t)warps;
        r.pattern = (uint32_t)pattern;
        r.adds_per_s = (double)red_rate_adds(iters, grid, threads) / (best * 1e-3);
      }
    }
  cudaFree(sink);
  if (e != cudaSuccess) return cuda_fail(e, "shared-atomic probe");
  return DD_OK;
}

int dd_measure_red_peak(dd_context* ctx, double* adds_per_s) {
  if (!ctx || !adds_per_s) { set_error("NULL argument"); return DD_ERR_INVALID_ARGUMENT; }
  dd_red_probe rows[64];
  uint32_t n = 0;
  const int st = dd_measure_red_sweep(ctx, rows, 64, &n);
  if (st != DD_OK) return st;
  double best = 0;
  for (uint32_t i = 0; i < n; ++i) best = std::max(best, rows[i].adds_per_s);
  *adds_per_s = best;
  return DD_OK;
}

}  // extern "C"

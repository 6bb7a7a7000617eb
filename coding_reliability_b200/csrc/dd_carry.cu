// dd_carry.cu — exact AN exhaustive histograms without visiting the pairs one by one.
//
// A codeword A*x with A odd and x in [0, 2^k) is fixed by its low k bits t (A is
// invertible mod 2^k, so t takes every value once): its high word is the c with
// t + 2^k c = 0 mod A, c in [0, A), that is
//     c(t) = psi(t mod A),   psi(v) = g v mod A,   g = -2^-k mod A.
// So the distance of two codewords is popc(t ^ t') + popc(psi(v) ^ psi(v')) with
// v = t mod A: 4^k pairs see only A^2 different high-word distances.  Written as
// a polynomial in z (coefficient of z^d = pairs at distance d) the histogram is
//     T = sum over t, t' of z^popc(t ^ t') Q(v, v'),  Q(v, v') = z^popc(psi(v) ^ psi(v')).
// Split t = 2^b q + r.  The sum over the low parts r, r' in [0, 2^b) is a window
//     G(v, v') = sum over r, r' of z^popc(r ^ r') Q(v + r, v' + r'),
// which b two-by-two steps build for all residue pairs at once, one per bit j:
//     H'(v, v') = H(v, v') + H(v+s, v'+s) + z (H(v, v'+s) + H(v+s, v')),  s = 2^j
// (the steps commute; they run from the largest s to s = 1).  Then
//     T = sum over q, q' in [0, 2^(k-b)) of z^popc(q ^ q') G(2^b q mod A, 2^b q' mod A),
// where residue v is hit by q = qinv v mod A, plus multiples of A below 2^(k-b).
// With b = k - bits(A) that is about b A^2 / 2 small steps instead of 4^k / 2 pairs
// (A = 58659, k = 22: 1.0e10 against 8.8e12), all in integers.
//
// Measured on B200 against the tcgen05 kernel: A = 62307, k = 22: 70 ms against 965 ms,
// k = 20: 20.6 against 63.5 ms; A = 867, k = 21: 0.32 against 231 ms, k = 16: 0.066
// against 0.37 ms.  Bound by instruction issue and its latencies at 12 warps an SM, the
// ALU and shared-memory pipes each a bit over half busy; DRAM carries nothing up to 4
// window bits and the staged histograms (24 bytes a residue pair, once each way) above.
//
// A histogram lives in registers, packed: four 8-bit counts per word while the
// counts stay within 4^4, two 16-bit counts per word up to 4^8.  The count 4^4 (4^8)
// itself does not fit its field: it needs all pairs of a window at one distance; the field would
// wrap, and the histogram's total with it, which the caller compares with the
// number of pairs (and computes the job on the direct kernels if they differ).
//
// Columns v' lie across threads, rows v are time, descending.  A step needs the
// neighbour column v'+s of the same row and both of row v+s, which are kept as
// Y = H(v, v'+s) + z H(v, v') in a ring of s rows.  Windows of up to 4 bits run in one
// kernel from the popcounts to the bins (carry_quad_kernel).  Longer ones run their
// largest steps first, in a kernel whose rows and columns are 16 residues apart, and
// stage the 8-bit histograms in memory; there a thread holds one column in words of
// every second (every fourth) bin, so that multiplying by z renames words and shifts
// only one word in two (in four).
#include <algorithm>

#include "dd_carry.cuh"

namespace dd {
namespace {

constexpr int kStageThreads = 512;  // staging kernel: 4 column residues mod 16 x 128 columns 16 apart
constexpr int kStageCols = kStageThreads / 4;
constexpr int kUnit = 16;           // residues between the staging kernel's rows and columns
constexpr int kFoldThreads = 192;   // folding kernel reading staged histograms
constexpr size_t kStageCells = 32u << 20;  // staged histograms of one round of blocks (768 MB)
constexpr int kLead = 8;            // rows above a step's own that its first level reads
constexpr int kAhead = 3;           // rows loaded ahead
constexpr int kSlots = kLead + 1 + kAhead;

// One block of residue pairs of one job: [row0, row0+rows) x [col0, col0+cols).
struct CarryEntry {
  uint32_t A, psi, qinv, nq, slices, wide;
  uint32_t row0, rows, col0, cols;
  uint32_t srows, scols;            // staged rows and columns (from row0, col0)
  uint32_t seg, segs, strips;       // folding: rows per CTA, CTAs down and across
  uint32_t stage_seg, stage_segs, stage_strips;
  uint32_t fold_end, stage_end;     // CTAs of the launch up to and including this entry
  uint4* st16;                      // staged histograms: words e0 e1 e2 o0 ...
  uint2* st8;                       // ... and o1 o2
  unsigned long long* acc;          // [0, kMaxBins): residue pairs v < v'; then v = v'
};

// Entries of one launch, in its parameters (short instances share a launch, and so
// fill the GPU together; 32 entries stay below the 4 KB every launch can pass).  64
// instances of 8-bit A, k = 14: 0.33 ms, 2.0 ms launched one by one; 256 at k = 16:
// 2.5 ms, popc kernel 123, tcgen05 81.
constexpr uint32_t kEntries = 32;
struct CarryBatch {
  uint32_t n;
  CarryEntry e[kEntries];
};
static_assert(sizeof(CarryBatch) <= 4096, "kernel parameters");

// One step in a running column: exchange with column c + s, combine, rotate the ring entry y.
template <int kLevel>
__device__ __forceinline__ Hist<kLevel> level(const Hist<kLevel - 1>& own, uint8_t* row, int c, int s,
                                              Hist<kLevel>& y) {
  put(row, c, own);
  __syncthreads();
  Hist<kLevel - 1> nb;
  get(row, c + s, nb);
  const Hist<kLevel> a = as_level<kLevel>(own), n = as_level<kLevel>(nb);
  const Hist<kLevel> r = add(add_z(a, n), y);
  y = add_z(n, a);
  return r;
}

// Shared bytes of the exchange rows: one per level after the first; with a single
// one, two that take turns (a row's only barrier then separates them).
template <int kBefore, int kLevels>
__host__ __device__ constexpr int exchange_bytes(int cols) {
  int n = 0;
  for (int i = 1; i < kLevels; ++i) n += (kBefore + i <= 4 ? 24 : 48) * cols;
  return kLevels == 2 ? 2 * n : n;
}

// ---------------------------------------------------------------- staging kernel
// The kLevels largest steps (s = 16 * 2^(kLevels-1) .. 16) for a block of residue
// pairs.  CTA: rows v = row0 + rho + 16 w for one rho and a run of w; columns v' =
// col0 + sigma + 16 w' for four neighbouring sigma (so that the stores of a warp
// fill sectors) and kStageCols consecutive w', of which the last 2^kLevels - 1
// only feed their neighbours.
template <int kLevels>
__global__ void __launch_bounds__(kStageThreads) carry_stage_kernel(const __grid_constant__ CarryBatch batch) {
  constexpr int kFirst = 1 << (kLevels - 1);
  constexpr int kWarm = kFirst - 1;
  constexpr int kUseful = kStageCols - ((1 << kLevels) - 1);
  constexpr int kUnroll = kLevels >= 3 ? kFirst / 2 : 1;
  constexpr int kCols = kStageThreads + 4 * kFirst;
  __shared__ __align__(16) uint8_t ex[exchange_bytes<0, kLevels>(kCols) + 16];

  uint32_t idx = 0;
  while (blockIdx.x >= batch.e[idx].stage_end) ++idx;
  const CarryEntry& a = batch.e[idx];
  const uint32_t cta = blockIdx.x - (idx ? batch.e[idx - 1].stage_end : 0);
  const uint32_t cx = cta % a.stage_strips, cy = cta / a.stage_strips;

  const int tid = threadIdx.x, sub = tid & 3, wi = tid >> 2;
  const uint32_t rho = cy % kUnit, seg = cy / kUnit;
  const uint32_t sigma = (cx & 3) * 4 + sub, w0 = (cx >> 2) * kUseful;
  const uint32_t wrows = (a.srows - rho + kUnit - 1) / kUnit;  // rows of this rho in the block
  const uint32_t wr0 = seg * a.stage_seg;
  if (wr0 >= wrows) return;
  const uint32_t wr1 = min(wrows, wr0 + a.stage_seg);
  // residue pairs v' < v are their mirror images; a final row reads staged rows up to 15 above it
  {
    const uint32_t vtop = a.col0 + (cx & 3) * 4 + 3 + kUnit * (w0 + kUseful - 1);
    if (vtop + 15 < a.row0 + rho + kUnit * wr0) return;
  }
  const uint32_t col = sigma + kUnit * (w0 + wi), vc = a.col0 + col;
  const bool store = wi < kUseful && col < a.scols;
  const uint32_t ca = mul_mod(a.psi, vc, a.A), cb = mul_mod(a.psi, vc + kUnit * kFirst, a.A);
  const int total = ((int)(wr1 - wr0) + kWarm + kUnroll - 1) / kUnroll * kUnroll;
  uint32_t w = wr0 + total - 1;  // descending
  const uint32_t step = mul_mod(a.psi, kUnit, a.A);
  uint32_t ra = mul_mod(a.psi, a.row0 + rho + kUnit * w, a.A);
  uint32_t rb = mul_mod(a.psi, a.row0 + rho + kUnit * (w + kFirst), a.A);

  H8 y4[4], y2[2], y1;
#pragma unroll
  for (int i = 0; i < 4; ++i) zero(y4[i]);
  zero(y2[0]); zero(y2[1]); zero(y1);
  for (int it = 0; it < total; it += kUnroll) {
#pragma unroll
    for (int u = 0; u < kUnroll; ++u, --w) {
      H8 h = first_level(ra, rb, ca, cb);
      ra = sub_mod(ra, step, a.A);
      rb = sub_mod(rb, step, a.A);
      uint8_t* row = ex;
      if constexpr (kLevels >= 4) { h = level<2>(h, row, tid, 4 * 4, y4[u & 3]); row += 24 * kCols; }
      if constexpr (kLevels >= 3) { h = level<2>(h, row, tid, 4 * 2, y2[u & 1]); row += 24 * kCols; }
      if constexpr (kLevels == 2) row += ((it + u) & 1) * 24 * kCols;
      if constexpr (kLevels >= 2) h = level<2>(h, row, tid, 4, y1);
      if (store && w < wr1) {
        const size_t at = (size_t)(rho + kUnit * w) * a.scols + col;
        a.st16[at] = make_uint4(h.e[0], h.e[1], h.e[2], h.o[0]);
        a.st8[at] = make_uint2(h.o[1], h.o[2]);
      }
    }
  }
}

// ---------------------------------------------------------------- folding kernel
__device__ __forceinline__ void copy_async16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}
__device__ __forceinline__ void copy_async8(void* dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int kPending>
__device__ __forceinline__ void copy_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(kPending) : "memory"); }

// Shared memory of the folding kernel: tables (U and D, twice for wide products),
// exchange rows, the ring of staged rows, and the q-distance counts of each thread (many).
template <int kBefore, int kLevels>
constexpr size_t fold_smem(bool many) {
  constexpr int cols = kFoldThreads + (1 << (kLevels - 1));
  return (size_t)kTabBytes * (many ? 4 : 2) + exchange_bytes<kBefore, kLevels>(cols) + (size_t)kSlots * cols * 24 +
         (many ? (size_t)(16 + 1) * kFoldThreads * 4 : 0);
}

// The last four steps (s = 8 .. 1) and the sum over q, q'.  kBefore: levels already in
// the staged input.  CTA: a
// strip of columns (one per thread, the last 2^kLevels - 1 only feed their
// neighbours) x a segment of rows.
template <int kBefore, int kLevels, bool kMany>
__global__ void __launch_bounds__(kFoldThreads, 2) carry_fold_kernel(const __grid_constant__ CarryBatch batch) {
  constexpr int kThreads = kFoldThreads;
  constexpr int kFirst = 1 << (kLevels - 1);
  constexpr int kWarm = kFirst - 1;
  constexpr int kUseful = kThreads - ((1 << kLevels) - 1);
  static_assert(kLevels == 4 && kFirst == kLead, "the staged input leaves four levels");
  constexpr int kUnroll = kFirst / 2;
  constexpr int kCols = kThreads + kFirst;
  constexpr int kL1 = kBefore + 1;
  constexpr int kLast = kBefore + kLevels;
  extern __shared__ __align__(16) uint8_t smem[];

  uint32_t idx = 0;
  while (blockIdx.x >= batch.e[idx].fold_end) ++idx;
  const CarryEntry& a = batch.e[idx];
  uint32_t cta = blockIdx.x - (idx ? batch.e[idx - 1].fold_end : 0);
  const uint32_t c0 = cta % a.strips * kUseful;
  cta /= a.strips;
  const uint32_t r0 = cta % a.segs * a.seg, slice = cta / a.segs;

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t r1 = min(a.rows, r0 + a.seg);
  if (a.col0 + min(a.cols, c0 + kUseful) <= a.row0 + r0) return;  // no v' >= v here

  // shared memory
  uint32_t* tab = reinterpret_cast<uint32_t*>(smem);  // U, D (and their high parts)
  uint8_t* ex = smem + kTabBytes * (kMany ? 4 : 2);
  uint4* in16 = reinterpret_cast<uint4*>(ex + exchange_bytes<kBefore, kLevels>(kCols));
  uint2* in8 = reinterpret_cast<uint2*>(in16 + kSlots * kCols);
  uint32_t* qd = reinterpret_cast<uint32_t*>(in8 + kSlots * kCols);
  for (int i = tid; i < kTabBytes * (kMany ? 4 : 2) / 4; i += kThreads) tab[i] = 0;
  if constexpr (kMany)
    for (int i = tid; i < 17 * kThreads; i += kThreads) qd[i] = 0;

  const uint32_t col = c0 + tid, vc = a.col0 + col;
  const bool mine = tid < kUseful && col < a.cols;
  const uint32_t qc = mul_mod(a.qinv, vc, a.A);
  const int total = ((int)(r1 - r0) + kWarm + kUnroll - 1) / kUnroll * kUnroll;
  uint32_t r = r0 + total - 1;  // descending, from row0
  uint32_t qr = mul_mod(a.qinv, a.row0 + r, a.A);
  const uint32_t tab_u = (uint32_t)__cvta_generic_to_shared(tab) + lane * 4u;

  // input: staged rows through a ring of kSlots rows
  int slot = 0;  // ring slot of load number it (row r + kLead of that step)
  const uint32_t scol = min(col, a.scols - 1);
  auto load = [&](int sl, uint32_t row) {
    const size_t at = (size_t)min(row, a.srows - 1) * a.scols;
    copy_async16(in16 + sl * kCols + tid, a.st16 + at + scol);
    copy_async8(in8 + sl * kCols + tid, a.st8 + at + scol);
    copy_commit();
  };
  for (int l = 0; l < kLead + kAhead; ++l) load(l, r + kLead - l);
  copy_wait<kAhead - 1>();
  __syncthreads();

  Hist<kLast - 2> y4[4];
  Hist<kLast - 1> y2[2];
  Hist<kLast> y1;
#pragma unroll
  for (int i = 0; i < 4; ++i) zero(y4[i]);
  zero(y2[0]); zero(y2[1]); zero(y1);

  for (int it = 0; it < total; it += kUnroll) {
#pragma unroll
    for (int u = 0; u < kUnroll; ++u, --r) {
      // first level
      auto fetch = [&](int sl, int c) {
        const uint4 x = in16[sl * kCols + c];
        const uint2 w = in8[sl * kCols + c];
        return as_level<kL1>(H8{{x.x, x.y, x.z}, {x.w, w.x, w.y}});
      };
      const int lo = slot, hi = slot + kLead < kSlots ? slot + kLead : slot + kLead - kSlots;
      const Hist<kL1> h1 =
          add_z(add(fetch(hi, tid), fetch(lo, tid + kFirst)), add(fetch(hi, tid + kFirst), fetch(lo, tid)));
      int nx = slot + kLead + kAhead;
      if (nx >= kSlots) nx -= kSlots;
      // row r + kLead - (kLead + kAhead); rows below the block's first are never used
      load(nx, r >= kAhead ? r - kAhead : 0u);
      slot = slot + 1 == kSlots ? 0 : slot + 1;
      copy_wait<kAhead - 1>();
      // remaining levels
      uint8_t* row = ex;
      const Hist<kLast - 2> h2 = level<kLast - 2>(h1, row, tid, 4, y4[u & 3]);
      row += slot_bytes<Hist<kL1>>() * kCols;
      const Hist<kLast - 1> h3 = level<kLast - 1>(h2, row, tid, 2, y2[u & 1]);
      row += slot_bytes<Hist<kLast - 2>>() * kCols;
      const Hist<kLast> g = level<kLast>(h3, row, tid, 1, y1);
      // fold: every q of row residue v with every q' of column residue v'
      const uint32_t v = a.row0 + r;
      if (mine && r < r1 && vc >= v) {
        const uint32_t at = tab_u + (vc == v ? kTabBytes : 0);
        if constexpr (!kMany) {
          const bool c2 = qc + a.A < a.nq;
          add_hist<kOne>(at + (__popc(qr ^ qc) << 7), 1, g);
          if (c2) add_hist<kOne>(at + (__popc(qr ^ (qc + a.A)) << 7), 1, g);
          if (qr + a.A < a.nq) {
            add_hist<kOne>(at + (__popc((qr + a.A) ^ qc) << 7), 1, g);
            if (c2) add_hist<kOne>(at + (__popc((qr + a.A) ^ (qc + a.A)) << 7), 1, g);
          }
        } else {
          volatile uint32_t* f = qd + tid;
          const uint32_t fa = (uint32_t)__cvta_generic_to_shared(qd + tid);
          for (uint32_t q = qr + slice * a.A; q < a.nq; q += a.slices * a.A)
            for (uint32_t p = qc; p < a.nq; p += a.A) red_add<0>(fa + __popc(q ^ p) * (kThreads * 4), 1);
          for (uint32_t d = 0; d <= 16; ++d) {
            const uint32_t x = f[d * kThreads];
            if (x) {
              f[d * kThreads] = 0;
              if (a.wide) add_hist<kWideProduct>(at + (d << 7), x, g);
              else add_hist<kNarrow>(at + (d << 7), x, g);
            }
          }
        }
      }
      qr = sub_mod(qr, a.qinv, a.A);
    }
  }
  copy_wait<0>();
  __syncthreads();
  // tables -> global sums
  for (int d = warp; d < 2 * kTabRows; d += kThreads / 32) {
    const uint32_t x = tab[d * 32 + lane];
    unsigned long long t = (unsigned long long)__reduce_add_sync(0xffffffffu, x & 0xFFFFu) +
                           ((unsigned long long)__reduce_add_sync(0xffffffffu, x >> 16) << 16);
    if constexpr (kMany) {
      const uint32_t y = tab[(2 * kTabRows + d) * 32 + lane];
      t += ((unsigned long long)__reduce_add_sync(0xffffffffu, y & 0xFFFFu) << 16) +
           ((unsigned long long)__reduce_add_sync(0xffffffffu, y >> 16) << 32);
    }
    if (lane == 0 && t) atomicAdd(a.acc + (d < kTabRows ? d : kMaxBins + d - kTabRows), t);
  }
}

// ---------------------------------------------------------------- windows of up to 4 bits
// Everything in one warp: a lane holds four neighbouring columns, one byte each, in
// one word per bin, so that z renames words, a step costs two additions per word for
// four residue pairs, and the neighbour columns come by shuffles (no barrier, no
// exchange through shared memory).  The last 2^kLevels - 1 of a warp's 128 columns only
// feed their neighbours.  The bins are folded two at a time: cell e of a lane's table
// holds distances e and e + 1 in its halves and is unpacked to 32 bits every
// kPackedRows rows.  A = 62307, k = 20: 28.5 ms with one column a thread (367 warp
// instructions per 32 residue pairs, neighbours through shared memory and a barrier a
// step), 20.6 ms (about 200); with the first ring in registers, too, 29 ms (254
// registers, 8 warps an SM, an unrolled loop past the instruction cache).
constexpr int kQuadWarps = 6;
constexpr int kCells = 37;                 // q distance <= 16, bins 0, 2, .. 20
constexpr int kDiscard = 21;               // cells for columns that do not count
constexpr int kPackedRows = 16;            // x 4 columns x 4 q pairs x 255 stays below 2^16
constexpr int kQuadRows = 40;               // distances of the tables U and D
constexpr int kQuadBytes = kCells * 128;
template <int kLevels>
__host__ __device__ constexpr int quad_smem() {  // U, D, the discarded; the warps' cells; the first ring (4 rows of 20 words a thread)
  return (2 * kQuadRows + kDiscard) * 128 + kQuadWarps * (kQuadBytes + (kLevels == 4 ? 4 * 5 * 16 * 32 : 0));
}
template <int kLevels>
__host__ __device__ constexpr uint32_t quad_useful() { return (128 - ((1 << kLevels) - 1)) / 4 * 4; }

template <int kN>
struct Quad {
  uint32_t w[kN];  // counts of bin d of four columns
};

// Adds the one-hot words of four distances 0..16 (bytes of h) to m[kFrom ..].
template <int kFrom, int kN>
__device__ __forceinline__ void count_bytes(uint32_t h, Quad<kN>& m) {
  constexpr uint32_t k1 = 0x01010101u;
  const uint32_t b0 = h & k1, b1 = (h >> 1) & k1, b2 = (h >> 2) & k1, b3 = (h >> 3) & k1, b4 = (h >> 4) & k1;
  const uint32_t lo[4] = {k1 & ~(b0 | b1), b0 & ~b1, b1 & ~b0, b0 & b1};
  const uint32_t hi[4] = {k1 & ~(b2 | b3 | b4), b2 & ~b3, b3 & ~b2, b2 & b3};
#pragma unroll
  for (int d = 0; d < 16; ++d) m.w[kFrom + d] += lo[d & 3] & hi[d >> 2];
  m.w[kFrom + 16] += b4;
}

// The word of the columns kShift to the right.
template <int kShift>
__device__ __forceinline__ uint32_t columns_at(uint32_t w) {
  if constexpr (kShift == 8) return __shfl_down_sync(0xffffffffu, w, 2);
  const uint32_t next = __shfl_down_sync(0xffffffffu, w, 1);
  if constexpr (kShift == 4) return next;
  else return __byte_perm(w, next, kShift == 2 ? 0x5432 : 0x4321);
}

__device__ __forceinline__ void load_quad(const uint4* p, Quad<19>& y) {
#pragma unroll
  for (int k = 0; k < 5; ++k) {
    const uint4 v = p[k * 32];
    y.w[4 * k] = v.x; y.w[4 * k + 1] = v.y; y.w[4 * k + 2] = v.z;
    if (k < 4) y.w[4 * k + 3] = v.w;
  }
}
__device__ __forceinline__ void store_quad(uint4* p, const Quad<19>& y) {
#pragma unroll
  for (int k = 0; k < 5; ++k)
    p[k * 32] = make_uint4(y.w[4 * k], y.w[4 * k + 1], y.w[4 * k + 2], k < 4 ? y.w[4 * k + 3] : 0u);
}

template <int kShift, int kN>
__device__ __forceinline__ Quad<kN + 1> quad_level(const Quad<kN>& a, Quad<kN + 1>& y) {
  Quad<kN> n;
#pragma unroll
  for (int d = 0; d < kN; ++d) n.w[d] = columns_at<kShift>(a.w[d]);
  Quad<kN + 1> r;
#pragma unroll
  for (int d = 0; d <= kN; ++d) {
    const uint32_t ad = d < kN ? a.w[d] : 0u, nd = d < kN ? n.w[d] : 0u;
    r.w[d] = ad + (d ? n.w[d - 1] : 0u) + y.w[d];
    y.w[d] = nd + (d ? a.w[d - 1] : 0u);
  }
  return r;
}

// Distances of row code r to the four column codes, one per byte.
__device__ __forceinline__ uint32_t distances(uint32_t r, const uint32_t (&c)[4]) {
  const uint32_t x = __byte_perm(__popc(r ^ c[0]), __popc(r ^ c[1]), 0x0040);
  const uint32_t y = __byte_perm(__popc(r ^ c[2]), __popc(r ^ c[3]), 0x0040);
  return __byte_perm(x, y, 0x5410);
}

__device__ __forceinline__ void red_at(uint32_t addr, uint32_t x) {
  asm volatile("red.shared.add.u32 [%0], %1;" ::"r"(addr), "r"(x) : "memory");
}

// Bins of the four columns, two per word, to the cells from at[i] (and at2[i]) on.
template <bool kTwice, int kN>
__device__ __forceinline__ void fold_quad(const Quad<kN>& g, const uint32_t (&at)[4], const uint32_t (&at2)[4]) {
#pragma unroll
  for (int d = 0; d < kN; d += 2) {
    const uint32_t x = g.w[d], y = d + 1 < kN ? g.w[d + 1] : 0u;
    const uint32_t xe = x & 0x00FF00FFu, xo = __byte_perm(x, 0, 0x4341);
    const uint32_t ye = y & 0x00FF00FFu, yo = __byte_perm(y, 0, 0x4341);
    const uint32_t v[4] = {__byte_perm(xe, ye, 0x5410), __byte_perm(xo, yo, 0x5410), __byte_perm(xe, ye, 0x7632),
                           __byte_perm(xo, yo, 0x7632)};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      red_at(at[i] + d * 128, v[i]);
      if constexpr (kTwice) red_at(at2[i] + d * 128, v[i]);
    }
  }
}

template <int kLevels>
__global__ void __launch_bounds__(kQuadWarps * 32, 2) carry_quad_kernel(const __grid_constant__ CarryBatch batch) {
  constexpr int kFirst = 1 << (kLevels - 1);
  constexpr int kWarm = kFirst - 1;
  constexpr uint32_t kUseful = quad_useful<kLevels>();
  constexpr int kUnroll = kLevels >= 3 ? 2 : 1;
  constexpr int kLast = 17 + kLevels;  // bins of the finished windows
  extern __shared__ __align__(16) uint8_t smem[];
  uint32_t idx = 0;
  while (blockIdx.x >= batch.e[idx].fold_end) ++idx;
  const CarryEntry& a = batch.e[idx];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t work = (blockIdx.x - (idx ? batch.e[idx - 1].fold_end : 0)) * kQuadWarps + warp;
  const uint32_t c0 = work % a.strips * kUseful, seg = work / a.strips;
  const uint32_t r0 = seg * a.seg;
  const uint32_t r1 = seg < a.segs && min(a.cols, c0 + kUseful) > r0 ? min(a.rows, r0 + a.seg) : r0;  // some v' >= v

  // the ring's first rows only reach rows that are not folded
  for (int i = threadIdx.x; i < quad_smem<0>() / 4; i += kQuadWarps * 32) reinterpret_cast<uint32_t*>(smem)[i] = 0;
  __syncthreads();
  const uint32_t tab_u = (uint32_t)__cvta_generic_to_shared(smem) + lane * 4u, tab_d = tab_u + kQuadRows * 128;
  const uint32_t discard = tab_d + kQuadRows * 128, cells = discard + kDiscard * 128 + warp * kQuadBytes;
  uint4* ring = reinterpret_cast<uint4*>(smem + (2 * kQuadRows + kDiscard) * 128 + kQuadWarps * kQuadBytes) + warp * (4 * 5 * 32) + lane;

  const uint32_t vc = c0 + 4u * lane;  // first of the lane's four residue columns
  uint32_t c[4], qc[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    c[i] = mul_mod(a.psi, vc + i, a.A);
    qc[i] = mul_mod(a.qinv, vc + i, a.A);
  }
  const uint32_t cols_end = 4u * lane < kUseful ? a.cols : 0u;  // columns of this lane that count: v' < cols_end
  const int total = r1 > r0 ? ((int)(r1 - r0) + kWarm + kUnroll - 1) / kUnroll * kUnroll : 0;
  uint32_t r = r0 + total - 1;  // descending
  uint32_t ra = mul_mod(a.psi, r, a.A), rb = mul_mod(a.psi, r + kFirst, a.A), qr = mul_mod(a.qinv, r, a.A);
  bool second = false;  // some column of the warp has a second q
#pragma unroll
  for (int i = 0; i < 4; ++i) second |= qc[i] + a.A < a.nq;
  second = __any_sync(0xffffffffu, second);

  auto unpack = [&]() {
    __syncwarp();
#pragma unroll 4
    for (int k = 0; k < kCells; ++k) {
      const uint32_t at = cells + k * 128;
      uint32_t x;
      asm volatile("ld.shared.u32 %0, [%1];" : "=r"(x) : "r"(at) : "memory");
      asm volatile("st.shared.u32 [%0], %1;" ::"r"(at), "r"(0u) : "memory");
      red_at(tab_u + k * 128, x & 0xFFFFu);
      red_at(tab_u + (k + 1) * 128, x >> 16);
    }
  };

  Quad<kLevels == 3 ? 19 : 20> y2[2];
  Quad<kLast> y1;
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int d = 0; d < (kLevels == 3 ? 19 : 20); ++d) y2[i].w[d] = 0;
#pragma unroll
  for (int d = 0; d < kLast; ++d) y1.w[d] = 0;
  int packed = 0;
  for (int it = 0; it < total; it += kUnroll) {
#pragma unroll
    for (int u = 0; u < kUnroll; ++u, --r) {
      const uint32_t ha = distances(ra, c), hd = distances(rb, c);
      Quad<18> h1;
#pragma unroll
      for (int d = 0; d < 18; ++d) h1.w[d] = 0;
      count_bytes<0>(ha, h1);
      count_bytes<1>(columns_at<kFirst>(ha), h1);
      count_bytes<1>(hd, h1);
      count_bytes<0>(columns_at<kFirst>(hd), h1);
      ra = sub_mod(ra, a.psi, a.A);
      rb = sub_mod(rb, a.psi, a.A);
      Quad<kLast> g;
      if constexpr (kLevels == 1) {
        g = h1;
      } else if constexpr (kLevels == 2) {
        g = quad_level<1>(h1, y1);
      } else if constexpr (kLevels == 3) {
        const Quad<19> h2 = quad_level<2>(h1, y2[u & 1]);
        g = quad_level<1>(h2, y1);
      } else {
        uint4* row = ring + ((it + u) & 3) * (5 * 32);
        Quad<19> y4;
        load_quad(row, y4);
        const Quad<19> h2 = quad_level<4>(h1, y4);
        store_quad(row, y4);
        const Quad<20> h3 = quad_level<2>(h2, y2[u & 1]);
        g = quad_level<1>(h3, y1);
      }
      if (r < r1) {
        // rows left of the strip need no test per column; lanes past the useful ones
        // count into columns of the table that nothing reads
        const bool inside = r < c0 && c0 + kUseful <= a.cols;
#pragma unroll 1
        for (uint32_t q = qr; q < a.nq; q += a.A) {
          uint32_t at[4], at2[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            at[i] = cells + (__popc(q ^ qc[i]) << 7);
            at2[i] = qc[i] + a.A < a.nq ? cells + (__popc(q ^ (qc[i] + a.A)) << 7) : discard;
          }
          if (!inside) {
#pragma unroll
            for (int i = 0; i < 4; ++i)
              if (vc + i <= r || vc + i >= cols_end) at[i] = at2[i] = discard;
            // the diagonal: both orders of two q of one residue, each q with itself
            if (r >= vc && r < vc + 4 && r < cols_end) {
              const uint32_t sh = (r - vc) * 8;
              for (uint32_t p = qr; p < a.nq; p += a.A)
#pragma unroll
                for (int d = 0; d < kLast; ++d) red_at(tab_d + (__popc(q ^ p) + d) * 128, (g.w[d] >> sh) & 0xFFu);
            }
          }
          if (second) fold_quad<true>(g, at, at2);
          else fold_quad<false>(g, at, at2);
        }
        if (++packed == kPackedRows) {
          unpack();
          packed = 0;
        }
      }
      qr = sub_mod(qr, a.qinv, a.A);
    }
  }
  unpack();
  __syncthreads();
  const uint32_t* tab = reinterpret_cast<const uint32_t*>(smem);
  for (int d = warp; d < 2 * kQuadRows; d += kQuadWarps) {
    const uint32_t x = 4u * lane < kUseful ? tab[d * 32 + lane] : 0u;
    const unsigned long long t = (unsigned long long)__reduce_add_sync(0xffffffffu, x & 0xFFFFu) +
                                 ((unsigned long long)__reduce_add_sync(0xffffffffu, x >> 16) << 16);
    if (lane == 0 && t) atomicAdd(a.acc + (d < kQuadRows ? d : kMaxBins + d - kQuadRows), t);
  }
}

// Residue pairs v < v' stand for one unordered pair of codewords each; pairs of
// one residue were counted in both orders, and each codeword with itself.
__global__ void carry_finish_kernel(const Job* jobs, const unsigned long long* acc) {
  const Job& j = jobs[blockIdx.x];
  const unsigned long long* t = acc + (size_t)blockIdx.x * 2 * kMaxBins;
  const uint32_t d = threadIdx.x;
  j.bins[d] = t[d] + (t[kMaxBins + d] - (d == 0 ? 1ull << j.n : 0ull)) / 2;
}

template <int kBefore, int kLevels, bool kMany>
cudaError_t run_fold(const CarryBatch& b, cudaStream_t stream) {
  constexpr size_t smem = fold_smem<kBefore, kLevels>(kMany);
  auto fn = carry_fold_kernel<kBefore, kLevels, kMany>;
  cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  fn<<<b.e[b.n - 1].fold_end, kFoldThreads, smem, stream>>>(b);
  return cudaGetLastError();
}

template <int kBefore, int kLevels>
cudaError_t run_batch(const CarryBatch& b, bool many, cudaStream_t stream) {
  carry_stage_kernel<kBefore><<<b.e[b.n - 1].stage_end, kStageThreads, 0, stream>>>(b);
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  return many ? run_fold<kBefore, kLevels, true>(b, stream) : run_fold<kBefore, kLevels, false>(b, stream);
}

template <int kLevels>
cudaError_t run_quad(const CarryBatch& b, cudaStream_t stream) {
  constexpr int smem = quad_smem<kLevels>();
  cudaError_t e = cudaFuncSetAttribute(carry_quad_kernel<kLevels>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return e;
  carry_quad_kernel<kLevels><<<b.e[b.n - 1].fold_end, kQuadWarps * 32, smem, stream>>>(b);
  return cudaGetLastError();
}

// With up to 4 window bits 2^s < 2 A, so a residue has at most two q (many is false).
cudaError_t run_batch(const CarryBatch& b, uint32_t levels, bool many, cudaStream_t stream) {
  switch (levels) {
    case 1: return run_quad<1>(b, stream);
    case 2: return run_quad<2>(b, stream);
    case 3: return run_quad<3>(b, stream);
    case 4: return run_quad<4>(b, stream);
    case 5: return run_batch<1, 4>(b, many, stream);
    case 6: return run_batch<2, 4>(b, many, stream);
    case 7: return run_batch<3, 4>(b, many, stream);
    default: return run_batch<4, 4>(b, many, stream);
  }
}

}  // namespace

bool carry_eligible(const Job& j) {
  if (j.kind != JOB_PAIRS || j.shape != SHAPE_TRIANGLE || j.row_kind != ROW_PROGRESSION ||
      j.col_kind != COL_PROGRESSION || j.tile_offset != 0 || j.A == 0 || (j.A >> 32) || j.n > 24)
    return false;
  const uint32_t a = bits_of(odd_part(j.A));
  return a <= 16 && j.n > a;
}

// Residue pairs cost about as much as the tcgen05 kernel's 16^2 codeword pairs
// (16-bit A: k = 19, 17.9 ms here and 15.3 ms there; k = 20, 26.8 and 63.5 ms); below
// k = 14 a launch of the popc kernel takes no longer than this path's three.
bool carry_wins(const Job& j) {
  const uint32_t a = bits_of(odd_part(j.A));
  return j.n >= a + 4 && j.n >= 14;
}

void carry_plan(const Job& j, CarryPlan& p) {
  p = CarryPlan();
  p.A = odd_part(j.A);
  p.k = j.n;
  p.b = std::min<uint32_t>(8, p.k - bits_of(p.A));
  p.s = p.k - p.b;
  p.staged = p.b > 4 ? p.b - 4 : 0;
  p.psi = (p.A - inverse_pow2(p.k, p.A)) % p.A;
  p.qinv = inverse_pow2(p.b, p.A);
  p.many = (1ull << p.s) > 2ull * p.A;
  p.side = p.A;
  if (p.staged) {
    const uint32_t useful = kStageCols - ((1u << p.staged) - 1);
    p.side = std::min(p.A, kUnit * useful * 2 - 15);
    p.cells = (size_t)(p.side + 15) * (p.side + 15);
  }
}

size_t carry_stage_bytes(const std::vector<CarryPlan>& plans) {
  size_t all = 0, one = 0;
  for (const CarryPlan& p : plans) {
    const size_t blocks = (p.A + p.side - 1) / p.side;
    all += p.cells * (blocks * (blocks + 1) / 2);
    one = std::max(one, p.cells);
  }
  // one round of blocks, at most kStageCells unless a single one is larger
  return std::max(one, std::min(all, kStageCells)) * 24;
}

cudaError_t launch_carry(const std::vector<CarryPlan>& plans, int num_sms, unsigned long long* acc, void* stage,
                         size_t stage_bytes, cudaStream_t stream) {
  uint4* st16 = static_cast<uint4*>(stage);
  const size_t cells = stage_bytes / 24;
  uint2* st8 = reinterpret_cast<uint2*>(st16 + cells);
  std::vector<bool> done(plans.size(), false);
  for (size_t first = 0; first < plans.size(); ++first) {
    if (done[first]) continue;
    // the jobs that run the same kernels, their blocks in rounds that fit the staging memory
    const uint32_t levels = plans[first].b, many = plans[first].many;
    size_t alike = 0;
    for (const CarryPlan& p : plans) alike += p.b == levels && p.many == many;
    CarryBatch b{};
    size_t used = 0;
    for (size_t i = first; i < plans.size(); ++i) {
      const CarryPlan& p = plans[i];
      if (done[i] || p.b != levels || p.many != many) continue;
      done[i] = true;
      if (b.n == kEntries) {  // the jobs left share the next launch
        const cudaError_t err = run_batch(b, levels, many != 0, stream);
        if (err != cudaSuccess) return err;
        b.n = 0;
        used = 0;
        alike -= std::min<size_t>(alike, kEntries);
      }
      for (uint32_t r0 = 0; r0 < p.A; r0 += p.side)
        for (uint32_t c0 = r0; c0 < p.A; c0 += p.side) {
          CarryEntry e{};
          e.A = p.A;
          e.psi = p.psi;
          e.qinv = p.qinv;
          e.nq = 1u << p.s;
          e.row0 = r0;
          e.col0 = c0;
          e.rows = std::min(p.side, p.A - r0);
          e.cols = std::min(p.side, p.A - c0);
          e.acc = acc + i * 2 * kMaxBins;
          const uint32_t useful = p.staged ? kFoldThreads - 15 : (128 - ((1u << p.b) - 1)) / 4 * 4;
          e.strips = (e.cols + useful - 1) / useful;
          // rows per CTA: long runs amortise the rows a segment computes twice; short
          // ones where the launch would leave SMs without a CTA
          // (strips x segments are CTAs of the folding kernel, warps of the other)
          const uint64_t want =
              std::max<uint64_t>(1, (p.staged ? 8ull : 24ull) * num_sms / std::min<size_t>(std::max<size_t>(alike, 1), kEntries));
          e.seg = 256;
          while (e.seg > 16 && (uint64_t)e.strips * ((e.rows + e.seg - 1) / e.seg) < want) e.seg /= 2;
          e.segs = (e.rows + e.seg - 1) / e.seg;
          e.slices = 1;
          if (p.many) {
            // every slice computes the windows again, so only as many as fill the GPU once
            // (A = 867, k = 21: 0.65 ms with four times as many, 0.32 ms)
            const uint64_t per = (e.nq + p.A - 1) / p.A, ctas = (uint64_t)e.strips * e.segs;
            e.slices = (uint32_t)std::min<uint64_t>(std::min<uint64_t>(per, 4096), std::max<uint64_t>(1, want / 4 / ctas));
            // a lane's 32-bit sums: rows x warps (x one lane) x q pairs x 4^b
            const uint64_t sum = (uint64_t)e.seg * (kFoldThreads / 32) * ((per + e.slices - 1) / e.slices) * per << (2 * p.b);
            e.wide = per > 4096 || sum > 0xFFFFFFFFull;
          }
          const size_t need = p.staged ? (size_t)(e.rows + 15) * (e.cols + 15) : 0;
          if (b.n == kEntries || (b.n && used + need > cells)) {
            const cudaError_t err = run_batch(b, levels, many != 0, stream);
            if (err != cudaSuccess) return err;
            b.n = 0;
            used = 0;
          }
          if (p.staged) {
            e.srows = e.rows + 15;
            e.scols = e.cols + 15;
            e.st16 = st16 + used;
            e.st8 = st8 + used;
            used += need;
            const uint32_t su = kStageCols - ((1u << p.staged) - 1);
            const uint32_t w = (e.scols + kUnit - 1) / kUnit, wr = (e.srows + kUnit - 1) / kUnit;
            e.stage_strips = 4 * ((w + su - 1) / su);
            e.stage_segs = (wr + 63) / 64;
            e.stage_seg = (wr + e.stage_segs - 1) / e.stage_segs;
          }
          const CarryEntry* before = b.n ? &b.e[b.n - 1] : nullptr;
          const uint32_t ctas = e.strips * e.segs * e.slices;
          e.fold_end = (before ? before->fold_end : 0) + (p.staged ? ctas : (ctas + kQuadWarps - 1) / kQuadWarps);
          e.stage_end = (before ? before->stage_end : 0) + e.stage_strips * e.stage_segs * kUnit;
          b.e[b.n++] = e;
        }
    }
    const cudaError_t err = run_batch(b, levels, many != 0, stream);
    if (err != cudaSuccess) return err;
  }
  return cudaSuccess;
}

cudaError_t launch_carry_finish(const Job* jobs, const unsigned long long* acc, uint32_t n, cudaStream_t stream) {
  carry_finish_kernel<<<n, kMaxBins, 0, stream>>>(jobs, acc);
  return cudaGetLastError();
}

}  // namespace dd

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
// Measured on B200 against the tcgen05 kernel: A = 58659, k = 22: 40.4 ms against 941 ms
// (965 ms before its generators were mended), k = 24: 85 ms against 15 s; A = 62307,
// k = 20: 20.6 against 59.2 ms; A = 867, k = 21: 0.18 against 193 ms, k = 16: 0.046
// against 0.28 ms.  Bound by instruction issue and its latencies at 12 to 18 warps an
// SM, the ALU (staging) and shared-memory (folding) pipes three quarters busy; DRAM
// carries nothing up to 4 window bits and the staged histograms (24 bytes a residue
// pair, once each way) above.
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
// kernel from the popcounts to the bins (carry_quad_kernel).  For longer ones the same
// four steps run first, in a kernel whose rows and columns are 2^(b-4) residues apart,
// and stage their 8-bit histograms in memory (carry_stage_kernel); the remaining small
// steps hold one column a thread in words of every fourth bin, so that multiplying by
// z renames words and shifts only one in four (carry_fold_kernel).
#include <algorithm>
#include <utility>

#include "dd_carry.cuh"

namespace dd {
namespace {

constexpr size_t kStageCells = 32u << 20;  // staged histograms of one round of blocks (768 MB)
constexpr uint32_t kStageSide = 3584;      // residues per side of a staged block, with the windows' overhang
constexpr int kAhead = 3;           // rows the folding kernels load ahead
constexpr int kFoldThreads = 192;
constexpr int kQuadWarps = 6;       // warps of a CTA where each works alone

// One block of residue pairs of one job: [row0, row0+rows) x [col0, col0+cols).
struct CarryEntry {
  uint32_t A, psi, qinv, nq, slices, wide;
  uint32_t row0, rows, col0, cols;
  uint32_t unit;                    // residues between the staging kernel's rows and columns: 2^(b-4)
  uint32_t srows, scols, pitch;     // staged rows and columns (from row0, col0); columns of one residue mod unit
  uint32_t seg, segs, strips;       // folding: rows per CTA, CTAs down and across
  uint32_t stage_seg, stage_segs, stage_strips;
  uint32_t fold_end, stage_end;     // CTAs of the launch up to and including this entry
  // staged histograms, row by row, a row's columns by their residue mod unit:
  uint4* st16;                      // words e0 e1 e2 o0 ...
  uint2* st8;                       // ... and o1 o2
  unsigned long long* acc;          // [0, kMaxBins): residue pairs v < v'; then v = v'
};

// Entries of one launch, in its parameters (short instances share a launch, and so
// fill the GPU together; 31 entries stay below the 4 KB every launch can pass).  64
// instances of 8-bit A, k = 14: 0.18 ms (0.33 when they first shared one, 2.0 launched one
// by one); 256 at k = 16: 1.9 ms, popc kernel 123, tcgen05 54.
constexpr uint32_t kEntries = 31;
struct CarryBatch {
  uint32_t n;
  CarryEntry e[kEntries];
};
static_assert(sizeof(CarryBatch) <= 4096, "kernel parameters");

// One step in a running column: exchange with column c + s, combine, rotate the ring entry y.
__device__ __forceinline__ H16 level(const H16& own, uint8_t* row, int c, int s, H16& y) {
  put(row, c, own);
  __syncthreads();
  H16 nb;
  get(row, c + s, nb);
  const H16 r = add(add_z(own, nb), y);
  y = add_z(nb, own);
  return r;
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

// One column's bins to the cells from at (and at2) on, in all words alike: most hold
// counts, and a test per word costs more than the empty additions.
template <int kBin>
__device__ __forceinline__ void fold_word(uint32_t w, uint32_t at, uint32_t at2, bool twice) {
  const uint32_t lo = w & 0xFFFFu, hi = w >> 16;
  red_add<kBin * 128>(at, lo);
  red_add<(kBin + 4) * 128>(at, hi);
  if (twice) {
    red_add<kBin * 128>(at2, lo);
    red_add<(kBin + 4) * 128>(at2, hi);
  }
}
template <bool kTwice>
__device__ __forceinline__ void fold_column(const H16& g, uint32_t at, uint32_t at2) {
  fold_word<0>(g.p0[0], at, at2, kTwice); fold_word<1>(g.p1[0], at, at2, kTwice);
  fold_word<2>(g.p2[0], at, at2, kTwice); fold_word<3>(g.p3[0], at, at2, kTwice);
  fold_word<8>(g.p0[1], at, at2, kTwice); fold_word<9>(g.p1[1], at, at2, kTwice);
  fold_word<10>(g.p2[1], at, at2, kTwice); fold_word<11>(g.p3[1], at, at2, kTwice);
  fold_word<16>(g.p0[2], at, at2, kTwice); fold_word<17>(g.p1[2], at, at2, kTwice);
  fold_word<18>(g.p2[2], at, at2, kTwice); fold_word<19>(g.p3[2], at, at2, kTwice);
  red_add<24 * 128>(at, g.p0[3]);  // bin 28 does not occur
  if (kTwice) red_add<24 * 128>(at2, g.p0[3]);
}

// The additions to the tables are the larger part of this kernel's shared-memory traffic
// (nearly every warp has a column with a second q, so 48 a row).  With up to six window
// bits a count stays below 2^12, so a word of an H16 (bins d and d + 4) goes to a cell as
// it is: cell e of a lane's packed table holds distances e and e + 4 (24 additions a row,
// and 9 to unpack).  k = 22, A = 58659 45.3 -> 40.3 ms, A = 40001 23.8 -> 20.2 ms; k = 21,
// A = 40001 20.1 -> 17.2 ms.  Seven window bits would need unpacking within a row.
// Two tables take turns of two rows; the one of the turn before is unpacked at the end of a
// turn, when every warp has left it (a barrier of this turn) and none has come back (the next
// turn's first).  So a field holds the counts of 6 warps x 2 rows; one table that is unpacked
// while others go on adding can hold 17 warps' rows, as their timing has it.  With five
// window bits a field is at most 12 x 4 q pairs x 4^5.  With six, an overflow takes four q
// pairs of one distance and most of every window's pairs in one bin: the fullest fields are
// those of A = 2^j + 1, 44,000 of 65,535 (62,600 with 17 rows), and as the rows of a turn are
// an odd one and the one below it, whatever the segments, they are the same in every run.
// An overflow would make the bins' sum wrong, and the caller counts on another kernel.
constexpr int kPackCells = 36;  // q distance <= 16, bins 0 .. 3, 8 .. 11, 16 .. 19 (and 4 more)
template <int kLevels, bool kMany>
__host__ __device__ constexpr bool fold_packed() { return kLevels <= 2 && !kMany; }
template <bool kTwice, int kBin>
__device__ __forceinline__ void pack_word(uint32_t w, uint32_t at, uint32_t at2) {
  red_add<kBin * 128>(at, w);
  if (kTwice) red_add<kBin * 128>(at2, w);
}
template <bool kTwice>
__device__ __forceinline__ void pack_column(const H16& g, uint32_t at, uint32_t at2) {
  pack_word<kTwice, 0>(g.p0[0], at, at2); pack_word<kTwice, 1>(g.p1[0], at, at2);
  pack_word<kTwice, 2>(g.p2[0], at, at2); pack_word<kTwice, 3>(g.p3[0], at, at2);
  pack_word<kTwice, 8>(g.p0[1], at, at2); pack_word<kTwice, 9>(g.p1[1], at, at2);
  pack_word<kTwice, 10>(g.p2[1], at, at2); pack_word<kTwice, 11>(g.p3[1], at, at2);
  pack_word<kTwice, 16>(g.p0[2], at, at2); pack_word<kTwice, 17>(g.p1[2], at, at2);
  pack_word<kTwice, 18>(g.p2[2], at, at2); pack_word<kTwice, 19>(g.p3[2], at, at2);
}
// A warp's share of a packed table to the 32-bit one; other warps may go on adding.  (An
// exchange also where none does: a load and a store take longer, k = 22 40.7 against 40.3 ms.)
__device__ __forceinline__ void unpack_cells(uint32_t cells, uint32_t tab, int warp) {
#pragma unroll
  for (int i = 0; i < kPackCells / (kFoldThreads / 32); ++i) {
    const uint32_t e = (uint32_t)(i * (kFoldThreads / 32) + warp) * 128;
    uint32_t x;
    asm volatile("atom.shared.exch.b32 %0, [%1], 0;" : "=r"(x) : "r"(cells + e) : "memory");
    red_add<0>(tab + e, x & 0xFFFFu);
    red_add<4 * 128>(tab + e, x >> 16);
  }
}
static_assert(kPackCells % (kFoldThreads / 32) == 0 && kPackCells + 4 <= kTabRows, "a warp's cells, unpacked");

// Many q: the counts of the 17 q distances (f, a stride of kStride words) times kN bins of
// a window from kFrom on.  The products are summed in registers, so that a residue pair
// costs 57 additions to the table in two parts (both at once would spill) instead of up to
// 17 x 25: A = 1019, k = 21 0.298 -> 0.188 ms, A = 867, k = 20 0.200 -> 0.128 ms, A = 61
// 0.133 -> 0.106 ms; shorter multipliers spend their time on the pairs of q.  The host
// sends sums that do not fit 32 bits to the wide products.
template <int kBin>
__device__ __forceinline__ uint32_t bin_of(const H16& g) {
  constexpr int j = kBin / 8, m = kBin % 4;
  const uint32_t w = m == 0 ? g.p0[j] : m == 1 ? g.p1[j % 3] : m == 2 ? g.p2[j % 3] : g.p3[j % 3];
  return kBin % 8 < 4 ? w & 0xFFFFu : w >> 16;
}
template <int kFrom, int... kI>
__device__ __forceinline__ void take_bins(const H16& g, uint32_t* x, std::integer_sequence<int, kI...>) {
  ((x[kI] = bin_of<kFrom + kI>(g)), ...);
}
template <int kFrom, int... kI>
__device__ __forceinline__ void add_sums(uint32_t at, const uint32_t* x, std::integer_sequence<int, kI...>) {
  (red_add<(kFrom + kI) * 128>(at, x[kI]), ...);
}
template <int kFrom, int kN, int kStride>
__device__ __forceinline__ void add_product(const volatile uint32_t* f, const H16& g, uint32_t at) {
  uint32_t x[kN], sum[kN + 16];
  take_bins<kFrom>(g, x, std::make_integer_sequence<int, kN>());
#pragma unroll
  for (int e = 0; e < kN + 16; ++e) sum[e] = 0;
#pragma unroll
  for (int d = 0; d <= 16; ++d) {
    const uint32_t n = f[d * kStride];
#pragma unroll
    for (int i = 0; i < kN; ++i) sum[d + i] += n * x[i];
  }
  add_sums<kFrom>(at, sum, std::make_integer_sequence<int, kN + 16>());
}

// The first level of the last kLevels reads its own row only, with a ring in registers;
// 8 rows of 16-bit histograms do not fit there, so kLevels = 4 reads row v + 8, too.
template <int kLevels>
__host__ __device__ constexpr int fold_lead() { return kLevels == 4 ? 8 : 0; }
template <int kLevels>
__host__ __device__ constexpr int fold_slots() { return fold_lead<kLevels>() + 1 + kAhead; }
// Exchange rows, one per level after the first; a single one has two that take turns
// (a row's only barrier then separates them).
template <int kLevels>
__host__ __device__ constexpr int fold_exchanges() { return kLevels == 2 ? 2 : kLevels - 1; }

// Shared memory of the folding kernel: tables (U, D and a spare, which a q' past the last
// reaches at distances up to 17; U and D twice for wide products; packed tables, two for U,
// beside U and D), exchange rows, the ring of staged rows, and the q-distance counts of each
// thread (many).
template <int kLevels, bool kMany>
__host__ __device__ constexpr int fold_tables() {
  return fold_packed<kLevels, kMany>() ? kTabBytes * 2 + (4 * kPackCells + 1) * 128 : kTabBytes * (kMany ? 4 : 3);
}
template <int kLevels, bool kMany>
constexpr size_t fold_smem() {
  constexpr int cols = kFoldThreads + (1 << (kLevels - 1));
  return (size_t)fold_tables<kLevels, kMany>() + (size_t)(48 * fold_exchanges<kLevels>() + 24 * fold_slots<kLevels>()) * cols +
         (kMany ? (size_t)(16 + 1) * kFoldThreads * 4 : 0);
}

// The last kLevels steps (s = 2^(kLevels-1) .. 1), from the staged 8-bit histograms to
// 16-bit ones, and the sum over q, q'.  CTA: a strip of columns (one per thread, the
// last 2^kLevels - 1 only feed their neighbours) x a segment of rows.  Measured and
// dropped: a warp alone with shuffles and tables of its own (k = 22 58.7 against 52.9 ms:
// fewer warps), CTAs of 256 threads (57 ms).
template <int kLevels, bool kMany>
__global__ void __launch_bounds__(kFoldThreads, kLevels <= 2 ? 3 : 2) carry_fold_kernel(const __grid_constant__ CarryBatch batch) {
  constexpr int kThreads = kFoldThreads;
  constexpr int kFirst = 1 << (kLevels - 1);
  constexpr int kLead = fold_lead<kLevels>(), kSlots = fold_slots<kLevels>();
  constexpr int kWarm = (kLead ? kFirst : 2 * kFirst) - 1;
  constexpr int kUseful = kThreads - ((1 << kLevels) - 1);
  constexpr int kUnroll = kLevels == 4 ? 4 : kFirst;  // the longest ring in registers
  constexpr int kCols = kThreads + kFirst;
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
  uint8_t* ex = smem + fold_tables<kLevels, kMany>();
  uint4* in16 = reinterpret_cast<uint4*>(ex + 48 * fold_exchanges<kLevels>() * kCols);
  uint2* in8 = reinterpret_cast<uint2*>(in16 + kSlots * kCols);
  uint32_t* qd = reinterpret_cast<uint32_t*>(in8 + kSlots * kCols);
  for (int i = tid; i < fold_tables<kLevels, kMany>() / 4; i += kThreads) tab[i] = 0;
  if constexpr (kMany)
    for (int i = tid; i < 17 * kThreads; i += kThreads) qd[i] = 0;

  const uint32_t col = c0 + tid, vc = a.col0 + col;
  const bool mine = tid < kUseful && col < a.cols;
  const uint32_t qc = mul_mod(a.qinv, vc, a.A);
  const int total = ((int)(r1 - r0) + kWarm + kUnroll - 1) / kUnroll * kUnroll;
  uint32_t r = r0 + total - 1;  // descending, from row0
  uint32_t qr = mul_mod(a.qinv, a.row0 + r, a.A);
  const uint32_t tab_u = (uint32_t)__cvta_generic_to_shared(tab) + lane * 4u;
  const bool two = qc + a.A < a.nq, second = __any_sync(0xffffffffu, two);  // a second q: here, in this warp
  // few q: the third table is not read
  constexpr bool kPacked = fold_packed<kLevels, kMany>();
  constexpr uint32_t kNext = kPacked ? kPackCells * 128 : kTabBytes;  // from a table to the next
  const uint32_t to_u0 = kPacked ? tab_u + 2 * kTabBytes : tab_u;     // U (packed: and U of the other turn)
  const uint32_t to_d = to_u0 + (kPacked ? 2 : 1) * kNext, spare = to_d + kNext;
  uint32_t to_u = to_u0;

  // input: staged rows through a ring of kSlots rows
  int slot = 0;  // ring slot of load number it (row r + kLead of that step)
  const uint32_t scol = min(col, a.scols - 1), cell = scol % a.unit * a.pitch + scol / a.unit;
  auto load = [&](int sl, uint32_t row) {
    const size_t at = (size_t)min(row, a.srows - 1) * (a.unit * a.pitch) + cell;
    copy_async16(in16 + sl * kCols + tid, a.st16 + at);
    copy_async8(in8 + sl * kCols + tid, a.st8 + at);
    copy_commit();
  };
  for (int l = 0; l < kLead + kAhead; ++l) load(l, r + kLead - l);
  copy_wait<kAhead - 1>();
  __syncthreads();

  H16 y4[4], y2[2], y1;  // the rings of the steps 4, 2, 1
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
        return widen(H8{{x.x, x.y, x.z}, {x.w, w.x, w.y}});
      };
      const int lo = slot, hi = slot + kLead < kSlots ? slot + kLead : slot + kLead - kSlots;
      H16 g;
      if constexpr (kLevels == 4) {
        g = add_z(add(fetch(hi, tid), fetch(lo, tid + kFirst)), add(fetch(hi, tid + kFirst), fetch(lo, tid)));
      } else {
        const H16 own = fetch(hi, tid), nb = fetch(hi, tid + kFirst);
        H16& y = kLevels == 3 ? y4[u & 3] : kLevels == 2 ? y2[u & 1] : y1;
        g = add(add_z(own, nb), y);
        y = add_z(nb, own);
      }
      int nx = slot + kLead + kAhead;
      if (nx >= kSlots) nx -= kSlots;
      // row r + kLead - (kLead + kAhead); rows below the block's first are never used
      load(nx, r >= kAhead ? r - kAhead : 0u);
      slot = slot + 1 == kSlots ? 0 : slot + 1;
      copy_wait<kAhead - 1>();
      // remaining levels
      uint8_t* row = ex;
      if constexpr (kLevels == 4) { g = level(g, row, tid, 4, y4[u & 3]); row += 48 * kCols; }
      if constexpr (kLevels >= 3) { g = level(g, row, tid, 2, y2[u & 1]); row += 48 * kCols; }
      if constexpr (kLevels == 2) row += ((it + u) & 1) * 48 * kCols;
      if constexpr (kLevels >= 2) g = level(g, row, tid, 1, y1);
      else __syncthreads();  // the row loaded ahead is complete for the neighbours
      if constexpr (kPacked) to_u = to_u0 + ((it + u) & 2 ? kNext : 0u);
      // fold: every q of row residue v with every q' of column residue v'
      const uint32_t v = a.row0 + r;
      if constexpr (!kMany) {
        if (r < r1)
#pragma unroll 1
          for (uint32_t q = qr; q < a.nq; q += a.A) {
            // columns that do not count here go to a spare column of the table
            const uint32_t to = !mine || vc < v ? spare : vc == v ? to_d : to_u;
            const uint32_t at = to + (__popc(q ^ qc) << 7);
            if constexpr (kPacked) {
              if (second) pack_column<true>(g, at, (two ? to : spare) + (__popc(q ^ (qc + a.A)) << 7));
              else pack_column<false>(g, at, at);
            } else if (second) fold_column<true>(g, at, (two ? to : spare) + (__popc(q ^ (qc + a.A)) << 7));
            else fold_column<false>(g, at, at);
          }
      } else if (mine && r < r1 && vc >= v) {
        const uint32_t at = tab_u + (vc == v ? kTabBytes : 0);
        {
          volatile uint32_t* f = qd + tid;
          const uint32_t fa = (uint32_t)__cvta_generic_to_shared(qd + tid);
          for (uint32_t q = qr + slice * a.A; q < a.nq; q += a.slices * a.A)
            for (uint32_t p = qc; p < a.nq; p += a.A) red_add<0>(fa + __popc(q ^ p) * (kThreads * 4), 1);
          if (!a.wide) {
            add_product<0, 13, kThreads>(f, g, at);
            add_product<13, 12, kThreads>(f, g, at);
#pragma unroll
            for (uint32_t d = 0; d <= 16; ++d) f[d * kThreads] = 0;
          } else {
            for (uint32_t d = 0; d <= 16; ++d) {
              const uint32_t x = f[d * kThreads];
              if (x) {
                f[d * kThreads] = 0;
                add_hist<kWideProduct>(at + (d << 7), x, g);
              }
            }
          }
        }
      }
      qr = sub_mod(qr, a.qinv, a.A);
    }
    if constexpr (kPacked) {
      // the other turn's table: every warp left it before a barrier of this turn, and enters
      // it past one that waits for this warp
      if (kUnroll == 2 || (it & 1)) unpack_cells(to_u0 + (it & 2 ? 0u : kNext), tab_u, warp);
      if ((it & 31) >= 32 - kUnroll) unpack_cells(to_d, tab_u + kTabBytes, warp);  // a row has one v = v', a lane every 32nd
    }
  }
  copy_wait<0>();
  __syncthreads();
  if constexpr (kPacked) {
    unpack_cells(to_u0, tab_u, warp);
    unpack_cells(to_u0 + kNext, tab_u, warp);
    unpack_cells(to_d, tab_u + kTabBytes, warp);
    __syncthreads();
  }
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

// ---------------------------------------------------------------- four steps in a warp
// Everything in one warp: a lane holds four neighbouring columns, one byte each, in
// one word per bin, so that z renames words, a step costs two additions per word for
// four residue pairs, and the neighbour columns come by shuffles (no barrier, no
// exchange through shared memory).  The last 2^kLevels - 1 of a warp's 128 columns only
// feed their neighbours.  The bins are folded two at a time: cell e of a lane's table
// holds distances e and e + 1 in its halves and is unpacked to 32 bits every
// kPackedRows rows.  A = 62307, k = 20: 28.5 ms with one column a thread (367 warp
// instructions per 32 residue pairs, neighbours through shared memory and a barrier a
// step), 20.6 ms so (229 at A = 30011, k = 19, margins included); with the first ring in
// registers, too, 29 ms (254 registers, 8 warps an SM, an unrolled loop past the
// instruction cache).
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

// ---------------------------------------------------------------- windows of 5 to 8 bits
// Their four largest steps, in the same way, for a block of residue pairs whose rows
// and columns are `unit` = 2^(b-4) apart: work of a warp is the rows v = row0 + rho +
// unit w, for one rho and a run of w, and the columns col0 + sigma + unit w' for one
// sigma and 128 consecutive w'.  The finished 8-bit histograms are stored column by
// column (a 4 x 4 byte transpose per four bins), 32 bytes a store.  159 warp
// instructions per 32 residue pairs at 62 % issue, the ALU pipe 70 % busy (A = 7151,
// k = 19).  Staging b - 4 levels and folding four took 70 ms where four staged and b - 4
// folded ones take 50 ms (A = 62307, k = 22).
constexpr int kStageRing = 4 * 5 * 16 * 32;  // a warp's first ring
constexpr int kStageBytes = kQuadWarps * kStageRing;

__device__ __forceinline__ void transpose_bytes(uint32_t w0, uint32_t w1, uint32_t w2, uint32_t w3, uint32_t (&col)[4]) {
  const uint32_t a = __byte_perm(w0, w1, 0x5140), b = __byte_perm(w2, w3, 0x5140);
  const uint32_t c = __byte_perm(w0, w1, 0x7362), d = __byte_perm(w2, w3, 0x7362);
  col[0] = __byte_perm(a, b, 0x5410);
  col[1] = __byte_perm(a, b, 0x7632);
  col[2] = __byte_perm(c, d, 0x5410);
  col[3] = __byte_perm(c, d, 0x7632);
}
__device__ __forceinline__ void store32(void* p, uint32_t a, uint32_t b, uint32_t c, uint32_t d, uint32_t e, uint32_t f,
                                        uint32_t g, uint32_t h) {
  asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "r"(a), "r"(b), "r"(c), "r"(d),
               "r"(e), "r"(f), "r"(g), "r"(h)
               : "memory");
}

__global__ void __launch_bounds__(kQuadWarps * 32, 2) carry_stage_kernel(const __grid_constant__ CarryBatch batch) {
  constexpr uint32_t kUseful = quad_useful<4>();
  extern __shared__ __align__(16) uint8_t smem[];
  uint32_t idx = 0;
  while (blockIdx.x >= batch.e[idx].stage_end) ++idx;
  const CarryEntry& a = batch.e[idx];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t work = (blockIdx.x - (idx ? batch.e[idx - 1].stage_end : 0)) * kQuadWarps + warp;
  const uint32_t w0 = work % a.stage_strips * kUseful;
  work /= a.stage_strips;
  const uint32_t sigma = work % a.unit;
  work /= a.unit;
  const uint32_t rho = work % a.unit, seg = work / a.unit;
  if (seg >= a.stage_segs) return;
  const uint32_t wrows = (a.srows - rho + a.unit - 1) / a.unit;  // rows of this rho in the block
  const uint32_t wr0 = seg * a.stage_seg, wr1 = min(wrows, wr0 + a.stage_seg);
  // residue pairs v' < v are their mirror images; a finished window reads unit - 1 past its own
  if (wr0 >= wr1 || a.col0 + sigma + a.unit * (w0 + kUseful) < a.row0 + rho + a.unit * wr0) return;
  uint4* ring = reinterpret_cast<uint4*>(smem + warp * kStageRing) + lane;

  const uint32_t w4 = w0 + 4u * lane;
  uint32_t c[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) c[i] = mul_mod(a.psi, a.col0 + sigma + a.unit * (w4 + i), a.A);
  const bool store = 4u * lane < kUseful && w4 < a.pitch;
  const int total = ((int)(wr1 - wr0) + 7 + 1) / 2 * 2;
  uint32_t w = wr0 + total - 1;  // descending
  const uint32_t step = mul_mod(a.psi, a.unit, a.A);
  uint32_t ra = mul_mod(a.psi, a.row0 + rho + a.unit * w, a.A), rb = mul_mod(a.psi, a.row0 + rho + a.unit * (w + 8), a.A);
  size_t at = ((size_t)(rho + a.unit * w) * a.unit + sigma) * a.pitch + w4;
  const size_t row_cells = (size_t)a.unit * a.unit * a.pitch;

  Quad<20> y2[2];
  Quad<21> y1;
#pragma unroll
  for (int d = 0; d < 20; ++d) y2[0].w[d] = y2[1].w[d] = 0;
#pragma unroll
  for (int d = 0; d < 21; ++d) y1.w[d] = 0;
  for (int it = 0; it < total; it += 2) {
#pragma unroll
    for (int u = 0; u < 2; ++u, --w, at -= row_cells) {
      const uint32_t ha = distances(ra, c), hd = distances(rb, c);
      Quad<18> h1;
#pragma unroll
      for (int d = 0; d < 18; ++d) h1.w[d] = 0;
      count_bytes<0>(ha, h1);
      count_bytes<1>(columns_at<8>(ha), h1);
      count_bytes<1>(hd, h1);
      count_bytes<0>(columns_at<8>(hd), h1);
      ra = sub_mod(ra, step, a.A);
      rb = sub_mod(rb, step, a.A);
      uint4* row = ring + ((it + u) & 3) * (5 * 32);
      Quad<19> y4;
      load_quad(row, y4);
      const Quad<19> h2 = quad_level<4>(h1, y4);
      store_quad(row, y4);
      const Quad<20> h3 = quad_level<2>(h2, y2[u & 1]);
      const Quad<21> g = quad_level<1>(h3, y1);
      if (store && w < wr1) {
        uint32_t e[3][4], o[3][4];
        transpose_bytes(g.w[0], g.w[2], g.w[4], g.w[6], e[0]);
        transpose_bytes(g.w[1], g.w[3], g.w[5], g.w[7], o[0]);
        transpose_bytes(g.w[8], g.w[10], g.w[12], g.w[14], e[1]);
        transpose_bytes(g.w[9], g.w[11], g.w[13], g.w[15], o[1]);
        transpose_bytes(g.w[16], g.w[18], g.w[20], 0u, e[2]);
        transpose_bytes(g.w[17], g.w[19], 0u, 0u, o[2]);
        store32(a.st16 + at, e[0][0], e[1][0], e[2][0], o[0][0], e[0][1], e[1][1], e[2][1], o[0][1]);
        store32(a.st16 + at + 2, e[0][2], e[1][2], e[2][2], o[0][2], e[0][3], e[1][3], e[2][3], o[0][3]);
        store32(a.st8 + at, o[1][0], o[2][0], o[1][1], o[2][1], o[1][2], o[2][2], o[1][3], o[2][3]);
      }
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

template <int kLevels, bool kMany>
cudaError_t run_staged(const CarryBatch& b, cudaStream_t stream) {
  cudaError_t e = cudaFuncSetAttribute(carry_stage_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kStageBytes);
  if (e != cudaSuccess) return e;
  carry_stage_kernel<<<b.e[b.n - 1].stage_end, kQuadWarps * 32, kStageBytes, stream>>>(b);
  if ((e = cudaGetLastError()) != cudaSuccess) return e;
  constexpr size_t smem = fold_smem<kLevels, kMany>();
  auto fn = carry_fold_kernel<kLevels, kMany>;
  if ((e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)) != cudaSuccess) return e;
  fn<<<b.e[b.n - 1].fold_end, kFoldThreads, smem, stream>>>(b);
  return cudaGetLastError();
}

template <int kLevels>
cudaError_t run_quad(const CarryBatch& b, cudaStream_t stream) {
  constexpr int smem = quad_smem<kLevels>();
  cudaError_t e = cudaFuncSetAttribute(carry_quad_kernel<kLevels>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return e;
  carry_quad_kernel<kLevels><<<b.e[b.n - 1].fold_end, kQuadWarps * 32, smem, stream>>>(b);
  return cudaGetLastError();
}

// With fewer than 8 window bits 2^s < 2 A, so a residue has at most two q (many is false).
cudaError_t run_batch(const CarryBatch& b, uint32_t levels, bool many, cudaStream_t stream) {
  switch (levels) {
    case 1: return run_quad<1>(b, stream);
    case 2: return run_quad<2>(b, stream);
    case 3: return run_quad<3>(b, stream);
    case 4: return run_quad<4>(b, stream);
    case 5: return run_staged<1, false>(b, stream);
    case 6: return run_staged<2, false>(b, stream);
    case 7: return run_staged<3, false>(b, stream);
    default: return many ? run_staged<4, true>(b, stream) : run_staged<4, false>(b, stream);
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

// A residue pair costs about as much as the tcgen05 kernel's 11^2 codeword pairs, so with
// three bits more than A's it depends on A itself (A of 16 bits, k = 19: A = 34407
// 7.0 ms here and 12.5 ms there, 42599 9.5, 49153 12.2, 55705 15.3; 15 bits, k = 18:
// 17203 2.1 and 3.2 ms, 21299 2.8, 24577 3.4; from 17 down a launch fills the GPU less,
// 14 bits, k = 17, A = 10649 1.02 and 0.90 ms), with four it always does (A = 62307,
// k = 20 20.6 and 59.2 ms).  Below k = 14 a launch of the popc kernel takes no longer
// than this path's three.
bool carry_wins(const Job& j) {
  const uint32_t odd = odd_part(j.A), a = bits_of(odd);
  if (j.n == a + 3 && j.n >= 18) return 5ull * odd <= 7ull << (a - 1);
  return j.n >= a + 4 && j.n >= 14;
}

// Staged columns of one residue mod unit (a lane stores four), and the histograms of a
// block of finished rows x cols.
static uint32_t staged_pitch(const CarryPlan& p, uint32_t cols) {
  const uint32_t unit = 1u << p.staged;
  return ((cols + unit - 1 + unit - 1) / unit + 3) / 4 * 4;
}
static size_t staged_cells(const CarryPlan& p, uint32_t rows, uint32_t cols) {
  return (size_t)(rows + (1u << p.staged) - 1) * (staged_pitch(p, cols) << p.staged);
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
    p.side = std::min(p.A, kStageSide - ((1u << p.staged) - 1));
    p.cells = staged_cells(p, p.side, p.side);
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

// Rows of a segment: long runs amortise the 7 to 15 rows a segment computes twice, down
// to 16 where the launch has fewer than want pieces.  A launch that does not fill the GPU
// once with 16 waits for one segment's chain of rows, so it goes on to 4 while it stays
// within one wave of few pieces (folding kernel, a residue with many q: A = 581, k = 21
// 0.31 -> 0.20 ms; quad kernels: A = 867, k = 14 0.046 -> 0.031 ms); more than a wave
// only computes rows again (A = 867, k = 18 0.078 -> 0.102 ms, 256 instances of an 8-bit
// A at k = 16 1.85 -> 2.07 ms; A = 1019, k = 21 0.299 -> 0.310 ms), and a few rows split
// badly (A = 9, k = 22 5.0 -> 6.2 ms).  Half of a block's pieces lie below its diagonal.
static uint32_t rows_per(uint32_t most, uint32_t rows, uint64_t across, uint64_t want, uint64_t few) {
  uint32_t seg = most;
  while (seg > 16 && across * ((rows + seg - 1) / seg) < want) seg /= 2;
  while (seg > 4 && seg <= 16 && rows > 10 && 2 * across * ((rows + seg - 1) / seg) <= few) seg /= 2;
  return seg;
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
          const uint32_t useful = p.staged ? kFoldThreads - ((1u << p.staged) - 1) : (128 - ((1u << p.b) - 1)) / 4 * 4;
          e.strips = (e.cols + useful - 1) / useful;
          // rows per CTA (of the folding kernel; per warp of the others)
          const uint64_t share = std::min<size_t>(std::max<size_t>(alike, 1), kEntries);
          const uint64_t want = std::max<uint64_t>(1, (p.staged ? 8ull : 24ull) * num_sms / share);
          const uint64_t warps = 10ull * num_sms / share;  // one wave of the quad kernels, nearly
          e.seg = rows_per(256, e.rows, e.strips, want, p.staged ? (p.many ? 4ull : 2ull) * num_sms / share : warps);
          e.segs = (e.rows + e.seg - 1) / e.seg;
          e.slices = 1;
          if (p.many) {
            // every slice computes the windows again, so only as many as fill the GPU once
            // (A = 867, k = 21: 0.65 ms with four times as many, 0.32 ms so, with segments of 16)
            const uint64_t per = (e.nq + p.A - 1) / p.A, ctas = (uint64_t)e.strips * e.segs;
            e.slices = (uint32_t)std::min<uint64_t>(std::min<uint64_t>(per, 4096), std::max<uint64_t>(1, want / 4 / ctas));
            // a lane's 32-bit sums: rows x warps (x one lane) x q pairs x 4^b
            const uint64_t sum = (uint64_t)e.seg * (kFoldThreads / 32) * ((per + e.slices - 1) / e.slices) * per << (2 * p.b);
            e.wide = per > 4096 || sum > 0xFFFFFFFFull;
          }
          const size_t need = p.staged ? staged_cells(p, e.rows, e.cols) : 0;
          if (b.n == kEntries || (b.n && used + need > cells)) {
            const cudaError_t err = run_batch(b, levels, many != 0, stream);
            if (err != cudaSuccess) return err;
            b.n = 0;
            used = 0;
          }
          if (p.staged) {
            e.unit = 1u << p.staged;
            e.srows = e.rows + e.unit - 1;
            e.scols = e.cols + e.unit - 1;
            e.pitch = staged_pitch(p, e.cols);
            e.st16 = st16 + used;
            e.st8 = st8 + used;
            used += need;
            const uint32_t wr = (e.srows + e.unit - 1) / e.unit, su = quad_useful<4>();
            e.stage_strips = (e.pitch + su - 1) / su;
            e.stage_seg = rows_per(128, wr, (uint64_t)e.stage_strips * e.unit * e.unit, want * 3 / 2, warps);
            e.stage_segs = (wr + e.stage_seg - 1) / e.stage_seg;
          }
          const CarryEntry* before = b.n ? &b.e[b.n - 1] : nullptr;
          const uint32_t ctas = e.strips * e.segs * e.slices;
          e.fold_end = (before ? before->fold_end : 0) + (p.staged ? ctas : (ctas + kQuadWarps - 1) / kQuadWarps);
          e.stage_end = (before ? before->stage_end : 0) +
                        (e.stage_strips * e.stage_segs * e.unit * e.unit + kQuadWarps - 1) / kQuadWarps;
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

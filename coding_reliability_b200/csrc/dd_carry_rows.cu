// dd_carry_rows.cu — exact 1-D grid histograms (lattice rows x every codeword)
// through residues of the columns.
//
// As in dd_carry.cu a codeword is its low k bits t with the high word c = -t 2^-k
// mod A, and distances add up over t and c.  A grid pairs m given rows (t, c) with all
// 2^k columns t'.  The window here is the top kB bits of t': t' = e' + 2^(k-kB) r',
// e' in [0, 2^(k-kB)).  In the column coordinate u' = 2^-(k-kB) t' mod A the window
// moves by r', and the high word is -2^-kB u' mod A; e' = 2^(k-kB) u' mod A, plus
// multiples of A, are the columns of residue u'.  For a row with t = e + 2^(k-kB) r
//     T = sum over u' of G(u') sum over its e' of z^popc(e ^ e'),
//     G(u') = sum over r' of z^popc(r ^ r') z^popc(c ^ c(u' + r')),
// and kB steps build G for all u': H'(u') = H(u') + z H(u' + s), s = 2^j, with the two
// exchanged where bit j of r is set.  So a row costs about 8 A steps, not 2^k pairs.
//
// Rows with a power-of-two stride 2^j come in blocks that share e and take every r
// once: the two rows that differ in one bit of r are added up before the next step,
// H' = lo(u') + z lo(u'+s) + hi(u'+s) + z hi(u'), a tree whose steps halve in number
// from level to level, so that a block of 64 rows costs about 64 first levels.
//
// Measured on B200 against the tcgen05 kernel: A = 62307, k = 24, m = 65536 14.8 ms
// against 126 ms, A = 867 0.35 against 116 ms; listed rows: A = 867, k = 24, m = 10001
// 0.43 against 18.7 ms, A = 62307, m = 1001 1.65 against 3.4 ms.  Bound by instruction
// issue, as the exhaustive form; DRAM carries nothing.
//
// Thread = column residue; the neighbour u' + s comes through shared memory.  The
// last 2^kB - 1 threads of a CTA only feed their neighbours.
#include <algorithm>
#include <type_traits>

#include "dd_carry.cuh"
#include "dd_device.cuh"

namespace dd {
namespace {

constexpr uint32_t kRowsMaxBits = 32;

struct RowsArgs {
  uint32_t A, k;
  uint32_t psi;              // high word of column u': psi * u' mod A
  uint32_t einv;             // first e' of column u': einv * u' mod A
  uint32_t ne;               // 2^(k-kB)
  uint32_t per;              // e' of a residue that one CTA takes (blockIdx.z: which ones)
  uint32_t seg;              // rows (blocks of rows) per CTA
  uint32_t stride_log;       // tree: rows are the multiples of 2^stride_log
  uint32_t uinv;             // tree: u of block q: uinv * q mod A
  uint64_t rows;             // rows (list), blocks (tree)
  uint64_t mult;             // list: odd part of the multiplier, 64-bit product with the lattice point
  double step;               // list: lattice point i is (uint64)(i * step)
  uint32_t shift[17];        // shift[L] = psi * 2^(kB-L) mod A (ring: 2^(b-L) mod A)
  uint32_t b, groups;        // ring: window bits, rows side by side in a CTA
  unsigned long long* bins;
};

// Window bits, threads and histogram types of the two forms.  A window of the tree
// counts 4^L pairs after L levels, one of the list 2^L.
template <bool kTree>
struct Form;
template <>
struct Form<true> {
  static constexpr int kB = 6, kThreads = 512, kExchange = 48;
  template <int L> using H = std::conditional_t<(L <= 4), H8, H16>;
};
template <>
struct Form<false> {
  static constexpr int kB = 8, kThreads = 1024, kExchange = 24;
  template <int L> using H = std::conditional_t<(L <= 7), H8, H16>;  // bin 24 exists at the last level only
};
template <bool kTree>
constexpr int rows_cols() { return Form<kTree>::kThreads + (1 << (Form<kTree>::kB - 1)); }
// Tables, exchange rows, and (many) each thread's counts of the distances 0 .. k - kB between e and e'.
template <bool kTree>
constexpr size_t rows_smem(bool many, uint32_t k) {
  return (size_t)kTabBytes + 2 * Form<kTree>::kExchange * rows_cols<kTree>() +
         (many ? (size_t)(k - Form<kTree>::kB + 1) * Form<kTree>::kThreads * 4 : 0);
}

__device__ __forceinline__ uint32_t add_mod(uint32_t x, uint32_t d, uint32_t A) {
  const uint32_t y = x + d;
  return y >= A ? y - A : y;
}

template <class To, class From>
__device__ __forceinline__ To widened(const From& h) {
  if constexpr (std::is_same_v<To, From>) return h;
  else return widen(h);
}

// A CTA's exchange rows take turns: a row is rewritten two exchanges later, past the
// barrier of the one in between, which follows every read.
struct Exchange {
  uint8_t* rows;
  uint32_t bytes, turn;
  int tid;
  template <class H>
  __device__ __forceinline__ H at(const H& own, int index) {
    uint8_t* row = rows + (turn ? bytes : 0);
    turn ^= 1;
    put(row, tid, own);
    __syncthreads();
    H nb;
    get(row, index, nb);
    return nb;
  }
  template <class H>
  __device__ __forceinline__ H with(const H& own, int s) { return at(own, tid + s); }
};

// Level L of the tree over the rows whose high words are c + (multiples of shift[1..L]).
template <int L>
__device__ __forceinline__ Form<true>::H<L> tree_node(const RowsArgs& a, uint32_t c, uint32_t ca, uint32_t cb,
                                                      Exchange& ex) {
  if constexpr (L == 1) {
    return first_level(c, add_mod(c, a.shift[1], a.A), ca, cb);
  } else {
    using To = Form<true>::H<L>;
    To x;
    auto half = [&](int h) {
      const auto own = tree_node<L - 1>(a, h ? add_mod(c, a.shift[L], a.A) : c, ca, cb, ex);
      const auto nb = ex.with(own, 1 << (Form<true>::kB - L));
      const To o = widened<To>(own), n = widened<To>(nb);
      if (h == 0) x = add_z(o, n);
      else x = add(x, add_z(n, o));
    };
    if constexpr (L <= 2) {
      half(0);
      half(1);
    } else {
#pragma unroll 1
      for (int h = 0; h < 2; ++h) half(h);
    }
    return x;
  }
}

// Level L of one row with window bits r.
template <int L>
__device__ __forceinline__ Form<false>::H<L> list_node(uint32_t c, uint32_t r, uint32_t ca, uint32_t cb, Exchange& ex) {
  constexpr int s = 1 << (Form<false>::kB - L);
  if constexpr (L == 1) {
    const bool set = (r & s) != 0;
    Nibbles same, cross;
    same.count(__popc(c ^ (set ? cb : ca)));
    cross.count(__popc(c ^ (set ? ca : cb)));
    return add_z(same.bytes(), cross.bytes());
  } else {
    using To = Form<false>::H<L>;
    const auto own = list_node<L - 1>(c, r, ca, cb, ex);
    const auto nb = ex.with(own, s);
    const To o = widened<To>(own), n = widened<To>(nb);
    return (r & s) ? add_z(n, o) : add_z(o, n);
  }
}

template <bool kTree, bool kMany>
__global__ void __launch_bounds__(Form<kTree>::kThreads, kTree ? 2 : 1) carry_rows_kernel(RowsArgs a) {
  using F = Form<kTree>;
  constexpr int kUseful = F::kThreads - ((1 << F::kB) - 1);
  constexpr int kCols = F::kThreads + (1 << (F::kB - 1));
  extern __shared__ __align__(16) uint8_t smem[];
  uint32_t* tab = reinterpret_cast<uint32_t*>(smem);
  uint32_t* ed = reinterpret_cast<uint32_t*>(smem + kTabBytes + 2 * F::kExchange * kCols);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (int i = tid; i < kTabRows * 32; i += F::kThreads) tab[i] = 0;
  if constexpr (kMany)
    for (uint32_t i = tid; i < (a.k - F::kB + 1) * F::kThreads; i += F::kThreads) ed[i] = 0;
  Exchange ex{smem + kTabBytes, (uint32_t)(F::kExchange * kCols), 0, tid};
  const uint32_t u = blockIdx.x * kUseful + tid;
  const bool mine = tid < kUseful && u < a.A;
  const uint32_t ca = mul_mod(a.psi, u, a.A), cb = mul_mod(a.psi, u + (1u << (F::kB - 1)), a.A);
  // this thread's e': from e0, at most `per` of them
  const uint64_t first = mul_mod(a.einv, u, a.A) + (uint64_t)blockIdx.z * a.per * a.A;
  const uint32_t e0 = (uint32_t)min(first, (uint64_t)a.ne);
  const uint32_t e1 = (uint32_t)min((uint64_t)a.ne, e0 + (uint64_t)a.per * a.A);
  const uint32_t at = (uint32_t)__cvta_generic_to_shared(tab) + lane * 4u;
  __syncthreads();

  const uint64_t i0 = (uint64_t)blockIdx.y * a.seg, i1 = min(a.rows, i0 + a.seg);
  for (uint64_t i = i0; i < i1; ++i) {
    uint32_t e;
    typename F::template H<F::kB> g;
    if constexpr (kTree) {
      e = (uint32_t)i << a.stride_log;
      const uint32_t c = mul_mod(a.psi, mul_mod(a.uinv, (uint32_t)i % a.A, a.A), a.A);
      g = tree_node<F::kB>(a, c, ca, cb, ex);
    } else {
      const uint64_t y = a.mult * (uint64_t)((double)i * a.step);
      const uint32_t t = (uint32_t)(y & ((1ull << a.k) - 1));
      e = t & (a.ne - 1);
      g = list_node<F::kB>((uint32_t)(y >> a.k), t >> (a.k - F::kB), ca, cb, ex);
    }
    if (mine) {
      if constexpr (!kMany) {
        for (uint32_t p = e0; p < e1; p += a.A) add_hist<kOne>(at + (__popc(e ^ p) << 7), 1, g);
      } else {
        volatile uint32_t* f = ed + tid;
        const uint32_t fa = (uint32_t)__cvta_generic_to_shared(ed + tid);
        for (uint32_t p = e0; p < e1; p += a.A) red_add<0>(fa + __popc(e ^ p) * (F::kThreads * 4), 1);
        for (uint32_t d = 0; d <= a.k - F::kB; ++d) {
          const uint32_t x = f[d * F::kThreads];
          if (x) {
            f[d * F::kThreads] = 0;
            add_hist<kNarrow>(at + (d << 7), x, g);
          }
        }
      }
    }
  }
  __syncthreads();
  for (int d = warp; d < kTabRows; d += F::kThreads / 32) {
    const uint32_t x = tab[d * 32 + lane];
    const unsigned long long t = (unsigned long long)__reduce_add_sync(0xffffffffu, x & 0xFFFFu) +
                                 ((unsigned long long)__reduce_add_sync(0xffffffffu, x >> 16) << 16);
    if (lane == 0 && t) atomicAdd(a.bins + d, t);
  }
}

// Listed rows of a short multiplier: the columns of all A residues fit a CTA, so the
// window closes on itself (no thread only feeds its neighbours) and may be as long as
// b = k - bits(A) bits (at most 16), which leaves about two columns a residue to visit
// instead of 2^(k-8) / A.  Several rows run side by side where A is at most half the CTA.
// A = 867, k = 24, 10,001 rows: 1.35 ms with a window of 8 bits, 0.43 ms.
template <int kThreads>
__global__ void __launch_bounds__(kThreads, 1024 / kThreads) carry_ring_kernel(const __grid_constant__ RowsArgs a) {
  extern __shared__ __align__(16) uint8_t smem[];
  uint32_t* tab = reinterpret_cast<uint32_t*>(smem);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (int i = tid; i < kTabRows * 32; i += kThreads) tab[i] = 0;
  Exchange ex{smem + kTabBytes, 48u * kThreads, 0, tid};
  const uint32_t group = tid / a.A, u = tid - group * a.A, first = group * a.A;
  const uint32_t ca = mul_mod(a.psi, u, a.A), cb = mul_mod(a.psi, u + (1u << (a.b - 1)), a.A);
  const uint32_t e0 = mul_mod(a.einv, u, a.A);
  const uint32_t at = (uint32_t)__cvta_generic_to_shared(tab) + lane * 4u;
  __syncthreads();
  auto next = [&](uint32_t L) {  // thread of the column shift[L] on
    const uint32_t v = u + a.shift[L];
    return (int)min(first + (v >= a.A ? v - a.A : v), (uint32_t)kThreads - 1);
  };
  const uint64_t i0 = (uint64_t)blockIdx.x * a.seg, i1 = min(a.rows, i0 + a.seg);
  for (uint64_t base = i0; base < i1; base += a.groups) {
    const uint64_t i = base + group;
    const uint64_t y = a.mult * (uint64_t)((double)i * a.step);
    const uint32_t t = (uint32_t)(y & ((1ull << a.k) - 1)), c = (uint32_t)(y >> a.k);
    const uint32_t r = t >> (a.k - a.b), e = t & (a.ne - 1);
    Nibbles same, cross;
    const bool set = (r >> (a.b - 1)) & 1;
    same.count(__popc(c ^ (set ? cb : ca)));
    cross.count(__popc(c ^ (set ? ca : cb)));
    H8 h = add_z(same.bytes(), cross.bytes());
    uint32_t L = 2;
#pragma unroll 1
    for (; L <= a.b && L <= 7; ++L) {
      const H8 nb = ex.at(h, next(L));
      h = (r >> (a.b - L)) & 1 ? add_z(nb, h) : add_z(h, nb);
    }
    H16 g = widen(h);
    if (L <= a.b) {
      const H16 nb = widen(ex.at(h, next(L)));
      g = (r >> (a.b - L)) & 1 ? add_z(nb, g) : add_z(g, nb);
#pragma unroll 1
      for (++L; L <= a.b; ++L) {
        const H16 n = ex.at(g, next(L));
        g = (r >> (a.b - L)) & 1 ? add_z(n, g) : add_z(g, n);
      }
    }
    if (group < a.groups && i < i1)
      for (uint32_t p = e0; p < a.ne; p += a.A) add_hist<kOne>(at + (__popc(e ^ p) << 7), 1, g);
  }
  __syncthreads();
  for (int d = warp; d < kTabRows; d += kThreads / 32) {
    const uint32_t x = tab[d * 32 + lane];
    const unsigned long long t = (unsigned long long)__reduce_add_sync(0xffffffffu, x & 0xFFFFu) +
                                 ((unsigned long long)__reduce_add_sync(0xffffffffu, x >> 16) << 16);
    if (lane == 0 && t) atomicAdd(a.bins + d, t);
  }
}

template <int kThreads>
cudaError_t run_ring(const RowsArgs& a, cudaStream_t stream) {
  constexpr int smem = kTabBytes + 2 * 48 * kThreads;
  cudaError_t e = cudaFuncSetAttribute(carry_ring_kernel<kThreads>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return e;
  carry_ring_kernel<kThreads><<<(uint32_t)((a.rows + a.seg - 1) / a.seg), kThreads, smem, stream>>>(a);
  return cudaGetLastError();
}

template <bool kTree, bool kMany>
cudaError_t run_rows(const RowsArgs& a, const RowsPlan& p, cudaStream_t stream) {
  using F = Form<kTree>;
  constexpr uint32_t useful = F::kThreads - ((1 << F::kB) - 1);
  const size_t smem = rows_smem<kTree>(kMany, a.k);
  auto fn = carry_rows_kernel<kTree, kMany>;
  // process-wide, so every caller sets the same limit: that of the longest k
  cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)rows_smem<kTree>(kMany, kRowsMaxBits));
  if (e != cudaSuccess) return e;
  const dim3 grid((a.A + useful - 1) / useful, (uint32_t)((a.rows + a.seg - 1) / a.seg), p.slices);
  fn<<<grid, F::kThreads, smem, stream>>>(a);
  return cudaGetLastError();
}

}  // namespace

bool rows_plan(const Job& j, int num_sms, RowsPlan& p) {
  p = RowsPlan();
  if (j.kind != JOB_PAIRS || j.shape != SHAPE_RECT || j.row_kind != ROW_LATTICE || j.col_kind != COL_PROGRESSION ||
      j.tile_offset != 0 || j.cols != 1ull << j.n || j.A == 0 || (j.A >> 32) || j.n < 12 || j.n > kRowsMaxBits || j.rows == 0 ||
      j.rows > j.cols)
    return false;
  p.A = odd_part(j.A);
  const uint32_t bits = bits_of(p.A);
  if (bits > 16) return false;
  // power-of-two stride: every multiple of it below 2^n is a row
  const double stride = j.row_step;
  const uint64_t st = stride >= 1 && stride < 4294967296.0 ? (uint64_t)stride : 0;
  p.tree = st && (double)st == stride && (st & (st - 1)) == 0 && j.rows == j.cols / st &&
           j.rows >= 1u << Form<true>::kB;
  if (!p.tree && p.A <= 1024 && j.n <= 24 && j.n > bits + 1) {
    // one wave of CTAs (two of 512 threads or one of 1024 an SM); a lane's column adds
    // the residue's columns x 2^16 a round of rows and warp (of 32), below 2^32
    p.ring = std::min<uint32_t>(16, j.n - bits);
    p.rows = j.rows;
    const uint32_t threads = p.A <= 512 ? 512 : 1024;
    p.groups = threads / p.A;
    const uint64_t ctas = (uint64_t)num_sms * (1024 / threads);
    const uint64_t columns = ((1ull << (j.n - p.ring)) + p.A - 1) / p.A;  // at most 256
    const uint64_t rounds = std::min<uint64_t>(2047 / columns, (p.rows + p.groups * ctas - 1) / (p.groups * ctas));
    p.seg = (uint32_t)rounds * p.groups;
    return true;
  }
  const uint32_t kb = p.tree ? Form<true>::kB : Form<false>::kB;
  while (p.tree && (1ull << p.stride_log) < st) ++p.stride_log;
  const uint64_t ne = 1ull << (j.n - kb), most = (ne + p.A - 1) / p.A;
  p.rows = p.tree ? j.rows >> kb : j.rows;
  p.slices = (uint32_t)((most + 4095) / 4096);
  if (p.slices > 65535) return false;
  p.per = (uint32_t)((most + p.slices - 1) / p.slices);
  p.many = p.per > 16;
  // rows per CTA: few enough to fill the GPU, and for a table's 32-bit sums (a lane's
  // column is shared by the CTA's warps; a row adds per * 4^kb, or per * 2^kb, a thread)
  const uint64_t threads = p.tree ? Form<true>::kThreads : Form<false>::kThreads;
  const uint64_t useful = threads - ((1u << kb) - 1), strips = (p.A + useful - 1) / useful;
  const uint64_t row_sum = (threads / 32) * p.per * (p.tree ? 1ull << (2 * kb) : 1ull << kb);
  const uint64_t bound = 0xFFFFFFFFull / row_sum;  // at least 15: per <= 4096
  uint64_t seg = p.tree ? 8 : 256;
  while (seg > 1 && strips * ((p.rows + seg - 1) / seg) * p.slices < 8ull * num_sms) seg /= 2;
  while ((p.rows + seg - 1) / seg > 65535) seg *= 2;
  seg = std::min(seg, bound);
  p.seg = (uint32_t)seg;
  return (p.rows + seg - 1) / seg <= 65535;
}

// The tree's residue pairs cost about as much as 30 codeword pairs of the tcgen05 kernel
// (A = 62307, m = 65536: k = 21, 34 a residue, 13.9 ms here and 15.8 ms there; k = 20,
// 13.9 and 7.9 ms), the list's about 170 (m = 10007: A = 62307, k = 22, 67 a residue,
// 13.8 and 5.2 ms; A = 8191, 512 a residue, 2.3 and 4.7 ms), the ring's as many (A = 867,
// m = 10001: k = 18, 302 a residue, 0.26 and 0.34 ms; k = 17, 0.23 and 0.19 ms); below 2^28 pairs the popc
// kernel's single launch is as fast.
// The shortest A leave most of a CTA without a residue, and a thread visits its columns one
// by one.  A tree's CTA of 4096 columns a residue takes 0.12 ms however few its rows, as
// long as the popc kernel takes for 2^29 pairs in whole row tiles (m = 128, k = 21: A = 13,
// 2521 columns, 0.086 and 0.080 ms, A = 15 0.075; k = 18, m = 1024, A = 1 0.121 and 0.081).
// A listed row past the ring's k takes A = 1 22 us at k = 25, A = 3 7.7, A = 5 4.4 and A = 7
// 3.3, the tcgen05 kernel 1.7 ms for up to 128 rows and 3.1 us for each more: as long with
// 72 rows at A = 1, 300 at A = 3, 550 at A = 5.
bool rows_win(const Job& j, const RowsPlan& p) {
  const double pairs = (double)j.rows * (double)j.cols;
  if (pairs < 268435456.0 || j.cols < (uint64_t)p.A * (p.tree ? 32 : p.ring ? 192 : 256)) return false;
  if (p.tree) return p.per <= 2300 || j.rows < 128 || pairs >= 536870912.0;
  return p.ring || p.A >= 7 || j.rows <= 120ull * p.A - 45;
}

cudaError_t launch_rows(const Job& j, const RowsPlan& p, cudaStream_t stream) {
  const uint32_t kb = p.ring ? p.ring : p.tree ? Form<true>::kB : Form<false>::kB;
  RowsArgs a{};
  a.A = p.A;
  a.k = j.n;
  a.psi = (p.A - inverse_pow2(kb, p.A)) % p.A;
  a.ne = 1u << (j.n - kb);
  a.einv = (uint32_t)(a.ne % p.A);
  a.per = p.per;
  a.seg = p.seg;
  a.rows = p.rows;
  a.mult = p.A;
  a.step = j.row_step;
  a.stride_log = p.stride_log;
  // block q: e = 2^stride_log q, u = 2^-(k-kb) e
  a.uinv = inverse_pow2(j.n - kb - (p.tree ? p.stride_log : 0), p.A);
  for (uint32_t L = 1; L <= kb; ++L) {
    const uint64_t s = (1ull << (kb - L)) % p.A;
    a.shift[L] = (uint32_t)(p.ring ? s : a.psi * s % p.A);
  }
  a.bins = j.bins;
  if (p.ring) {
    a.b = p.ring;
    a.groups = p.groups;
    return p.A <= 512 ? run_ring<512>(a, stream) : run_ring<1024>(a, stream);
  }
  if (p.tree) return p.many ? run_rows<true, true>(a, p, stream) : run_rows<true, false>(a, p, stream);
  return p.many ? run_rows<false, true>(a, p, stream) : run_rows<false, false>(a, p, stream);
}

}  // namespace dd

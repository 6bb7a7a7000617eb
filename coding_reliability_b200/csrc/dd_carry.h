// dd_carry.h — AN histograms through residues: exhaustive (dd_carry.cu), 1-D grids (dd_carry_rows.cu).
#pragma once
#include <cuda_runtime.h>
#include <cstddef>
#include <cstdint>
#include <vector>

#include "dd_jobs.h"

namespace dd {

// One job as the carry kernels run it.
struct CarryPlan {
  uint32_t A = 0;       // odd part of the multiplier
  uint32_t k = 0;       // data bits
  uint32_t b = 0;       // window bits: levels of the pair recursion
  uint32_t s = 0;       // k - b: bits enumerated at the end
  uint32_t staged = 0;  // levels the staging kernel computes (b - 4 when b > 4, else 0)
  uint32_t psi = 0;     // high word of t: psi * t mod A
  uint32_t qinv = 0;    // first q of residue v: qinv * v mod A
  uint32_t many = 0;    // a residue has more than two q
  uint32_t side = 0;    // residues per side of a block
  size_t cells = 0;     // staged histograms of one block
};

// AN exhaustive jobs over the whole instance, A's odd part of at most 16 bits, k <= 24.
bool carry_eligible(const Job& j);
// The rule that picks this path for an eligible job under AUTO.
bool carry_wins(const Job& j);
void carry_plan(const Job& j, CarryPlan& p);
// Bytes of staging memory that serve any launch of these plans (0: none).
size_t carry_stage_bytes(const std::vector<CarryPlan>& plans);
// Enqueues the jobs' kernels: job i's sums are added to acc + i * 2 * kMaxBins (zeroed
// by the caller).
cudaError_t launch_carry(const std::vector<CarryPlan>& plans, int num_sms, unsigned long long* acc, void* stage,
                         size_t stage_bytes, cudaStream_t stream);
// acc of n jobs (2 x kMaxBins each) -> their bins; jobs: the device's table entries.
cudaError_t launch_carry_finish(const Job* jobs, const unsigned long long* acc, uint32_t n, cudaStream_t stream);

// One 1-D grid job as carry_rows_kernel or carry_ring_kernel runs it.
struct RowsPlan {
  uint32_t A = 0;           // odd part of the multiplier
  uint32_t tree = 0;        // rows with a power-of-two stride, in blocks
  uint32_t stride_log = 0;  // tree: log2 of the stride
  uint32_t ring = 0;        // window bits of carry_ring_kernel (0: carry_rows_kernel)
  uint32_t groups = 0;      // ring: rows side by side
  uint32_t many = 0;        // a residue stands for more columns than are worth visiting one by one
  uint32_t per = 0;         // columns of a residue per CTA
  uint32_t slices = 1;      // CTAs that share a residue's columns
  uint32_t seg = 0;         // rows (blocks) per CTA
  uint64_t rows = 0;        // rows (list) or blocks of rows (tree)
};
// False where the job is no 1-D grid this path runs (whole instances, A's odd part of
// at most 16 bits, 12 <= n <= 32).
bool rows_plan(const Job& j, int num_sms, RowsPlan& p);
// The rule that picks this path under AUTO.
bool rows_win(const Job& j, const RowsPlan& p);
// Adds the job's histogram to its (zeroed) bins.
cudaError_t launch_rows(const Job& j, const RowsPlan& p, cudaStream_t stream);

}  // namespace dd

"""What happens to a residue-route instance whose bins lack pairs: the host rules
(dd_rules.cpp, no CUDA) compiled with a driver that stands in for the kernels.  Only the
short instances are computed again, on a pair kernel and with their own requests; the other
results stay as they are; the times of a recounted one are those of both passes; an error
of the second pass is the call's."""
import shutil
import subprocess

import pytest

from conftest import ROOT

CSRC = ROOT / "coding_reliability_b200" / "csrc"

DRIVER = r"""
#include <cstdio>
#include <cstring>
#include "dd_host.h"
namespace dd { void set_error(const std::string&) {} }
using namespace dd;
#define CHECK(x) do { if (!(x)) { std::printf("line %d: %s\n", __LINE__, #x); return 1; } } while (0)
int main() {
  // totals: exact, one pair short, a byte's and a half word's overflow, above 2^64
  uint64_t raw[kMaxBins] = {0};
  raw[1] = 5; raw[40] = 7; raw[63] = 1;
  CHECK(holds_all_pairs(raw, 13));
  CHECK(!holds_all_pairs(raw, 14) && !holds_all_pairs(raw, 12));
  raw[2] = 1000;
  CHECK(holds_all_pairs(raw, 1013));
  raw[2] -= 255;
  CHECK(!holds_all_pairs(raw, 1013));
  raw[2] += 255; raw[3] = 1 << 20;
  raw[3] -= 65535;
  CHECK(!holds_all_pairs(raw, 1013 + (1 << 20)));
  uint64_t big[kMaxBins] = {0};
  big[7] = big[8] = ~0ull;
  CHECK(holds_all_pairs(big, ((u128)1 << 65) - 2) && !holds_all_pairs(big, ~(uint64_t)0 - 1));

  dd_request reqs[4];
  dd_result res[4], before[4];
  std::memset(reqs, 0, sizeof(reqs));
  std::memset(res, 0, sizeof(res));
  for (uint32_t i = 0; i < 4; ++i) {
    reqs[i].A = 101 + 2 * i;
    reqs[i].n = 14;
    reqs[i].kernel = i == 3 ? DD_KERNEL_CARRY : DD_KERNEL_AUTO;
    reqs[i].user_tag = 70 + i;
    res[i].kernel_used = DD_KERNEL_CARRY;
    res[i].kernel_ms = 2.0;
    res[i].total_ms = 3.0;
    res[i].raw[5] = 900 + i;
  }
  std::memcpy(before, res, sizeof(res));
  std::vector<uint64_t> seen;
  auto run = [&](const dd_request& q, dd_result& r) {
    seen.push_back(q.A);
    if (q.kernel != DD_KERNEL_MMA || q.n != 14) return (int)DD_ERR_INVALID_ARGUMENT;
    std::memset(&r, 0, sizeof(r));
    r.kernel_used = q.kernel;
    r.user_tag = q.user_tag;
    r.raw[5] = 10 * q.A;
    r.kernel_ms = 40.0;
    r.total_ms = 50.0;
    return (int)DD_OK;
  };
  CHECK(recount(reqs, res, {}, run) == DD_OK && seen.empty() && !std::memcmp(before, res, sizeof(res)));
  CHECK(recount(reqs, res, {1, 3}, run) == DD_OK);
  CHECK((seen == std::vector<uint64_t>{103, 107}));
  for (uint32_t i = 0; i < 4; ++i) {
    if (i % 2 == 0) {
      CHECK(!std::memcmp(&before[i], &res[i], sizeof(res[i])));
      continue;
    }
    CHECK(res[i].kernel_used == DD_KERNEL_MMA && res[i].user_tag == 70 + i && res[i].raw[5] == 10 * reqs[i].A);
    CHECK(res[i].kernel_ms == 42.0 && res[i].total_ms == 53.0);
    CHECK(reqs[i].kernel == (i == 3 ? DD_KERNEL_CARRY : DD_KERNEL_AUTO));
  }
  seen.clear();
  auto fail = [&](const dd_request& q, dd_result&) { seen.push_back(q.A); return (int)DD_ERR_TIMEOUT; };
  CHECK(recount(reqs, res, {0, 2}, fail) == DD_ERR_TIMEOUT && seen.size() == 1);
  std::puts("ok");
  return 0;
}
"""


@pytest.mark.skipif(not shutil.which("g++"), reason="needs g++")
def test_recount(tmp_path):
    src, exe = tmp_path / "driver.cpp", tmp_path / "driver"
    src.write_text(DRIVER)
    subprocess.run(["g++", "-std=c++17", "-O1", f"-I{CSRC}", str(src), str(CSRC / "dd_rules.cpp"), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.stdout.strip() == "ok" and out.returncode == 0, out.stdout

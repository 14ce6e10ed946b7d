// The choice of rays of the binary pass after a wide one (TEST INFRASTRUCTURE ONLY): every entry
// gives its ray, and an index past the batch is flagged and left out.
#include <cstdio>
#include <vector>

#include "layout.h"
#include "trace_core.cuh"

int main() {
  const uint32_t n = 1000;
  std::vector<uint32_t> perm(n);
  for (uint32_t i = 0; i < n; ++i) perm[i] = n - 1 - i;
  const uint32_t unc[4] = {0, 999, 1000, 0xFFFFFFFFu}, redo[3] = {5, 7777777, 999};
  int bad = 0;
  auto expect = [&](uint32_t idx, uint32_t rays, bool scan, const uint32_t *p, uint32_t want,
                    bool flagged) {
    uint32_t err = 0;
    const uint32_t got = bzr::handed_on_ray(idx, rays, scan, unc, redo, p, n, &err);
    if (got != want || err != (flagged ? bzr::kErrRayIndex : 0u)) {
      std::printf("entry %u of %u (scan %d): %u, error word %u\n", idx, rays, scan, got, err);
      ++bad;
    }
  };
  expect(0, 4, false, nullptr, 0, false);
  expect(1, 4, false, perm.data(), 999, false);
  expect(2, 4, false, nullptr, bzr::kNoRay, true);   // one past the batch
  expect(3, 4, false, nullptr, bzr::kNoRay, true);
  expect(4, 4, false, nullptr, 5, false);
  expect(5, 4, false, nullptr, bzr::kNoRay, true);   // of a larger batch
  expect(6, 4, false, nullptr, 999, false);
  expect(0, 0, false, nullptr, 5, false);            // none uncovered
  expect(999, n, true, nullptr, 999, false);
  expect(0, n, true, perm.data(), 999, false);
  expect(n, n, true, nullptr, 5, false);
  expect(n + 1, n, true, perm.data(), bzr::kNoRay, true);
  return bad;
}

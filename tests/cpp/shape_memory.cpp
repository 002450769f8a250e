// The memory of shape sets over fake_cudart.cpp: what the library's C entries do to the device's memory and in
// which order. Prints "ok" or what went wrong.
#include <algorithm>
#include <cstdio>
#include <cstring>
#include <string>
#include <vector>

#include "../../include/curvami_gb300.h"

namespace fake {
extern std::vector<std::string> log;
extern size_t limit, held, idle, peak;
}  // namespace fake

#define CHECK(x) do { if (!(x)) { std::printf("line %d: %s (%s)\n", __LINE__, #x, cgb_last_error(ctx)); return 1; } } while (0)

// A wait for all work on the device.
static bool waits(const std::string& s) { return s == "cudaFree" || s == "cudaDeviceSynchronize"; }

int main(int argc, char** argv) {
  const std::string what = argc > 1 ? argv[1] : "";
  cgb_context* ctx = nullptr;
  if (cgb_create(0, &ctx) != CGB_OK) return 2;
  std::vector<double> xy;
  for (int i = 0; i < 400; ++i) { xy.push_back(i % 20); xy.push_back(i / 20); }
  CHECK(cgb_set_nodes(ctx, xy.data(), 400) == CGB_OK);
  const int n = 1000;
  std::vector<int64_t> ptr(n + 1);
  std::vector<int32_t> idx(4 * n, 7);
  std::vector<double> v(12 * n, 1.0);
  for (int g = 0; g <= n; ++g) ptr[g] = 4 * g;
  cgb_shape* sh = nullptr;
  auto first_after = [](size_t at, auto&& is) {
    return std::find_if(fake::log.begin() + at, fake::log.end(), is) - fake::log.begin();
  };
  auto given = [](const std::string& s) { return s == "cudaFreeAsync"; };

  if (what == "failed_set") {   // no room for the last array: the copies into the others may be in flight
    const size_t all = 8 * (n + 1) + 4 * 4 * n + 8 * 4 * n * 6;
    fake::limit = fake::held + all - 8;
    fake::log.clear();
    CHECK(cgb_shape_from_host(ctx, n, ptr.data(), idx.data(), v.data(), v.data(), v.data(), &sh) == CGB_ERR_CUDA);
    size_t copy = 0;
    for (size_t k = 0; k < fake::log.size(); ++k) if (fake::log[k] == "cudaMemcpyAsync") copy = k;
    const size_t wait = first_after(copy, waits), free_at = first_after(copy, given);
    CHECK(free_at < fake::log.size());
    CHECK(wait < free_at);
  } else if (what == "destroy") {   // waits, but not with a call that another thread's capture forbids
    CHECK(cgb_shape_from_host(ctx, n, ptr.data(), idx.data(), v.data(), v.data(), v.data(), &sh) == CGB_OK);
    fake::log.clear();
    CHECK(cgb_shape_destroy(sh) == CGB_OK);
    CHECK(std::find(fake::log.begin(), fake::log.end(), "cudaDeviceSynchronize") == fake::log.end());
    CHECK(first_after(0, waits) < first_after(0, given));
  } else if (what == "room" || what == "scratch" || what == "trim") {
    const int np = 200000;
    std::vector<double> pts(2 * np, 5.5);
    cgb_shape_params prm;
    std::memset(&prm, 0, sizeof(prm));
    prm.rho = 3.0;
    prm.order = 2;
    const size_t small = fake::held, scratch = size_t(np) * (90 + 36) * 8;   // moment sums and polynomials
    CHECK(cgb_shape_build(ctx, pts.data(), np, &prm, nullptr, 0, &sh) == CGB_OK);
    const size_t peak = fake::peak;
    CHECK(peak > small + scratch);
    CHECK(cgb_shape_destroy(sh) == CGB_OK);
    if (what == "room") {   // other arrays find the room that destroyed sets and the scratch had
      fake::limit = fake::held;
      std::vector<double> more(2000000, 1.0);
      CHECK(cgb_set_nodes(ctx, more.data(), 1000000) == CGB_OK);
    } else {
      CHECK(cgb_trim(ctx) == CGB_OK);
      CHECK(fake::idle == 0 && fake::held < small + (8u << 20));
      if (what == "scratch") {    // fewer points at a time
        fake::limit = peak - scratch / 3;
        CHECK(cgb_shape_build(ctx, pts.data(), np, &prm, nullptr, 0, &sh) == CGB_OK);
        CHECK(cgb_shape_destroy(sh) == CGB_OK);
      }
    }
  } else {
    std::printf("unknown\n");
    return 2;
  }
  cgb_destroy(ctx);
  CHECK(fake::held == 0);
  std::printf("ok\n");
  return 0;
}

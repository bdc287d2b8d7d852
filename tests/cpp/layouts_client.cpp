/*
 * layouts_client.cpp - decodes the frames of layouts.hpp through the C API on
 * the GPU, each as it is planned (by regions, where the planner gives them)
 * and traced (by chains and done flags), and compares the planes (test
 * infrastructure). Prints "ok" at the end; exits non-zero on a difference or
 * an error.
 */
#include <cstdio>

#include "layouts.hpp"

static int decode(av1b_decoder* d, const LayoutFrame& f, bool traced, std::vector<uint16_t> (&planes)[3]) {
  if (av1b_set_unit_trace(d, traced ? 1 : 0)) return -1;
  av1b_planes out;
  for (int p = 0; p < 3; ++p) {
    const int w = p ? (f.width + f.ss_x) >> f.ss_x : f.width, h = p ? (f.height + f.ss_y) >> f.ss_y : f.height;
    planes[p].assign(static_cast<size_t>(w) * h, 0);
    out.plane[p] = planes[p].data();
    out.stride[p] = w;
  }
  const av1b_frame_syntax s = f.syntax();
  char error[256] = "";
  const int rc = av1b_decode(d, &s, 0, &out, nullptr, error, sizeof(error));
  if (rc) std::printf("%s: %d %s\n", f.name.c_str(), rc, error);
  return rc;
}

int main() {
  av1b_decoder* d = nullptr;
  if (av1b_decoder_create(0, 0, &d)) return 1;
  int bad = 0;
  for (int i = 0; i < layout_count(); ++i) {
    const LayoutFrame f = layout_frame(i);
    std::vector<uint16_t> a[3], b[3];
    if (decode(d, f, false, a) || decode(d, f, true, b)) {
      ++bad;
      continue;
    }
    for (int p = 0; p < 3; ++p)
      if (a[p] != b[p]) {
        std::printf("%s %d: plane %d differs\n", f.name.c_str(), i, p);
        ++bad;
      }
  }
  av1b_decoder_destroy(d);
  if (bad) return 1;
  std::printf("ok\n");
  return 0;
}

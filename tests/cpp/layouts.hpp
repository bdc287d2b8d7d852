/*
 * layouts.hpp - hand-made and random intra frames whose block layouts and
 * coding orders no encoder's partition tree gives, all of them valid input of
 * the API: any block of 2 to 64 samples a side at any place, in any order
 * (test infrastructure).
 *
 * Blocks tile every plane; a block reads its left column, above row and
 * corner only where all of them were coded before it, so that the picture
 * does not depend on anything but the layout. Each has one transform of its
 * size, most of them.
 */
#ifndef AV1B_TEST_LAYOUTS_HPP
#define AV1B_TEST_LAYOUTS_HPP

#include <algorithm>
#include <cstdint>
#include <cstring>
#include <string>
#include <vector>

#include "../../include/av1b.h"

struct LayoutFrame {
  std::string name;
  int width = 0, height = 0, bit_depth = 8, ss_x = 1, ss_y = 1;
  std::vector<av1b_block> blocks;
  std::vector<av1b_transform> transforms;
  std::vector<int32_t> coefficients;

  av1b_frame_syntax syntax() const {
    av1b_frame_syntax s;
    std::memset(&s, 0, sizeof(s));
    s.width = width;
    s.height = height;
    s.bit_depth = bit_depth;
    s.ss_x = ss_x;
    s.ss_y = ss_y;
    s.base_q_idx = 100;
    s.enable_intra_edge_filter = 1;
    s.blocks = blocks.data();
    s.n_blocks = blocks.size();
    s.transforms = transforms.data();
    s.n_transforms = transforms.size();
    s.coefficients = coefficients.data();
    s.n_coefficients = coefficients.size();
    return s;
  }
};

class LayoutBuilder {
 public:
  LayoutBuilder(const std::string& name, int w, int h, int bit_depth, int ss_x, int ss_y, uint64_t seed) : seed_(seed) {
    f_.name = name;
    f_.width = w;
    f_.height = h;
    f_.bit_depth = bit_depth;
    f_.ss_x = ss_x;
    f_.ss_y = ss_y;
    for (int p = 0; p < 3; ++p) {
      gw_[p] = p ? ((w + 7) & ~7) >> ss_x : (w + 7) & ~7;
      gh_[p] = p ? ((h + 7) & ~7) >> ss_y : (h + 7) & ~7;
      done_[p].assign(static_cast<size_t>(gw_[p]) * gh_[p], 0);
    }
  }

  int gw(int p) const { return gw_[p]; }
  int gh(int p) const { return gh_[p]; }
  int pick(int lo, int hi) {
    seed_ = seed_ * 6364136223846793005ull + 1442695040888963407ull;
    return lo + static_cast<int>((seed_ >> 33) % static_cast<uint64_t>(hi - lo + 1));
  }

  /* The next block in coding order; mode -1: any but chroma from luma. */
  void block(int plane, int x, int y, int w, int h, int mode = -1) {
    av1b_block b;
    std::memset(&b, 0, sizeof(b));
    b.plane = plane;
    b.x = x;
    b.y = y;
    b.w = w;
    b.h = h;
    b.bit_depth = f_.bit_depth;
    b.is_intra = 1;
    b.mode = mode >= 0 ? mode : (pick(0, 2) ? pick(1, 8) : pick(0, 12));
    if (b.mode >= 1 && b.mode <= 8) b.angle_delta = pick(-3, 3);
    b.cfl_alpha = b.mode == 13 ? pick(-16, 16) : 0;
    const bool corner = x == 0 || y == 0 || at(plane, x - 1, y - 1);
    bool left = x > 0, above = y > 0;
    for (int k = 0; left && k < h && y + k < gh_[plane]; ++k) left = at(plane, x - 1, y + k);
    for (int k = 0; above && k < w && x + k < gw_[plane]; ++k) above = at(plane, x + k, y - 1);
    b.have_left = left && (!above || corner);
    b.have_above = above && (!left || corner);
    b.have_above_right = b.have_below_left = -1;
    b.ref[0] = b.ref[1] = -1;
    b.tx_first = static_cast<int32_t>(f_.transforms.size());
    if (w >= 4 && h >= 4 && pick(0, 4)) {
      av1b_transform t;
      std::memset(&t, 0, sizeof(t));
      t.w = w;
      t.h = h;
      t.denominator = 1;
      t.qm_off = -1;
      t.coef_offset = static_cast<int32_t>(f_.coefficients.size());
      t.eob = 3;
      const int cw = std::min(w, 32), ch = std::min(h, 32);
      f_.coefficients.resize(f_.coefficients.size() + static_cast<size_t>(cw) * ch, 0);
      int32_t* c = f_.coefficients.data() + t.coef_offset;
      c[0] = pick(-400, 400);
      c[1] = pick(-200, 200);
      c[cw] = pick(-200, 200);
      f_.transforms.push_back(t);
      b.tx_count = 1;
    }
    f_.blocks.push_back(b);
    for (int yy = y; yy < std::min(y + h, gh_[plane]); ++yy)
      for (int xx = x; xx < std::min(x + w, gw_[plane]); ++xx) done_[plane][static_cast<size_t>(yy) * gw_[plane] + xx] = 1;
  }

  /* The plane's samples not coded yet, in blocks of w x h from (x0, y0) on,
   * row by row. */
  void fill(int plane, int x0, int y0, int x1, int y1, int w, int h, int mode = -1) {
    for (int y = y0; y < y1; y += h)
      for (int x = x0; x < x1; x += w)
        if (!at(plane, x, y)) block(plane, x, y, w, h, mode);
  }
  void chroma() { chroma(0, 0, f_.width, f_.height); }
  /* the chroma of [x0, x1) x [y0, y1) of luma */
  void chroma(int x0, int y0, int x1, int y1, int mode = -1) {
    for (int p = 1; p < 3; ++p)
      fill(p, x0 >> f_.ss_x, y0 >> f_.ss_y, std::min(gw_[p], x1 >> f_.ss_x), std::min(gh_[p], y1 >> f_.ss_y), 16, 16,
           mode);
  }

  /* A random tiling of [x, x + w) x [y, y + h): split in two, in either
   * order, or a block. */
  void random(int plane, int x, int y, int w, int h, int least) {
    if (x >= gw_[plane] || y >= gh_[plane]) return;
    const bool inside = x + w <= gw_[plane] && y + h <= gh_[plane];
    const bool fits = w <= 64 && h <= 64 && std::max(w, h) <= 4 * std::min(w, h);
    if (fits && (inside || std::max(w, h) <= least) && (std::max(w, h) <= least || pick(0, 2) == 0)) {
      block(plane, x, y, w, h);
      return;
    }
    const bool across = w > least && (h <= least || (w > h ? pick(0, 3) > 0 : pick(0, 3) == 0));
    const bool back = pick(0, 5) == 0;
    for (int k = 0; k < 2; ++k) {
      const int q = back ? 1 - k : k;
      if (across) random(plane, x + q * (w / 2), y, w / 2, h, least);
      else random(plane, x, y + q * (h / 2), w, h / 2, least);
    }
  }

  LayoutFrame take() { return std::move(f_); }

 private:
  bool at(int p, int x, int y) const { return done_[p][static_cast<size_t>(y) * gw_[p] + x] != 0; }

  LayoutFrame f_;
  uint64_t seed_;
  int gw_[3], gh_[3];
  std::vector<uint8_t> done_[3];
};

static const int kHandLayouts = 7, kRandomLayouts = 60;
inline int layout_count() { return kHandLayouts + kRandomLayouts; }

inline LayoutFrame layout_frame(int i) {
  if (i >= kHandLayouts) {
    static const int kSs[3][2] = {{1, 1}, {1, 0}, {0, 0}};
    const int k = i - kHandLayouts;
    const int* ss = kSs[k % 3];
    LayoutBuilder b("random", 64 + 40 * (k % 5), 72 + 56 * (k % 3), k % 2 ? 10 : 8, ss[0], ss[1],
                    1000 + static_cast<uint64_t>(k));
    const int side = k % 4 == 0 ? 128 : 64;
    for (int y = 0; y < b.gh(0); y += side)
      for (int x = 0; x < b.gw(0); x += side)
        for (int p = 0; p < 3; ++p) {
          const int sx = p ? ss[0] : 0, sy = p ? ss[1] : 0;
          b.random(p, x >> sx, y >> sy, side >> sx, side >> sy, 8);
        }
    return b.take();
  }
  switch (i) {
    case 0: {  /* a block across two regions, its above row inside the first */
      LayoutBuilder b("rows off the regions", 64, 128, 8, 1, 1, 1);
      b.block(0, 0, 0, 64, 16);
      b.block(0, 0, 16, 64, 64, 3);
      b.block(0, 0, 80, 64, 32);
      b.block(0, 0, 112, 64, 16);
      b.chroma();
      return b.take();
    }
    case 1: {  /* the right square first: above right at its inner rows */
      LayoutBuilder b("right square first", 128, 64, 10, 1, 1, 2);
      for (int x : {64, 0}) {
        for (int y = 0; y < 64; y += 16)
          for (int k = 0; k < 64; k += 16) b.block(0, x + k, y, 16, 16, 8);
        b.chroma(x, 0, x + 64, 64);
      }
      return b.take();
    }
    case 2: {  /* a block across two regions, its left column inside the first */
      LayoutBuilder b("columns off the regions", 64, 128, 8, 1, 1, 3);
      b.fill(0, 0, 0, 32, 64, 32, 32);
      b.block(0, 32, 0, 32, 32);
      b.chroma(0, 0, 64, 64);
      b.block(0, 32, 32, 32, 64, 6);
      b.fill(0, 0, 64, 32, 128, 32, 32);
      b.block(0, 32, 96, 32, 32);
      b.chroma();
      return b.take();
    }
    case 3: {  /* chroma blocks across two regions, side by side */
      LayoutBuilder b("chroma rows off the regions", 128, 64, 8, 1, 1, 4);
      b.fill(0, 0, 0, 64, 64, 32, 32);
      b.fill(0, 64, 0, 128, 64, 32, 32);
      for (int p = 1; p < 3; ++p) {
        b.block(p, 0, 0, 32, 16);
        b.block(p, 32, 0, 32, 16);
        b.block(p, 0, 16, 64, 16, 3);
      }
      return b.take();
    }
    case 4: {  /* the lower square first: below left at inner columns */
      LayoutBuilder b("lower square first", 64, 128, 8, 0, 0, 5);
      for (int y : {64, 0}) {
        for (int x = 0; x < 64; x += 16)
          for (int k = 0; k < 64; k += 16) b.block(0, x, y + k, 16, 16, 7);
        b.chroma(0, y, 64, y + 64);
      }
      return b.take();
    }
    case 5: {  /* the mode of chroma from luma on a luma block, the samples at
                  twice its place coded before it */
      LayoutBuilder b("luma by the chroma from luma mode", 128, 128, 8, 1, 1, 6);
      static const int kOrder[4][2] = {{64, 64}, {0, 0}, {64, 0}, {0, 64}};
      for (const int* at : kOrder) {
        if (at[0] + at[1] == 0) b.block(0, 48, 48, 16, 16, 13);
        b.fill(0, at[0], at[1], at[0] + 64, at[1] + 64, 16, 16, 0);
        b.chroma(at[0], at[1], at[0] + 64, at[1] + 64, 0);
      }
      return b.take();
    }
    default: {  /* squares of one block and of many, in coding order */
      LayoutBuilder b("squares", 256, 192, 12, 1, 1, 7);
      for (int y = 0; y < 192; y += 64)
        for (int x = 0; x < 256; x += 64) {
          const int side = 64 >> ((x / 64 + y / 64) % 4);
          b.fill(0, x, y, x + 64, y + 64, side, side);
          for (int p = 1; p < 3; ++p) {
            const int half = std::max(4, side / 2);
            b.fill(p, x / 2, y / 2, x / 2 + 32, y / 2 + 32, half, half);
          }
        }
      return b.take();
    }
  }
}

#endif

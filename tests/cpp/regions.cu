/*
 * regions.cu - host-only check of phase B's regions (test infrastructure; no
 * GPU needed).
 *
 * Plans seeded synthetic frames, and frames of hand-made layouts
 * (layouts.hpp), with the planner compiled here and checks what lets a region
 * run in one CTA and every wait end: each phase B block is in the region its
 * samples lie in, as items that are each of its parts once; every sample it
 * waits for is either of an item earlier in its own region, or of an item of a
 * region listed before and in that region's last row or column (the only
 * samples that are tagged); what a chroma-from-luma block waits for by tags
 * lies in its region's luma tile; and a part's residual fits a warp's scratch.
 * A frame with inter blocks in phase B or a block off its cells has no
 * regions. Prints "ok" at the end; exits non-zero on a failure.
 */
#define main plan_invariants_main
#include "plan_invariants.cu"
#undef main
#include "layouts.hpp"

namespace {

size_t with_regions = 0, parted = 0, shared = 0, across = 0;

/* What a frame's regions are to be: none, some, or either (a layout that the
 * planner may send to the chains). */
enum Want { kNone, kSome, kEither };

void check_syntax(av1b_decoder* d, WorkPool* pool, const av1b_frame_syntax& s, const char* name, int k, Want want) {
  PlanCtx c;
  const int cw = (s.coded_width <= 0 || s.coded_width > s.width) ? s.width : s.coded_width;
  c.L = make_layout(s.width, s.height, cw, s.bit_depth, s.ss_x, s.ss_y);
  for (int i = 0; i < kSlots; ++i) {
    c.slot_used[i] = c.slot_valid[i] = i < 4;
    c.slot_width[i] = s.width;
    c.slot_height[i] = s.height;
  }
  PlanScratch scratch;
  PlanLists lists;
  c.pool = pool;
  c.scratch = &scratch;
  Plan P;
  P.R = &lists;
  const int rc = build_plan(d, c, s, &P);
  CHECK(rc == 0, "%s frame %d: planning failed (%d)", name, k, rc);
  if (rc) return;
  if (want == kEither && lists.regions.empty()) return;
  if (want == kNone || P.units_inter || lists.units.empty()) {
    CHECK(lists.regions.empty(), "%s frame %d: regions", name, k);
    return;
  }
  CHECK(!lists.regions.empty(), "%s frame %d: no regions", name, k);
  ++with_regions;
  const Layout& L = c.L;
  const auto& B = lists.blocks;
  constexpr int kMask = (1 << AV1B_ITEM_SHIFT) - 1;
  int sh[3], gw[3];
  for (int p = 0; p < 3; ++p) {
    sh[p] = p == 0 ? 2 : ((p == 1 ? L.ss_x : L.ss_y) ? 1 : 2);
    gw[p] = (L.p[p].grid_w + (1 << sh[p]) - 1) >> sh[p];
  }
  /* a block's last item and the parts seen */
  std::vector<int> last(B.size(), -1), seen(B.size(), 0);
  int place = 0;
  for (const int4& r : lists.regions) {
    CHECK(r.x == place && r.y > 0 && r.y <= region_items(L, P.region_log2), "%s frame %d: a region's items", name, k);
    place += r.y;
    for (int i = r.x; i < r.x + r.y; ++i) {
      const int bi = lists.items[i] & kMask, part = lists.items[i] >> AV1B_ITEM_SHIFT;
      const BlockRec& b = B[bi];
      const int sx = b.plane ? L.ss_x : 0, sy = b.plane ? L.ss_y : 0;
      const int tw = (1 << P.region_log2) >> sx, th = (1 << P.region_log2) >> sy;
      const int cols = b.w < tw ? b.w : tw, over = b.parts > 1 ? b.w / cols : 1, rows = b.h / (b.parts / over);
      const int x0 = b.x + part % over * cols, y0 = b.y + part / over * rows;
      CHECK(part < b.parts && !(seen[bi] >> part & 1), "%s frame %d: block %d part %d", name, k, bi, part);
      seen[bi] |= 1 << part;
      if (over > 1 || y0 + b.h > (r.w + 1) * th) ++shared;
      CHECK(cols * over == b.w && rows * (b.parts / over) == b.h && x0 >= r.z * tw && x0 + cols <= (r.z + 1) * tw &&
                y0 >= r.w * th && y0 + rows <= (r.w + 1) * th,
            "%s frame %d: block %d part %d is not in its region", name, k, bi, part);
      if (b.parts > 1) {
        ++parted;
        CHECK(rows * cols <= 1024 && !(b.sync & AV1B_SYNC_FLAG) &&
                  (b.tx_count == 0 || b.res_one) && b.fuse_res && (b.palette || (b.mode != 13 && b.fi_mode < 0)),
              "%s frame %d: block %d in parts", name, k, bi);
      }
      if (!(b.sync & AV1B_SYNC_TAGS))
        for (int j = 0; j < b.dep_count; ++j) {
          const int o = lists.deps[b.dep_first + j];
          CHECK(last[o] >= 0 && seen[o] == (1 << B[o].parts) - 1, "%s frame %d: block %d waits for a later item of %d",
                name, k, bi, o);
        }
      last[bi] = i;
      /* sample (x, y) of the block's plane, which the item waits for */
      bool ok = true;
      auto awaited = [&](int x, int y) {
        const int o = scratch.owner[b.plane][static_cast<size_t>(y >> sh[b.plane]) * gw[b.plane] + (x >> sh[b.plane])];
        const BlockRec& ob = B[o];
        const bool same = x >= r.z * tw && x < (r.z + 1) * tw && y >= r.w * th && y < (r.w + 1) * th;
        if (!same) ++across;
        /* the part of the owner that the sample is in is an earlier item */
        const int oc = ob.w < tw ? ob.w : tw, oo = ob.parts > 1 ? ob.w / oc : 1, orow = ob.h / (ob.parts / oo);
        const int opart = (y - ob.y) / orow * oo + (x - ob.x) / oc;
        if (!(seen[o] >> opart & 1)) ok = false;
        if (!same && x % tw != tw - 1 && y % th != th - 1) ok = false;
      };
      if (b.sync & AV1B_SYNC_TAGS) {
        const int cell = 1 << sh[b.plane];
        for (int q = 0; q < 64; ++q)
          for (int e = 0; e < cell; ++e) {
            const int at = q * cell + e;
            if (((b.wait_cells[0][q >> 5] >> (q & 31)) & 1) && b.x + at < L.p[b.plane].grid_w) awaited(b.x + at, b.y - 1);
            if (((b.wait_cells[1][q >> 5] >> (q & 31)) & 1) && b.y + at < L.p[b.plane].grid_h) awaited(b.x - 1, b.y + at);
          }
        if (b.sync & AV1B_SYNC_CORNER) awaited(b.x - 1, b.y - 1);
      }
      CHECK(ok, "%s frame %d: block %d part %d waits for a sample nobody tags", name, k, bi, part);
      if (b.sync & AV1B_SYNC_LUMA) {
        const int side = 1 << P.region_log2;
        const int lx = (b.x - r.z * tw) << L.ss_x, ly = (b.y - r.w * th) << L.ss_y;
        CHECK(lx >= 0 && ly >= 0 && lx + (b.w << L.ss_x) <= side && ly + (b.h << L.ss_y) <= side,
              "%s frame %d: block %d's luma is outside its region's tile", name, k, bi);
      }
    }
  }
  CHECK(static_cast<size_t>(place) == lists.items.size(), "%s frame %d: items outside regions", name, k);
  for (int bi : lists.units) CHECK(seen[bi] == (1 << B[bi].parts) - 1, "%s frame %d: block %d is not run", name, k, bi);
}

void check_frame(av1b_decoder* d, WorkPool* pool, uint8_t* blob, size_t len, const char* name, int k, Want want) {
  int32_t refs[8];
  const int n = av1b_blob_get_refs(blob, len, refs, 8);
  int32_t slots[8];
  for (int i = 0; i < n; ++i) slots[i] = ((k - refs[i]) % 4 + 4) % 4;
  av1b_blob_set_refs(blob, len, slots, n);
  av1b_frame_syntax s;
  av1b_syntax_view(blob, len, &s);
  check_syntax(d, pool, s, name, k, want);
  av1b_blob_set_refs(blob, len, refs, n);
}

}  // namespace

int main() {
  av1b_decoder* d = new av1b_decoder;
  WorkPool pool(3);
  struct Case {
    const char* name;
    int w, h, cw, bd, sb, tools, frames;
  };
  const int all = (1 << 16) - 1 - (1 << 13) - (1 << 11) - (1 << 12);
  const Case cases[] = {
      {"720p basic", 1280, 720, 0, 8, 64, 0, 2},
      {"odd size", 998, 514, 750, 12, 128, all & ~(1 << 14), 3},
      {"tiny", 16, 16, 0, 8, 64, all, 2},
      {"raw residuals", 240, 136, 0, 10, 64, all, 3},
      {"4K superres", 3840, 2160, 2880, 10, 128, all & ~(1 << 14), 2},
      {"inter blocks in phase B", 640, 360, 0, 8, 64, (1 << 16) - 1 - (1 << 13), 2},
      {"4:2:2", 338, 206, 0, 8, 64, all | (1 << 18), 3},
      {"4:4:4", 338, 206, 0, 10, 64, all | (1 << 19), 3},
  };
  for (const Case& cs : cases)
    for (int k = 0; k < cs.frames; ++k) {
      uint8_t* blob = nullptr;
      size_t len = 0;
      if (av1s_synth_frame_ex(cs.w, cs.h, cs.cw, cs.bd, cs.sb, cs.tools, 5, k, 30, &blob, &len) != AV1B_OK) return 1;
      check_frame(d, &pool, blob, len, cs.name, k, kSome);
      av1s_blob_free(blob);
    }
  const size_t synthetic = with_regions;
  for (int i = 0; i < layout_count(); ++i) {
    const LayoutFrame f = layout_frame(i);
    check_syntax(d, &pool, f.syntax(), f.name.c_str(), i, kEither);
  }
  std::printf("%zu frames by regions, %zu items of parted blocks, %zu of them of blocks regions share, %zu cells across\n",
              with_regions, parted, shared, across);
  std::printf("%zu of %d layouts by regions\n", with_regions - synthetic, layout_count());
  if (failures || synthetic < 8 || with_regions - synthetic < 8 || !parted || !shared || !across) return 1;
  std::printf("ok\n");
  return 0;
}

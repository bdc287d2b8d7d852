/*
 * regions.cu - host-only check of phase B's regions (test infrastructure; no
 * GPU needed).
 *
 * Plans seeded synthetic frames with the planner compiled here and checks
 * what lets a region run in one CTA and every wait end: each phase B block is
 * in the region its samples lie in, as items that are each of its parts once;
 * every block it waits for has all its items earlier in its own region or in
 * a region listed before; the cells it waits on outside its region are the
 * last row or column of another region (the only samples that are tagged);
 * and a part's residual fits a warp's scratch. A frame with inter blocks in
 * phase B or a block off its cells has no regions. Prints "ok" at the end;
 * exits non-zero on a failure.
 */
#define main plan_invariants_main
#include "plan_invariants.cu"
#undef main

namespace {

size_t with_regions = 0, parted = 0, shared = 0, across = 0;

void check_frame(av1b_decoder* d, WorkPool* pool, uint8_t* blob, size_t len, const char* name, int k, bool none) {
  int32_t refs[8];
  const int n = av1b_blob_get_refs(blob, len, refs, 8);
  int32_t slots[8];
  for (int i = 0; i < n; ++i) slots[i] = ((k - refs[i]) % 4 + 4) % 4;
  av1b_blob_set_refs(blob, len, slots, n);
  av1b_frame_syntax s;
  av1b_syntax_view(blob, len, &s);
  av1b_blob_set_refs(blob, len, refs, n);
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
  if (none || P.units_inter || lists.units.empty()) {
    CHECK(lists.regions.empty(), "%s frame %d: regions", name, k);
    return;
  }
  CHECK(!lists.regions.empty(), "%s frame %d: no regions", name, k);
  ++with_regions;
  const Layout& L = c.L;
  const auto& B = lists.blocks;
  constexpr int kMask = (1 << AV1B_ITEM_SHIFT) - 1;
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
      for (int j = 0; j < b.dep_count; ++j) {
        const int o = lists.deps[b.dep_first + j];
        CHECK(last[o] >= 0 && seen[o] == (1 << B[o].parts) - 1, "%s frame %d: block %d waits for a later item of %d", name, k,
              bi, o);
      }
      last[bi] = i;
      const int cell = b.plane == 0 ? 4 : ((b.plane == 1 ? L.ss_x : L.ss_y) ? 2 : 4);
      for (int q = 0; q < 64; ++q) {
        const bool above = (b.wait_cells[0][q >> 5] >> (q & 31)) & 1, left = (b.wait_cells[1][q >> 5] >> (q & 31)) & 1;
        if (above && b.y % th == 0) {
          ++across;
          CHECK(b.y > 0, "%s frame %d: block %d waits above the picture", name, k, bi);
        }
        if (above && b.x + q * cell >= (r.z + 1) * tw) CHECK(b.y % th == 0, "%s frame %d: block %d above", name, k, bi);
        if (left && b.y + q * cell >= (r.w + 1) * th) CHECK(b.x % tw == 0, "%s frame %d: block %d left", name, k, bi);
      }
    }
  }
  CHECK(static_cast<size_t>(place) == lists.items.size(), "%s frame %d: items outside regions", name, k);
  for (int bi : lists.units) CHECK(seen[bi] == (1 << B[bi].parts) - 1, "%s frame %d: block %d is not run", name, k, bi);
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
  };
  for (const Case& cs : cases)
    for (int k = 0; k < cs.frames; ++k) {
      uint8_t* blob = nullptr;
      size_t len = 0;
      if (av1s_synth_frame_ex(cs.w, cs.h, cs.cw, cs.bd, cs.sb, cs.tools, 5, k, 30, &blob, &len) != AV1B_OK) return 1;
      check_frame(d, &pool, blob, len, cs.name, k, false);
      av1s_blob_free(blob);
    }
  std::printf("%zu frames by regions, %zu items of parted blocks, %zu of them of blocks regions share, %zu cells across\n",
              with_regions, parted, shared, across);
  if (failures || with_regions < 8 || !parted || !shared || !across) return 1;
  std::printf("ok\n");
  return 0;
}

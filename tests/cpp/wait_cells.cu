/*
 * wait_cells.cu - host-only check of what a phase B block waits on by its
 * tagged samples (test infrastructure; no GPU needed).
 *
 * Plans seeded synthetic frames with the planner compiled here, and compares
 * the cell masks it gives a block with the general rule, the block's
 * dependency list: of the cells of its above row, left column and corner that
 * its prediction reads, exactly those whose owner is on the list are waited
 * on; the samples of a chroma-from-luma block are waited on by their tags
 * only where every luma cell's owner is on the list and inside the grid; and
 * every block named by a list that is waited on by done flags publishes one.
 * A frame with a block off its plane's owner cells uses no tags. Prints "ok"
 * at the end; exits non-zero on a failure.
 */
#define main plan_invariants_main
#include "plan_invariants.cu"
#undef main

namespace {

size_t tagged = 0, by_luma = 0, by_flag = 0;

void check_frame(av1b_decoder* d, WorkPool* pool, uint8_t* blob, size_t len, const char* name, int k,
                 bool shift) {
  int32_t refs[8];
  const int n = av1b_blob_get_refs(blob, len, refs, 8);
  int32_t slots[8];
  for (int i = 0; i < n; ++i) slots[i] = ((k - refs[i]) % 4 + 4) % 4;
  av1b_blob_set_refs(blob, len, slots, n);
  av1b_frame_syntax s;
  av1b_syntax_view(blob, len, &s);
  av1b_blob_set_refs(blob, len, refs, n);
  std::vector<av1b_block> moved(s.blocks, s.blocks + s.n_blocks);
  if (shift) {
    for (av1b_block& b : moved)
      if (b.is_intra && b.x > 0 && b.tx_count == 0) {
        b.x -= 1;
        break;
      }
    s.blocks = moved.data();
  }
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
  const Layout& L = c.L;
  const auto& B = lists.blocks;
  int sh[3], gw[3], gh[3];
  for (int p = 0; p < 3; ++p) {
    sh[p] = p == 0 ? 2 : ((p == 1 ? L.ss_x : L.ss_y) ? 1 : 2);
    gw[p] = (L.p[p].grid_w + (1 << sh[p]) - 1) >> sh[p];
    gh[p] = (L.p[p].grid_h + (1 << sh[p]) - 1) >> sh[p];
  }
  auto owner = [&](int p, int x, int y) {
    if (x < 0 || y < 0 || x >= L.p[p].grid_w || y >= L.p[p].grid_h) return -1;
    return scratch.owner[p][static_cast<size_t>(y >> sh[p]) * gw[p] + (x >> sh[p])];
  };
  std::vector<uint8_t> flagged(B.size(), 0);
  for (int bi : lists.units) {
    const BlockRec& b = B[bi];
    const int* dep = lists.deps.data() + b.dep_first;
    auto waits = [&](int o) { return o >= 0 && std::binary_search(dep, dep + b.dep_count, o); };
    if (!(b.sync & AV1B_SYNC_TAGS)) {
      for (int j = 0; j < b.dep_count; ++j) flagged[dep[j]] = 1;
      ++by_flag;
      continue;
    }
    CHECK(!shift, "%s frame %d: block %d waits on tags in a frame off the cells", name, k, bi);
    CHECK(b.kind == AV1B_U_INTRA, "%s frame %d: block %d waits on tags and is not intra", name, k, bi);
    ++tagged;
    const int p = b.plane, cell = 1 << sh[p];
    const uint64_t above = b.wait_cells[0][0] | (static_cast<uint64_t>(b.wait_cells[0][1]) << 32);
    const uint64_t left = b.wait_cells[1][0] | (static_cast<uint64_t>(b.wait_cells[1][1]) << 32);
    if (b.palette) {
      CHECK(above == 0 && left == 0 && !(b.sync & AV1B_SYNC_CORNER), "%s frame %d: palette block %d waits", name,
            k, bi);
      continue;
    }
    static const int kAngle[9] = {0, 90, 180, 45, 135, 113, 157, 203, 67};
    const int angle = b.mode >= 1 && b.mode <= 8 ? kAngle[b.mode] + 3 * b.angle_delta : 0;
    const int na = b.w * (angle > 0 && angle < 90 && b.have_ar ? 2 : 1);
    const int nl = b.h * (angle > 180 && b.have_bl ? 2 : 1);
    for (int i = 0; i < 64; ++i) {
      const bool wa = i * cell < na && waits(owner(p, b.x + i * cell, b.y - 1));
      const bool wl = i * cell < nl && waits(owner(p, b.x - 1, b.y + i * cell));
      CHECK(((above >> i) & 1) == wa, "%s frame %d: block %d above cell %d", name, k, bi, i);
      CHECK(((left >> i) & 1) == wl, "%s frame %d: block %d left cell %d", name, k, bi, i);
    }
    CHECK(((b.sync & AV1B_SYNC_CORNER) != 0) == waits(owner(p, b.x - 1, b.y - 1)), "%s frame %d: block %d corner",
          name, k, bi);
    if (b.mode == 13) {
      bool all = b.w * b.h <= 1024;
      for (int y = b.y << L.ss_y; y < (b.y + b.h) << L.ss_y; ++y)
        for (int x = b.x << L.ss_x; x < (b.x + b.w) << L.ss_x; ++x) all = all && waits(owner(0, x, y));
      CHECK(all && (b.sync & AV1B_SYNC_LUMA), "%s frame %d: block %d reads luma it does not wait for", name, k, bi);
      ++by_luma;
    }
  }
  for (size_t i = 0; i < B.size(); ++i)
    CHECK(!flagged[i] == !(B[i].sync & AV1B_SYNC_FLAG), "%s frame %d: block %zu's done flag", name, k, i);
}

}  // namespace

int main() {
  av1b_decoder* d = new av1b_decoder;
  WorkPool pool(3);
  struct Case {
    const char* name;
    int w, h, cw, bd, sb, tools, frames;
    bool shift;
  };
  const int all = (1 << 16) - 1 - (1 << 13);
  const Case cases[] = {
      {"720p basic", 1280, 720, 0, 8, 64, 0, 2, false},
      {"odd size, every tool", 998, 514, 750, 12, 128, all | (1 << 11) | (1 << 12) | (1 << 14), 3, false},
      {"tiny", 16, 16, 0, 8, 64, all, 2, false},
      {"1080p, every tool", 1920, 1080, 0, 10, 64, all, 2, false},
      {"a block off its cells", 320, 180, 0, 8, 64, all, 2, true},
  };
  for (const Case& cs : cases)
    for (int k = 0; k < cs.frames; ++k) {
      uint8_t* blob = nullptr;
      size_t len = 0;
      if (av1s_synth_frame_ex(cs.w, cs.h, cs.cw, cs.bd, cs.sb, cs.tools, 5, k, 30, &blob, &len) != AV1B_OK) return 1;
      check_frame(d, &pool, blob, len, cs.name, k, cs.shift);
      av1s_blob_free(blob);
    }
  std::printf("%zu blocks by tags, %zu of them chroma from luma, %zu by flags\n", tagged, by_luma, by_flag);
  if (failures || !tagged || !by_luma || !by_flag) return 1;
  std::printf("ok\n");
  return 0;
}

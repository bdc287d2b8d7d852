/*
 * kernels.cu - the sm_100a kernels of one frame step.
 *
 * Reconstruction runs in two phases. Phase A is everything that reads only
 * reference pictures: the inter prediction of every inter block (one warp per
 * 16x8 tile), then every inverse transform (one warp per transform) - added
 * to the picture for inter blocks, left in a buffer for the rest. Phase B is
 * the dependency-scheduled rest: intra blocks, inter-intra blocks and intra
 * block copies, by a persistent kernel whose warps claim blocks from a device
 * queue, wait for the blocks whose samples they read and add the residual
 * computed ahead. What each block waits for comes from the planner, which
 * resolves the reference's owner grids and edge scans (engine.cpp:719-924)
 * into a short list per block and orders the claims by dependency depth: the
 * host launches nothing per wave.
 *
 * Waiting is safe without a cooperative launch: a block only ever waits on
 * blocks claimed before it, each by a warp that is already running (or has
 * finished it), so the first unfinished block in claim order always has
 * everything it needs. Every wait is bounded (one second of globaltimer); on
 * expiry the kernel records AV1B_STATUS_TIMEOUT in the status word and
 * carries on, and the host fails the frame.
 */
#include <cuda_runtime.h>

#include <algorithm>
#include <utility>

#include "dev_common.cuh"
#include "dev_filters.cuh"
#include "dev_inter.cuh"
#include "dev_intra.cuh"
#include "dev_itx.cuh"
#include "kernels.h"
#include "batch.h"

namespace av1b {

/* ---- helpers --------------------------------------------------------------------- */
__device__ __forceinline__ unsigned ld_relaxed(const unsigned* p) {
  unsigned v;
  asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ unsigned ld_acquire(const unsigned* p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void fence_acq_rel() { asm volatile("fence.acq_rel.gpu;" ::: "memory"); }
__device__ __forceinline__ void st_release(unsigned* p, unsigned v) {
  asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

/* Programmatic dependent launch: `deps_may_start` lets the next kernel of the
 * stream, launched with that attribute, take the SMs this one leaves;
 * `deps_done` waits there for the kernels before it (a no-op in a kernel
 * launched without). Every kernel that is launched with the attribute waits:
 * before it reads what they wrote or, one that reads nothing of theirs, before
 * it ends, since what comes after it takes its end for theirs. For that its
 * last CTA waits (ends_after_deps): the others leave the SMs to what comes
 * next (every CTA waiting: an inter pass at 1080p 497 us instead of 467). What
 * the kernels before wrote is read through plain pointers: a __restrict__
 * const pointer or __ldg says that the data is constant for as long as the
 * kernel runs, and such a load may be moved above the wait. */
__device__ __forceinline__ void deps_may_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void deps_done() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void ends_after_deps() {
  if (blockIdx.x == gridDim.x - 1) deps_done();
}

__device__ __forceinline__ const px_t* ref_plane(const FrameArgs& a, int slot, int plane) {
  const px_t* base = slot >= 0 ? a.slot_ptr[slot] : a.cur;
  return base + a.L.p[plane].off;
}

/* Builds the resolved inter job of a block. */
__device__ void make_inter_job(const FrameArgs& a, const BlockRec& b, InterJob* j) {
  const int p = b.plane;
  const PlaneGeom& g = a.L.p[p];
  j->x = b.x;
  j->y = b.y;
  j->w = b.w;
  j->h = b.h;
  j->plane = p;
  j->ctx.sub_x = p > 0 ? a.L.ss_x : 0;
  j->ctx.sub_y = p > 0 ? a.L.ss_y : 0;
  j->ctx.bitdepth = a.L.bit_depth;
  if (b.kind == AV1B_U_INTRABC) {
    /* a block copy reads this frame: the 4-rounded coded size, unscaled */
    j->ctx.ref_w = ((a.L.p[0].coded_w + 3) & ~3) >> j->ctx.sub_x;
    j->ctx.ref_h = ((a.L.p[0].coded_h + 3) & ~3) >> j->ctx.sub_y;
    j->ctx.scale_x = AV1B_SCALE_ONE;
    j->ctx.scale_y = AV1B_SCALE_ONE;
  } else {
    j->ctx.ref_w = g.out_w;
    j->ctx.ref_h = g.out_h;
    j->ctx.scale_x = a.scale_x;
    j->ctx.scale_y = a.scale_y;
  }
  j->ref[0] = ref_plane(a, b.ref_slot[0], p);
  j->ref[1] = ref_plane(a, b.ref_slot[1], p);
  j->ref_stride = g.stride;
  for (int r = 0; r < 2; ++r) {
    j->mv[r][0] = b.mv[r][0];
    j->mv[r][1] = b.mv[r][1];
  }
  j->filt = b.filt;
  j->filt_v = b.filt_v;
  j->compound = b.compound;
  j->w0 = b.w0;
  j->w1 = b.w1;
  j->mask_kind = b.mask_kind;
  j->mask_sign = b.mask_sign;
  j->wedge_dir = b.wedge_dir;
  j->wedge_xoff = b.wedge_xoff;
  j->wedge_yoff = b.wedge_yoff;
  j->wedge_flip = b.wedge_flip;
  j->warp[0] = b.warp0;
  j->warp[1] = b.warp1;
  j->mask_warp[0] = b.mask_warp0;
  j->mask_warp[1] = b.mask_warp1;
  j->model[0] = a.warps + (b.warp_idx[0] >= 0 ? b.warp_idx[0] : 0);
  j->model[1] = a.warps + (b.warp_idx[1] >= 0 ? b.warp_idx[1] : 0);
  j->luma_ref[0] = ref_plane(a, b.ref_slot[0], 0);
  j->luma_ref[1] = ref_plane(a, b.ref_slot[1], 0);
  j->luma_stride = a.L.p[0].stride;
  j->luma_x = b.x << (p > 0 ? a.L.ss_x : 0);
  j->luma_y = b.y << (p > 0 ? a.L.ss_y : 0);
  j->luma_ref_w = a.L.p[0].out_w;
  j->luma_ref_h = a.L.p[0].out_h;
  j->interintra = b.interintra;
  j->ii_mode = b.ii_mode;
  j->ii_wedge = b.ii_wedge;
  j->have_left = b.have_left;
  j->have_above = b.have_above;
  j->max_x = g.grid_w - 1;
  j->max_y = g.grid_h - 1;
  j->cur = a.cur + g.off + b.y * g.stride + b.x;
  j->cur_stride = g.stride;
  j->obmc = a.obmc + b.obmc_first;
  j->obmc_count = b.obmc_count;
  for (int k = 0; k < 8; ++k)
    j->obmc_ref[k] = k < b.obmc_count ? ref_plane(a, a.obmc[b.obmc_first + k].ref_slot, p) : j->ref[0];
  j->maxv = a.maxv;
}

/* ---- phase A ------------------------------------------------------------------------ */

/* The compound mask of a block the lean kernel predicts, its fields read
 * once into registers (the mask pool's byte stores could alias the block
 * record, so fields read from it would be loaded again after every store). */
struct LeanMask {
  int kind, sign, role, off, mw, dir, xoff, yoff, flip;
  __device__ __forceinline__ explicit LeanMask(const BlockRec& b)
      : kind(b.compound ? b.mask_kind : 0), sign(b.mask_sign), role(b.mask_role), off(b.mask_off),
        mw(b.mask_w), dir(b.wedge_dir), xoff(b.wedge_xoff), yoff(b.wedge_yoff), flip(b.wedge_flip) {}
};

/* The mask (0..64) of sample (x, y): a wedge (a chroma sample averages the
 * luma positions it covers), a luma difference-weighted mask from the two
 * predictions - written to the mask pool when chroma blocks read it - or a
 * chroma difference-weighted mask read from the pool its luma block wrote. */
__device__ __forceinline__ int lean_mask(const FrameArgs& a, const LeanMask& k, int plane, int sub_x,
                                         int sub_y, int bitdepth, int x, int y, int v0, int v1) {
  if (k.kind == 2 && plane == 0) {
    const int sh = 7 - (bitdepth >= 12 ? 5 : 3) + (bitdepth - 8);
    const int m = diffwtd_m(absi(v0 - v1), sh, k.sign);
    if (k.role == 1) a.mask_pool[k.off + y * k.mw + x] = static_cast<unsigned char>(m);
    return m;
  }
  const int nx = sub_x + 1, ny = sub_y + 1;
  int sum = 0;
  for (int jj = 0; jj < ny; ++jj)
    for (int ii = 0; ii < nx; ++ii) {
      const int lx = (x << sub_x) + ii, ly = (y << sub_y) + jj;
      if (k.kind == 1) {
        const int m = wedge_px(k.dir, k.xoff, k.yoff, k.flip, ly, lx);
        sum += k.sign ? 64 - m : m;
      } else {
        sum += a.mask_pool[k.off + ly * k.mw + lx];
      }
    }
  const int n = nx * ny;
  return n == 1 ? sum : (n == 2 ? (sum + 1) >> 1 : (sum + 2) >> 2);
}

/* Sample (x, y) of a block's job (a reference, or an OBMC strip, whose own
 * coordinates these then are), by mc_tap, out of line: the lean kernel's way
 * for windows that do not fit its buffers, which no reference of a valid
 * stream has. */
__device__ __noinline__ int mc_tap_far(const FrameArgs& a, const BlockRec& b, int job, int x, int y) {
  const int p = b.plane;
  const PlaneGeom& g = a.L.p[p];
  InterCtx c;
  c.sub_x = p > 0 ? a.L.ss_x : 0;
  c.sub_y = p > 0 ? a.L.ss_y : 0;
  c.ref_w = g.out_w;
  c.ref_h = g.out_h;
  c.bitdepth = a.L.bit_depth;
  c.scale_x = a.scale_x;
  c.scale_y = a.scale_y;
  const int nref = b.compound ? 2 : 1;
  if (job < nref)
    return mc_tap(c, ref_plane(a, b.ref_slot[job], p), g.stride, b.x, b.y, b.w, b.h, b.mv[job][0],
                  b.mv[job][1], b.filt, b.filt_v, x, y, b.compound != 0);
  const ObmcRec& o = a.obmc[b.obmc_first + job - nref];
  return mc_tap(c, ref_plane(a, o.ref_slot, p), g.stride, b.x + o.x, b.y + o.y, o.w, o.h, o.mv_x, o.mv_y,
                o.filt, o.filt_v, x, y, 0);
}

/* Inter prediction of the phase A blocks but inter-intra ones and chroma
 * blocks of difference-weighted compounds without a luma mask to read (they
 * take the full kernel): one warp per 16x8 tile, each reference through
 * mc_rect or, for a globally warped one, warp_block8, then the blend, then
 * the OBMC strips in order, each neighbour's prediction of the strip through
 * mc_rect. It carries none of the full kernel's state, so it runs with a
 * fraction of its registers and many more warps in flight. Two builds: the
 * average and distance-weighted blends (MASK false: translation, global
 * warp and OBMC blocks, almost every tile), and the masked blends (MASK
 * true: wedge and difference-weighted compounds) - the mask code in the
 * first build slows its tiles by a fifth. */
template <bool MASK>
__device__ __forceinline__ void inter_simple_tile(const FrameArgs& a, int tile, McTileBuf (&buf)[2],
                                                  int lane) {
  const int2 t = a.inter_tiles[tile];
  const BlockRec& b = a.blocks[t.x];
  const int p = b.plane;
  const PlaneGeom& g = a.L.p[p];
  InterCtx c;
  c.sub_x = p > 0 ? a.L.ss_x : 0;
  c.sub_y = p > 0 ? a.L.ss_y : 0;
  c.ref_w = g.out_w;
  c.ref_h = g.out_h;
  c.bitdepth = a.L.bit_depth;
  c.scale_x = a.scale_x;
  c.scale_y = a.scale_y;
  const bool scaled = c.scale_x != AV1B_SCALE_ONE;
  const int x0 = t.y & 0xffff, y0 = t.y >> 16;
  const int tw = mini(16, b.w - x0), th = mini(8, b.h - y0);
  /* the lane's samples: columns col, col + 1 of rows row, row + 1 */
  const int col = (lane & 7) * 2, row = (lane >> 3) * 2;
  const int compound = b.compound;
  const int nref = compound ? 2 : 1;
  const int jobs = nref + b.obmc_count;
  const int post = 7 - (c.bitdepth >= 12 ? 5 : 3);
  int v0[4] = {0, 0, 0, 0}, acc[4] = {0, 0, 0, 0};
  McReq cur{}, nxt{};
  /* what a job is: 0 nothing of the tile, 1 a window on its way, 2 a warped
   * reference, 3 a translation the window does not fit */
  int kind = 0, kind_next = 0;
  /* The references, then the OBMC strips in order, each blended onto the
   * samples it covers; a job's window is started before the one before it is
   * filtered. */
  for (int job = -1; job < jobs; ++job) {
    kind_next = 0;
    if (job + 1 < jobs) {
      const int n = job + 1;
      McTileBuf& dst = buf[n & 1];
      if (n < nref) {
        if (n == 0 ? b.warp0 : b.warp1) {
          kind_next = 2;
        } else {
          kind_next = mc_request(c, ref_plane(a, b.ref_slot[n], p), g.stride, b.x, b.y, b.w, b.h,
                                 b.mv[n][0], b.mv[n][1], b.filt, b.filt_v, x0, y0, tw, th, 0, 0, dst, nxt, lane)
                          ? 1
                          : 3;
        }
      } else {
        const ObmcRec& o = a.obmc[b.obmc_first + n - nref];
        const int ix0 = maxi(o.x, x0), ix1 = mini(o.x + o.w, x0 + tw);
        const int iy0 = maxi(o.y, y0), iy1 = mini(o.y + o.h, y0 + th);
        if (ix0 < ix1 && iy0 < iy1) {
          const int c0 = (ix0 - x0) & ~1, r0 = (iy0 - y0) & ~1;
          kind_next = mc_request(c, ref_plane(a, o.ref_slot, p), g.stride, b.x + o.x, b.y + o.y, o.w, o.h,
                                 o.mv_x, o.mv_y, o.filt, o.filt_v, x0 + c0 - o.x, y0 + r0 - o.y,
                                 ix1 - x0 - c0, iy1 - y0 - r0, c0, r0, dst, nxt, lane)
                          ? 1
                          : 3;
        }
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    if (job >= 0) {
      McTileBuf& src = buf[job & 1];
      int out[4] = {0, 0, 0, 0};
      if (kind == 1) {
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncwarp();
        mc_filter(cur, scaled, src, c.bitdepth, job < nref ? compound : 0, col, row, out, lane);
      } else if (kind == 2) {
        /* one or two whole 8x8 warp blocks (x0 is a multiple of 16, y0 of 8) */
        const int wi = b.warp_idx[job];
        const WarpRec& m = a.warps[wi >= 0 ? wi : 0];
        for (int bx = 0; bx < tw; bx += 8)
          warp_block8(c.sub_x, c.sub_y, c.ref_w, c.ref_h, m, ref_plane(a, b.ref_slot[job], p), g.stride,
                      b.x, b.y, x0 + bx, y0, c.bitdepth, compound != 0, src.wwin, src.wmid,
                      src.wout + bx, 16, mini(8, tw - bx), th, lane);
#pragma unroll
        for (int e = 0; e < 4; ++e) out[e] = src.wout[(row + (e >> 1)) * 16 + col + (e & 1)];
        __syncwarp();
      }
      if (job < nref) {
        if (kind == 3) {
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int x = col + (e & 1), y = row + (e >> 1);
            if (x < tw && y < th)
              out[e] = mc_tap_far(a, b, job, x0 + x, y0 + y);
          }
        }
        if (job + 1 < nref) {
#pragma unroll
          for (int e = 0; e < 4; ++e) v0[e] = out[e];
        } else if constexpr (MASK) {
          const LeanMask mk(b);
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int x = col + (e & 1), y = row + (e >> 1);
            if (x >= tw || y >= th) continue;
            const int m = lean_mask(a, mk, p, c.sub_x, c.sub_y, c.bitdepth, x0 + x, y0 + y, v0[e], out[e]);
            acc[e] = clampi((m * v0[e] + (64 - m) * out[e] + (1 << (5 + post))) >> (6 + post), 0, a.maxv);
          }
        } else {
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            int v = out[e];
            if (compound == 1) v = (v0[e] + v + (1 << post)) >> (1 + post);
            else if (compound) v = (b.w0 * v0[e] + b.w1 * v + (1 << (3 + post))) >> (4 + post);
            acc[e] = clampi(v, 0, a.maxv);
          }
        }
      } else if (kind) {
        const ObmcRec& o = a.obmc[b.obmc_first + job - nref];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int x = x0 + col + (e & 1) - o.x, y = y0 + row + (e >> 1) - o.y;
          if (x < 0 || x >= o.w || y < 0 || y >= o.h || col + (e & 1) >= tw || row + (e >> 1) >= th) continue;
          const int pv = kind == 1 ? out[e]
                                   : mc_tap_far(a, b, job, x, y);
          acc[e] = obmc_blend(o, x, y, acc[e], pv, a.maxv);
        }
      }
    }
    cur = nxt;
    kind = kind_next;
  }
  px_t* dst = a.cur + g.off + (b.y + y0 + row) * g.stride + b.x + x0 + col;
#pragma unroll
  for (int r = 0; r < 2; ++r, dst += g.stride) {
    if (row + r >= th || col >= tw) continue;
    if (col + 1 < tw && (reinterpret_cast<uintptr_t>(dst) & 3) == 0) {
      *reinterpret_cast<unsigned*>(dst) = static_cast<unsigned>(acc[2 * r]) | (static_cast<unsigned>(acc[2 * r + 1]) << 16);
    } else {
      dst[0] = static_cast<px_t>(acc[2 * r]);
      if (col + 1 < tw) dst[1] = static_cast<px_t>(acc[2 * r + 1]);
    }
  }
}

/* Tiles [first, end) of the lean kernel's: the unmasked tiles listed first;
 * the masked build takes the wedge and luma difference-weighted tiles listed
 * next and (a launch of their own, after the luma tiles that write the
 * masks) the chroma tiles that read a luma mask, listed last. */
template <bool MASK>
__global__ void __launch_bounds__(128, 5) k_inter_simple(const __grid_constant__ FrameArgs a, int first,
                                                      int end) {
  __shared__ McTileBuf buf[4][2];
  deps_may_start();
  const int wib = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int warp = first + blockIdx.x * 4 + wib;
  if (warp < end) inter_simple_tile<MASK>(a, warp, buf[wib], lane);
  ends_after_deps();
}

/* Both of the lean kernel's luma-side ranges in one launch, for frames with
 * few tiles: there the launches, not the tiles, take the time (240x136: 41 ->
 * 27 us a frame for the stage; 360p, above the rule's line, 54 -> 39 by
 * running the two launches side by side). */
__global__ void __launch_bounds__(128, 5) k_inter_lean(const __grid_constant__ FrameArgs a, int n_unmasked,
                                                       int end) {
  __shared__ McTileBuf buf[4][2];
  const int wib = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int warp = blockIdx.x * 4 + wib;
  if (warp >= end) return;
  if (warp < n_unmasked) inter_simple_tile<false>(a, warp, buf[wib], lane);
  else inter_simple_tile<true>(a, warp, buf[wib], lane);
}

/* Inter prediction of phase A blocks: one warp per 16x8 tile. Translation
 * predictions (and OBMC strips) go through mc_rect, warped ones through
 * warp_block8; the composition and the OBMC blends run per sample on
 * registers. A chroma tile whose compound mask is difference-weighted takes
 * its mask from the luma predictions of the area it covers (up to 32x16
 * luma samples), computed the same separable way into shared memory. */
__device__ __forceinline__ void inter_full_tile(const FrameArgs& a, int tile, McScratch& scr,
                                                int (&pred)[2][8 * 16],
                                                int (&lpred)[2][4 * 8 * 16], int lane) {
  const int2 t = a.inter_tiles[tile];
  const BlockRec& b = a.blocks[t.x];
  InterJob j;
  make_inter_job(a, b, &j);
  const int x0 = t.y & 0xffff, y0 = t.y >> 16;
  const int tw = mini(16, b.w - x0), th = mini(8, b.h - y0);
  /* k / tw for the tile's k < 128 as a multiply and a shift (exact there) */
  const int tmul = (65536 + tw - 1) / tw;
  const PlaneGeom& g = a.L.p[b.plane];
  px_t* dst = a.cur + g.off + (b.y + y0) * g.stride + b.x + x0;
  if (j.interintra) {
    /* inter-intra reads this frame: scheduled with the dependency phase */
    for (int k = lane; k < tw * th; k += 32) {
      const int yy = k / tw, xx = k - yy * tw;
      int v = inter_core(j, x0 + xx, y0 + yy);
      v = inter_finish(j, x0 + xx, y0 + yy, v, 0);
      dst[yy * g.stride + xx] = (px_t)v;
    }
    return;
  }
  const int nref = j.compound ? 2 : 1;
  for (int r = 0; r < nref; ++r) {
    int* pr = pred[r];
    if (j.warp[r]) {
      /* the tile is one or two whole 8x8 warp blocks (x0 is a multiple of
       * 16, y0 of 8) */
      for (int bx = 0; bx < tw; bx += 8)
        warp_block8(j.ctx.sub_x, j.ctx.sub_y, j.ctx.ref_w, j.ctx.ref_h, *j.model[r], j.ref[r],
                    j.ref_stride, j.x, j.y, x0 + bx, y0, j.ctx.bitdepth, j.compound != 0, scr.win,
                    scr.mid, pr + bx, 16, mini(8, tw - bx), th, lane);
      continue;
    }
    const bool ok = mc_rect(j.ctx, j.ref[r], j.ref_stride, j.x, j.y, j.w, j.h, j.mv[r][0],
                            j.mv[r][1], j.filt, j.filt_v, j.compound != 0, x0, y0, tw, th, scr,
                            pr, lane);
    if (!ok) {
      for (int k = lane; k < tw * th; k += 32) {
        const int yy = k / tw, xx = k - yy * tw;
        pr[yy * 16 + xx] = inter_ref(j, r, x0 + xx, y0 + yy);
      }
      __syncwarp();
    }
  }
  const bool luma_mask = j.compound && j.mask_kind == 2 && b.plane > 0;
  /* the luma block is the same prediction and has written its mask */
  const bool shared_mask = luma_mask && b.mask_role == 2;
  if (luma_mask && !shared_mask) {
    InterCtx l;
    l.sub_x = l.sub_y = 0;
    l.ref_w = j.luma_ref_w;
    l.ref_h = j.luma_ref_h;
    l.bitdepth = j.ctx.bitdepth;
    l.scale_x = j.ctx.scale_x;
    l.scale_y = j.ctx.scale_y;
    const int lx0 = x0 << j.ctx.sub_x, ly0 = y0 << j.ctx.sub_y;
    const int lw = tw << j.ctx.sub_x, lh = th << j.ctx.sub_y;
    const int ew = j.w << j.ctx.sub_x, eh = j.h << j.ctx.sub_y;
    for (int r = 0; r < 2; ++r)
      for (int qy = 0; qy < lh; qy += 8)
        for (int qx = 0; qx < lw; qx += 16) {
          int* out = lpred[r] + ((qy >> 3) * 2 + (qx >> 4)) * 128;
          const int rw = mini(16, lw - qx), rh = mini(8, lh - qy);
          if (j.mask_warp[r]) {
            for (int bx = 0; bx < rw; bx += 8)
              warp_block8(0, 0, j.luma_ref_w, j.luma_ref_h, *j.model[r], j.luma_ref[r],
                          j.luma_stride, j.luma_x, j.luma_y, lx0 + qx + bx, ly0 + qy,
                          j.ctx.bitdepth, 1, scr.win, scr.mid, out + bx, 16, mini(8, rw - bx), rh, lane);
          } else if (!mc_rect(l, j.luma_ref[r], j.luma_stride, j.luma_x, j.luma_y, ew, eh,
                              j.mv[r][0], j.mv[r][1], j.filt, j.filt_v, 1, lx0 + qx, ly0 + qy, rw,
                              rh, scr, out, lane)) {
            for (int k = lane; k < rw * rh; k += 32) {
              const int yy = k / rw, xx = k - yy * rw;
              out[yy * 16 + xx] = mc_tap(l, j.luma_ref[r], j.luma_stride, j.luma_x, j.luma_y, ew,
                                         eh, j.mv[r][0], j.mv[r][1], j.filt, j.filt_v,
                                         lx0 + qx + xx, ly0 + qy + yy, 1);
            }
            __syncwarp();
          }
        }
  }
  int acc[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int k = lane + 32 * q;
    if (k < tw * th) {
      const int yy = (k * tmul) >> 16, xx = k - yy * tw;
      const int v0 = pred[0][yy * 16 + xx], v1 = nref > 1 ? pred[1][yy * 16 + xx] : 0;
      if (luma_mask) {
        /* the chroma sample's mask: the mean over the luma samples it covers,
         * from the luma block's mask or from the luma predictions */
        const int sh = 7 - (j.ctx.bitdepth >= 12 ? 5 : 3) + (j.ctx.bitdepth - 8);
        const int nx = j.ctx.sub_x + 1, ny = j.ctx.sub_y + 1;
        int sum = 0;
        for (int jj = 0; jj < ny; ++jj)
          for (int ii = 0; ii < nx; ++ii) {
            const int lx = (xx << j.ctx.sub_x) + ii, ly = (yy << j.ctx.sub_y) + jj;
            if (shared_mask) {
              const int bx = (x0 << j.ctx.sub_x) + lx, by = (y0 << j.ctx.sub_y) + ly;
              sum += a.mask_pool[b.mask_off + by * b.mask_w + bx];
            } else {
              const int idx = ((ly >> 3) * 2 + (lx >> 4)) * 128 + (ly & 7) * 16 + (lx & 15);
              sum += diffwtd_m(absi(lpred[0][idx] - lpred[1][idx]), sh, j.mask_sign);
            }
          }
        const int n = nx * ny;
        const int m = n == 1 ? sum : (n == 2 ? (sum + 1) >> 1 : (sum + 2) >> 2);
        acc[q] = blend_mask(j, v0, v1, m);
      } else {
        acc[q] = inter_compose(j, x0 + xx, y0 + yy, v0, v1);
        if (b.mask_role == 1) {
          /* the mask its chroma blocks read (the one inter_compose blends with) */
          const int sh = 7 - (j.ctx.bitdepth >= 12 ? 5 : 3) + (j.ctx.bitdepth - 8);
          a.mask_pool[b.mask_off + (y0 + yy) * b.mask_w + x0 + xx] =
              static_cast<unsigned char>(diffwtd_m(absi(v0 - v1), sh, j.mask_sign));
        }
      }
    }
  }
  __syncwarp();
  for (int kk = 0; kk < j.obmc_count; ++kk) {
    const ObmcRec& c = j.obmc[kk];
    const int ix0 = maxi(c.x, x0), ix1 = mini(c.x + c.w, x0 + tw);
    const int iy0 = maxi(c.y, y0), iy1 = mini(c.y + c.h, y0 + th);
    if (ix0 >= ix1 || iy0 >= iy1) continue;
    int* tmp = pred[0];
    const bool ok = mc_rect(j.ctx, j.obmc_ref[kk], j.ref_stride, j.x + c.x, j.y + c.y, c.w, c.h,
                            c.mv_x, c.mv_y, c.filt, c.filt_v, 0, ix0 - c.x, iy0 - c.y, ix1 - ix0,
                            iy1 - iy0, scr, tmp, lane);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int k = lane + 32 * q;
      if (k >= tw * th) continue;
      const int yy = (k * tmul) >> 16, xx = k - yy * tw;
      const int x = x0 + xx, y = y0 + yy;
      if (x < ix0 || x >= ix1 || y < iy0 || y >= iy1) continue;
      const int pv = ok ? tmp[(y - iy0) * 16 + x - ix0]
                        : mc_tap(j.ctx, j.obmc_ref[kk], j.ref_stride, j.x + c.x, j.y + c.y, c.w,
                                 c.h, c.mv_x, c.mv_y, c.filt, c.filt_v, x - c.x, y - c.y, 0);
      acc[q] = obmc_blend(c, x - c.x, y - c.y, acc[q], pv, j.maxv);
    }
    __syncwarp();
  }
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int k = lane + 32 * q;
    if (k < tw * th) {
      const int yy = (k * tmul) >> 16, xx = k - yy * tw;
      dst[yy * g.stride + xx] = (px_t)acc[q];
    }
  }
}

/* Tiles [first, end) of the full kernel's (between the lean kernel's two
 * ranges). */
__global__ void __launch_bounds__(128, 4) k_inter(const __grid_constant__ FrameArgs a, int first, int end) {
  __shared__ McScratch scr[4];
  __shared__ int pred[4][2][8 * 16];
  __shared__ int lpred[4][2][4 * 8 * 16];   /* luma predictions, four 16x8 quarters */
  const int wib = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int warp = first + blockIdx.x * 4 + wib;
  if (warp >= end) return;
  inter_full_tile(a, warp, scr[wib], pred[wib], lpred[wib], lane);
}

/* Adds one transform's residual (or a raw residual block) to the picture. */
template <bool CG>
__device__ void apply_tx(const FrameArgs& a, const BlockRec& b, const TxRec& tx, int* tmp,
                         int lane) {
  const PlaneGeom& g = a.L.p[b.plane];
  px_t* dst = a.cur + g.off + (b.y + tx.y) * g.stride + b.x + tx.x;
  if (b.residual_provided || tx.pre_off >= 0) {
    const int* res = b.residual_provided ? a.residual + tx.coef_off : a.pre_res + tx.pre_off;
    for (int k = lane; k < tx.w * tx.h; k += 32) {
      const int yy = k / tx.w, xx = k - yy * tx.w;
      px_t* q = dst + yy * g.stride + xx;
      const int old = CG ? (int)__ldcg(q) : (int)*q;
      *q = (px_t)clampi(old + res[yy * tx.w + xx], 0, a.maxv);
    }
    __syncwarp();
    return;
  }
  ItxParams p;
  p.lw = tx.log2w;
  p.lh = tx.log2h;
  p.type = tx.type;
  p.lossless = b.lossless;
  p.row_shift = tx.row_shift;
  p.bitdepth = a.L.bit_depth;
  itx_warp<CG>(p, a.coef + tx.coef_off, tmp, dst, g.stride, a.maxv, lane);
}

/* Dequantisation on the device: a frame's coded levels, in scan order, into
 * the raster the inverse transforms read (the reference front end's
 * dequantise_tile fill, dequant.hpp:317-345, with dequantise_level,
 * dequant.hpp:94-106). One warp per coded transform: the raster is cleared
 * with vector stores, then the lanes place the levels through the scan. It
 * runs on the planner's upload stream right after the levels arrive, so it
 * overlaps the frames still decoding; the rasters it writes are what the
 * ITX kernels read next, mostly out of L2. */
__global__ void __launch_bounds__(256) k_dequant(const DqRec* __restrict__ jobs, int n,
                                                 const short* __restrict__ levels,
                                                 const unsigned char* __restrict__ qm,
                                                 int* __restrict__ coef, int bit_depth) {
  const int j = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (j >= n) return;
  const DqRec r = jobs[j];
  const int area = 1 << (r.alw + r.alh);
  int* raster = coef + r.coef_off;
  if ((r.coef_off & 3) == 0) {
    int4* v = reinterpret_cast<int4*>(raster);
    for (int k = lane; k < (area >> 2); k += 32) v[k] = make_int4(0, 0, 0, 0);
  } else {
    for (int k = lane; k < area; k += 32) raster[k] = 0;
  }
  __syncwarp();
  const short* lv = levels + r.level_off;
  const unsigned short* scan = kScans + r.scan_off;
  const unsigned char* m = r.qm_off >= 0 ? qm + r.qm_off : nullptr;
  const int hi = (1 << (7 + bit_depth)) - 1, lo = -(1 << (7 + bit_depth));
  for (int i = lane; i < r.count; i += 32) {
    const int level = lv[i];
    const int pos = scan[i];
    if (level == 0 || pos >= area) continue;
    int step = pos == 0 ? r.dc_step : r.ac_step;
    if (m) step = (step * m[pos] + 16) >> 5;
    const long long prod = static_cast<long long>(level) * step;
    const unsigned mag = static_cast<unsigned>((prod < 0 ? -prod : prod) & 0xFFFFFF);
    const int scaled = static_cast<int>(mag / r.denom);
    raster[pos] = clampi(prod < 0 ? -scaled : scaled, lo, hi);
  }
}

cudaError_t launch_dequant(const DqRec* jobs, int n, const short* levels, const unsigned char* qm,
                           int* coef, int bit_depth, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  k_dequant<<<(n + 7) / 8, 256, 0, s>>>(jobs, n, levels, qm, coef, bit_depth);
  return cudaGetLastError();
}

/* Inverse transforms, in batches of one size class: a warp runs 32 / S
 * transforms whose longer side is S (S = 4, 8, 16, 32; one of 64), one lane
 * group of S lanes each, so a 4x4 transform no longer leaves 28 lanes idle.
 * One launch per class (CLS = log2 S), each instantiating only its class's
 * transform lengths: the small classes, most of the transforms, run with a
 * fraction of the registers of the 64-point ones and so with many more warps
 * in flight. The planner sorts the transforms by class, shape and type, so
 * the groups of a warp mostly take the same path. Those of phase A blocks add
 * into the picture; those of phase B blocks leave their residual in the
 * precomputed buffer, so the dependency-scheduled kernel only predicts and
 * adds (the residual does not depend on the prediction). Raw residual blocks
 * (class 7) add with the whole warp. */
/* Scratch ints a warp of class CLS needs. */
template <int CLS>
struct ItxScratch {
  static constexpr int S = 1 << (CLS < 7 ? CLS : 5);
  /* a transform's intermediate: at most 32 rows of the class's longest */
  static constexpr int PER_TX = (S < 32 ? S : 32) * itx_stride(CLS < 7 ? CLS : 6);
  static constexpr int PER_WARP = CLS >= 6 ? PER_TX : 32 / S * PER_TX;
};

/* One batch of class CLS (`bt`: first job, jobs, class) with the warp's
 * scratch `wsm`. */
template <int CLS>
__device__ __forceinline__ void itx_batch(const FrameArgs& a, const int4 bt, int* wsm, int lane) {
  constexpr int S = ItxScratch<CLS>::S, STEP = S < 32 ? S : 32;
  if constexpr (CLS == 7) {
    const int2 t = a.itx_jobs[bt.x];
    apply_tx<false>(a, a.blocks[t.x], a.txs[t.y], wsm, lane);
  } else {
    const int g = lane / STEP, sub = lane - g * STEP;
    const bool active = g < bt.y;
    const int2 t = a.itx_jobs[bt.x + (active ? g : 0)];
    const BlockRec& b = a.blocks[t.x];
    const TxRec& tx = a.txs[t.y];
    ItxParams p;
    p.lw = tx.log2w;
    p.lh = tx.log2h;
    p.type = tx.type;
    p.lossless = b.lossless;
    p.row_shift = tx.row_shift;
    p.bitdepth = a.L.bit_depth;
    int* tmp = wsm + (S <= 32 ? g * ItxScratch<CLS>::PER_TX : 0);
    const PlaneGeom& gm = a.L.p[b.plane];
    px_t* dst = a.cur + gm.off + (b.y + tx.y) * gm.stride + b.x + tx.x;
    int* res = tx.pre_off >= 0 ? a.pre_res + tx.pre_off : nullptr;
    itx_group_cls<CLS, false>(p, a.coef + tx.coef_off, tmp, dst, gm.stride, a.maxv, res, sub, STEP,
                              active);
  }
}

/* CTAs an SM of a class's kernels: the registers its transforms need with
 * little to spare (unbounded, the compiler takes up to twice that for
 * scheduling, and the small classes live on warps in flight). */
constexpr int kItxCtas[8] = {0, 0, 10, 8, 5, 4, 3, 3};

template <int CLS>
__global__ void __launch_bounds__(128, kItxCtas[CLS]) k_itx(const __grid_constant__ FrameArgs a, int first,
                                             int count) {
  extern __shared__ int smem[];
  deps_may_start();
  const int wib = threadIdx.x >> 5;
  const int bi = blockIdx.x * (blockDim.x >> 5) + wib;
  const int lane = threadIdx.x & 31;
  if (bi < count) itx_batch<CLS>(a, a.itx_batches[first + bi], smem + wib * ItxScratch<CLS>::PER_WARP, lane);
  ends_after_deps();
}

/* Every class in one launch, the longest transforms first (they take the
 * longest): for frames whose batches all fit the GPU at once at this kernel's
 * registers, the largest class's, so that the stage takes as long as its
 * longest class instead of the sum of six launches (a 240x136 frame 37 -> 19
 * us, 360p 47 -> 26). Larger frames launch a kernel a class, each with its own
 * registers, side by side where no two transforms of a block share samples
 * (1080p 65 -> 37 us, 4K 100 -> 64). */
__global__ void __launch_bounds__(128, AV1B_ITX_ALL_CTAS) k_itx_all(const __grid_constant__ FrameArgs a, int n) {
  extern __shared__ int smem[];
  const int wib = threadIdx.x >> 5;
  const int bi = blockIdx.x * 4 + wib;
  const int lane = threadIdx.x & 31;
  if (bi >= n) return;
  const int4 bt = a.itx_batches[n - 1 - bi];
  int* wsm = smem + wib * ItxScratch<6>::PER_WARP;
  switch (bt.z) {
    case 2: itx_batch<2>(a, bt, wsm, lane); break;
    case 3: itx_batch<3>(a, bt, wsm, lane); break;
    case 4: itx_batch<4>(a, bt, wsm, lane); break;
    case 5: itx_batch<5>(a, bt, wsm, lane); break;
    case 6: itx_batch<6>(a, bt, wsm, lane); break;
    default: itx_batch<7>(a, bt, wsm, lane); break;
  }
}

static inline unsigned cdiv(long long a, long long b) { return (unsigned)((a + b - 1) / b); }

/* Launches a kernel that may start once the one before it in the stream lets
 * it (deps_may_start), and that waits for it itself (deps_done,
 * ends_after_deps). */
template <class... P, class... A>
static cudaError_t launch_chained(bool early, void (*k)(P...), dim3 grid, int block, size_t smem,
                                  cudaStream_t s, A&&... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(static_cast<unsigned>(block));
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &at;
  cfg.numAttrs = early ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, k, std::forward<A>(args)...);
}

/* `early`: beside the class launched before it (they write other samples). */
template <int CLS>
static cudaError_t launch_itx_class(const FrameArgs& a, bool* early, cudaStream_t s) {
  const int first = a.itx_class_first[CLS], count = a.itx_class_count[CLS];
  if (count <= 0) return cudaSuccess;
  constexpr size_t smem = 4 * ItxScratch<CLS>::PER_WARP * sizeof(int);
  const cudaError_t e = launch_chained(*early, k_itx<CLS>, (count + 3) / 4, 128, smem, s, a, first, count);
  *early = !a.itx_overlap;
  return e;
}

/* ---- phase B -------------------------------------------------------------------------- */

/* How a dependency wait polls: with AV1B_POLL_ACQUIRE every poll is an
 * acquire load (the load that sees the flag orders what follows, no separate
 * fence); without, relaxed polls and one acquire fence once the flag is seen.
 * Between polls the warp sleeps, backing off to AV1B_POLL_PAUSE_MAX ns (0: no
 * sleep). Acquire polls take about 6 % off the dependency-scheduled phase
 * (the fence after a relaxed poll is a round trip of its own on the path).
 * Shorter pauses gain nothing on one stream, and with many streams' chains
 * waiting at once (a batched key frame-set) 64 ns pauses saw occasional
 * steps of twice the usual time, 256 ns none. */
#ifndef AV1B_POLL_ACQUIRE
#define AV1B_POLL_ACQUIRE 1
#endif
#ifndef AV1B_POLL_PAUSE_MAX
#define AV1B_POLL_PAUSE_MAX 256
#endif

__device__ __forceinline__ bool flag_seen(const unsigned* flag, unsigned want) {
#if AV1B_POLL_ACQUIRE
  return ld_acquire(flag) == want;
#else
  if (ld_relaxed(flag) != want) return false;
  fence_acq_rel();
  return true;
#endif
}

/* Waits until *flag == want, for at most limit_ns of globaltimer. Once any
 * wait has given up (AV1B_STATUS_TIMEOUT in *status), nothing waits any more:
 * the frame has failed and the kernel only has to run to its end. The status
 * word and the clock are read every 16th poll. */
__device__ bool bounded_wait(const unsigned* flag, unsigned want, int* status, int* status_host,
                             unsigned long long limit_ns) {
  if (flag_seen(flag, want)) return true;
  const unsigned long long t0 = global_ns();
  unsigned pause = AV1B_POLL_PAUSE_MAX < 32 ? AV1B_POLL_PAUSE_MAX : 32;
  for (unsigned it = 1;; ++it) {
    if (flag_seen(flag, want)) return true;
    if ((it & 15) == 0) {
      if (ld_relaxed(reinterpret_cast<const unsigned*>(status)) & AV1B_STATUS_TIMEOUT) return false;
      if (global_ns() - t0 > limit_ns) {
        wait_failed(status, status_host);
        return false;
      }
    }
    if (AV1B_POLL_PAUSE_MAX > 0) __nanosleep(pause);
    if (pause < AV1B_POLL_PAUSE_MAX) pause <<= 1;
  }
}

/* Waits until block `o` is reconstructed. Returns false on timeout. */
__device__ bool wait_block(const FrameArgs& a, int o) {
  return bounded_wait(a.done + (size_t)o * AV1B_FLAG_STRIDE, a.epoch, a.status, a.status_host, a.wait_ns);
}

/* A wait on a flag nothing sets: the failure-detection self test. */
__global__ void k_selftest_wait(const unsigned* flag, int* status, unsigned long long limit_ns) {
  if (threadIdx.x == 0) bounded_wait(flag, 1u, status, nullptr, limit_ns);
}

cudaError_t launch_selftest_wait(const unsigned* flag, int* status, unsigned long long limit_ns,
                                 cudaStream_t s) {
  k_selftest_wait<<<1, 32, 0, s>>>(flag, status, limit_ns);
  return cudaGetLastError();
}

/* The persistent dependency-scheduled kernel: each warp claims chains of
 * blocks in the planner's order (chains start in order of dependency depth)
 * and runs a chain's blocks one after another: for each it waits for the
 * blocks its list names - except the one before it in the chain, its own
 * work - and reconstructs. Everything that does not depend on other blocks - the
 * block record, its dependency list, its residual - is loaded before the
 * wait. An intra block waits on the samples it reads, by their tags
 * (FrameArgs::tags): a step of the critical path is then one store and one
 * load through L2 and the prediction, where the done flag added the writer's
 * fence, its store, the poll and the acquire before the samples could be
 * loaded (a 4K key frame's phase, 1,372 steps: 6.28 -> 4.18 ms, 4.6 -> 3.0 us
 * a step; 1080p 3.74 -> 2.51; 720p 2.53 -> 1.67). Shared memory per warp: three edge buffers and a 64x64 scratch (the
 * block's residual image, or the transform scratch). */
/* Adds a phase B transform's residual - precomputed by k_itx, or the raw
 * residual of a residual-provided block - to the reconstructed prediction
 * (read back through L2). No transform code here: the kernel stays small. */
__device__ void add_residual_cg(const FrameArgs& a, const BlockRec& b, const TxRec& tx, int lane) {
  const PlaneGeom& g = a.L.p[b.plane];
  px_t* dst = a.cur + g.off + (b.y + tx.y) * g.stride + b.x + tx.x;
  const int* res = b.residual_provided ? a.residual + tx.coef_off : a.pre_res + tx.pre_off;
  /* four samples a lane at a time, every load before any store: the loads
   * read the picture the stores write, so the compiler cannot overlap one
   * sample's load with another's store by itself */
  const int n = tx.w * tx.h;
  for (int k0 = lane; k0 < n; k0 += 4 * 32) {
    int v[4];
    int o[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int k = k0 + 32 * q;
      if (k < n) {
        const int yy = k / tx.w, xx = k - yy * tx.w;
        o[q] = yy * g.stride + xx;
        v[q] = (int)__ldcg(dst + o[q]) + res[k];
      }
    }
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if (k0 + 32 * q < n) dst[o[q]] = (px_t)clampi(v[q], 0, a.maxv);
  }
  __syncwarp();
}

/* Starts the copies of the residual of an intra block's `rows` rows from row0
 * and `cols` columns from col0 on into `tmp` (row-major; asynchronous,
 * committed). The common block has one transform of its size: runs of 16-byte
 * copies, its place in the block's record. Only such a block comes in parts. */
__device__ __forceinline__ void fetch_residual(const FrameArgs& a, const BlockRec& b, int* tmp, int row0, int rows,
                                               int col0, int cols, int lane) {
  const int* pool = b.residual_provided ? a.residual : a.pre_res;
  const int w = b.w, n = rows * cols;
  const int* src0 = pool + b.res_off + row0 * w + col0;
  if (b.res_one && ((cols | w) & 3) == 0 && (reinterpret_cast<uintptr_t>(src0) & 15) == 0) {
    const int lc = ilog2(cols);
    for (int k = lane * 4; k < n; k += 128) {
      const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(tmp + k));
      const int* src = src0 + (k >> lc) * w + (k & (cols - 1));
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
    }
  } else {
    for (int k = lane; k < n; k += 32) tmp[k] = 0;
    __syncwarp();
    for (int t = 0; t < b.tx_count; ++t) {
      const TxRec tx = a.txs[b.tx_first + t];
      const int* src = pool + (b.residual_provided ? tx.coef_off : tx.pre_off);
      for (int k = lane; k < tx.w * tx.h; k += 32) {
        const int yy = k / tx.w, xx = k - yy * tx.w;
        const int row = tx.y + yy - row0, col = tx.x + xx - col0;
        if (row < 0 || row >= rows || col < 0 || col >= cols) continue;
        const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(tmp + row * cols + col));
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(d), "l"(src + k) : "memory");
      }
    }
  }
  asm volatile("cp.async.commit_group;" ::: "memory");
}

/* An intra block's prediction job and its tagged samples (`tagged`: at its
 * top-left sample; `write`: its samples are final as they are predicted). */
__device__ __forceinline__ IntraJob intra_job(const FrameArgs& a, const BlockRec& b) {
  const PlaneGeom& g = a.L.p[b.plane];
  IntraJob j;
  j.x = b.x;
  j.y = b.y;
  j.w = b.w;
  j.h = b.h;
  j.mode = b.mode;
  j.angle = b.angle_delta;
  j.bitdepth = a.L.bit_depth;
  j.maxv = a.maxv;
  j.have_left = b.have_left;
  j.have_above = b.have_above;
  j.have_ar = b.have_ar;
  j.have_bl = b.have_bl;
  j.filter_type = b.filter_type;
  j.filter_intra = b.fi_mode >= 0;
  j.fi_mode = b.fi_mode >= 0 ? b.fi_mode : 0;
  j.cfl_alpha = b.cfl_alpha;
  j.max_x = g.grid_w - 1;
  j.max_y = g.grid_h - 1;
  j.ss_x = a.L.ss_x;
  j.ss_y = a.L.ss_y;
  j.palette = b.palette;
  j.palette_off = b.palette_off;
  j.palette_stride = b.palette_stride;
  return j;
}

__device__ __forceinline__ TagIo tag_io(const FrameArgs& a, const BlockRec& b, unsigned* tagged, bool write) {
  const int p = b.plane;
  const PlaneGeom& g = a.L.p[p];
  TagIo t;
  t.write = write ? tagged : nullptr;
  t.at = tagged;
  t.stride = g.grid_w;
  t.luma_at = a.tags ? a.tags + a.tag_off[0] : nullptr;
  t.luma_stride = a.L.p[0].grid_w;
  t.tag = a.tag;
  t.wait = a.tags && (b.sync & AV1B_SYNC_TAGS);
  t.luma = a.tags && (b.sync & AV1B_SYNC_LUMA);
  t.corner = (b.sync & AV1B_SYNC_CORNER) != 0;
  t.cell = p == 0 ? 2 : ((p == 1 ? a.L.ss_x : a.L.ss_y) ? 1 : 2);
  t.above = b.wait_cells[0][0] | (static_cast<unsigned long long>(b.wait_cells[0][1]) << 32);
  t.left = b.wait_cells[1][0] | (static_cast<unsigned long long>(b.wait_cells[1][1]) << 32);
  t.clip_w = mini(b.w, g.grid_w - b.x);
  t.clip_h = mini(b.h, g.grid_h - b.y);
  t.status = a.status;
  t.status_host = a.status_host;
  t.limit_ns = a.wait_ns;
  return t;
}

/* INTER: some frame of the launch has phase B inter blocks (inter-intra, intra
 * block copy); a batched step of intra blocks only runs the instantiation
 * without the inter prediction code. A single frame by chains has one build:
 * a key frame takes as long with it as without that code (720p 1.86 ms, 1080p
 * 2.55).
 *
 * Runs chain `c` of the frame: its blocks one after another, each after the
 * blocks it waits for. `edges` and `tmp` are the warp's shared memory. */
template <bool INTER>
__device__ __forceinline__ void run_chain(const FrameArgs& a, int c, int* edges, int* tmp,
                                          int lane) {
  {
    const int u_end = a.chains[c + 1];
    int prev = -1;
    /* the next block's record is loaded while this one runs: in a chain the
     * next block usually starts as soon as this one is published (not in
     * the kernel with inter prediction, whose registers it would spill) */
    int bi_next = a.units[a.chains[c]];
    BlockRec b_next = a.blocks[bi_next];
    for (int u = a.chains[c]; u < u_end; ++u) {
      const int bi = bi_next;
      const BlockRec b = INTER ? a.blocks[bi] : b_next;
      if (u + 1 < u_end) {
        bi_next = a.units[u + 1];
        if (!INTER) b_next = a.blocks[bi_next];
      }
      const int p = b.plane;
      const PlaneGeom& g = a.L.p[p];
      const bool fused = b.kind == AV1B_U_INTRA && b.fuse_res;

      /* the residual image, copied asynchronously: it arrives while the
       * block waits and reads its edges (intra_predict waits for it) */
      const bool has_res = fused && b.tx_count > 0;
      if (has_res) fetch_residual(a, b, tmp, 0, b.h, 0, b.w, lane);

      /* the blocks this one reads from: each lane's acquire load of a done flag
       * orders the samples that block published before that lane's later
       * reads, and the warp barrier extends the order to every lane (all
       * picture reads go through L2, never a stale L1 line) */
      unsigned long long t_claim = 0;
      if (a.trace) t_claim = global_ns();
      /* the block before this one in the chain is this warp's own work, already
       * ordered by the warp barrier that ended it */
      if (!(a.tags && (b.sync & AV1B_SYNC_TAGS))) {
        for (int k = lane; k < b.dep_count; k += 32) {
          const int o = a.deps[b.dep_first + k];
          if (o != prev) wait_block(a, o);
        }
      }
      __syncwarp();
      if (a.trace) {
        /* the dependency published last (its record was written before its
         * flag, so the acquire above made it visible) */
        unsigned long long last = 0, who = ~0ull;
        for (int k = lane; k < b.dep_count; k += 32) {
          const int o = a.deps[b.dep_first + k];
          const unsigned long long t = __ldcg(a.trace + 4 * (size_t)o + 2);
          if (t >= last) {
            last = t;
            who = static_cast<unsigned long long>(o);
          }
        }
        for (int s = 16; s > 0; s >>= 1) {
          const unsigned long long lo = __shfl_down_sync(0xffffffffu, last, s);
          const unsigned long long wo = __shfl_down_sync(0xffffffffu, who, s);
          if (lo > last) {
            last = lo;
            who = wo;
          }
        }
        if (lane == 0) {
          a.trace[4 * (size_t)bi + 0] = t_claim;
          a.trace[4 * (size_t)bi + 1] = global_ns();
          a.trace[4 * (size_t)bi + 3] = who;
        }
      }

      px_t* dst = a.cur + g.off + b.y * g.stride + b.x;
      /* the tagged samples: written with the prediction where it is final */
      unsigned* tagged = a.tags ? a.tags + a.tag_off[p] + b.y * g.grid_w + b.x : nullptr;
      const bool tag_last = tagged && !(b.kind == AV1B_U_INTRA && fused);
      if (b.kind == AV1B_U_INTRA) {
        TagIo t = tag_io(a, b, tagged, !tag_last);
        t.tile = nullptr;
        t.luma_tile = nullptr;
        t.tile_x = t.tile_y = t.tile_w = t.tile_h = t.luma_tile_w = 0;
        t.row0 = 0;
        t.row1 = b.h;
        t.col0 = 0;
        t.cols = b.w;
        /* filter intra (at most 32x32) keeps its predictions after the
         * residual image: tmp[1024 ..] */
        intra_predict(intra_job(a, b), dst, g.stride, a.cur + a.L.p[0].off, a.L.p[0].stride, a.palette_map,
                      a.palette_colors + 8 * b.palette_color_idx, edges, lane, t,
                      has_res ? tmp : nullptr, reinterpret_cast<short*>(tmp + 1024), has_res, [] {});
      } else if constexpr (INTER) {
        InterJob j;
        make_inter_job(a, b, &j);
        int dc = 0;
        if (b.interintra && b.ii_mode == 0) dc = ii_dc(j);
        for (int k = lane; k < b.w * b.h; k += 32) {
          const int yy = k / b.w, xx = k - yy * b.w;
          int v = b.kind == AV1B_U_INTRABC ? inter_core<true>(j, xx, yy) : inter_core(j, xx, yy);
          v = inter_finish(j, xx, yy, v, dc);
          dst[yy * g.stride + xx] = (px_t)v;
        }
      }
      __syncwarp();
      if (!fused)
        for (int t = 0; t < b.tx_count; ++t) add_residual_cg(a, b, a.txs[b.tx_first + t], lane);
      if (tag_last) {
        /* a block whose samples are final only now: its tags from the picture */
        __syncwarp();
        const int tw = mini(b.w, g.grid_w - b.x), th = mini(b.h, g.grid_h - b.y);
        for (int y = 0; y < th; ++y)
          for (int x = lane; x < tw; x += 32)
            st_tag(tagged + y * g.grid_w + x, a.tag | static_cast<unsigned>(ldpx(dst + y * g.stride + x)));
      }

      /* publish, for the blocks that wait on the done flag: the barrier
       * orders every lane's stores before lane 0's release, whose fence
       * (cumulative) makes them visible at GPU scope to any warp that
       * acquires the flag */
      __syncwarp();
      if (a.trace && lane == 0) a.trace[4 * (size_t)bi + 2] = global_ns();
      if (lane == 0 && (!a.tags || (b.sync & AV1B_SYNC_FLAG)))
        st_release(a.done + (size_t)bi * AV1B_FLAG_STRIDE, a.epoch);
      prev = bi;
    }
  }
}

/* What k_regions does not take: frames with inter blocks in phase B or with
 * blocks off the cell grid, and traced ones. */
__global__ void __launch_bounds__(128, AV1B_UNIT_CTAS_PER_SM) k_units(const __grid_constant__ FrameArgs a) {
  extern __shared__ int smem[];
  const int wib = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  int* edges = smem + wib * (3 * AV1B_EDGE_LEN + AV1B_UNIT_SCRATCH);
  int* tmp = edges + 3 * AV1B_EDGE_LEN;
  for (;;) {
    int c = 0;
    /* every warp makes one claim past the last chain and ends: a frame adds
     * its chains and its warps to the counter, which is never reset */
    if (lane == 0) c = static_cast<int>(atomicAdd(a.queue, 1u) - a.queue_base);
    c = __shfl_sync(0xffffffffu, c, 0);
    if (c >= a.n_chains) break;
    run_chain<true>(a, c, edges, tmp, lane);
  }
}

/* Phase B by regions: a CTA claims a region of 64x64 or 128x128 luma samples
 * (in an order in which every region comes after those its blocks wait for)
 * and its warps claim the region's items in order of dependency depth, so
 * every wait is on an item claimed before and the earliest unfinished item
 * always progresses. The path through a frame is a chain of small blocks, most
 * of them neighbours: a step through the tagged words in L2 took a store and a
 * polled load (about 1 us of the 2.0 us step of a 4x4 block) where two blocks
 * of a region now hand their samples over in shared memory. A block of more
 * than AV1B_ITEM_SAMPLES samples is several items of some rows each, and one
 * that several regions share is items in each; they gather its edges each for
 * themselves. (One warp alone took 21 us for a 64x64 block.) An item's record
 * is loaded while the one before it is predicted. Key frames, a pass: 720p
 * 1,128 -> 585 us, 1080p 2,170 -> 1,360, 4K 3,838 -> 2,455. */
struct RegionSmem {
  static constexpr int PER_WARP = 3 * AV1B_EDGE_LEN + AV1B_REGION_SCRATCH;   /* ints */
  int warp[AV1B_REGION_WARPS][PER_WARP];
  BlockRec rec[AV1B_REGION_WARPS];
  int region, next, pad[2];
};

/* then the tiles, and the items */
static size_t region_smem(const Layout& L, int log2) {
  return sizeof(RegionSmem) + region_samples(L, log2) * sizeof(px_t) + region_items(L, log2) * sizeof(int);
}

/* Its CTAs: as many as an SM's shared memory holds, but one on one SM, where
 * the grain templates' CTA runs beside them. */
static int region_ctas(const FrameArgs& a, int n_sm) {
  const int fit = 2 * (region_smem(a.L, a.region_log2) + 1024) <= 228 * 1024 ? 2 * n_sm - 1 : n_sm;
  return a.n_regions < fit ? a.n_regions : fit;
}
unsigned unit_claims(const FrameArgs& a, int n_sm) {
  return units_by_region(a) ? static_cast<unsigned>(a.n_regions + region_ctas(a, n_sm))
                            : static_cast<unsigned>(a.n_chains) + 4u * AV1B_UNIT_CTAS_PER_SM * n_sm;
}

template <class Ahead>
__device__ __forceinline__ void run_item(const FrameArgs& a, const BlockRec& b, int part, int bi, const int4& reg,
                                         volatile unsigned short* tiles, int* edges, int* tmp, int lane,
                                         Ahead&& ahead) {
  const int p = b.plane;
  const PlaneGeom& g = a.L.p[p];
  const int ss_x = p ? a.L.ss_x : 0, ss_y = p ? a.L.ss_y : 0;
  const int tile_w = (1 << a.region_log2) >> ss_x, tile_h = (1 << a.region_log2) >> ss_y;
  /* the part: a column of regions' width of the block, and some of its rows */
  const int cols = mini(b.w, tile_w), across = b.parts > 1 ? b.w / cols : 1;
  const int rows = b.h / (b.parts / across);
  /* the scratch holds a residual of 1024 samples */
  const bool fused = b.fuse_res && (b.tx_count == 0 || rows * cols <= 1024);
  const bool has_res = fused && b.tx_count > 0;
  const int row0 = part / across * rows, col0 = part % across * cols;
  if (has_res) fetch_residual(a, b, tmp, row0, rows, col0, cols, lane);
  /* a block that does not wait on samples: the done flags of the list */
  if (!(b.sync & AV1B_SYNC_TAGS)) {
    for (int k = lane; k < b.dep_count; k += 32) wait_block(a, a.deps[b.dep_first + k]);
    __syncwarp();
  }
  px_t* dst = a.cur + g.off + b.y * g.stride + b.x;
  unsigned* tagged = a.tags + a.tag_off[p] + b.y * g.grid_w + b.x;
  TagIo t = tag_io(a, b, tagged, fused);
  t.tile_w = tile_w;
  t.tile_h = tile_h;
  t.tile_x = b.x - reg.z * tile_w;
  t.tile_y = b.y - reg.w * tile_h;
  t.tile = tiles + (p == 0 ? 0 : (1 << (2 * a.region_log2)) + (p - 1) * t.tile_w * t.tile_h);
  t.luma_tile_w = 1 << a.region_log2;
  t.luma_tile = tiles + (t.tile_y << a.L.ss_y) * t.luma_tile_w + (t.tile_x << a.L.ss_x);
  t.row0 = row0;
  t.row1 = row0 + rows;
  t.col0 = col0;
  t.cols = cols;
  intra_predict(intra_job(a, b), dst, g.stride, a.cur + a.L.p[0].off, a.L.p[0].stride, a.palette_map,
                a.palette_colors + 8 * b.palette_color_idx, edges, lane, t, has_res ? tmp : nullptr,
                reinterpret_cast<short*>(tmp + 1024), has_res, ahead);
  __syncwarp();
  if (!fused) {
    for (int k = 0; k < b.tx_count; ++k) add_residual_cg(a, b, a.txs[b.tx_first + k], lane);
    __syncwarp();
    for (int y = 0; y < t.clip_h; ++y)
      for (int x = lane; x < t.clip_w; x += 32) {
        const unsigned v = static_cast<unsigned>(ldpx(dst + y * g.stride + x));
        t.tile[(t.tile_y + y) * t.tile_w + t.tile_x + x] = static_cast<unsigned short>(v);
        if (t.tile_y + y == t.tile_h - 1 || t.tile_x + x == t.tile_w - 1)
          st_tag(tagged + y * g.grid_w + x, a.tag | v);
      }
  }
  __syncwarp();
  if (lane == 0 && (b.sync & AV1B_SYNC_FLAG)) st_release(a.done + (size_t)bi * AV1B_FLAG_STRIDE, a.epoch);
  __syncwarp();   /* the caller replaces the record */
}

__global__ void __launch_bounds__(32 * AV1B_REGION_WARPS, 1) k_regions(const __grid_constant__ FrameArgs a) {
  extern __shared__ __align__(16) unsigned char region_mem[];
  RegionSmem& m = *reinterpret_cast<RegionSmem*>(region_mem);
  const int n_samples = region_samples(a.L, a.region_log2);
  volatile unsigned short* tiles = reinterpret_cast<volatile unsigned short*>(&m + 1);
  int* items = reinterpret_cast<int*>(&m + 1) + n_samples / 2;
  const int wib = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int* edges = m.warp[wib];
  int* tmp = edges + 3 * AV1B_EDGE_LEN;
  BlockRec& b = m.rec[wib];
  constexpr int kBlockMask = (1 << AV1B_ITEM_SHIFT) - 1;
  for (;;) {
    if (threadIdx.x == 0) {
      /* every CTA makes one claim past the last region and ends */
      m.region = static_cast<int>(atomicAdd(a.queue, 1u) - a.queue_base);
      m.next = 0;
    }
    uint4* clear = reinterpret_cast<uint4*>(region_mem + sizeof(RegionSmem));
    for (int k = threadIdx.x; k < n_samples / 8; k += blockDim.x)
      clear[k] = make_uint4(~0u, ~0u, ~0u, ~0u);
    __syncthreads();
    const int r = m.region;
    if (r >= a.n_regions) break;
    const int4 reg = a.regions[r];
    for (int k = threadIdx.x; k < reg.y; k += blockDim.x) items[k] = a.items[reg.x + k];
    __syncthreads();
    auto claim = [&] {
      int u = 0;
      if (lane == 0) u = atomicAdd(&m.next, 1);
      u = __shfl_sync(0xffffffffu, u, 0);
      return u < reg.y ? items[u] : -1;
    };
    /* a record, a word a lane */
    constexpr int kWords = sizeof(BlockRec) / sizeof(int);
    static_assert(kWords <= 32 && sizeof(BlockRec) % sizeof(int) == 0, "a record is a word a lane");
    auto record = [&](int item) {
      return lane < kWords ? reinterpret_cast<const int*>(a.blocks + (item & kBlockMask))[lane] : 0;
    };
    int item = claim();
    int word = item >= 0 ? record(item) : 0;
    while (item >= 0) {
      if (lane < kWords) reinterpret_cast<int*>(&b)[lane] = word;
      __syncwarp();
      /* the next item is claimed once this one's edges are there */
      int next = -1;
      run_item(a, b, item >> AV1B_ITEM_SHIFT, item & kBlockMask, reg, tiles, edges, tmp, lane, [&] {
        next = claim();
        if (next >= 0) word = record(next);
      });
      item = next;
    }
    /* the tiles and the items are read until every warp is through */
    __syncthreads();
  }
}

/* ---- deblocking ---------------------------------------------------------------------- */
/* Deblocks records recs[0 .. m), m <= AV1B_DB_GROUP, with the warp's lanes
 * spread over their samples: most edges are 4 or 8 samples long, so a warp
 * per edge would leave three lanes of four idle. Lane j < m holds record j;
 * an inclusive scan of the lengths maps each sample to its record, whose
 * fields the sample's lane takes by shuffle, and the warp steps 32 samples at
 * a time. The edges of one pass never filter the same sample (a filter is
 * never longer than the transforms on its sides), so their samples run in
 * any order. */
template <int G = AV1B_DB_GROUP>
__device__ __forceinline__ void deblock_group(px_t* pic, const DeblockRec* recs, int m, int sharpness,
                                              int bd, int maxv, int lane) {
  DeblockRec r{};
  int len = 0;
  if (lane < m) {
    r = recs[lane];
    len = r.len;
  }
  int cum = len;
#pragma unroll
  for (int o = 1; o < G; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, cum, o);
    if (lane >= o) cum += v;
  }
  const int total = __shfl_sync(0xffffffffu, cum, G - 1);
  const int fc = r.filter_size | (r.chroma << 8);
  for (int base = 0; base < total; base += 32) {
    const int t = base + lane;
    int j = 0;
#pragma unroll
    for (int q = 0; q < G - 1; ++q) j += __shfl_sync(0xffffffffu, cum, q) <= t;
    const int start = __shfl_sync(0xffffffffu, cum - len, j);
    const int p_off = __shfl_sync(0xffffffffu, r.p_off, j);
    const int across = __shfl_sync(0xffffffffu, r.across, j);
    const int along = __shfl_sync(0xffffffffu, r.along, j);
    const int level = __shfl_sync(0xffffffffu, static_cast<int>(r.level), j);
    const int fcj = __shfl_sync(0xffffffffu, fc, j);
    if (t < total)
      deblock_px(pic + p_off + (t - start) * along, across, level, sharpness, fcj & 255, fcj >> 8, bd,
                 maxv);
  }
}

/* A warp per G records. */
template <int G>
__global__ void k_deblock(px_t* pic, const DeblockRec* recs, int n, int sharpness, int bd,
                          int maxv) {
  deps_may_start();
  deps_done();
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  const long long r0 = static_cast<long long>(warp) * G;
  if (r0 >= n) return;
  deblock_group<G>(pic, recs + r0, mini(G, n - static_cast<int>(r0)), sharpness, bd, maxv, lane);
}

/* ---- CDEF ------------------------------------------------------------------------------ */
/* CDEF direction search (av1gpu_kernels.h:2601-2660), one thread per 8x8 luma
 * block: the 90 partial sums of the eight directions stay in registers (the
 * loops unroll, so every bin index is a constant). The result packs
 * (variance << 3) | direction. Threads [0, n_grid) search the cells of the
 * 8x8 grid (result index = cell), the rest the listed positions off the grid
 * (result index grid_n + k). Chroma blocks read the search of their luma
 * block, so each luma block is searched once. */
__device__ __forceinline__ void cdef_search_one(const px_t* src, int grid_w, int grid_n,
                                                int n_grid, const unsigned* __restrict__ pos,
                                                int* out, const Layout& L, int t) {
  int x, y, o;
  if (t < n_grid) {
    y = (t / grid_w) << 3;
    x = (t - (t / grid_w) * grid_w) << 3;
    o = t;
  } else {
    const unsigned q = pos[t - n_grid];
    x = q & 0xffff;
    y = q >> 16;
    o = grid_n + (t - n_grid);
  }
  const int stride = L.p[0].stride, cs = L.bit_depth - 8;
  const px_t* b = src + L.p[0].off + y * stride + x;
  int p0[15] = {}, p1[11] = {}, p2[8] = {}, p3[11] = {}, p4[15] = {}, p5[11] = {}, p6[8] = {},
      p7[11] = {};
  const bool vec = ((L.p[0].off + y * stride + x) & 7) == 0;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    int v[8];
    if (vec) {
      const uint4 w = *reinterpret_cast<const uint4*>(b + i * stride);
      const unsigned u[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        v[2 * k] = u[k] & 0xffff;
        v[2 * k + 1] = u[k] >> 16;
      }
    } else {
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] = b[i * stride + j];
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int s = (v[j] >> cs) - 128;
      p0[i + j] += s;
      p1[i + j / 2] += s;
      p2[i] += s;
      p3[3 + i - j / 2] += s;
      p4[7 + i - j] += s;
      p5[3 - i / 2 + j] += s;
      p6[j] += s;
      p7[i / 2 + j] += s;
    }
  }
  const int div[9] = {0, 840, 420, 280, 210, 168, 140, 120, 105};
  int cost[8];
  cost[2] = cost[6] = 0;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    cost[2] += p2[i] * p2[i];
    cost[6] += p6[i] * p6[i];
  }
  cost[2] *= div[8];
  cost[6] *= div[8];
  cost[0] = p0[7] * p0[7] * div[8];
  cost[4] = p4[7] * p4[7] * div[8];
#pragma unroll
  for (int i = 0; i < 7; ++i) {
    cost[0] += (p0[i] * p0[i] + p0[14 - i] * p0[14 - i]) * div[i + 1];
    cost[4] += (p4[i] * p4[i] + p4[14 - i] * p4[14 - i]) * div[i + 1];
  }
  int* odd[4] = {p1, p3, p5, p7};
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int* pt = odd[k];
    int c = 0;
#pragma unroll
    for (int j = 0; j < 5; ++j) c += pt[3 + j] * pt[3 + j];
    c *= div[8];
#pragma unroll
    for (int j = 0; j < 3; ++j) c += (pt[j] * pt[j] + pt[10 - j] * pt[10 - j]) * div[2 * j + 2];
    cost[2 * k + 1] = c;
  }
  int best = 0, d = 0;
#pragma unroll
  for (int i = 0; i < 8; ++i)
    if (cost[i] > best) {
      best = cost[i];
      d = i;
    }
  int opp = 0;
#pragma unroll
  for (int i = 0; i < 8; ++i)
    if (i == ((d + 4) & 7)) opp = cost[i];
  out[o] = (((best - opp) >> 10) << 3) | d;
}

__global__ void __launch_bounds__(128) k_cdef_search(const px_t* src, int grid_w,
                                                     int grid_n, int n_grid,
                                                     const unsigned* __restrict__ pos, int n_extra,
                                                     int* out, const __grid_constant__ Layout L) {
  deps_may_start();
  deps_done();
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n_grid + n_extra) return;
  cdef_search_one(src, grid_w, grid_n, n_grid, pos, out, L, t);
}

__constant__ signed char kCdefDirs[8][2][2] = {
    {{-1, 1}, {-2, 2}}, {{0, 1}, {-1, 2}}, {{0, 1}, {0, 2}}, {{0, 1}, {1, 2}},
    {{1, 1}, {2, 2}},   {{1, 0}, {2, 1}},  {{1, 0}, {2, 0}}, {{1, 0}, {2, -1}},
};
__constant__ unsigned char kCdefUvDir[2][2][8] = {{{0, 1, 2, 3, 4, 5, 6, 7}, {1, 2, 2, 2, 3, 4, 6, 0}},
                                                  {{7, 0, 2, 4, 5, 6, 6, 6}, {0, 1, 2, 3, 4, 5, 6, 7}}};

/* CDEF filter (av1gpu_kernels.h:2662-2775), one half-warp per block: the
 * block and its 2-sample halo staged in shared memory, then 4 samples a lane
 * (luma 8x8) or 1 (4:2:0 chroma 4x4), so chroma blocks leave no lane idle.
 * Everything per block is resolved once before the sample loop: the tap
 * offsets of the three directions, each strength's damping shift (the
 * constrain function's floor_log2), and whether every tap of the block lies
 * inside the plane (then no per-tap bound checks). */
__device__ __forceinline__ int cdef_cst(int diff, int th, int sh) {
  const int m = absi(diff);
  const int v = clampi(th - (m >> sh), 0, m);
  return diff < 0 ? -v : v;
}

/* The same with the hardware's three-input and add-min-relu integer
 * instructions (max(min(th - s, m), 0) is the clamp of th - s to [0, m] for
 * m >= 0). */
__device__ __forceinline__ int cdef_cst3(int diff, int th, int sh) {
  const int m = absi(diff);
  const int v = __viaddmin_s32_relu(th, -(m >> sh), m);
  return diff < 0 ? -v : v;
}

template <bool EDGE>
__device__ __forceinline__ void cdef_samples(const int* win, px_t* d, int stride, int w, int h,
                                             int hl, int x0, int y0, int pw, int ph,
                                             const int (&oy)[6], const int (&ox)[6], int pri,
                                             int psh, int sec, int ssh, int pt0, int pt1,
                                             int maxv) {
  for (int k = hl; k < w * h; k += 16) {
    const int i = k >> (w == 8 ? 3 : (w == 4 ? 2 : 1)), j = k & (w - 1);
    if (EDGE && (y0 + i >= ph || x0 + j >= pw)) continue;
    const int x = win[(i + 2) * 12 + j + 2];
    int sum = 0, lo = x, hi = x;
    if (!EDGE) {
      /* every tap lies in the plane: both taps of a direction at once */
#pragma unroll
      for (int q = 0; q < 6; ++q) {
        const int tap = q == 0 ? pt0 : (q == 1 ? pt1 : (q & 1 ? 1 : 2));
        const int th = q < 2 ? pri : sec, sh = q < 2 ? psh : ssh;
        const int o = oy[q] * 12 + ox[q];
        const int va = win[(i + 2) * 12 + j + 2 - o], vb = win[(i + 2) * 12 + j + 2 + o];
        if (th) sum += tap * (cdef_cst3(va - x, th, sh) + cdef_cst3(vb - x, th, sh));
        lo = __vimin3_s32(lo, va, vb);
        hi = __vimax3_s32(hi, va, vb);
      }
      d[i * stride + j] = (px_t)clampi(clampi(x + ((8 + sum - (sum < 0)) >> 4), lo, hi), 0, maxv);
      continue;
    }
#pragma unroll
    for (int q = 0; q < 6; ++q) {
      const int tap = q == 0 ? pt0 : (q == 1 ? pt1 : (q & 1 ? 1 : 2));
      const int th = q < 2 ? pri : sec, sh = q < 2 ? psh : ssh;
#pragma unroll
      for (int sg = -1; sg <= 1; sg += 2) {
        const int dy = sg * oy[q], dx = sg * ox[q];
        if (EDGE) {
          const int px = x0 + j + dx, py = y0 + i + dy;
          if (px < 0 || px >= pw || py < 0 || py >= ph) continue;
        }
        const int v = win[(i + 2 + dy) * 12 + j + 2 + dx];
        if (th) sum += tap * cdef_cst(v - x, th, sh);
        lo = mini(lo, v);
        hi = maxi(hi, v);
      }
    }
    d[i * stride + j] = (px_t)clampi(clampi(x + ((8 + sum - (sum < 0)) >> 4), lo, hi), 0, maxv);
  }
}

/* One CDEF record by a half-warp (lanes `hmask`, this thread `hl`) with its
 * 12x12 window `win` in shared memory. */
__device__ __forceinline__ void cdef_record(const px_t* __restrict__ src, px_t* dst,
                                            const CdefRec& r, const int* __restrict__ search,
                                            const Layout& L, int* win, int hl, unsigned hmask) {
  const int p = r.plane;
  const bool uv = p > 0;
  const PlaneGeom& g = L.p[p];
  const int bd = L.bit_depth, maxv = (1 << bd) - 1, cs = bd - 8;
  const int w = uv ? (8 >> L.ss_x) : 8, h = uv ? (8 >> L.ss_y) : 8;
  const int pw = g.grid_w, ph = g.grid_h;
  /* the block and its halo; rows and columns above or left of the buffer
   * clamp into it (taps outside the plane are never used) */
  for (StepWalk wk(hl, 16, w + 4); wk.k < (h + 4) * (w + 4); wk.next()) {
    const int i = wk.r, j = wk.q;
    const int y = maxi(r.y - 2 + i, 0), x = maxi(r.x - 2 + j, 0);
    win[i * 12 + j] = src[g.off + y * g.stride + x];
  }
  int pri = r.pri << cs, sec = r.sec << cs;
  const int damping = r.damping + cs - (uv ? 1 : 0);
  int dir = r.dir;
  if (dir < 0) {
    const int sr = search[r.search];
    const int ydir = sr & 7, var = sr >> 3;
    if (uv) {
      dir = pri == 0 ? 0 : kCdefUvDir[L.ss_x][L.ss_y][ydir];
    } else {
      const int vs = (var >> 6) ? mini(floor_log2(var >> 6), 12) : 0;
      dir = pri == 0 ? 0 : ydir;
      pri = var ? ((pri * (4 + vs) + 8) >> 4) : 0;
    }
  }
  __syncwarp(hmask);
  px_t* d = dst + g.off + r.y * g.stride + r.x;
  if (pri == 0 && sec == 0) {
    for (int k = hl; k < w * h; k += 16) {
      const int i = k / w, j = k - i * w;
      if (r.y + i < ph && r.x + j < pw) d[i * g.stride + j] = (px_t)win[(i + 2) * 12 + j + 2];
    }
    return;
  }
  const int ts = (pri >> cs) & 1;
  const int pt0 = ts ? 3 : 4, pt1 = ts ? 3 : 2;
  const int psh = pri ? maxi(0, damping - floor_log2(pri)) : 0;
  const int ssh = sec ? maxi(0, damping - floor_log2(sec)) : 0;
  /* taps: primary (dir) k = 0, 1; secondary (dir - 2, dir + 2) k = 0, 1 */
  int oy[6], ox[6];
#pragma unroll
  for (int q = 0; q < 6; ++q) {
    const int dd = q < 2 ? dir : (q < 4 ? (dir + 6) & 7 : (dir + 2) & 7);
    const int t = q & 1;
    oy[q] = kCdefDirs[dd][t][0];
    ox[q] = kCdefDirs[dd][t][1];
  }
  const bool interior = r.x >= 2 && r.y >= 2 && r.x + w + 2 <= pw && r.y + h + 2 <= ph;
  if (interior)
    cdef_samples<false>(win, d, g.stride, w, h, hl, r.x, r.y, pw, ph, oy, ox, pri, psh, sec, ssh,
                        pt0, pt1, maxv);
  else
    cdef_samples<true>(win, d, g.stride, w, h, hl, r.x, r.y, pw, ph, oy, ox, pri, psh, sec, ssh,
                       pt0, pt1, maxv);
}

__global__ void __launch_bounds__(128) k_cdef(const px_t* __restrict__ src, px_t* dst,
                                              const CdefRec* recs, int n,
                                              const int* __restrict__ search,
                                              const __grid_constant__ Layout L) {
  __shared__ int sw[8][12 * 12];
  const int hw = threadIdx.x >> 4, hl = threadIdx.x & 15;
  const unsigned hmask = 0xffffu << (threadIdx.x & 16);
  const int ri = blockIdx.x * 8 + hw;
  if (ri >= n) return;
  const CdefRec r = recs[ri];
  cdef_record(src, dst, r, search, L, sw[hw], hl, hmask);
}

/* ---- CDEF by tiles ----------------------------------------------------------------------- */
/* The filter of a whole picture, out of place: a CTA takes 64x32 samples of a
 * plane (three planes of cells say how each 8x8 luma block, or the chroma it
 * covers, is filtered), stages them and their 2-sample halo once with 16-byte
 * loads, and copies what no block filters, so the picture needs no snapshot
 * before and the tiles' halos add an eighth to what is read; a half-warp per
 * block staged 144 samples for 64, or 64 for 16, a sample a load.
 *
 * A thread filters four samples of a row as two words of two 16-bit samples.
 * A tap's part is clamp(v, x - l, x + l) with l = max(th - (|v - x| >> sh), 0)
 * - the constrained difference added to x - summed with its weight; the sum
 * less x times the weights is the reference's (the sums of 8- and 10-bit
 * samples, at most 24 x 1023, fit 16 bits; 12-bit ones are summed apart,
 * WIDE). With one of the two strengths zero the other's taps alone cannot
 * leave their own range (weights of 12 / 16), so the zero strength's taps,
 * which would only widen the clip, are not read. Samples outside the plane
 * are staged as 0xffff and take x's place (EDGE tiles only). The CDEF stage of
 * a frame with its search: 4K (coded 2880 wide) 126 -> 79 us, 1080p 51 -> 35,
 * and the copy before it gone; 16 streams 0.69 -> 0.43 ms a step, copies
 * 0.16 ms less. */
#define AV1B_CDEF_PITCH 80
struct CdefTileSmem {
  uint4 win[(AV1B_CDEF_TH + 4) * AV1B_CDEF_PITCH / 8];
};

struct CdefTap {
  int sh;
  unsigned mask, thp1, nth;
  __device__ __forceinline__ CdefTap(int th, int damping) {
    sh = mini(maxi(0, damping - (31 - __clz(th | 1))), 15);
    mask = (0xffffu >> sh) * 0x10001u;
    thp1 = static_cast<unsigned>(th + 1) * 0x10001u;
    nth = (static_cast<unsigned>(-th) & 0xffffu) * 0x10001u;
  }
  /* clamp(v, x - l, x + l) of two samples */
  __device__ __forceinline__ unsigned pull(unsigned x, unsigned v) const {
    const unsigned m = __vmaxu2(v, x) - __vminu2(v, x);
    const unsigned s = (m >> sh) & mask;
    const unsigned l = __viaddmax_s16x2(~s, thp1, 0u);
    const unsigned nl = __viaddmin_s16x2(s, nth, 0u);
    return __viaddmax_s16x2(x, nl, __viaddmin_s16x2(x, l, v));
  }
};

/* Four samples from sample `k` of the window's words on (k of any parity). */
__device__ __forceinline__ void cdef_load4(const unsigned short* win, int k, unsigned* a, unsigned* b) {
  const unsigned* w = reinterpret_cast<const unsigned*>(win) + (k >> 1);
  const unsigned w0 = w[0], w1 = w[1], w2 = w[2];
  const int sh = (k & 1) * 16;
  *a = __funnelshift_r(w0, w1, sh);
  *b = __funnelshift_r(w1, w2, sh);
}

/* x where v is outside the plane. */
__device__ __forceinline__ unsigned cdef_inside(unsigned v, unsigned x) {
  unsigned m = 0;
  if ((v & 0xffffu) == 0xffffu) m = 0xffffu;
  if (v >= 0xffff0000u) m |= 0xffff0000u;
  return (v & ~m) | (x & m);
}

template <bool EDGE, bool WIDE>
__device__ __forceinline__ void cdef_tile_filter(const unsigned short* win, px_t* __restrict__ dst,
                                                 const unsigned* __restrict__ cells,
                                                 const int* search, int search_w,
                                                 const Layout& L, int p, int x0, int y0) {
  const PlaneGeom& g = L.p[p];
  const bool uv = p > 0;
  const int cs = L.bit_depth - 8;
  const int lw = uv ? 3 - L.ss_x : 3, lh = uv ? 3 - L.ss_y : 3;
  const int gw = L.p[0].grid_w >> 3;
  /* four-sample pieces of a cell: a cell's run together */
  const int lp = lw + lh - 2;
  for (int t = threadIdx.x; t < AV1B_CDEF_TW * AV1B_CDEF_TH / 4; t += blockDim.x) {
    const int cell = t >> lp, piece = t & ((1 << lp) - 1);
    const int cx = cell & ((AV1B_CDEF_TW >> lw) - 1), cy = cell >> (6 - lw);
    const int i = (cy << lh) + (piece >> (lw - 2));
    const int j = (cx << lw) + (piece & ((1 << (lw - 2)) - 1)) * 4;
    const int x = x0 + j, y = y0 + i;
    if (x >= g.grid_w || y >= g.grid_h) continue;
    const int ac = (x0 >> lw) + cx, ar = (y0 >> lh) + cy;
    const unsigned word = cells[ar * gw + ac];
    const int k0 = (i + 2) * AV1B_CDEF_PITCH + j + 8;
    const uint2 xv = *reinterpret_cast<const uint2*>(win + k0);
    uint2 out = xv;
    int pri = (word & 255) << cs;
    const int sec = ((word >> 8) & 255) << cs;
    const int damping = static_cast<int>((word >> 16) & 255) + cs - (uv ? 1 : 0);
    int dir = static_cast<int>(word >> 24) - 2;
    if (dir == -1) {
      const int sr = search[ar * search_w + ac];
      const int ydir = sr & 7, var = sr >> 3;
      if (uv) {
        dir = pri == 0 ? 0 : kCdefUvDir[L.ss_x][L.ss_y][ydir];
      } else {
        const int vs = (var >> 6) ? mini(31 - __clz(var >> 6), 12) : 0;
        dir = pri == 0 ? 0 : ydir;
        pri = var ? ((pri * (4 + vs) + 8) >> 4) : 0;
      }
    }
    if (word != 0 && (pri | sec) != 0) {
      unsigned lo0 = xv.x, hi0 = xv.x, lo1 = xv.y, hi1 = xv.y;
      unsigned a0 = 0, a1 = 0, b0 = 0, b1 = 0;   /* sums; WIDE: the high halves' in b */
      int weights = 0;
      const auto taps = [&](const CdefTap& c, int dd, int tap0, int tap1) {
#pragma unroll
        for (int n = 0; n < 2; ++n) {
          const unsigned tap = n ? tap1 : tap0;
          const int o = kCdefDirs[dd][n][0] * AV1B_CDEF_PITCH + kCdefDirs[dd][n][1];
          unsigned va0, va1, vb0, vb1;
          cdef_load4(win, k0 - o, &va0, &va1);
          cdef_load4(win, k0 + o, &vb0, &vb1);
          if (EDGE) {
            va0 = cdef_inside(va0, xv.x);
            va1 = cdef_inside(va1, xv.y);
            vb0 = cdef_inside(vb0, xv.x);
            vb1 = cdef_inside(vb1, xv.y);
          }
          lo0 = __vimin3_u16x2(lo0, va0, vb0);
          hi0 = __vimax3_u16x2(hi0, va0, vb0);
          lo1 = __vimin3_u16x2(lo1, va1, vb1);
          hi1 = __vimax3_u16x2(hi1, va1, vb1);
          /* two pulled samples add up to at most 13 bits a half */
          const unsigned s0 = c.pull(xv.x, va0) + c.pull(xv.x, vb0);
          const unsigned s1 = c.pull(xv.y, va1) + c.pull(xv.y, vb1);
          if (WIDE) {
            a0 += tap * (s0 & 0xffffu);
            b0 += tap * (s0 >> 16);
            a1 += tap * (s1 & 0xffffu);
            b1 += tap * (s1 >> 16);
          } else {
            a0 += tap * s0;
            a1 += tap * s1;
          }
        }
        weights += 2 * (tap0 + tap1);
      };
      if (pri) {
        const int ts = (pri >> cs) & 1;
        taps(CdefTap(pri, damping), dir, ts ? 3 : 4, ts ? 3 : 2);
      }
      if (sec) {
        const CdefTap c(sec, damping);
        taps(c, (dir + 6) & 7, 2, 1);
        taps(c, (dir + 2) & 7, 2, 1);
      }
      const auto finish = [&](unsigned xx, unsigned acc, unsigned lo, unsigned hi) {
        const int v = static_cast<int>(xx), sum = static_cast<int>(acc) - v * weights;
        return static_cast<unsigned>(
            clampi(v + ((8 + sum - (sum < 0)) >> 4), static_cast<int>(lo), static_cast<int>(hi)));
      };
      if (!WIDE) {
        b0 = a0 >> 16;
        b1 = a1 >> 16;
        a0 &= 0xffffu;
        a1 &= 0xffffu;
      }
      out.x = finish(xv.x & 0xffffu, a0, lo0 & 0xffffu, hi0 & 0xffffu) |
              (finish(xv.x >> 16, b0, lo0 >> 16, hi0 >> 16) << 16);
      out.y = finish(xv.y & 0xffffu, a1, lo1 & 0xffffu, hi1 & 0xffffu) |
              (finish(xv.y >> 16, b1, lo1 >> 16, hi1 >> 16) << 16);
    }
    *reinterpret_cast<uint2*>(dst + g.off + y * g.stride + x) = out;
  }
}

/* One tile (bx, by, bz). Early returns are uniform over the CTA. */
__device__ __forceinline__ void cdef_tile_item(const px_t* src, px_t* __restrict__ dst,
                                               const unsigned* __restrict__ cells,
                                               const int* search, int search_w,
                                               const Layout& L, int bx, int by, int bz,
                                               CdefTileSmem& sm) {
  int p = bz;
  if (p > 0) {
    const int t1 = (L.p[1].grid_w + AV1B_CDEF_TW - 1) / AV1B_CDEF_TW;
    if (bx >= t1) {
      bx -= t1;
      p = 2;
    }
  }
  const PlaneGeom& g = L.p[p];
  const int x0 = bx * AV1B_CDEF_TW, y0 = by * AV1B_CDEF_TH;
  if (x0 >= g.grid_w || y0 >= g.grid_h) return;
  /* columns x0 - 8 .. x0 + 71, eight at a time (16 bytes: rows start on
   * 128-byte boundaries); a grid is a multiple of 4 samples wide */
  constexpr int kGroups = AV1B_CDEF_PITCH / 8;
  for (int k = threadIdx.x; k < (AV1B_CDEF_TH + 4) * kGroups; k += blockDim.x) {
    const int i = k / kGroups, q = k - i * kGroups;
    const int y = y0 - 2 + i, x = x0 - 8 + 8 * q;
    uint4 v = make_uint4(~0u, ~0u, ~0u, ~0u);
    if (y >= 0 && y < g.grid_h && x >= 0 && x < g.grid_w) {
      v = *reinterpret_cast<const uint4*>(src + g.off + y * g.stride + x);
      if (x + 8 > g.grid_w) v.z = v.w = ~0u;
    }
    sm.win[i * kGroups + q] = v;
  }
  __syncthreads();
  const unsigned short* win = reinterpret_cast<const unsigned short*>(sm.win);
  cells += p * cdef_cells(L);
  const bool edge = x0 == 0 || y0 == 0 || x0 + AV1B_CDEF_TW + 2 > g.grid_w || y0 + AV1B_CDEF_TH + 2 > g.grid_h;
  if (L.bit_depth > 10)
    cdef_tile_filter<true, true>(win, dst, cells, search, search_w, L, p, x0, y0);
  else if (edge)
    cdef_tile_filter<true, false>(win, dst, cells, search, search_w, L, p, x0, y0);
  else
    cdef_tile_filter<false, false>(win, dst, cells, search, search_w, L, p, x0, y0);
}

__global__ void __launch_bounds__(256) k_cdef_tile(const px_t* src, px_t* __restrict__ dst,
                                                   const unsigned* __restrict__ cells,
                                                   const int* search, int search_w,
                                                   const __grid_constant__ Layout L) {
  __shared__ CdefTileSmem sm;
  deps_may_start();
  deps_done();
  cdef_tile_item(src, dst, cells, search, search_w, L, blockIdx.x, blockIdx.y, blockIdx.z, sm);
}

/* ---- superres ------------------------------------------------------------------------- */
/* One CTA of 128 threads per 512 output samples of a row, a thread per 4
 * (CTAs of half that, 64 threads, took 11 % longer: twice the CTAs,
 * each staging the taps and its span). The source span those outputs read (a
 * superres step is at most one source sample, so at most 512 + 8 samples) is
 * staged in shared memory once, with
 * the clamp to the coded row applied while staging, and the 8-tap phases
 * beside it; each output then reads its taps there. Grid rows: the luma
 * rows, then the chroma rows with plane 1's segments and plane 2's side by
 * side. `border_rows`: only the rows within two of a loop restoration stripe
 * boundary (the rows the restoration reads from the pre-CDEF picture,
 * av1gpu_kernels.h:2832-2845); the reference upscales the whole pre-CDEF
 * picture and reads only these. */
#define AV1B_UP_SPAN 544
/* One CTA item (segment xb of grid row yb): the caller has filled `taps`
 * (the 64 filter phases); the body stages the source span, meets the CTA
 * barrier and writes. Early returns are either uniform over the CTA or after
 * its last barrier. */
__device__ __forceinline__ void upscale_item(const px_t* src, px_t* __restrict__ dst, const Layout& L,
                                             const UpscaleArgs& u, int maxv, int border_rows,
                                             int rows0, int xb, int yb, const short* taps,
                                             px_t* span) {
  int y = yb, p = 0;
  if (y >= rows0) {
    y -= rows0;
    const int xb1 = (L.p[1].out_w + AV1B_UP_OUT - 1) / AV1B_UP_OUT;
    p = 1;
    if (xb >= xb1) {
      xb -= xb1;
      p = 2;
    }
  }
  const PlaneGeom& g = L.p[p];
  if (border_rows) {
    const int sub_y = p > 0 ? L.ss_y : 0;
    const int b = (64 * (y / 4 + 1) - 8) >> sub_y;
    y = b - 2 + (y & 3);
    if (y < 0) return;
  }
  const int xs = xb * AV1B_UP_OUT;
  if (y >= g.out_h || xs >= g.out_w) return;  /* uniform over the CTA */
  const px_t* row = src + g.off + y * g.stride;
  px_t* out = dst + g.off + y * g.stride;
  const int last = g.coded_w - 1;
  const int step = u.step[p], init = u.initial[p] - (1 << 14);
  const int xe = min(xs + AV1B_UP_OUT, g.out_w) - 1;
  const int p0 = (init + xs * step) >> 14;
  const int n = ((init + xe * step) >> 14) - p0 + 8;
  const bool staged = n <= AV1B_UP_SPAN;
  if (staged)
    for (int i = threadIdx.x; i < n; i += blockDim.x) span[i] = row[clampi(p0 - 3 + i, 0, last)];
  __syncthreads();
  const int x0 = xs + threadIdx.x * 4;
  if (x0 > xe) return;
  int o[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int x = min(x0 + q, xe);  /* past the row's end: a repeat, not stored */
    const int sx = init + x * step;
    const int px = sx >> 14;
    const int4 fv = *reinterpret_cast<const int4*>(taps + ((sx & ((1 << 14) - 1)) >> 8) * 8);
    const int f[8] = {(short)fv.x, fv.x >> 16, (short)fv.y, fv.y >> 16,
                      (short)fv.z, fv.z >> 16, (short)fv.w, fv.w >> 16};
    int sum = 0;
    if (staged) {
      const px_t* sp = span + (px - p0);
#pragma unroll
      for (int k = 0; k < 8; ++k) sum += (int)sp[k] * f[k];
    } else {
#pragma unroll
      for (int k = 0; k < 8; ++k) sum += (int)row[clampi(px + k - 3, 0, last)] * f[k];
    }
    o[q] = clampi(rnd2(sum, 7), 0, maxv);
  }
  if (x0 + 3 <= xe && (reinterpret_cast<uintptr_t>(out) & 7) == 0) {
    uint2 v;
    v.x = (unsigned)o[0] | ((unsigned)o[1] << 16);
    v.y = (unsigned)o[2] | ((unsigned)o[3] << 16);
    *reinterpret_cast<uint2*>(out + x0) = v;
  } else {
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if (x0 + q <= xe) out[x0 + q] = (px_t)o[q];
  }
}

__global__ void __launch_bounds__(128) k_upscale(const px_t* src, px_t* __restrict__ dst,
                                                const __grid_constant__ Layout L,
                                                const __grid_constant__ UpscaleArgs u, int maxv,
                                                int border_rows, int rows0) {
  __shared__ __align__(16) short taps[512];
  __shared__ px_t span[AV1B_UP_SPAN];
  deps_may_start();
  for (int i = threadIdx.x; i < 512; i += blockDim.x) taps[i] = kUpscaleFilter[i];
  deps_done();
  upscale_item(src, dst, L, u, maxv, border_rows, rows0, blockIdx.x, blockIdx.y, taps, span);
}

/* ---- loop restoration --------------------------------------------------------------------- */
/* Loop restoration by tiles: one CTA per (plane, stripe piece, 32 columns).
 * A stripe piece is the rows of one 64-row luma stripe (offset by 8), so every
 * sample of the tile reads through the same stripe mapping (get_source_sample,
 * av1gpu_kernels.h:2832-2845), and a 32-column tile lies in one restoration
 * unit (units are 32..256 wide; the last one of a row extends to the edge).
 * The source window (3 samples of margin) is staged in shared memory once.
 * Wiener runs as a horizontal pass into an intermediate (rounded and clipped
 * like the reference's) and a vertical pass. Self-guided computes A and B of
 * every box position the tile needs once - the reference recomputes them nine
 * times per output sample (av1gpu_kernels.h:2928-2970) - then projects. */
#define AV1B_LR_MAXR 64
#define AV1B_LR_WR (AV1B_LR_MAXR + 6)
#define AV1B_LR_WC (AV1B_LR_TW + 6)
#define AV1B_LR_AR (AV1B_LR_MAXR + 2)
#define AV1B_LR_AC (AV1B_LR_TW + 2)

/* A and B of one self-guided box position (i, j) from its box sums `sq`
 * (squares) and `sb` (samples). */
__device__ __forceinline__ void sgr_ab(unsigned sq, int sb, int bd, int n, long long mtable, int one_over_n,
                                       const short* xbyx1, int* a_out, int* b_out) {
  const long long sa = rnd2llz(static_cast<long long>(sq), 2 * (bd - 8));
  const long long sbs = rnd2z(sb, bd - 8);
  long long pv = sa * n - sbs * sbs;
  if (pv < 0) pv = 0;
  const int z = rnd2ll(pv * mtable, 20);
  const int a2 = xbyx1[mini(z, 255)];
  const long long b2 = (long long)(256 - a2) * sb * one_over_n;
  *a_out = a2;
  *b_out = rnd2ll(b2, 12);
}

/* The box sums of a self-guided pass of radius RAD, register blocked: a
 * thread takes one column and LR_G box positions STEP rows apart (the first
 * pass of radius 2 keeps every other row, the second of radius 1 every row),
 * sums each window row it needs across the box once, and adds those row sums
 * down each box - (2 RAD + 1) (STEP (LR_G - 1) + 2 RAD + 1) loads for LR_G
 * positions instead of (2 RAD + 1)^2 each. Positions i = first, first + STEP,
 * ... below `ar` and columns below `ac`; window rows below `wr` are read. */
#define AV1B_LR_G 4
template <int RAD, int STEP>
__device__ __forceinline__ void sgr_box_pass(const int* win, int* a_out, int* b_out, int first, int ar,
                                             int ac, int wr, int bd, int n, long long mtable,
                                             int one_over_n, const short* xbyx1) {
  constexpr int NR = STEP * (AV1B_LR_G - 1) + 2 * RAD + 1;
  const int rows = ar > first ? (ar - first + STEP - 1) / STEP : 0;
  const int groups = (rows + AV1B_LR_G - 1) / AV1B_LR_G;
  for (int it = threadIdx.x; it < groups * ac; it += blockDim.x) {
    const int g = it / ac, j = it - g * ac;
    const int i0 = first + g * AV1B_LR_G * STEP;
    int hs[NR];
    unsigned hq[NR];
#pragma unroll
    for (int t = 0; t < NR; ++t) {
      const int row = i0 + 2 - RAD + t;
      int sum = 0;
      unsigned sq = 0;
      if (row < wr) {
        const int* w = win + row * AV1B_LR_WC + j + 2 - RAD;
#pragma unroll
        for (int dx = 0; dx <= 2 * RAD; ++dx) {
          const int c = w[dx];
          sum += c;
          sq += static_cast<unsigned>(c * c);
        }
      }
      hs[t] = sum;
      hq[t] = sq;
    }
#pragma unroll
    for (int k = 0; k < AV1B_LR_G; ++k) {
      const int i = i0 + k * STEP;
      if (i < ar) {
        int sb = 0;
        unsigned sq = 0;   /* at most 25 * 4095^2 */
#pragma unroll
        for (int t = 0; t <= 2 * RAD; ++t) {
          sb += hs[k * STEP + t];
          sq += hq[k * STEP + t];
        }
        sgr_ab(sq, sb, bd, n, mtable, one_over_n, xbyx1, a_out + i * AV1B_LR_AC + j,
               b_out + i * AV1B_LR_AC + j);
      }
    }
  }
}

/* Shared memory of one loop restoration tile. */
struct LrSmem {
  int win[AV1B_LR_WR * AV1B_LR_WC];
  int aux[2][2][AV1B_LR_AR * AV1B_LR_AC];  /* Wiener: aux[0][0] = intermediate */
  short xbyx1[256];   /* a2 = ((z << 8) + z / 2) / (z + 1), by z */
};

/* One tile (bx, stripe, bz). Early returns are uniform over the CTA or after
 * its last barrier. */
__device__ __forceinline__ void lr_tile_item(const px_t* cdef, const px_t* curr, px_t* __restrict__ dst,
                                             const Layout& L, const LrArgs& r, int maxv,
                                             int copy_rest, int bx, int stripe, int bz,
                                             LrSmem& sm) {
  int* win = sm.win;
  auto& aux = sm.aux;
  short* xbyx1 = sm.xbyx1;
  /* grid z: luma, then chroma with plane 1's tiles and plane 2's side by side */
  int p = bz;
  if (p > 0) {
    const int t1 = (L.p[1].out_w + AV1B_LR_TW - 1) / AV1B_LR_TW;
    if (bx >= t1) {
      bx -= t1;
      p = 2;
    }
  }
  const PlaneGeom& g = L.p[p];
  const int sub_y = p > 0 ? L.ss_y : 0;
  const int x0 = bx * AV1B_LR_TW;
  if (x0 >= g.out_w) return;
  /* the stripe piece */
  const int s0 = (-8 + stripe * 64) >> sub_y;
  const int s1 = s0 + (64 >> sub_y) - 1;
  const int y0 = maxi(s0, 0), y1 = mini(g.out_h, s1 + 1);
  if (y0 >= y1) return;
  const int tw = mini(AV1B_LR_TW, g.out_w - x0), th = y1 - y0;
  LrUnitRec u{};
  if (r.type[p]) {
    const int us = r.unit_size[p];
    const int urow = mini(r.unit_rows[p] - 1, ((((y0 << sub_y) + 8) >> sub_y) / us));
    const int ucol = mini(r.unit_cols[p] - 1, x0 / us);
    const int idx = urow * r.unit_cols[p] + ucol;
    if (idx < r.n_units[p]) u = r.units[p][idx];
  }
  if (u.type != 1 && u.type != 2) {
    /* not restored: with `copy_rest` (the source is not the destination's
     * own content) the tile passes through */
    if (copy_rest && (tw & 7) == 0) {
      /* eight samples a load: tiles start on multiples of 32 samples of rows
       * that start on 128-byte boundaries */
      const int groups = tw >> 3;
      for (int k = threadIdx.x; k < th * groups; k += blockDim.x) {
        const int i = k / groups, o = g.off + (y0 + i) * g.stride + x0 + 8 * (k - i * groups);
        *reinterpret_cast<uint4*>(dst + o) = *reinterpret_cast<const uint4*>(cdef + o);
      }
    } else if (copy_rest) {
      for (StepWalk wk(threadIdx.x, blockDim.x, tw); wk.k < th * tw; wk.next())
        dst[g.off + (y0 + wk.r) * g.stride + x0 + wk.q] = cdef[g.off + (y0 + wk.r) * g.stride + x0 + wk.q];
    }
    return;
  }
  const int wr = th + 6, wc = tw + 6;
  const px_t* pc = cdef + g.off;
  const px_t* pp = curr + g.off;
  /* source window: rows y0-3 .., columns x0-3 .. */
  for (StepWalk wk(threadIdx.x, blockDim.x, wc); wk.k < wr * wc; wk.next()) {
    const int i = wk.r, j = wk.q;
    const int x = clampi(x0 - 3 + j, 0, g.out_w - 1);
    const int y = clampi(y0 - 3 + i, 0, g.out_h - 1);
    int v;
    if (y < s0) v = pp[maxi(y, s0 - 2) * g.stride + x];
    else if (y > s1) v = pp[mini(y, s1 + 2) * g.stride + x];
    else v = pc[y * g.stride + x];
    win[i * AV1B_LR_WC + j] = v;
  }
  __syncthreads();
  const int bd = L.bit_depth;
  px_t* out = dst + g.off + y0 * g.stride + x0;
  if (u.type == 1) {
    const int r0 = bd == 12 ? 5 : 3, r1 = bd == 12 ? 9 : 11;
    const int offset = 1 << (bd + 7 - r0 - 1);
    const int limit = (1 << (bd + 1 + 7 - r0)) - 1;
    int ht[7], vt[7];
    for (int t = 0; t < 3; ++t) {
      ht[t] = ht[6 - t] = u.hf[t];
      vt[t] = vt[6 - t] = u.vf[t];
    }
    ht[3] = 128 - 2 * (u.hf[0] + u.hf[1] + u.hf[2]);
    vt[3] = 128 - 2 * (u.vf[0] + u.vf[1] + u.vf[2]);
    /* the intermediate has up to 70 rows: it spans aux[0][0] and aux[0][1] */
    static_assert(AV1B_LR_WR * AV1B_LR_AC <= 2 * AV1B_LR_AR * AV1B_LR_AC, "Wiener intermediate");
    int* mid = &aux[0][0][0];
    for (StepWalk wk(threadIdx.x, blockDim.x, tw); wk.k < wr * tw; wk.next()) {
      const int i = wk.r, j = wk.q;
      const int* w = win + i * AV1B_LR_WC + j;
      int acc = 0;
#pragma unroll
      for (int t = 0; t < 7; ++t) acc += ht[t] * w[t];
      mid[i * AV1B_LR_AC + j] = clampi(rnd2(acc, r0), -offset, limit - offset);
    }
    __syncthreads();
    for (StepWalk wk(threadIdx.x, blockDim.x, tw); wk.k < th * tw; wk.next()) {
      const int i = wk.r, j = wk.q;
      int acc = 0;
#pragma unroll
      for (int t = 0; t < 7; ++t) acc += vt[t] * mid[(i + t) * AV1B_LR_AC + j];
      out[i * g.stride + j] = (px_t)clampi(rnd2(acc, r1), 0, maxv);
    }
    return;
  }
  /* self-guided: A and B of both passes on rows y0-1 .. y1, columns x0-1 .. */
  for (int z = threadIdx.x; z < 256; z += blockDim.x)
    xbyx1[z] = static_cast<short>(z >= 255 ? 256 : (z == 0 ? 1 : ((z << 8) + (z / 2)) / (z + 1)));
  __syncthreads();
  const int ar = th + 2, ac = tw + 2;
  /* unrolled: the unit record stays in registers (indexed by a loop
   * variable it would live in local memory) */
#pragma unroll
  for (int pass = 0; pass < 2; ++pass) {
    const int rad = u.r[pass];
    if (rad == 0) continue;
    const int n = (2 * rad + 1) * (2 * rad + 1);
    const long long n2e = (long long)n * n * u.e[pass];
    const long long mtable = ((1LL << 20) + n2e / 2) / n2e;
    const int one_over_n = ((1 << 12) + (n / 2)) / n;
    /* the first pass keeps the odd rows of the picture only */
    if (pass == 0 && rad == 2) {
      sgr_box_pass<2, 2>(win, aux[0][0], aux[0][1], y0 & 1, ar, ac, wr, bd, n, mtable, one_over_n, xbyx1);
      continue;
    }
    if (pass == 1 && rad == 1) {
      sgr_box_pass<1, 1>(win, aux[1][0], aux[1][1], 0, ar, ac, wr, bd, n, mtable, one_over_n, xbyx1);
      continue;
    }
    for (StepWalk wk(threadIdx.x, blockDim.x, ac); wk.k < ar * ac; wk.next()) {
      const int i = wk.r, j = wk.q;
      /* the first pass reads odd rows only */
      if (pass == 0 && !((y0 - 1 + i) & 1)) continue;
      unsigned sq = 0;   /* at most 25 * 4095^2 */
      int sb = 0;
      for (int dy = -rad; dy <= rad; ++dy) {
        const int* w = win + (i + 2 + dy) * AV1B_LR_WC + j + 2;
        for (int dx = -rad; dx <= rad; ++dx) {
          const int c = w[dx];
          sq += static_cast<unsigned>(c * c);
          sb += c;
        }
      }
      sgr_ab(sq, sb, bd, n, mtable, one_over_n, xbyx1, &aux[pass][0][i * AV1B_LR_AC + j],
             &aux[pass][1][i * AV1B_LR_AC + j]);
    }
  }
  __syncthreads();
  const int w0 = u.xqd[0], w1 = u.xqd[1], w2 = 128 - w0 - w1;
  for (StepWalk wk(threadIdx.x, blockDim.x, tw); wk.k < th * tw; wk.next()) {
    const int i = wk.r, j = wk.q;
    const int y = y0 + i;
    const int v = win[(i + 3) * AV1B_LR_WC + j + 3];
    int flt[2] = {0, 0};
#pragma unroll
    for (int pass = 0; pass < 2; ++pass) {
      if (u.r[pass] == 0) continue;
      int a = 0, b = 0;
      for (int dy = -1; dy <= 1; ++dy)
        for (int dx = -1; dx <= 1; ++dx) {
          int wgt;
          if (pass == 0) wgt = ((y + dy) & 1) ? (dx == 0 ? 6 : 5) : 0;
          else wgt = (dx == 0 || dy == 0) ? 4 : 3;
          if (!wgt) continue;
          const int o = (i + 1 + dy) * AV1B_LR_AC + j + 1 + dx;
          a += wgt * aux[pass][0][o];
          b += wgt * aux[pass][1][o];
        }
      const int shift = (pass == 0 && (y & 1)) ? 4 : 5;
      flt[pass] = rnd2ll((long long)a * v + b, 8 + shift - 4);
    }
    const int vs = v << 4;
    long long t = (long long)w1 * vs;
    t += (long long)w0 * (u.r[0] ? flt[0] : vs);
    t += (long long)w2 * (u.r[1] ? flt[1] : vs);
    out[i * g.stride + j] = (px_t)clampi(rnd2ll(t, 11), 0, maxv);
  }
}

__global__ void __launch_bounds__(256) k_lr_tile(const px_t* cdef, const px_t* curr, px_t* __restrict__ dst,
                                                 const __grid_constant__ Layout L,
                                                 const __grid_constant__ LrArgs r, int maxv,
                                                 int copy_rest) {
  __shared__ LrSmem sm;
  deps_may_start();
  deps_done();
  lr_tile_item(cdef, curr, dst, L, r, maxv, copy_rest, blockIdx.x, blockIdx.y, blockIdx.z, sm);
}

/* ---- film grain ------------------------------------------------------------------------------- */

/* Generates the three grain templates (7.18.3.3): Gaussian noise from the LFSR
 * (every draw independent through the orbit table) on all threads of the
 * block, then the auto-regressive filters, one warp a template: a sample
 * reads the samples of its own row to its left and of the rows above within
 * +-lag columns, so with row y starting LAG + 1 steps after row y - 1 every
 * step has one sample of each row, and a warp holds the rows of one step in
 * its lanes. */

/* The position stride of the templates in shared memory, all three planes. */
#define AV1B_GRAIN_W 82

/* One template's auto-regressive filter by one warp, LAG 2 or 3 (shorter
 * lags run as LAG 2 with zero taps). Lane l takes rows l, l + 32, ..: at step
 * t the row's column x = t - S y, S = LAG + 1 (a row is finished before the
 * lane's next one starts: 82 columns and the lead-in of LAG are fewer than
 * 32 S steps). The value above at column x + LAG, the newest one a sample
 * reads, is the output of the lane below's step before, taken by shuffle;
 * the rows further up were written at least LAG + 2 steps ago and come from
 * shared memory, loaded a step ahead. Each arriving value is added, weighted,
 * to the sums of the 2 LAG + 1 positions that read it; the sums rotate
 * through registers, a block of 2 LAG + 1 steps unrolled so that their
 * indexes are constants. What bounds it is the chain of one step - shuffle,
 * multiply-add, round, clip - times 82 + S (rows - 1) steps; a thread a row
 * with every tap a shared-memory read and a block barrier a step took 0.27 us
 * a step (150 us a frame's templates). */
template <int LAG, bool CHROMA>
struct GrainWave {
  static constexpr int R = 2 * LAG + 1, S = LAG + 1;
  int co[LAG + 1][R];        /* taps by rows up, then column; row 0: the left ones */
  int luma_co;
  int acc[R];
  int x, y, prev;
  int noise, up2, up3;       /* of the coming step, loaded ahead */

  __device__ __forceinline__ void taps(const int* c, int lag, int lane) {
#pragma unroll
    for (int dr = 0; dr <= LAG; ++dr)
#pragma unroll
      for (int k = 0; k < R; ++k) {
        const int dc = k - LAG;
        const bool in = dr <= lag && dc >= -lag && dc <= lag && (dr > 0 || dc < 0);
        co[dr][k] = in ? c[(lag - dr) * (2 * lag + 1) + dc + lag] : 0;
      }
    luma_co = CHROMA ? c[2 * lag * (lag + 1)] : 0;
#pragma unroll
    for (int k = 0; k < R; ++k) acc[k] = 0;
    y = lane;
    x = -3 - S * lane;
    prev = noise = up2 = up3 = 0;
  }

  /* Template entry (row, col) or, outside the template, any entry: those only
   * reach positions that keep their noise. */
  static __device__ __forceinline__ int at(const short* t, int row, int col) {
    return t[maxi(0, mini(row * AV1B_GRAIN_W + col, AV1B_GRAIN_W * 73 - 1))];
  }

  /* R steps. gw x gh: the template; luma: its luma template when the chroma
   * filter reads it. */
  __device__ __forceinline__ void steps(short* tmpl, int gw, int gh, const short* luma, int sx, int sy,
                                        int arshift, int gmin, int gmax, int lane) {
#pragma unroll
    for (int q = 0; q < R; ++q) {
      const int above = __shfl_sync(0xffffffffu, prev, (lane + 31) & 31);
      int base = acc[q] + ((noise * 2 + 1) << (arshift - 1));
      if (CHROMA && luma) {
        const int lx = mini(maxi(((x - 3) << sx) + 3, 0), AV1B_GRAIN_W - 1 - sx);
        const int ly = mini(maxi(((y - 3) << sy) + 3, 0), 72 - sy);
        const short* lp = luma + ly * AV1B_GRAIN_W + lx;
        int v = lp[0];
        if (sx) v += lp[1];
        if (sy) v += lp[AV1B_GRAIN_W] + (sx ? lp[AV1B_GRAIN_W + 1] : 0);
        base += rnd2z(v, sx + sy) * luma_co;
      }
      /* this step's sum first: the older rows, the left neighbour, and last
       * the neighbour above, whose shuffle is the longest wait */
      base += up2 * co[2][R - 1 - 0] + prev * co[0][LAG - 1];
      if (LAG == 3) base += up3 * co[LAG][R - 1];
      const int sum = base + above * co[1][R - 1];
      const bool keep = x < 3 || x >= gw - 3 || y < 3;
      const int out = keep ? noise : clampi(sum >> arshift, gmin, gmax);
      if (!keep && y < gh) tmpl[y * AV1B_GRAIN_W + x] = static_cast<short>(out);
      /* the positions after this one that read the same values */
#pragma unroll
      for (int k = 1; k < R; ++k) {
        int v = above * co[1][R - 1 - k] + up2 * co[2][R - 1 - k];
        if (LAG == 3) v += up3 * co[LAG][R - 1 - k];
        if (k < LAG) v += prev * co[0][LAG - 1 - k];
        acc[(q + k) % R] += v;
      }
      acc[q] = 0;
      prev = out;
      if (++x == gw) {
        x -= 32 * S;
        y += 32;
      }
      noise = at(tmpl, y, x);
      up2 = at(tmpl, y - 2, x + LAG);
      if (LAG == 3) up3 = at(tmpl, y - 3, x + LAG);
      __syncwarp();
    }
  }
};

/* The auto-regressive filters of the three templates (7.18.3.3) by warps 0
 * (luma), 1 and 2 (chroma) of the block; `tid` < 96. Chroma trails luma: in
 * iteration k, between two barriers of the three warps, luma runs its steps
 * 2R k .. 2R (k + 1) - 1 and chroma, from k = 1 on, R (k - 1) .. R k - 1 where
 * chroma is subsampled (its sample of step s reads luma of step 2s - 5 at
 * most), 2R (k - 1) .. 2R k - 1 where it is not (step s). */
template <int LAG>
__device__ __forceinline__ void grain_ar(const GrainParamsDev& prm, short* luma, short* cb, short* cr,
                                         int cw, int ch, bool chroma, int arshift, int gmin, int gmax,
                                         int tid) {
  constexpr int R = 2 * LAG + 1, S = LAG + 1;
  const int warp = tid >> 5, lane = tid & 31, lag = prm.ar_coeff_lag;
  const bool do_luma = prm.num_y_points > 0;
  const int sx = prm.ss_x, sy = prm.ss_y;
  const int per = sx || sy ? 1 : 2;   /* chroma's blocks of R steps an iteration */
  const int luma_it = do_luma ? (3 + AV1B_GRAIN_W + S * 72 + 2 * R - 1) / (2 * R) : 0;
  const int chroma_it = chroma ? (3 + cw + S * (ch - 1) + per * R - 1) / (per * R) + 1 : 0;
  const int its = maxi(luma_it, chroma_it);
  if (warp == 0) {
    GrainWave<LAG, false> w;
    w.taps(prm.ar_y, lag, lane);
    for (int k = 0; k < its; ++k) {
      if (k < luma_it) {
#pragma unroll 1
        for (int r = 0; r < 2; ++r)
          w.steps(luma, AV1B_GRAIN_W, 73, nullptr, 0, 0, arshift, gmin, gmax, lane);
      }
      if (chroma) asm volatile("bar.sync 1, 96;" ::: "memory");
    }
  } else if (chroma) {
    GrainWave<LAG, true> w;
    short* t = warp == 1 ? cb : cr;
    w.taps(warp == 1 ? prm.ar_cb : prm.ar_cr, lag, lane);
    for (int k = 0; k < its; ++k) {
      if (k >= 1 && k < chroma_it) {
#pragma unroll 1
        for (int r = 0; r < per; ++r)
          w.steps(t, cw, ch, do_luma ? luma : nullptr, sx, sy, arshift, gmin, gmax, lane);
      }
      asm volatile("bar.sync 1, 96;" ::: "memory");
    }
  }
}

/* The templates live in shared memory while the auto-regressive wavefront
 * runs (hundreds of dependent steps: every tap a shared-memory read, not a
 * global one) and are written out at the end. */
struct GrainTemplateSmem {
  short luma[82 * 73], cb[82 * 73], cr[82 * 73];
};

/* Every thread of the CTA runs it (the filters on its first three warps);
 * it has no early return. */
__device__ __forceinline__ void grain_template_body(GrainState* gs, const int* gs_src,
                                                    const GrainParamsDev& prm, const uint16_t* orbit,
                                                    const uint16_t* pos, GrainTemplateSmem& sm) {
  /* the frame's grain constants and scaling tables, from its plan (null: in
   * place already) */
  if (gs_src) {
    constexpr int tail = static_cast<int>(offsetof(GrainState, lut));
    constexpr int words = static_cast<int>((sizeof(GrainState) - tail) / 4);
    int* dst = reinterpret_cast<int*>(reinterpret_cast<char*>(gs) + tail);
    for (int k = threadIdx.x; k < words; k += blockDim.x) dst[k] = gs_src[k];
  }
  short* s_luma = sm.luma;
  short* s_cb = sm.cb;
  short* s_cr = sm.cr;
  const int tid = threadIdx.x;
  const int bd = prm.bitdepth;
  const int shift = 12 - bd + prm.grain_scale_shift;
  const int gmin = -(128 << (bd - 8)), gmax = (256 << (bd - 8)) - 1 - (128 << (bd - 8));
  const int cw = prm.ss_x ? 44 : AV1B_GRAIN_W, ch = prm.ss_y ? 38 : 73;
  short* luma = s_luma;
  short* cb = s_cb;
  short* cr = s_cr;
  /* Gaussian fill: draw k is the LFSR's state k + 1 steps after its seed */
  const auto draw = [&](unsigned seed, unsigned first, int k) {
    const int st = seed ? orbit[(first + static_cast<unsigned>(k) + 1u) % 65535u] : 0;
    return rnd2z(kGaussianSequence[(st >> 5) & 2047], shift);
  };
  {
    const bool on = prm.num_y_points > 0;
    const unsigned seed = (unsigned)prm.seed & 0xffffu, first = pos[seed];
#pragma unroll 8
    for (int k = tid; k < 82 * 73; k += blockDim.x)
      luma[k] = static_cast<short>(on ? draw(seed, first, k) : 0);
  }
  const bool chroma = prm.chroma_scaling_from_luma || prm.num_cb_points > 0 || prm.num_cr_points > 0;
  if (chroma) {
    const bool acb = prm.num_cb_points > 0 || prm.chroma_scaling_from_luma;
    const bool acr = prm.num_cr_points > 0 || prm.chroma_scaling_from_luma;
    const unsigned sb = ((unsigned)prm.seed ^ 0xb524u) & 0xffffu, sr = ((unsigned)prm.seed ^ 0x49d8u) & 0xffffu;
    const unsigned fb = pos[sb], fr = pos[sr];
#pragma unroll 4
    for (int k = tid; k < cw * ch; k += blockDim.x) {
      const int y = k / cw, o = y * AV1B_GRAIN_W + k - y * cw;
      cb[o] = static_cast<short>(acb ? draw(sb, fb, k) : 0);
      cr[o] = static_cast<short>(acr ? draw(sr, fr, k) : 0);
    }
  }
  __syncthreads();
  const int arshift = prm.ar_coeff_shift_minus_6 + 6;
  if (tid < 96) {
    if (prm.ar_coeff_lag >= 3)
      grain_ar<3>(prm, luma, cb, cr, cw, ch, chroma, arshift, gmin, gmax, tid);
    else
      grain_ar<2>(prm, luma, cb, cr, cw, ch, chroma, arshift, gmin, gmax, tid);
  }
  __syncthreads();
  for (int k = tid; k < 82 * 73; k += blockDim.x) gs->luma[k] = luma[k];
  if (chroma)
    for (int k = tid; k < cw * ch; k += blockDim.x) {
      const int y = k / cw, o = y * AV1B_GRAIN_W + k - y * cw;
      gs->cb[k] = cb[o];
      gs->cr[k] = cr[o];
    }
}

__global__ void __launch_bounds__(256) k_grain_template(GrainState* gs, const int* gs_src,
                                                        const __grid_constant__ GrainParamsDev prm,
                                                        const uint16_t* orbit, const uint16_t* pos) {
  __shared__ GrainTemplateSmem sm;
  grain_template_body(gs, gs_src, prm, orbit, pos, sm);
}

/* The stripe values of plane `p` (7.18.3.5, the horizontal half: the grain
 * block that covers the column, blended with the previous block at the two -
 * one for subsampled chroma - overlap columns) of four samples
 * x0 .. x0 + 3 of one row, x0 a multiple of 4: they lie in one grain block,
 * whose random offset is computed once; only a group starting a block has
 * overlap columns. */
__device__ __forceinline__ void grain_stripe4(const GrainState* gs, const short* grain, int src_w,
                                              int sub_x, int sub_y, int s, int row, int x0,
                                              const uint16_t* orbit, const uint16_t* pos, int gmin,
                                              int gmax, bool overlap, int n[4]) {
  unsigned st0 = (unsigned)gs->seed & 0xffffu;
  st0 ^= (unsigned)(((s * 37 + 178) & 255) << 8);
  st0 ^= (unsigned)((s * 173 + 105) & 255);
  st0 &= 0xffffu;
  const int bw_log = sub_x ? 4 : 5;
  const int k = x0 >> bw_log, j0 = x0 & ((1 << bw_log) - 1);
  auto block_row = [&](int blk) {
    const int r = (lfsr_after(orbit, pos, st0, blk + 1) >> 8) & 255;
    const int ox = r >> 4, oy = r & 15;
    const int src_x = sub_x ? 6 + ox : 9 + ox * 2;
    const int src_y = sub_y ? 6 + oy : 9 + oy * 2;
    return grain + (src_y + row) * src_w + src_x;
  };
  const short* cur = block_row(k) + j0;
#pragma unroll
  for (int q = 0; q < 4; ++q) n[q] = cur[q];
  if (overlap && k > 0 && j0 == 0) {
    const short* prev = block_row(k - 1);
    if (!sub_x) {
      n[0] = clampi(rnd2z((int)prev[32] * 27 + n[0] * 17, 5), gmin, gmax);
      n[1] = clampi(rnd2z((int)prev[33] * 17 + n[1] * 27, 5), gmin, gmax);
    } else {
      n[0] = clampi(rnd2z((int)prev[16] * 23 + n[0] * 22, 5), gmin, gmax);
    }
  }
}

/* Film grain blend, out of place: `src` is the decoded picture (luma read
 * before any grain), `dst` gets the output picture. One thread per four
 * samples of a row (8-byte loads and stores; a chroma group reads its luma as
 * one 8- or 16-byte load); the arithmetic per sample is that of
 * 7.18.3.5 (the no-allocation entry point's grain_sample is the same per
 * sample). Grid rows are the luma rows, then the chroma rows
 * with plane 1's groups and plane 2's side by side, so a chroma row of
 * 4:2:0 fills a grid row as a luma row does. */
/* The film grain output of four samples x0 .. x0 + 3 (x0 a multiple of 4) of
 * row y of plane p, from their decoded values `orig` (7.18.3.5); `src` is the
 * picture before grain (a chroma sample reads its luma there), `vec` whether
 * it is 16-byte aligned. */
__device__ __forceinline__ void grain_group4(const px_t* __restrict__ src, const Layout& L,
                                             const GrainState* gs, const uint16_t* orbit,
                                             const uint16_t* pos, int p, int y, int x0, bool vec,
                                             const int (&orig)[4], int (&out)[4]) {
  const int bd = gs->bitdepth;
#pragma unroll
  for (int q = 0; q < 4; ++q) out[q] = orig[q];
  const bool active = p == 0 ? gs->num_points[0] > 0 : (gs->chroma_from_luma || gs->num_points[p] > 0);
  if (active) {
    const int sub_x = p ? L.ss_x : 0, sub_y = p ? L.ss_y : 0;
    const int gmin = -(128 << (bd - 8)), gmax = (256 << (bd - 8)) - 1 - (128 << (bd - 8));
    const short* grain = p == 0 ? gs->luma : (p == 1 ? gs->cb : gs->cr);
    const int src_w = p == 0 ? 82 : gs->chroma_w;
    const bool overlap = gs->overlap != 0;
    /* vertical half: stripes of 32 (16) rows, blended with the stripe above */
    const int sh = 5 - sub_y;
    const int s = y >> sh, row = y - (s << sh);
    int n[4];
    grain_stripe4(gs, grain, src_w, sub_x, sub_y, s, row, x0, orbit, pos, gmin, gmax, overlap, n);
    if (overlap && s > 0) {
      if (!sub_y && row < 2) {
        int old[4];
        grain_stripe4(gs, grain, src_w, sub_x, sub_y, s - 1, row + 32, x0, orbit, pos, gmin, gmax,
                      overlap, old);
#pragma unroll
        for (int q = 0; q < 4; ++q)
          n[q] = clampi(rnd2z(row == 0 ? old[q] * 27 + n[q] * 17 : old[q] * 17 + n[q] * 27, 5), gmin,
                        gmax);
      } else if (sub_y && row == 0) {
        int old[4];
        grain_stripe4(gs, grain, src_w, sub_x, sub_y, s - 1, 16, x0, orbit, pos, gmin, gmax, overlap,
                      old);
#pragma unroll
        for (int q = 0; q < 4; ++q) n[q] = clampi(rnd2z(old[q] * 23 + n[q] * 22, 5), gmin, gmax);
      }
    }
    int index[4];
    if (p == 0) {
#pragma unroll
      for (int q = 0; q < 4; ++q) index[q] = orig[q];
    } else {
      /* the co-located luma sample and its right neighbour (clamped to the
       * luma width), before grain */
      const PlaneGeom& gl = L.p[0];
      const int ly = y << L.ss_y, lx0 = x0 << L.ss_x;
      const px_t* lrow = src + gl.off + ly * gl.stride;
      int lum[8];
      if (vec && L.ss_x) {
        const uint4 v = *reinterpret_cast<const uint4*>(lrow + lx0);
        lum[0] = v.x & 0xffff;
        lum[1] = v.x >> 16;
        lum[2] = v.y & 0xffff;
        lum[3] = v.y >> 16;
        lum[4] = v.z & 0xffff;
        lum[5] = v.z >> 16;
        lum[6] = v.w & 0xffff;
        lum[7] = v.w >> 16;
      } else if (vec) {
        const uint2 v = *reinterpret_cast<const uint2*>(lrow + lx0);
        lum[0] = v.x & 0xffff;
        lum[1] = v.x >> 16;
        lum[2] = v.y & 0xffff;
        lum[3] = v.y >> 16;
        lum[4] = lum[5] = lum[6] = lum[7] = 0;
      } else {
#pragma unroll
        for (int q = 0; q < 8; ++q) lum[q] = (L.ss_x || q < 4) ? lrow[min(lx0 + q, gl.out_w - 1)] : 0;
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        int avg;
        if (L.ss_x) {
          const int lx = lx0 + 2 * q;
          const int l0 = lum[2 * q];
          const int l1 = lx + 1 < gl.out_w ? lum[2 * q + 1] : l0;
          avg = rnd2z(l0 + l1, 1);
        } else {
          avg = lum[q];
        }
        if (gs->chroma_from_luma) {
          index[q] = avg;
        } else {
          const int comb = avg * (gs->luma_mult[p] - 128) + orig[q] * (gs->mult[p] - 128);
          index[q] = clampi((comb >> 6) + (gs->offset[p] - 256) * (1 << (bd - 8)), 0, (1 << bd) - 1);
        }
      }
    }
    const int hi = p == 0 ? gs->max_luma : gs->max_chroma;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int scaled = rnd2z(grain_scale_lut(gs->lut[p], index[q], bd) * n[q], gs->scaling_shift);
      out[q] = clampi(orig[q] + scaled, gs->min_value, hi);
    }
  }
}

/* One thread's four samples: group gi of grid row y (no barrier). */
__device__ __forceinline__ void grain_blend_item(const px_t* __restrict__ src, px_t* dst,
                                                 const Layout& L, const GrainState* gs,
                                                 const uint16_t* orbit, const uint16_t* pos,
                                                 int gi, int y) {
  int p = 0;
  if (y >= L.p[0].out_h) {
    y -= L.p[0].out_h;
    const int g1 = (L.p[1].out_w + 3) >> 2;
    p = 1;
    if (gi >= g1) {
      gi -= g1;
      p = 2;
    }
  }
  const PlaneGeom& g = L.p[p];
  const int x0 = gi * 4;
  if (x0 >= g.out_w || y >= g.out_h) return;
  const int idx = g.off + y * g.stride + x0;
  const bool vec = ((reinterpret_cast<uintptr_t>(src) | reinterpret_cast<uintptr_t>(dst)) & 15) == 0;
  const int nq = min(4, g.out_w - x0);
  int orig[4];
  if (vec) {
    const uint2 v = *reinterpret_cast<const uint2*>(src + idx);
    orig[0] = v.x & 0xffff;
    orig[1] = v.x >> 16;
    orig[2] = v.y & 0xffff;
    orig[3] = v.y >> 16;
  } else {
#pragma unroll
    for (int q = 0; q < 4; ++q) orig[q] = q < nq ? src[idx + q] : 0;
  }
  int out[4];
  grain_group4(src, L, gs, orbit, pos, p, y, x0, vec, orig, out);
  if (vec && nq == 4) {
    uint2 v;
    v.x = (unsigned)out[0] | ((unsigned)out[1] << 16);
    v.y = (unsigned)out[2] | ((unsigned)out[3] << 16);
    *reinterpret_cast<uint2*>(dst + idx) = v;
  } else {
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if (q < nq) dst[idx + q] = (px_t)out[q];
  }
}

__global__ void k_grain_blend(const px_t* __restrict__ src, px_t* dst,
                              const __grid_constant__ Layout L,
                              const GrainState* gs, const uint16_t* orbit, const uint16_t* pos) {
  grain_blend_item(src, dst, L, gs, orbit, pos, blockIdx.x * blockDim.x + threadIdx.x, blockIdx.y);
}

/* ---- output packing ---------------------------------------------------------------------------- */

/* NV12: one thread per 8 output bytes of a `pitch`-byte row; rows [0, h) are
 * luma, then (h + 1) / 2 rows of interleaved Cb, Cr. Padding is zero.
 *
 * The reference packs a copy of the picture gathered row by row at the
 * *coded* width into a display-sized frame that starts out zero
 * (cpu_backend.cpp:576-584), so for a superres frame every sample right of the
 * coded width packs as 0. This kernel reproduces that byte for byte. */
/* One thread's eight bytes at byte x0 of NV12 row `row` (no barrier). */
__device__ __forceinline__ void nv12_item(const px_t* __restrict__ pic, uint8_t* out, const Layout& L,
                                          int pitch, int x0, int row) {
  if (x0 >= pitch) return;
  const int w = L.p[0].out_w, h = L.p[0].out_h;
  const int shift = L.bit_depth - 8;
  uint8_t v[8];
  if (row < h) {
    const px_t* src = pic + L.p[0].off + row * L.p[0].stride;
    const int lim = mini(w, L.p[0].coded_w);
#pragma unroll
    for (int k = 0; k < 8; ++k) v[k] = x0 + k < lim ? (uint8_t)(src[x0 + k] >> shift) : 0;
  } else {
    const int cr = row - h;
    const int cw = (w + 1) >> 1;
    const int ccw = L.p[1].coded_w;
    const px_t* u = pic + L.p[1].off + cr * L.p[1].stride;
    const px_t* vv = pic + L.p[2].off + cr * L.p[2].stride;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const int x = x0 + k;
      v[k] = (x < 2 * cw && (x >> 1) < ccw) ? (uint8_t)(((x & 1) ? vv[x >> 1] : u[x >> 1]) >> shift) : 0;
    }
  }
  uint8_t* d = out + (size_t)row * pitch + x0;
  if (x0 + 8 <= pitch && ((reinterpret_cast<uintptr_t>(d) & 7) == 0)) {
    uint2 pk;
    pk.x = v[0] | (v[1] << 8) | (v[2] << 16) | ((unsigned)v[3] << 24);
    pk.y = v[4] | (v[5] << 8) | (v[6] << 16) | ((unsigned)v[7] << 24);
    *reinterpret_cast<uint2*>(d) = pk;
  } else {
    for (int k = 0; k < 8 && x0 + k < pitch; ++k) d[k] = v[k];
  }
}

__global__ void k_nv12(const px_t* __restrict__ pic, uint8_t* out, const __grid_constant__ Layout L,
                       int pitch) {
  nv12_item(pic, out, L, pitch, (blockIdx.x * blockDim.x + threadIdx.x) * 8, blockIdx.y);
}

/* NV12 with the film grain of the packed samples applied while packing:
 * eight bytes of row `row` at byte x0, from the picture before grain. The
 * same arithmetic per sample as grain_blend_item followed by nv12_item. */
__device__ __forceinline__ void nv12_grain_item(const px_t* __restrict__ pic, uint8_t* out,
                                                const Layout& L, int pitch, int x0, int row,
                                                const GrainState* gs, const uint16_t* orbit,
                                                const uint16_t* pos) {
  if (x0 >= pitch) return;
  const int w = L.p[0].out_w, h = L.p[0].out_h;
  const int shift = L.bit_depth - 8;
  const bool vec = (reinterpret_cast<uintptr_t>(pic) & 15) == 0;
  uint8_t v[8];
  if (row < h) {
    const px_t* src = pic + L.p[0].off + row * L.p[0].stride;
    const int lim = mini(w, L.p[0].coded_w);
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      const int xs = x0 + 4 * half;
      int orig[4] = {0, 0, 0, 0}, o[4] = {0, 0, 0, 0};
      if (xs < lim) {
#pragma unroll
        for (int q = 0; q < 4; ++q) orig[q] = xs + q < w ? src[xs + q] : 0;
        grain_group4(pic, L, gs, orbit, pos, 0, row, xs, vec, orig, o);
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) v[4 * half + q] = xs + q < lim ? (uint8_t)(o[q] >> shift) : 0;
    }
  } else {
    const int cr = row - h;
    const int cw = (w + 1) >> 1;
    const int ccw = L.p[1].coded_w;
    const int cx0 = x0 >> 1;
    int ou[4] = {0, 0, 0, 0}, ov[4] = {0, 0, 0, 0};
    if (cx0 < mini(cw, ccw)) {
      const px_t* u = pic + L.p[1].off + cr * L.p[1].stride;
      const px_t* vv = pic + L.p[2].off + cr * L.p[2].stride;
      int origu[4], origv[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        origu[q] = cx0 + q < L.p[1].out_w ? u[cx0 + q] : 0;
        origv[q] = cx0 + q < L.p[2].out_w ? vv[cx0 + q] : 0;
      }
      grain_group4(pic, L, gs, orbit, pos, 1, cr, cx0, vec, origu, ou);
      grain_group4(pic, L, gs, orbit, pos, 2, cr, cx0, vec, origv, ov);
    }
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const int x = x0 + k;
      const int c = (x >> 1) - cx0;
      v[k] = (x < 2 * cw && (x >> 1) < ccw) ? (uint8_t)(((x & 1) ? ov[c] : ou[c]) >> shift) : 0;
    }
  }
  uint8_t* d = out + (size_t)row * pitch + x0;
  if (x0 + 8 <= pitch && ((reinterpret_cast<uintptr_t>(d) & 7) == 0)) {
    uint2 pk;
    pk.x = v[0] | (v[1] << 8) | (v[2] << 16) | ((unsigned)v[3] << 24);
    pk.y = v[4] | (v[5] << 8) | (v[6] << 16) | ((unsigned)v[7] << 24);
    *reinterpret_cast<uint2*>(d) = pk;
  } else {
    for (int k = 0; k < 8 && x0 + k < pitch; ++k) d[k] = v[k];
  }
}

/* NV12 of a picture whose film grain was not applied yet (its decode read
 * nothing back): the grain of each packed sample is computed while packing,
 * and the display picture is not written. */
__global__ void k_nv12_grain(const px_t* __restrict__ pic, uint8_t* out,
                             const __grid_constant__ Layout L, int pitch, const GrainState* gs,
                             const uint16_t* orbit, const uint16_t* pos) {
  nv12_grain_item(pic, out, L, pitch, (blockIdx.x * blockDim.x + threadIdx.x) * 8, blockIdx.y, gs,
                  orbit, pos);
}

__global__ void k_rgb(const px_t* __restrict__ pic, uint8_t* out, const __grid_constant__ Layout L,
                      const __grid_constant__ RgbArgs m) {
  const int x = blockIdx.x * blockDim.x + threadIdx.x;
  const int y = blockIdx.y;
  const int w = L.p[0].out_w;
  if (x >= w) return;
  /* zero right of the coded width, as in the reference's gathered frame */
  const int yy = x < L.p[0].coded_w ? pic[L.p[0].off + y * L.p[0].stride + x] : 0;
  const int cx = x >> L.ss_x;
  const int ci = (y >> L.ss_y) * L.p[1].stride + cx;
  const int uu = cx < L.p[1].coded_w ? pic[L.p[1].off + ci] : 0;
  const int vv = cx < L.p[2].coded_w ? pic[L.p[2].off + ci] : 0;
  const int r = (m.m[0] * yy + m.m[1] * vv + m.o[0]) >> 16;
  const int g = (m.m[2] * yy + m.m[3] * uu + m.m[4] * vv + m.o[1]) >> 16;
  const int b = (m.m[5] * yy + m.m[6] * uu + m.o[2]) >> 16;
  uint8_t* d = out + ((size_t)y * w + x) * 3;
  d[0] = (uint8_t)clampi(r, 0, 255);
  d[1] = (uint8_t)clampi(g, 0, 255);
  d[2] = (uint8_t)clampi(b, 0, 255);
}

/* ---- launchers ------------------------------------------------------------------------------------ */

cudaError_t launch_recon_stage(int stage, const FrameArgs& a, int n_sm, cudaStream_t s) {
  switch (stage) {
    case 1:
      if (a.n_inter_tiles > 0) {
        const int lm_end = a.n_inter_simple + a.n_inter_lmask;
        const int cm_first = a.n_inter_tiles - a.n_inter_cmask;
        /* the ranges before the last one write different samples and read
         * only other pictures: they run side by side */
        cudaError_t e = cudaSuccess;
        bool early = false;
        if (inter_one_launch(a, n_sm)) {
          k_inter_lean<<<cdiv(lm_end, 4), 128, 0, s>>>(a, a.n_inter_simple, lm_end);
        } else {
          if (a.n_inter_simple > 0) {
            k_inter_simple<false><<<cdiv(a.n_inter_simple, 4), 128, 0, s>>>(a, 0, a.n_inter_simple);
            early = true;
          }
          if (a.n_inter_lmask > 0)
            e = launch_chained(early, k_inter_simple<true>, cdiv(a.n_inter_lmask, 4), 128, 0, s, a,
                               a.n_inter_simple, lm_end);
        }
        if (e != cudaSuccess) return e;
        /* the full kernel's tiles, then the chroma tiles that read the masks
         * the luma tiles wrote */
        if (cm_first > lm_end) k_inter<<<cdiv(cm_first - lm_end, 4), 128, 0, s>>>(a, lm_end, cm_first);
        if (a.n_inter_cmask > 0)
          k_inter_simple<true><<<cdiv(a.n_inter_cmask, 4), 128, 0, s>>>(a, cm_first, a.n_inter_tiles);
      }
      break;
    case 2:
      if (a.n_itx_batches > 0) {
        if (itx_one_launch(a, n_sm)) {
          k_itx_all<<<cdiv(a.n_itx_batches, 4), 128, 4 * ItxScratch<6>::PER_WARP * sizeof(int), s>>>(
              a, a.n_itx_batches);
          break;
        }
        cudaError_t e;
        bool early = false;
        if ((e = launch_itx_class<6>(a, &early, s)) != cudaSuccess ||
            (e = launch_itx_class<5>(a, &early, s)) != cudaSuccess ||
            (e = launch_itx_class<4>(a, &early, s)) != cudaSuccess ||
            (e = launch_itx_class<3>(a, &early, s)) != cudaSuccess ||
            (e = launch_itx_class<2>(a, &early, s)) != cudaSuccess ||
            (e = launch_itx_class<7>(a, &early, s)) != cudaSuccess)
          return e;
      }
      break;
    default:
      if (a.n_units > 0) {
        if (units_by_region(a)) {
          k_regions<<<region_ctas(a, n_sm), 32 * AV1B_REGION_WARPS, region_smem(a.L, a.region_log2), s>>>(a);
        } else {
          const size_t smem = 4 * (3 * AV1B_EDGE_LEN + AV1B_UNIT_SCRATCH) * sizeof(int);
          k_units<<<AV1B_UNIT_CTAS_PER_SM * n_sm, 128, smem, s>>>(a);
        }
      }
      break;
  }
  return cudaGetLastError();
}

/* A frame's deblocking edges and CDEF blocks, converted where the caller's
 * lists were uploaded: one thread per record validates and converts it
 * (prep_edge / prep_cdef, the checks the host planner runs too). Edges are
 * compacted into the V and H lists with one atomic per warp: the edges of one
 * direction are independent, so their order in a list does not matter. A CDEF
 * block off the 8x8 search grid gets a search of its own, listed after the
 * grid. `out` (zeroed by the caller) gets the counts and the invalid flag. */
__global__ void __launch_bounds__(256) k_prep_filters(
    const av1b_deblock_edge* __restrict__ de, int nde, const av1b_cdef_block* __restrict__ cb,
    int ncb, const Layout L, int grid_w, int grid_n, DeblockRec* __restrict__ v,
    DeblockRec* __restrict__ h, CdefRec* __restrict__ cdef, unsigned* __restrict__ cells,
    unsigned* __restrict__ extra, PrepOut* __restrict__ out) {
  const long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  const int lane = threadIdx.x & 31;
  const bool is_edge = i < nde, is_cdef = !is_edge && i < static_cast<long long>(nde) + ncb;
  int code = kPrepSkip, vert = 0, off_grid = 0;
  DeblockRec er{};
  CdefRec cr{};
  unsigned pos = 0;
  if (is_edge) {
    code = prep_edge(L, de[i], &er, &vert);
  } else if (is_cdef) {
    const av1b_cdef_block& c = cb[i - nde];
    code = prep_cdef(L, c, grid_w, &cr, &off_grid);
    if (code == kPrepOk && off_grid) {
      const int sx = c.plane ? L.ss_x : 0, sy = c.plane ? L.ss_y : 0;
      pos = static_cast<unsigned>(c.x << sx) | (static_cast<unsigned>(c.y << sy) << 16);
    }
  }
  const bool ok = code == kPrepOk;
  bool irregular = false;
  if (is_cdef && ok) {
    const int lw = cr.plane ? 3 - L.ss_x : 3, lh = cr.plane ? 3 - L.ss_y : 3;
    const PlaneGeom& g = L.p[cr.plane];
    if ((cr.x & ((1 << lw) - 1)) || (cr.y & ((1 << lh) - 1)) || cr.x >= g.grid_w || cr.y >= g.grid_h)
      irregular = true;
    else
      irregular = atomicExch(cells + cr.plane * cdef_cells(L) + (cr.y >> lh) * (L.p[0].grid_w >> 3) +
                                 (cr.x >> lw),
                             cdef_cell_word(cr)) != 0;
  }
  const unsigned mi = __ballot_sync(0xffffffffu, irregular);
  const unsigned mv = __ballot_sync(0xffffffffu, is_edge && ok && vert);
  const unsigned mh = __ballot_sync(0xffffffffu, is_edge && ok && !vert);
  const unsigned me = __ballot_sync(0xffffffffu, is_cdef && ok && off_grid);
  const unsigned mg = __ballot_sync(0xffffffffu, is_cdef && ok && !off_grid && cr.dir < 0);
  const unsigned mb = __ballot_sync(0xffffffffu, code >= kPrepErrFirst);
  unsigned bv = 0, bh = 0, be = 0;
  if (lane == 0) {
    if (mv) bv = atomicAdd(&out->n_v, __popc(mv));
    if (mh) bh = atomicAdd(&out->n_h, __popc(mh));
    if (me) be = atomicAdd(&out->n_extra, __popc(me));
    if (mg) atomicOr(&out->any_grid, 1u);
    if (mb) atomicOr(&out->bad, 1u);
    if (mi) atomicOr(&out->irregular, 1u);
  }
  bv = __shfl_sync(0xffffffffu, bv, 0);
  bh = __shfl_sync(0xffffffffu, bh, 0);
  be = __shfl_sync(0xffffffffu, be, 0);
  const unsigned below = (1u << lane) - 1u;
  if (is_edge && ok) {
    if (vert)
      v[bv + __popc(mv & below)] = er;
    else
      h[bh + __popc(mh & below)] = er;
  } else if (is_cdef && ok) {
    if (off_grid) {
      const unsigned k = be + __popc(me & below);
      cr.search = grid_n + static_cast<int>(k);
      extra[k] = pos;
    }
    cdef[i - nde] = cr;
  }
}

cudaError_t launch_prep_filters(const av1b_deblock_edge* edges, int n_edges, const av1b_cdef_block* cdef,
                                int n_cdef, const Layout& L, int grid_w, int grid_n, DeblockRec* v,
                                DeblockRec* h, CdefRec* cdef_out, unsigned* cells, unsigned* extra,
                                PrepOut* out, cudaStream_t s) {
  const long long n = static_cast<long long>(n_edges) + n_cdef;
  if (n <= 0) return cudaSuccess;
  k_prep_filters<<<cdiv(n, 256), 256, 0, s>>>(edges, n_edges, cdef, n_cdef, L, grid_w, grid_n, v, h,
                                              cdef_out, cells, extra, out);
  return cudaGetLastError();
}

cudaError_t launch_deblock(px_t* pic, const DeblockRec* recs, int n, int sharpness, int bd, int maxv,
                           bool early, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  const unsigned grid = cdiv(cdiv(n, AV1B_DB_PLAIN) * 32, 256);
  return launch_chained(early, k_deblock<AV1B_DB_PLAIN>, grid, 256, 0, s, pic, recs, n, sharpness, bd, maxv);
}

cudaError_t launch_cdef(const px_t* src, px_t* dst, const CdefRec* recs, int n, int grid_w,
                        int grid_n, bool grid, const unsigned* extra_pos, int n_extra, int* search,
                        const Layout& L, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  const int n_grid = grid ? grid_n : 0;
  if (n_grid + n_extra > 0)
    k_cdef_search<<<cdiv(n_grid + n_extra, 128), 128, 0, s>>>(src, grid_w, grid_n, n_grid, extra_pos,
                                                               n_extra, search, L);
  k_cdef<<<cdiv(n, 8), 128, 0, s>>>(src, dst, recs, n, search, L);
  return cudaGetLastError();
}

cudaError_t launch_cdef_tiles(const px_t* src, px_t* dst, const unsigned* cells, int grid_w, int grid_n,
                              bool grid, int* search, const Layout& L, bool early, cudaStream_t s) {
  if (grid) {
    const cudaError_t e = launch_chained(early, k_cdef_search, cdiv(grid_n, 128), 128, 0, s, src, grid_w, grid_n,
                                         grid_n, nullptr, 0, search, L);
    if (e != cudaSuccess) return e;
    early = true;
  }
  int tx, ty;
  cdef_tile_grid(L, &tx, &ty);
  return launch_chained(early, k_cdef_tile, dim3(tx, ty, L.p[1].grid_w > 0 ? 2 : 1), 256, 0, s, src, dst, cells, search,
                      grid_w, L);
}

cudaError_t launch_upscale(const px_t* src, px_t* dst, const Layout& L, int maxv, bool border_rows,
                           bool early, cudaStream_t s) {
  UpscaleArgs u;
  for (int p = 0; p < 3; ++p) superres_params(L.p[p].coded_w, L.p[p].out_w, &u.step[p], &u.initial[p]);
  /* grid rows: the luma rows, then the chroma rows (planes 1 and 2 side by side) */
  const int rows0 = border_rows ? 4 * ((L.p[0].out_h + 8) / 64 + 1) : L.p[0].out_h;
  const int rows1 = L.p[1].out_h > 0 ? (border_rows ? rows0 : L.p[1].out_h) : 0;
  const int segs = maxi(cdiv(L.p[0].out_w, AV1B_UP_OUT), 2 * cdiv(L.p[1].out_w, AV1B_UP_OUT));
  return launch_chained(early, k_upscale, dim3(segs, rows0 + rows1), 128, 0, s, src, dst, L, u, maxv, border_rows ? 1 : 0,
                      rows0);
}

cudaError_t launch_lr(const px_t* cdef, const px_t* curr, px_t* dst, const Layout& L,
                      const LrArgs& r, int maxv, bool copy_rest, bool early, cudaStream_t s) {
  const int stripes = (L.p[0].out_h + 8 + 63) / 64;
  const int tiles = maxi(cdiv(L.p[0].out_w, AV1B_LR_TW), 2 * cdiv(L.p[1].out_w, AV1B_LR_TW));
  return launch_chained(early, k_lr_tile, dim3(tiles, stripes, 2), 256, 0, s, cdef, curr, dst, L, r, maxv, copy_rest ? 1 : 0);
}

cudaError_t launch_grain_template(GrainState* gs, const int* gs_src, const GrainParamsDev& prm,
                                  const uint16_t* orbit, const uint16_t* pos, cudaStream_t s) {
  k_grain_template<<<1, 256, 0, s>>>(gs, gs_src, prm, orbit, pos);
  return cudaGetLastError();
}

cudaError_t launch_grain_blend(const px_t* src, px_t* dst, const Layout& L, const GrainState* gs,
                               const uint16_t* orbit, const uint16_t* pos, cudaStream_t s) {
  /* grid rows: the luma rows, then the chroma rows (planes 1 and 2 side by side) */
  const int groups = maxi(cdiv(L.p[0].out_w, 4), 2 * cdiv(L.p[1].out_w, 4));
  const int rows = L.p[0].out_h + L.p[1].out_h;
  k_grain_blend<<<dim3(cdiv(groups, 128), rows), 128, 0, s>>>(src, dst, L, gs, orbit, pos);
  return cudaGetLastError();
}

cudaError_t launch_nv12(const px_t* pic, uint8_t* out, const Layout& L, int pitch, cudaStream_t s) {
  const int rows = L.p[0].out_h + (L.p[0].out_h + 1) / 2;
  k_nv12<<<dim3(cdiv(cdiv(pitch, 8), 128), rows), 128, 0, s>>>(pic, out, L, pitch);
  return cudaGetLastError();
}

cudaError_t launch_nv12_grain(const px_t* pic, uint8_t* out, const Layout& L, int pitch,
                              const GrainState* gs, const uint16_t* orbit, const uint16_t* pos,
                              cudaStream_t s) {
  const int rows = L.p[0].out_h + (L.p[0].out_h + 1) / 2;
  k_nv12_grain<<<dim3(cdiv(cdiv(pitch, 8), 128), rows), 128, 0, s>>>(pic, out, L, pitch, gs, orbit, pos);
  return cudaGetLastError();
}

cudaError_t launch_rgb(const px_t* pic, uint8_t* out, const Layout& L, const RgbArgs& m,
                       cudaStream_t s) {
  k_rgb<<<dim3(cdiv(L.p[0].out_w, 128), L.p[0].out_h), 128, 0, s>>>(pic, out, L, m);
  return cudaGetLastError();
}

/* Loads every kernel of this file now. With lazy module loading (the CUDA
 * 12 default) a kernel's first launch loads its code, and a load waits for
 * the kernels already running; decoder creation loading them all keeps that
 * wait out of every frame. */
template <class K>
static cudaError_t load_kernel(K k) {
  cudaFuncAttributes fa;
  return cudaFuncGetAttributes(&fa, reinterpret_cast<const void*>(k));
}

static cudaError_t load_all_kernels() {
  cudaError_t e;
  if ((e = load_kernel(k_inter_simple<false>)) != cudaSuccess ||
      (e = load_kernel(k_inter_simple<true>)) != cudaSuccess || (e = load_kernel(k_inter)) != cudaSuccess ||
      (e = load_kernel(k_inter_lean)) != cudaSuccess || (e = load_kernel(k_itx_all)) != cudaSuccess ||
      (e = load_kernel(k_itx<2>)) != cudaSuccess || (e = load_kernel(k_itx<3>)) != cudaSuccess ||
      (e = load_kernel(k_itx<4>)) != cudaSuccess || (e = load_kernel(k_itx<5>)) != cudaSuccess ||
      (e = load_kernel(k_itx<6>)) != cudaSuccess || (e = load_kernel(k_itx<7>)) != cudaSuccess ||
      (e = load_kernel(k_units)) != cudaSuccess || (e = load_kernel(k_regions)) != cudaSuccess ||
      (e = load_kernel(k_selftest_wait)) != cudaSuccess || (e = load_kernel(k_deblock<AV1B_DB_PLAIN>)) != cudaSuccess ||
      (e = load_kernel(k_cdef_search)) != cudaSuccess || (e = load_kernel(k_cdef)) != cudaSuccess ||
      (e = load_kernel(k_cdef_tile)) != cudaSuccess ||
      (e = load_kernel(k_upscale)) != cudaSuccess || (e = load_kernel(k_lr_tile)) != cudaSuccess ||
      (e = load_kernel(k_grain_template)) != cudaSuccess || (e = load_kernel(k_grain_blend)) != cudaSuccess ||
      (e = load_kernel(k_nv12)) != cudaSuccess || (e = load_kernel(k_nv12_grain)) != cudaSuccess ||
      (e = load_kernel(k_rgb)) != cudaSuccess ||
      (e = load_kernel(k_dequant)) != cudaSuccess || (e = load_kernel(k_prep_filters)) != cudaSuccess)
    return e;
  return cudaSuccess;
}

cudaError_t set_kernel_attributes() {
  {
    const cudaError_t e = load_all_kernels();
    if (e != cudaSuccess) return e;
  }
  cudaError_t e = cudaFuncSetAttribute(k_units, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       4 * (3 * AV1B_EDGE_LEN + AV1B_UNIT_SCRATCH) * (int)sizeof(int));
  if (e != cudaSuccess) return e;
  Layout full{}, half{};   /* the largest tiles: 64x64 in 4:4:4, 128x128 in 4:2:0 */
  half.ss_x = half.ss_y = 1;
  const size_t most = std::max(region_smem(full, 6), region_smem(half, 7));
  if ((e = cudaFuncSetAttribute(k_regions, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                static_cast<int>(most))) != cudaSuccess)
    return e;
  /* phase B's picture reads bypass L1: the SM's memory goes to shared memory,
   * so two CTAs fit */
  if ((e = cudaFuncSetAttribute(k_units, cudaFuncAttributePreferredSharedMemoryCarveout,
                                cudaSharedmemCarveoutMaxShared)) != cudaSuccess ||
      (e = cudaFuncSetAttribute(k_regions, cudaFuncAttributePreferredSharedMemoryCarveout,
                                cudaSharedmemCarveoutMaxShared)) != cudaSuccess)
    return e;
  return cudaSuccess;
}

/* ---- batched form: the stage kernels of many streams ------------------------------------- */
#include "batch_kernels.cuh"

}  // namespace av1b

/*
 * dev_intra.cuh - intra prediction of one transform block by one warp
 * (specification 7.11.2).
 *
 * The reference predicts a row per thread and gathers and filters the whole
 * edge again in every thread (av1_cuda.cu:70-117). Here the warp gathers the
 * block's two edges once into shared memory, runs the edge filter and the
 * upsampler with one lane per edge sample, and then predicts the block with
 * one lane per output sample. The arithmetic of every step is the
 * reference's (av1gpu_kernels.h:1108-1677):
 *   - edge gather and the stand-in values for missing neighbours (1108-1151);
 *   - corner fix, edge filter strength and upsampling selection (1193-1239,
 *     1452-1481);
 *   - directional, smooth, Paeth, DC, recursive filter, palette and
 *     chroma-from-luma predictors (1245-1447, 1578-1677).
 * Reads of the picture being reconstructed go through L2 (ld.cg), because
 * another SM produced them and published them with a release flag.
 */
#ifndef AV1B_DEV_INTRA_CUH
#define AV1B_DEV_INTRA_CUH

#include "dev_common.cuh"

namespace av1b {

#define AV1B_EDGE_LEN 288
#define AV1B_EDGE_OFF 16

/* The tagged samples a block reads and writes (FrameArgs::tags): words at its
 * top-left sample and the luma plane's origin, with the words a row; null
 * `write`: untagged. `wait`: the edges are read by their tags, the cells (of
 * 1 << cell samples) of `cells` only - the others are final already; `luma`:
 * so are the chroma-from-luma samples. Waits give up after limit_ns or once
 * one has given up (AV1B_STATUS_TIMEOUT, bit 0 of *status). */
#define AV1B_TILE_EMPTY 0xffffu
struct TagIo {
  unsigned* write;
  const unsigned* at;
  const unsigned* luma_at;
  int stride, luma_stride;
  unsigned tag;               /* in the high half */
  bool wait, luma, corner;
  int cell;
  unsigned long long above, left;
  int clip_w, clip_h;         /* the block's samples inside the grid */
  /* The region form: the samples of the region's phase B blocks, in shared
   * memory, tile_w a row (AV1B_TILE_EMPTY until reconstructed); tile_x and
   * tile_y are the block's place in it. What a block waits for inside its
   * region it reads there; the tagged words then serve other regions, which
   * read the last row and column only. Null: no region. */
  volatile unsigned short* tile;
  volatile const unsigned short* luma_tile;   /* at the block's first luma sample */
  int tile_x, tile_y, tile_w, tile_h, luma_tile_w;
  int row0, row1;             /* the rows and columns of the block this warp */
  int col0, cols;             /* predicts (a power of two of columns) */
  int* status;
  int* status_host;           /* page-locked; null: none */
  unsigned long long limit_ns;
};

/* A wait has given up: in the status word the other waits read, and in the
 * host's copy. */
__device__ __forceinline__ void wait_failed(int* status, int* status_host) {
  atomicOr(status, 1);
  if (status_host) {
    *reinterpret_cast<volatile int*>(status_host) = 1;
    __threadfence_system();
  }
}

__device__ __forceinline__ unsigned ld_tag(const unsigned* p) {
  unsigned v;
  asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_tag(unsigned* p, unsigned v) {
  asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

/* Four consecutive tagged words (16-byte aligned): one access, but each word
 * is valid by its own tag. */
__device__ __forceinline__ void st_tag4(unsigned* p, unsigned a, unsigned b, unsigned c, unsigned d) {
  asm volatile("st.relaxed.gpu.global.v4.u32 [%0], {%1, %2, %3, %4};" ::"l"(p), "r"(a), "r"(b), "r"(c), "r"(d)
               : "memory");
}

/* Between two rounds of loads of a warp whose samples have not all arrived:
 * a pause that backs off to `most` ns; every 128th round the status word and
 * the clock. Returns false when the wait has given up (the same for every
 * lane). */
struct TagBackoff {
  unsigned it = 0, pause = 0;
  unsigned long long t0 = 0;
  __device__ __forceinline__ bool next(const TagIo& g, int lane, unsigned most) {
    ++it;
    if ((it & 127) == 0) {
      int give_up = 0;
      if (lane == 0) {
        unsigned long long now;
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(now));
        if (t0 == 0) t0 = now;
        if (ld_tag(reinterpret_cast<const unsigned*>(g.status)) & 1u) {
          give_up = 1;
        } else if (now - t0 > g.limit_ns) {
          wait_failed(g.status, g.status_host);
          give_up = 1;
        }
      }
      if (__shfl_sync(0xffffffffu, give_up, 0)) return false;
    }
    if (pause) __nanosleep(pause);
    if (it >= 4) pause = mini(pause ? pause << 1 : 16, most);
    return true;
  }
};

/* Everything the intra predictor needs for one block, resolved. */
struct IntraJob {
  int x, y, w, h;
  int mode, angle, bitdepth, maxv;
  int have_left, have_above, have_ar, have_bl;
  int filter_type;     /* -1: the sequence disables the intra edge filter */
  int filter_intra, fi_mode;
  int cfl_alpha;
  int max_x, max_y;
  int ss_x, ss_y;
  int palette, palette_off, palette_stride;
};


AV1B_DEV int edge_strength(int w, int h, int filter_type, int delta) {
  const int d = absi(delta);
  const int blk = w + h;
  int s = 0;
  if (filter_type == 0) {
    if (blk <= 8) {
      if (d >= 56) s = 1;
    } else if (blk <= 16) {
      if (d >= 40) s = 1;
    } else if (blk <= 24) {
      if (d >= 8) s = 1;
      if (d >= 16) s = 2;
      if (d >= 32) s = 3;
    } else if (blk <= 32) {
      s = 1;
      if (d >= 4) s = 2;
      if (d >= 32) s = 3;
    } else {
      s = 3;
    }
  } else {
    if (blk <= 8) {
      if (d >= 40) s = 1;
      if (d >= 64) s = 2;
    } else if (blk <= 16) {
      if (d >= 20) s = 1;
      if (d >= 48) s = 2;
    } else if (blk <= 24) {
      if (d >= 4) s = 3;
    } else {
      s = 3;
    }
  }
  return s;
}

AV1B_DEV int upsample_sel(int w, int h, int filter_type, int delta) {
  const int d = absi(delta);
  if (d <= 0 || d >= 40) return 0;
  return filter_type == 0 ? (w + h <= 16) : (w + h <= 8);
}

/* The gather below for a block that waits on the samples themselves: a
 * sample of a block it waits for is loaded with its tag until the tag is this
 * frame's, any other from the picture. The wait and the read are one round
 * trip; with done flags they were a poll, then the loads, and on the writing
 * side a fence before the flag. A sample of the block's own region is read
 * from the region's tile in shared memory instead. NQ: samples of each edge
 * a lane takes (edges of up to 32 * NQ). */
template <int NQ>
AV1B_DEV void intra_edges_tagged(const IntraJob& j, const px_t* p, int stride, int* above, int* left,
                                 const TagIo& g, int lane) {
  constexpr int E = 2 * NQ + 1;
  const int n = j.w + j.h;
  const int mid = 1 << (j.bitdepth - 1);
  const int alimit = mini(j.max_x, j.x + (j.have_ar ? 2 * j.w : j.w) - 1);
  const int llimit = mini(j.max_y, j.y + (j.have_bl ? 2 * j.h : j.h) - 1);
  /* entries 2q: above, 2q + 1: left, of sample lane + 32 q; last: the corner */
  int v[E], o[E];
  unsigned pend = 0, in_tile = 0;
  auto want = [&](int e, bool have, int dy, int dx, bool tagged, int none) {
    v[e] = none;
    o[e] = 0;
    if (!have) return;
    if (!tagged) {
      v[e] = ldpx(p + dy * stride + dx);
      return;
    }
    pend |= 1u << e;
    if (g.tile) {
      const int ty = g.tile_y + dy, tx = g.tile_x + dx;
      if (static_cast<unsigned>(ty) < static_cast<unsigned>(g.tile_h) &&
          static_cast<unsigned>(tx) < static_cast<unsigned>(g.tile_w)) {
        in_tile |= 1u << e;
        o[e] = ty * g.tile_w + tx;
        return;
      }
    }
    o[e] = dy * g.stride + dx;
  };
  const bool above0 = g.above & 1, left0 = g.left & 1;
#pragma unroll
  for (int q = 0; q < NQ; ++q) {
    v[2 * q] = v[2 * q + 1] = o[2 * q] = o[2 * q + 1] = 0;
    const int i = lane + 32 * q;
    if (i < n) {
      if (j.have_above) {
        const int k = mini(j.x + i, alimit) - j.x;
        want(2 * q, true, -1, k, (g.above >> (k >> g.cell)) & 1, 0);
      } else {
        want(2 * q, j.have_left, 0, -1, left0, mid - 1);
      }
      if (j.have_left) {
        const int k = mini(j.y + i, llimit) - j.y;
        want(2 * q + 1, true, k, -1, (g.left >> (k >> g.cell)) & 1, 0);
      } else {
        want(2 * q + 1, j.have_above, -1, 0, above0, mid + 1);
      }
    }
  }
  v[E - 1] = mid;
  o[E - 1] = 0;
  if (lane == 0) {
    if (j.have_above && j.have_left) want(E - 1, true, -1, -1, g.corner, 0);
    else if (j.have_above) want(E - 1, true, -1, 0, above0, 0);
    else want(E - 1, j.have_left, 0, -1, left0, mid);
  }
  TagBackoff back;
  for (;;) {
    unsigned w[E];
#pragma unroll
    for (int e = 0; e < E; ++e)
      if (pend >> e & 1) {
        if (in_tile >> e & 1) {
          const unsigned t = g.tile[o[e]];
          w[e] = t == AV1B_TILE_EMPTY ? 0 : g.tag | t;
        } else {
          w[e] = ld_tag(g.at + o[e]);
        }
      }
#pragma unroll
    for (int e = 0; e < E; ++e)
      if ((pend >> e & 1) && (w[e] & 0xffff0000u) == g.tag) {
        v[e] = static_cast<int>(w[e] & 0xffffu);
        pend &= ~(1u << e);
      }
    if (!__any_sync(0xffffffffu, pend)) break;
    /* short pauses once only the tile is waited for: its reads are cheap */
    const unsigned most = __any_sync(0xffffffffu, pend & ~in_tile) ? 128 : 32;
    if (!back.next(g, lane, most)) break;
  }
#pragma unroll
  for (int q = 0; q < NQ; ++q) {
    const int i = lane + 32 * q;
    if (i < n) {
      above[i] = v[2 * q];
      left[i] = v[2 * q + 1];
    }
  }
  if (lane == 0) {
    above[-1] = v[E - 1];
    left[-1] = v[E - 1];
  }
  __syncwarp();
}

/* Gathers AboveRow[-1 .. w+h-1] and LeftCol[-1 .. w+h-1]. `p` is the block's
 * top-left sample in the plane. */
AV1B_DEV void intra_edges(const IntraJob& j, const px_t* p, int stride, int* above, int* left,
                          const TagIo& g, int lane) {
  if (g.wait) {
    if (j.w + j.h <= 32) intra_edges_tagged<1>(j, p, stride, above, left, g, lane);
    else intra_edges_tagged<4>(j, p, stride, above, left, g, lane);
    return;
  }
  const int n = j.w + j.h;
  const int mid = 1 << (j.bitdepth - 1);
  const int alimit = mini(j.max_x, j.x + (j.have_ar ? 2 * j.w : j.w) - 1);
  const int llimit = mini(j.max_y, j.y + (j.have_bl ? 2 * j.h : j.h) - 1);
  /* every load of the edges (at most 128 + 128 samples and the corner) is
   * issued before any is used: one round trip to L2, not one per sample */
  int a[4], l[4], c = mid;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int i = lane + 32 * q;
    a[q] = mid - 1;
    l[q] = mid + 1;
    if (i < n) {
      if (!j.have_above) a[q] = j.have_left ? ldpx(p - 1) : mid - 1;
      else a[q] = ldpx(p - stride + (mini(j.x + i, alimit) - j.x));
      if (!j.have_left) l[q] = j.have_above ? ldpx(p - stride) : mid + 1;
      else l[q] = ldpx(p + (mini(j.y + i, llimit) - j.y) * stride - 1);
    }
  }
  if (lane == 0) {
    if (j.have_above && j.have_left) c = ldpx(p - stride - 1);
    else if (j.have_above) c = ldpx(p - stride);
    else if (j.have_left) c = ldpx(p - 1);
  }
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int i = lane + 32 * q;
    if (i < n) {
      above[i] = a[q];
      left[i] = l[q];
    }
  }
  if (lane == 0) {
    above[-1] = c;
    left[-1] = c;
  }
  __syncwarp();
}

/* The 5-tap intra edge filter over buf[-1 .. sz-2] (entry i-1 is edge sample
 * i; sample 0, the corner, is read but not written), of both edges at once: a
 * warp barrier serves both. Strength 0: the edge stays. */
#define AV1B_EDGE_TMP 144
AV1B_DEV void edge_filter(int* above, int asz, int astrength, int* left, int lsz, int lstrength, int* tmp,
                          int lane) {
  if ((astrength | lstrength) == 0) return;
  if (astrength)
    for (int i = lane; i < asz; i += 32) tmp[i] = above[i - 1];
  if (lstrength)
    for (int i = lane; i < lsz; i += 32) tmp[AV1B_EDGE_TMP + i] = left[i - 1];
  __syncwarp();
  auto run = [&](int* buf, int sz, int strength, const int* t) {
    /* kernels (0 4 8 4 0), (0 5 6 5 0), (2 4 4 4 2) */
    const int k1 = strength == 2 ? 5 : 4, k2 = strength == 1 ? 8 : (strength == 2 ? 6 : 4);
    const int k0 = strength == 3 ? 2 : 0;
    for (int i = 1 + lane; i < sz; i += 32) {
      const int s = k0 * (t[maxi(i - 2, 0)] + t[mini(i + 2, sz - 1)]) +
                    k1 * (t[i - 1] + t[mini(i + 1, sz - 1)]) + k2 * t[i];
      buf[i - 1] = (s + 8) >> 4;
    }
  };
  if (astrength) run(above, asz, astrength, tmp);
  if (lstrength) run(left, lsz, lstrength, tmp + AV1B_EDGE_TMP);
  __syncwarp();
}

/* Doubles the resolution of an edge of at most 16 samples: buf[-2 .. 2*num-2].
 * The samples pass between lanes (lane i: sample i - 1), no scratch. */
AV1B_DEV void edge_upsample(int* buf, int num, int maxv, int lane) {
  const int at = mini(lane, num) - 1;
  const int v = buf[at];
  /* of the samples -1, -1, 0, .., num - 1, num - 1: lane i has the four from
   * its own on */
  const int d0 = __shfl_up_sync(0xffffffffu, v, 1), d2 = __shfl_down_sync(0xffffffffu, v, 1);
  const int d3 = __shfl_down_sync(0xffffffffu, v, 2);
  __syncwarp();
  if (lane < num) {
    const int s = -(lane == 0 ? v : d0) + 9 * v + 9 * d2 - d3;
    buf[2 * lane - 1] = clampi(rnd2(s, 4), 0, maxv);
    buf[2 * lane] = d2;
  }
  if (lane == 0) buf[-2] = v;
  __syncwarp();
}

AV1B_DEV int warp_sum(int v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
AV1B_DEV long long warp_sum64(long long v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

/* DC of whichever edges exist. */
AV1B_DEV int intra_dc(const IntraJob& j, const int* above, const int* left, int lane) {
  int s = 0;
  if (j.have_above)
    for (int k = lane; k < j.w; k += 32) s += above[k];
  if (j.have_left)
    for (int k = lane; k < j.h; k += 32) s += left[k];
  s = warp_sum(s);
  if (j.have_above && j.have_left)
    return static_cast<int>(static_cast<unsigned>(s + ((j.w + j.h) >> 1)) / static_cast<unsigned>(j.w + j.h));
  if (j.have_left) return (s + (j.h >> 1)) >> ilog2(j.h);
  if (j.have_above) return (s + (j.w >> 1)) >> ilog2(j.w);
  return 1 << (j.bitdepth - 1);
}

/* One directional sample (the reference's av1g_intra_directional_row). */
AV1B_DEV int dir_sample(const int* above, const int* left, int w, int h, int pangle, int dx,
                        int dy, int ua, int ul, int i, int jj) {
  if (pangle < 90) {
    const int max_base = (w + h - 1) << ua;
    const int idx = (i + 1) * dx;
    const int base = (idx >> (6 - ua)) + (jj << ua);
    const int shift = ((idx << ua) >> 1) & 0x1F;
    if (base < max_base) return rnd2(above[base] * (32 - shift) + above[base + 1] * shift, 5);
    return above[max_base];
  }
  if (pangle > 90 && pangle < 180) {
    int idx = (jj << 6) - (i + 1) * dx;
    int base = idx >> (6 - ua);
    if (base >= -(1 << ua)) {
      const int shift = ((idx * (1 << ua)) >> 1) & 0x1F;
      return rnd2(above[base] * (32 - shift) + above[base + 1] * shift, 5);
    }
    idx = (i << 6) - (jj + 1) * dy;
    base = idx >> (6 - ul);
    const int shift = ((idx * (1 << ul)) >> 1) & 0x1F;
    return rnd2(left[base] * (32 - shift) + left[base + 1] * shift, 5);
  }
  if (pangle > 180) {
    const int idx = (jj + 1) * dy;
    const int base = (idx >> (6 - ul)) + (i << ul);
    const int shift = ((idx << ul) >> 1) & 0x1F;
    return rnd2(left[base] * (32 - shift) + left[base + 1] * shift, 5);
  }
  return pangle == 90 ? above[jj] : left[i];
}

/* Predicts one intra block into `dst` (the block's top-left sample in its
 * plane, global memory). `plane` points at the plane origin (for CFL's luma,
 * `luma` at the luma plane origin). `scratch` is warp-private shared memory of
 * 3 * AV1B_EDGE_LEN ints. */
/* The pause of one lane's chroma-from-luma wait after its `it`-th round;
 * false when the wait has given up. */
AV1B_DEV bool luma_backoff(const TagIo& g, unsigned it, unsigned long long* t0) {
  if ((it & 127) == 127) {
    unsigned long long now;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(now));
    if (*t0 == 0) *t0 = now;
    if (ld_tag(reinterpret_cast<const unsigned*>(g.status)) & 1u) return false;
    if (now - *t0 > g.limit_ns) {
      wait_failed(g.status, g.status_host);
      return false;
    }
  }
  if (it >= 3) __nanosleep(g.tile ? 32 : 64);
  return true;
}

/* Waits for the asynchronous copies this thread issued (cp.async), then
 * for the warp: every lane's copies are in shared memory. */
AV1B_DEV void async_copies_done() {
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncwarp();
}

template <class Ahead>
AV1B_DEV void intra_predict(const IntraJob& j, px_t* dst, int stride, const px_t* luma,
                            int luma_stride, const uint8_t* palette_map,
                            const int* palette_colors, int* scratch, int lane,
                            const TagIo& g, const int* res, short* fi_pred, bool res_in_flight,
                            Ahead&& ahead) {
  /* `res_in_flight`: the caller's residual image is still arriving by
   * asynchronous copies; it is waited for after the edges are read (the two
   * fetches overlap), before the first sample is written. `ahead`: called
   * once the edges are there, to start loads for what comes after */
  const int w = j.w, h = j.h, n = w * h;
  const int lw = ilog2(w);
  /* the reconstructed sample: the prediction plus, when the caller fused the
   * residual in (`res`, the block's residual, w x h row-major), that residual,
   * clipped - what adding the transforms afterwards gives */
  const int row0 = g.row0, col0 = g.col0, cols = g.cols, lc = ilog2(cols);
  const int n_rows = (g.row1 - g.row0) << lc;
  auto put = [&](int i, int jj, int v) {
    if (res) v = clampi(v + res[(i - row0) * cols + jj - col0], 0, j.maxv);
    dst[i * stride + jj] = (px_t)v;
    if (g.write && jj < g.clip_w && i < g.clip_h) {
      if (g.tile) {
        const int ty = g.tile_y + i, tx = g.tile_x + jj;
        g.tile[ty * g.tile_w + tx] = static_cast<unsigned short>(v);
        if (ty != g.tile_h - 1 && tx != g.tile_w - 1) return;
      }
      st_tag(g.write + i * g.stride + jj, g.tag | v);
    }
  };
  /* four samples of a row at once where everything they are stored to is
   * aligned for it (blocks lie on a grid of 4 samples; odd callers' may not) */
  const bool vec = n_rows > 32 && cols >= 4 &&
                   ((static_cast<unsigned>(reinterpret_cast<uintptr_t>(dst)) & 7) | (stride & 3)) == 0 &&
                   (!g.write || ((static_cast<unsigned>(reinterpret_cast<uintptr_t>(g.write)) & 15) |
                                 (g.stride & 3) | (g.clip_w & 3) | (g.tile ? g.tile_x & 3 : 0)) == 0);
  auto put4 = [&](int i, int jj, int v0, int v1, int v2, int v3) {
    if (res) {
      const int4 r = *reinterpret_cast<const int4*>(res + (i - row0) * cols + jj - col0);
      v0 = clampi(v0 + r.x, 0, j.maxv);
      v1 = clampi(v1 + r.y, 0, j.maxv);
      v2 = clampi(v2 + r.z, 0, j.maxv);
      v3 = clampi(v3 + r.w, 0, j.maxv);
    }
    const uint2 two = make_uint2(static_cast<unsigned>(v0 | (v1 << 16)), static_cast<unsigned>(v2 | (v3 << 16)));
    *reinterpret_cast<uint2*>(dst + i * stride + jj) = two;
    if (g.write && jj < g.clip_w && i < g.clip_h) {
      if (g.tile) {
        const int ty = g.tile_y + i, tx = g.tile_x + jj;
        volatile unsigned* t = reinterpret_cast<volatile unsigned*>(g.tile + ty * g.tile_w + tx);
        t[0] = two.x;
        t[1] = two.y;
        if (ty != g.tile_h - 1) {
          if (tx + 3 == g.tile_w - 1) st_tag(g.write + i * g.stride + jj + 3, g.tag | v3);
          return;
        }
      }
      st_tag4(g.write + i * g.stride + jj, g.tag | v0, g.tag | v1, g.tag | v2, g.tag | v3);
    }
  };
  /* every sample the warp predicts from pred(row, column): four a lane (their
   * loads all before the first store, which no load can be moved across) or,
   * of up to 32 samples, one */
  auto each = [&](auto&& pred) {
    if (vec) {
      for (int k = lane * 4; k < n_rows; k += 128) {
        const int i = row0 + (k >> lc), jj = col0 + (k & (cols - 1));
        const int v0 = pred(i, jj), v1 = pred(i, jj + 1), v2 = pred(i, jj + 2), v3 = pred(i, jj + 3);
        put4(i, jj, v0, v1, v2, v3);
      }
    } else {
      for (int k = lane; k < n_rows; k += 32) {
        const int i = row0 + (k >> lc), jj = col0 + (k & (cols - 1));
        put(i, jj, pred(i, jj));
      }
    }
  };
  if (j.palette) {
    ahead();
    if (res_in_flight) async_copies_done();
    const uint8_t* map = palette_map + j.palette_off;
    each([&](int i, int jj) { return palette_colors[map[i * j.palette_stride + jj]]; });
    return;
  }
  int* above = scratch + AV1B_EDGE_OFF;
  int* left = scratch + AV1B_EDGE_LEN + AV1B_EDGE_OFF;
  int* tmp = scratch + 2 * AV1B_EDGE_LEN;
  intra_edges(j, dst, stride, above, left, g, lane);
  ahead();
  if (res_in_flight) async_copies_done();

  if (j.mode == 13 && fi_pred && n <= 1024) {
    /* chroma from luma, each sample's luma value read once: kept in the
     * filter-intra buffer (unused by a CFL block) between the average and the
     * prediction. The (up to four) luma samples of a chroma sample are read
     * from neighbouring positions clamped to the block: every load of an
     * iteration is issued before any is used (one round trip to L2, not one
     * per sample), four iterations at a time. */
    const int dc = intra_dc(j, above, left, lane);
    const int sx = j.ss_x, sy = j.ss_y;
    const int lxl = ((j.x + w) << sx) - (1 << sx);
    const int lyl = ((j.y + h) << sy) - (1 << sy);
    long long sum = 0;
    unsigned long long luma_t0 = 0;
#pragma unroll 2
    for (int k = lane; k < n; k += 32) {
      const int i = k >> lw, jj = k & (w - 1);
      const int ly = mini((j.y + i) << sy, lyl), lx = mini((j.x + jj) << sx, lxl);
      int v00, v01, v10, v11;
      if (g.luma && g.tile) {
        volatile const unsigned short* p0 =
            g.luma_tile + (ly - (j.y << sy)) * g.luma_tile_w + lx - (j.x << sx);
        volatile const unsigned short* p1 = p0 + (sy ? g.luma_tile_w : 0);
        for (unsigned it = 0;; ++it) {
          v00 = p0[0];
          v01 = p0[sx];
          v10 = p1[0];
          v11 = p1[sx];
          if (maxi(maxi(v00, v01), maxi(v10, v11)) != static_cast<int>(AV1B_TILE_EMPTY)) break;
          if (!luma_backoff(g, it, &luma_t0)) break;
        }
      } else if (g.luma) {
        const unsigned* p0 = g.luma_at + ly * g.luma_stride + lx;
        const unsigned* p1 = p0 + (sy ? g.luma_stride : 0);
        unsigned a, b, c, d;
        /* a lane's own wait: lanes leave the loop as their samples arrive */
        for (unsigned it = 0;; ++it) {
          a = ld_tag(p0);
          b = ld_tag(p0 + sx);
          c = ld_tag(p1);
          d = ld_tag(p1 + sx);
          if ((((a ^ g.tag) | (b ^ g.tag) | (c ^ g.tag) | (d ^ g.tag)) & 0xffff0000u) == 0) break;
          if (!luma_backoff(g, it, &luma_t0)) break;
        }
        v00 = static_cast<int>(a & 0xffffu);
        v01 = static_cast<int>(b & 0xffffu);
        v10 = static_cast<int>(c & 0xffffu);
        v11 = static_cast<int>(d & 0xffffu);
      } else {
        const px_t* p0 = luma + ly * luma_stride + lx;
        const px_t* p1 = p0 + (sy ? luma_stride : 0);
        v00 = ldpx(p0);
        v01 = ldpx(p0 + sx);
        v10 = ldpx(p1);
        v11 = ldpx(p1 + sx);
      }
      /* the sum of the 1, 2 or 4 samples the subsampling averages, scaled to 8x */
      int t;
      if (sx && sy) t = (v00 + v01 + v10 + v11) << 1;
      else if (sx) t = (v00 + v01) << 2;
      else if (sy) t = (v00 + v10) << 2;
      else t = v00 << 3;
      fi_pred[k] = static_cast<short>(t);   /* at most 8 * 4095 */
      sum += t;
    }
    sum = warp_sum64(sum);
    const int shift = lw + ilog2(h);
    const int avg = (int)((sum + (1LL << (shift - 1))) >> shift);
    __syncwarp();
    each([&](int i, int jj) {
      return clampi(dc + rnd2s(j.cfl_alpha * (fi_pred[(i << lw) + jj] - avg), 6), 0, j.maxv);
    });
    return;
  }
  if (j.mode == 13) { /* chroma from luma */
    const int dc = intra_dc(j, above, left, lane);
    const int sx = j.ss_x, sy = j.ss_y;
    const int lxl = ((j.x + w) << sx) - (1 << sx);
    const int lyl = ((j.y + h) << sy) - (1 << sy);
    long long sum = 0;
    for (int k = lane; k < n; k += 32) {
      const int i = k >> lw, jj = k & (w - 1);
      const int ly = mini((j.y + i) << sy, lyl), lx = mini((j.x + jj) << sx, lxl);
      int t = 0;
      for (int a = 0; a <= sy; ++a)
        for (int b = 0; b <= sx; ++b) t += ldpx(luma + (ly + a) * luma_stride + lx + b);
      sum += t << (3 - sx - sy);
    }
    sum = warp_sum64(sum);
    const int shift = lw + ilog2(h);
    const int avg = (int)((sum + (1LL << (shift - 1))) >> shift);
    for (int k = lane; k < n; k += 32) {
      const int i = k >> lw, jj = k & (w - 1);
      const int ly = mini((j.y + i) << sy, lyl), lx = mini((j.x + jj) << sx, lxl);
      int t = 0;
      for (int a = 0; a <= sy; ++a)
        for (int b = 0; b <= sx; ++b) t += ldpx(luma + (ly + a) * luma_stride + lx + b);
      const int v = t << (3 - sx - sy);
      put(i, jj, clampi(dc + rnd2s(j.cfl_alpha * (v - avg), 6), 0, j.maxv));
    }
    return;
  }

  if (j.filter_intra && w >= 4 && h >= 2) {
    /* recursive filter: 4x2 cells along anti-diagonals; a cell reads the row
     * above it (cells up-left and up) and the column left of it - the
     * predictions of this block, kept in `fi_pred` (w x h, shared memory) so
     * the recursion never round-trips through global memory; the block is
     * written (with its residual when fused) once every cell is done */
    const int cw = w >> 2, ch = h >> 1;
    const signed char* taps = kFilterIntraTaps + j.fi_mode * 56;
    for (int d = 0; d < cw + ch - 1; ++d) {
      const int c0 = maxi(0, d - (ch - 1)), c1 = mini(d, cw - 1);
      const int cells = c1 - c0 + 1;
      for (int k = lane; k < cells * 8; k += 32) {
        const int j4 = c0 + (k >> 3), i2 = d - j4;
        const int pos = k & 7, i1 = pos >> 2, j1 = pos & 3;
        int pv[7];
        for (int t = 0; t < 5; ++t) {
          if (i2 == 0) pv[t] = above[(j4 << 2) + t - 1];
          else if (j4 == 0 && t == 0) pv[t] = left[(i2 << 1) - 1];
          else pv[t] = fi_pred[((i2 << 1) - 1) * w + (j4 << 2) + t - 1];
        }
        for (int t = 5; t < 7; ++t) {
          if (j4 == 0) pv[t] = left[(i2 << 1) + t - 5];
          else pv[t] = fi_pred[((i2 << 1) + t - 5) * w + (j4 << 2) - 1];
        }
        int pr = 0;
        for (int t = 0; t < 7; ++t) pr += taps[pos * 7 + t] * pv[t];
        fi_pred[((i2 << 1) + i1) * w + (j4 << 2) + j1] = static_cast<short>(clampi(rnd2(pr, 4), 0, j.maxv));
      }
      __syncwarp();
    }
    each([&](int i, int jj) { return static_cast<int>(fi_pred[(i << lw) + jj]); });
    return;
  }

  const int mode = j.mode;
  if (mode >= 1 && mode <= 8) {
    const int pangle = kModeAngle[mode] + j.angle * 3;
    int ua = 0, ul = 0;
    if (j.filter_type >= 0 && pangle != 90 && pangle != 180) {
      if (pangle > 90 && pangle < 180 && w + h >= 24) {
        if (lane == 0) {
          const int c = rnd2(left[0] * 5 + above[-1] * 6 + above[0] * 5, 4);
          above[-1] = c;
          left[-1] = c;
        }
        __syncwarp();
      }
      const int as = j.have_above ? edge_strength(w, h, j.filter_type, pangle - 90) : 0;
      const int ls = j.have_left ? edge_strength(w, h, j.filter_type, pangle - 180) : 0;
      edge_filter(above, mini(w, j.max_x - j.x + 1) + (pangle < 90 ? h : 0) + 1, as, left,
                  mini(h, j.max_y - j.y + 1) + (pangle > 180 ? w : 0) + 1, ls, tmp, lane);
      ua = upsample_sel(w, h, j.filter_type, pangle - 90);
      if (ua) edge_upsample(above, w + (pangle < 90 ? h : 0), j.maxv, lane);
      ul = upsample_sel(w, h, j.filter_type, pangle - 180);
      if (ul) edge_upsample(left, h + (pangle > 180 ? w : 0), j.maxv, lane);
    }
    int dx = 0, dy = 0;
    if (pangle < 90) dx = kDrDeriv[pangle];
    else if (pangle > 90 && pangle < 180) dx = kDrDeriv[180 - pangle];
    if (pangle > 90 && pangle < 180) dy = kDrDeriv[pangle - 90];
    else if (pangle > 180) dy = kDrDeriv[270 - pangle];
    each([&](int i, int jj) {
      return clampi(dir_sample(above, left, w, h, pangle, dx, dy, ua, ul, i, jj), 0, j.maxv);
    });
    return;
  }
  if (mode >= 9 && mode <= 11) {
    const int bl = left[h - 1], tr = above[w - 1];
    each([&](int i, int jj) {
      int pred;
      if (mode == 9) {
        const int wy = sm_weight(h, i), wx = sm_weight(w, jj);
        pred = rnd2(wy * above[jj] + (256 - wy) * bl + wx * left[i] + (256 - wx) * tr, 9);
      } else if (mode == 10) {
        const int wy = sm_weight(h, i);
        pred = rnd2(wy * above[jj] + (256 - wy) * bl, 8);
      } else {
        const int wx = sm_weight(w, jj);
        pred = rnd2(wx * left[i] + (256 - wx) * tr, 8);
      }
      return clampi(pred, 0, j.maxv);
    });
    return;
  }
  if (mode == 12) {
    const int tl = above[-1];
    each([&](int i, int jj) {
      const int base = above[jj] + left[i] - tl;
      const int pl = absi(base - left[i]), pt = absi(base - above[jj]), ptl = absi(base - tl);
      const int v = (pl <= pt && pl <= ptl) ? left[i] : (pt <= ptl ? above[jj] : tl);
      return clampi(v, 0, j.maxv);
    });
    return;
  }
  const int dc = clampi(intra_dc(j, above, left, lane), 0, j.maxv);
  each([&](int, int) { return dc; });
}

}  // namespace av1b

#endif

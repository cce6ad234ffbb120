// lr.cu — loop restoration (7.17): Wiener and self-guided filters.
//
// Reference: rivet-av1 src/decoder/postfilter.rs:568-1004 (LrCtx::sample,
// loop_restoration, lr_stripe, lr_unit_cols, restore_stripe, lr_window,
// restore_rect_from_window, box_filter_rect, wiener_coefficient).
//
// A team of threads restores one rectangle: the rows of one stripe (64 luma
// rows, offset by 8) and up to 64 columns of one restoration unit. The team is
// a CTA of 128 threads, or for 4:2:0 chroma, whose stripes have 32 rows, half a
// CTA: one item then holds the U and the V rectangle of a place. The window the
// rectangle reads (3-sample border, the stripe-boundary rule of LrCtx::sample)
// is staged in shared memory with one row-uniform source choice per row, behind
// the only barrier. After it the team's groups work on their own: a group is
// the lanes across the rectangle, two columns a lane (32 lanes; 16 for
// rectangles of up to 32 columns), and a run of its rows, which the group
// walks down with everything it reuses in registers.
//   Wiener: the horizontal filter of a row, then the vertical filter over the
//   last seven rows' results. The horizontal taps are 16-bit by 8-bit dot
//   products on the window's packed samples.
//   Self-guided, two rows a step: box sums from the rows' horizontal sums
//   (radius 2 and 1 at once), each position's A and B packed in a word, the
//   words' neighbours from the lanes on either side, then both filters. The
//   positions one column outside the group, which no lane owns, are worked out
//   by the group beforehand, a lane a row.
// Rectangles of units without restoration (and planes or frames without it)
// pass their samples through, so the kernel writes the whole visible area of
// the reference frame and, for a frame without film grain, the packed output
// frame too, so such a frame needs no output pass.
//
// What bounds it: instruction issue and latency (each CTA's chain of item, unit
// and window loads, then a group's serial walk), at 16 warps on an SM. Against
// CTAs of 288 threads that passed A, B and the Wiener intermediate through 64 KB
// of shared memory behind a barrier a phase: 1080p 10-bit 37.5 -> 27.5 us (under
// ncu), 14.5 M -> 9.4 M warp instructions; the chain call 57.0 -> 51.8 us, 4K
// 10-bit with superres and grain 231 -> 213 us, 4K 12-bit 4:4:4 478 -> 456 us.
// 128 registers (4 CTAs a SM): at 96 or 80 the walks spill, and 1080p takes 54.2
// and 61 us. Items of whole stripes (16 rows a group) instead of 32 rows: 67 us,
// too few and too long CTAs.
#include "common.cuh"
#include "kernels.h"
#include "lr_walk.cuh"

namespace av1pf {

namespace {
constexpr A2Table make_a2() {
  A2Table t{};
  for (int z = 0; z < 256; z++) t.v[z] = z >= 255 ? 256 : (z == 0 ? 1 : ((z << 8) + z / 2) / (z + 1));
  return t;
}

constexpr int32_t kSgrParams AV1T_SGR_PARAMS_DIMS = AV1T_SGR_PARAMS;
constexpr LrConst make_lr_const() {
  LrConst t{};
  for (int set = 0; set < 16; set++)
    for (int k = 0; k < 2; k++) {
      const int n = k ? 9 : 25, n2e = n * n * kSgrParams[set][2 * k + 1];
      t.s12[set][k] = n2e ? uint32_t(((1 << 20) + n2e / 2) / n2e) << 12 : 0u;
    }
  for (int n = 1; n < 50; n++) t.inv[n] = ((1u << 22) + n - 1) / n;
  return t;
}
}  // namespace

__device__ const A2Table g_sgr_a2 = make_a2();
__constant__ LrConst c_lr = make_lr_const();

// A rectangle without restoration: its samples of the upscaled CDEF frame
// go straight to the reference frame and (frames without film grain) the
// packed frame, 8 samples per thread and step, two steps' loads in flight.
__device__ __forceinline__ void pass_through(const FrameDesc& f, int p, int x0, int y0, int w, int h, const Team& tm) {
  const int sb = f.sb, bps = f.bd > 8 ? 2 : 1;
  const uint8_t* src = f.up[p].p + (int64_t(y0) * f.up[p].stride + x0) * sb;
  const int64_t spitch = f.up[p].stride * sb, dpitch = f.ref[p].stride * sb;
  uint8_t* dst = f.ref[p].p + int64_t(y0) * dpitch + x0 * sb;
  const int64_t opitch = int64_t((f.uw + plane_ssx(f, p)) >> plane_ssx(f, p)) * bps;
  uint8_t* out = f.lr_pack ? f.frame_out + f.out_off[p] + int64_t(y0) * opitch + x0 * bps : nullptr;
  const int ng = (w + 7) >> 3;  // 8-sample chunks a row, at most 8
  const uint32_t inv = c_lr.inv[ng];
  const bool sv = ((reinterpret_cast<uintptr_t>(src) | uintptr_t(spitch)) & uintptr_t(8 * sb - 1)) == 0;
  constexpr int kBatch = 2;
#pragma unroll 1
  for (int k0 = tm.t; k0 < h * ng; k0 += kBatch * tm.n) {
    uint4 q[kBatch];  // two samples to a word
#pragma unroll
    for (int m = 0; m < kBatch; m++) {
      const int k = k0 + m * tm.n;
      if (k >= h * ng) continue;
      const int r = int((uint32_t(k) * inv) >> 22), c = (k - r * ng) * 8;
      const uint8_t* sp = src + int64_t(r) * spitch + c * sb;
      if (sv && c + 8 <= w) {
        if (sb == 2) {
          q[m] = *reinterpret_cast<const uint4*>(sp);
        } else {
          const uint2 b = *reinterpret_cast<const uint2*>(sp);
          q[m] = make_uint4(__byte_perm(b.x, 0, 0x4140), __byte_perm(b.x, 0, 0x4342), __byte_perm(b.y, 0, 0x4140),
                            __byte_perm(b.y, 0, 0x4342));
        }
      } else {
        uint32_t v[8];
#pragma unroll
        for (int e = 0; e < 8; e++) v[e] = c + e < w ? uint32_t(ld_row(sp, sb, e)) : 0u;
        q[m] = make_uint4(v[0] | (v[1] << 16), v[2] | (v[3] << 16), v[4] | (v[5] << 16), v[6] | (v[7] << 16));
      }
    }
#pragma unroll
    for (int m = 0; m < kBatch; m++) {
      const int k = k0 + m * tm.n;
      if (k >= h * ng) continue;
      const int r = int((uint32_t(k) * inv) >> 22), c = (k - r * ng) * 8, n = min(8, w - c);
      auto put = [&](uint8_t* at, int width) {
        if (n == 8 && (reinterpret_cast<uintptr_t>(at) & uintptr_t(8 * width - 1)) == 0) {
          if (width == 2)
            *reinterpret_cast<uint4*>(at) = q[m];
          else
            *reinterpret_cast<uint2*>(at) =
                make_uint2(__byte_perm(q[m].x, q[m].y, 0x6420), __byte_perm(q[m].z, q[m].w, 0x6420));
        } else {
          const uint32_t wd[4] = {q[m].x, q[m].y, q[m].z, q[m].w};
#pragma unroll
          for (int e = 0; e < 8; e++) {
            if (e >= n) continue;
            const uint32_t v = (e & 1) ? wd[e >> 1] >> 16 : wd[e >> 1];
            if (width == 2)
              reinterpret_cast<uint16_t*>(at)[e] = uint16_t(v);
            else
              at[e] = uint8_t(v);
          }
        }
      };
      put(dst + int64_t(r) * dpitch + c * sb, sb);
      if (out) put(out + int64_t(r) * opitch + c * bps, bps);
    }
  }
}

// What a group restores: rows i0 .. of the rectangle, `per` of them walked (the
// same for a warp's groups) and `left` of them written; the lane's columns c and
// c + 1, and where they go: the next row in the reference frame and (not null)
// the packed frame, in samples of rw and ow bytes.
struct Group {
  int i0, per, left, c;
  int cols;             // how many of the lane's columns are inside the rectangle
  const uint16_t* win;  // window row 0, column c
  int ws;
  uint8_t *ref, *out;
  int64_t ref_pitch, out_pitch;
  int rw, ow;
};

// Writes the next row's samples. PAIRS: both of every lane's are written, and
// are aligned as a pair in every row.
template <bool PAIRS>
__device__ __forceinline__ void emit(Group& g, uint32_t a, uint32_t b) {
  auto put = [&](uint8_t* at, int width) {
    if (PAIRS) {
      if (width == 2)
        *reinterpret_cast<uint32_t*>(at) = a | (b << 16);
      else
        *reinterpret_cast<uint16_t*>(at) = uint16_t(a | (b << 8));
      return;
    }
    if (width == 2) {
      if (g.cols > 0) reinterpret_cast<uint16_t*>(at)[0] = uint16_t(a);
      if (g.cols > 1) reinterpret_cast<uint16_t*>(at)[1] = uint16_t(b);
    } else {
      if (g.cols > 0) at[0] = uint8_t(a);
      if (g.cols > 1) at[1] = uint8_t(b);
    }
  };
  if (g.left > 0) {
    put(g.ref, g.rw);
    if (g.out) {
      put(g.out, g.ow);
      g.out += g.out_pitch;
    }
  }
  g.left--;
  g.ref += g.ref_pitch;
}

// postfilter.rs:795-822
template <bool PAIRS>
__device__ __forceinline__ void wiener_group(Group& g, const av1pf_lr_unit& u, int bd) {
  wiener_walk(g.win, g.ws, g.i0, g.per, u.wiener[0][0], u.wiener[0][1], u.wiener[0][2], u.wiener[1][0], u.wiener[1][1],
              u.wiener[1][2], bd, [](int) {}, [&](int, uint32_t a, uint32_t b) { emit<PAIRS>(g, a, b); });
}

// postfilter.rs:823-851
template <bool DEEP, bool PAIRS>
__device__ __forceinline__ void sgr_group(Group& g, const av1pf_lr_unit& u, int bd, GroupEdges& edges, int gl, int gn) {
  const int set = u.sgr_set & 15;
  const int r0 = c_sgr_params[set][0], r1 = c_sgr_params[set][2];
  // the weights of the first filter, the sample and the second filter; a filter
  // that is off (radius 0) gives the sample, whose weight then takes its own
  int w0 = u.sgr_xqd[0], w1 = u.sgr_xqd[1], w2 = (1 << 7) - w0 - w1;
  if (!r0) {
    w1 += w0;
    w0 = 0;
  }
  if (!r1) {
    w1 += w2;
    w2 = 0;
  }
  w1 *= 16;
  const int maxv = (1 << bd) - 1;
  auto finish = [&](uint32_t cd, int flt0, int flt1) {
    return uint32_t(clip3(0, maxv, (w1 * int(cd) + (1 << 10) + w0 * flt0 + w2 * flt1) >> 11));
  };
  sgr_walk<DEEP>(g.win, g.ws, g.c, g.i0, g.per, r0, r1, c_lr.s12[set][0], c_lr.s12[set][1], bd - 8, edges, gl, gn,
                 [&](uint32_t ca, uint32_t cb, int f0a, int f0b, int f1a, int f1b) {
                   emit<PAIRS>(g, finish(ca, f0a, f1a), finish(cb, f0b, f1b));
                 });
}

// With readiness flags: waits (team threads 0..15, one flag each) for the CDEF
// half superblocks under a rectangle: the stripe's rows y0 .. y1, which it
// reads from the CDEF planes, over its columns and 3 on either side. (The
// rows past the stripe come from the loop filter's output: the half
// superblocks at the stripe's first and last rows waited for the tiles
// under their windows, which reach 2 rows further.)
__device__ __forceinline__ void lr_wait_cdef(const FrameDesc& f, const SyncFlags& flags, int p, const LrGeom& geo, int x0,
                                             int w, int tid) {
  if (tid >= 16) return;
  const int sx = plane_ssx(f, p), sy = plane_ssy(f, p);
  const int xa = max(x0 - 3, 0), xb = min(x0 + w + 2, geo.pex);
  // (an item of part of a stripe reads 3 more of the stripe's rows on either side)
  const int ya = max(geo.y0 - 3, max(geo.ss, 0)), yb = min(geo.y1 + 3, min(geo.se, geo.pey));
  const int h0 = (ya << sy) >> 5, h1 = ((yb << sy) + sy) >> 5;
  const int c0 = (xa << sx) >> 6, c1 = min(((xb << sx) + sx) >> 6, f.cdef_sbc - 1);
  const int hr = h0 + (tid >> 2), c = c0 + (tid & 3);
  if (hr > h1 || c > c1) return;
  flag_wait(flags.p + f.cdef_flag_base + hr * f.cdef_sbc + c, flags.epoch);
}

// Item: the rectangle x0 .. x1 - 1 of stripe a and unit column b of `plane`;
// kind 1: of planes 1 and 2, the CTA's halves a plane each (at most 32 columns
// and rows).
template <class F>
__global__ void __launch_bounds__(kLrThreads, 4) lr_kernel(const __grid_constant__ F one, const FrameDesc* __restrict__ frames,
                                                      const Item* __restrict__ items, int n_items, SyncFlags flags) {
  AV1PF_TRACE_BEGIN();
  __shared__ __align__(16) uint16_t window[kWinBytes / 2];
  __shared__ GroupEdges edges[kLrThreads / 16];
  __shared__ const uint8_t* rows[2][kMaxH + 6];
  const int tid = threadIdx.x;

  FOR_EACH_ITEM(it, n_items) {
    const Item item = items[it];
    const FrameDesc& f = frame_of(one, frames, item.frame);
    const bool pair = item.kind != 0;
    Team tm;
    const int half = pair ? tid >> 6 : 0;
    tm.t = pair ? tid & 63 : tid;
    tm.n = pair ? 64 : kLrThreads;
    tm.bar = 1 + half;
    const int p = item.plane + half;
    const int sx = plane_ssx(f, p), sy = plane_ssy(f, p);
    // lr_stripe (postfilter.rs:640-661)
    LrGeom geo;
    const int s = item.a;
    geo.pey = ((f.fh + sy) >> sy) - 1;
    geo.pex = ((f.uw + sx) >> sx) - 1;
    geo.ss = (-8 + s * 64) >> sy;
    geo.se = geo.ss + (64 >> sy) - 1;
    geo.y0 = max(geo.ss, 0);
    geo.y1 = min(geo.se, geo.pey);
    const int x0 = item.x0, w = int(item.x1) - int(item.x0);
    // the item's rows of the stripe
    geo.y0 += item.y0;
    geo.y1 = min(geo.y1, geo.y0 + int(item.y1) - int(item.y0) - 1);
    const int h = geo.y1 - geo.y0 + 1;
    if (h <= 0 || w <= 0) {
      // without flags every CTA waits, so the kernel never completes before
      // its predecessor
      if (flags.p)
        pdl_trigger();
      else
        pdl_wait();
      continue;
    }
    int type = AV1PF_RESTORE_NONE;
    av1pf_lr_unit unit{};
    if (f.lr_on && f.lr_type[p] != AV1PF_RESTORE_NONE) {
      const int unit_size = f.lr_unit_size[p];
      const int luma_row = max(s * 64 - 8, 0);
      const int unit_row = min(f.lr_unit_rows[p] - 1, ((luma_row + 8) >> sy) >> floor_log2(uint32_t(unit_size)));  // 32 .. 256
      unit = f.lru[p][unit_row * f.lr_unit_cols[p] + item.b];
      type = unit.type;
    }
    // the descriptor and the unit are inputs of the chain; the planes below
    // are the previous stage's output: all of it, or with readiness flags
    // the half superblocks under the rectangle
    if (flags.p) {
      pdl_trigger();
      lr_wait_cdef(f, flags, p, geo, x0, w, tm.t);
      // the previous call may write the same planes
      if (flags.ahead && tm.t == 32) flag_wait(flags.complete, flags.epoch - 1);
    } else {
      pdl_wait();
    }
    const bool restores = type == AV1PF_RESTORE_WIENER || type == AV1PF_RESTORE_SGRPROJ;
    if (restores) {
      LrSrc src;
      src.up = f.up[p].p;
      src.cur = f.cur[p].p;
      // superres: upscaled boundary rows; fused horizontal LF pass: the
      // loop filter's boundary rows; else the loop-filtered plane itself
      const DPlane& lines = f.sr_on ? f.lines[p] : f.prelf[p];
      src.lines = lines.p;
      src.up_pitch = int32_t(f.up[p].stride * f.sb);
      src.cur_pitch = int32_t(f.cur[p].stride * f.sb);
      src.lines_pitch = int32_t(lines.stride * f.sb);
      src.sr = f.sr_on != 0 || f.prelf[p].p != nullptr;
      window_rows(src, rows[half], geo, s, h, tm);
    }
    tm.sync();  // (also: the team is done with the previous item's window)
    if (!restores) {
      pass_through(f, p, x0, geo.y0, w, h, tm);
      continue;
    }
    const bool wide = w > 32;
    Group g;
    g.ws = wide ? kWideWS : kSlimWS;
    uint16_t* win = window + half * kSlimTeamWin;
    stage_window(win, g.ws, rows[half], f.sb, geo.pex, x0, w, h, tm);
    const int gs = wide ? 5 : 4, gn = 1 << gs;  // lanes of a group
    const int gl = tm.t & (gn - 1), gi = tm.t >> gs, lgroups = (pair ? 6 : 7) - gs;
    // an even number of rows a group (y0 is even: row i has the parity of y0 + i)
    g.per = (((h + (1 << lgroups) - 1) >> lgroups) + 1) & ~1;
    g.i0 = gi * g.per;
    g.left = min(h - g.i0, g.per);
    g.c = 2 * gl;
    g.cols = min(w - g.c, 2);
    g.win = win + g.c;
    const int bd = f.bd;
    const int y = geo.y0 + g.i0, x = x0 + g.c;
    g.rw = f.sb;
    g.ref_pitch = f.ref[p].stride * g.rw;
    g.ref = f.ref[p].p + y * g.ref_pitch + x * g.rw;
    // the packed frame: u8 samples at 8 bits, little-endian u16 above
    // (frame.rs:153-158), rows of the plane's width (decoder/mod.rs:846-917)
    g.ow = bd > 8 ? 2 : 1;
    g.out_pitch = int64_t(geo.pex + 1) * g.ow;
    g.out = f.lr_pack ? f.frame_out + f.out_off[p] + y * g.out_pitch + x * g.ow : nullptr;
    const bool odd = ((reinterpret_cast<uintptr_t>(g.ref) | uintptr_t(g.ref_pitch)) & uintptr_t(2 * g.rw - 1)) != 0 ||
                     (g.out && ((reinterpret_cast<uintptr_t>(g.out) | uintptr_t(g.out_pitch)) & uintptr_t(2 * g.ow - 1)) != 0);
    const bool pairs = __all_sync(0xffffffffu, g.cols > 1 && !odd);
    tm.sync();
    GroupEdges& ed = edges[tid >> gs];
    if (type == AV1PF_RESTORE_WIENER)
      pairs ? wiener_group<true>(g, unit, bd) : wiener_group<false>(g, unit, bd);
    else if (bd > 10)
      pairs ? sgr_group<true, true>(g, unit, bd, ed, gl, gn) : sgr_group<true, false>(g, unit, bd, ed, gl, gn);
    else
      pairs ? sgr_group<false, true>(g, unit, bd, ed, gl, gn) : sgr_group<false, false>(g, unit, bd, ed, gl, gn);
  }
  AV1PF_TRACE_END(3);
}

void launch_lr(const FrameSet& frames, const Item* items, int n_items, SyncFlags flags, cudaStream_t s) {
  if (n_items <= 0) return;
  // one CTA per item: the block scheduler hands items of uneven cost (copy,
  // Wiener, self-guided) to SMs as they free up
  launch_frames(frames, lr_kernel<NoFrame>, lr_kernel<OneFrame>, min(n_items, kItemGrid), kLrThreads, 0, s, items, n_items,
                flags);
}

}  // namespace av1pf

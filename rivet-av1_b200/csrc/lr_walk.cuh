// lr_walk.cuh — what the decoder's loop restoration (lr.cu) and the encoder's
// search for it (lr_search.cu) share: staging a rectangle's window, and the
// self-guided filters walked down its rows in registers.
//
// Reference: rivet-av1 src/decoder/postfilter.rs:581-597, 765-777, 884-991.
#pragma once

#include <cstdint>

#include "common.cuh"

namespace av1pf {

constexpr int kLrThreads = 128;
constexpr int kMaxH = 64;  // rows per stripe
// window row strides (u16): rectangles of up to 64 columns (w + 6 <= 70), and of
// up to 32, whose two groups a warp read rows 8 apart: 8 x 22 words are 16 mod
// 32 banks
constexpr int kWideWS = 72, kSlimWS = 44;
// a team's window: 70 wide rows, or two of 38 slim ones (the last rows' loads
// reach past their columns)
constexpr int kWinBytes = (kMaxH + 6) * kWideWS * 2 + 16;
constexpr int kSlimTeamWin = (kMaxH / 2 + 6) * kSlimWS + 8;  // u16
// per group: the packed A / B of the columns on either side, for the first
// filter's rows and the second's
constexpr int kEdgeRows = 18;
struct GroupEdges {
  uint32_t first[kEdgeRows / 2][2], second[kEdgeRows][2];
};

// SGR_A2 (postfilter.rs:884-898), built at compile time into global memory:
// the self-guided passes read it through the L1, so no CTA sets it up.
struct A2Table {
  int32_t v[256];
};
extern __device__ const A2Table g_sgr_a2;
// The scale s of each self-guided parameter set's two filters, times 2^12
// (postfilter.rs:903-918: ((1 << 20) + n^2 eps / 2) / (n^2 eps)), and 2^22 / n
// rounded up, for quotients k / n of k < 2^22 / n without a division (chunks of
// eight columns of a unit of up to 383, in 70 rows).
struct LrConst {
  uint32_t s12[16][2];
  uint32_t inv[50];
};
extern __constant__ LrConst c_lr;

// The threads that restore one rectangle: `t` of `n`, meeting at barrier `bar`.
struct Team {
  int t, n, bar;
  __device__ __forceinline__ void sync() const {  // (constant barrier names: a kernel that computes them holds all 16)
    if (bar == 1)
      asm volatile("bar.sync 1, %0;" ::"r"(n) : "memory");
    else
      asm volatile("bar.sync 2, %0;" ::"r"(n) : "memory");
  }
};

struct LrGeom {
  int ss, se, y0, y1, pex, pey;
};

// The three sources LrCtx::sample (postfilter.rs:584-596) draws rows from,
// read once per rectangle: the upscaled CDEF plane, the loop-filtered plane
// and (with superres) the line buffer of upscaled pre-CDEF rows.
struct LrSrc {
  const uint8_t* up;
  const uint8_t* cur;
  const uint8_t* lines;
  int32_t up_pitch, cur_pitch, lines_pitch;  // bytes
  bool sr;  // the pre-CDEF rows come from `lines` (4 per stripe boundary), not `cur`
};

// The row LrCtx::sample reads for window row y of stripe `s`. With superres
// (or with the loop filter's horizontal pass run inside the CDEF kernel) the
// pre-CDEF rows come from a line buffer, 4 rows per stripe boundary:
// boundary b (the first row B of stripe b) holds rows B-2 .. B+1 at line
// rows (b-1)*4 ...
__device__ __forceinline__ const uint8_t* lr_row(const LrSrc& src, const LrGeom& g, int s, int y) {
  y = max(min(y, g.pey), 0);
  if (y < g.ss) {
    const int yy = max(g.ss - 2, y);
    return src.sr ? src.lines + int64_t((s - 1) * 4 + (yy - (g.ss - 2))) * src.lines_pitch
                  : src.cur + int64_t(yy) * src.cur_pitch;
  }
  if (y > g.se) {
    const int yy = min(g.se + 2, y);
    return src.sr ? src.lines + int64_t(s * 4 + (yy - (g.se - 1))) * src.lines_pitch
                  : src.cur + int64_t(yy) * src.cur_pitch;
  }
  return src.up + int64_t(y) * src.up_pitch;
}

__device__ __forceinline__ int ld_row(const uint8_t* row, int sb, int x) {
  return sb == 1 ? int(row[x]) : int(reinterpret_cast<const uint16_t*>(row)[x]);
}

// Where the window's rows come from: rows[r] is the start of the plane row that
// window row r reads.
__device__ __forceinline__ void window_rows(const LrSrc& src, const uint8_t** rows, const LrGeom& geo, int s, int h,
                                            const Team& tm) {
  for (int r = tm.t; r < h + 6; r += tm.n) rows[r] = lr_row(src, geo, s, geo.y0 + r - 3);
}

// lr_window (postfilter.rs:765-777): window row r, columns 8q .. 8q+7 (samples
// x0-3+8q ..) per task. Where the two aligned 8-sample chunks that hold them
// lie inside the plane row (and the row is 16-byte aligned) they come as two
// vector loads and are shifted into place; other chunks (the plane's left and
// right edges) take one clamped scalar load per sample. The loads of two
// tasks issue before their stores.
__device__ __forceinline__ void stage_window(uint16_t* win, int ws, const uint8_t* const* rows, int sb, int pex, int x0,
                                             int w, int h, const Team& tm) {
  const int ww = w + 6, wh = h + 6;
  const int nq = (ww + 7) >> 3;  // chunks per window row
  const uint32_t inv = c_lr.inv[nq];
  const int ntask = wh * nq;
  constexpr int kBatch = 2;
#pragma unroll 1
  for (int k0 = tm.t; k0 < ntask; k0 += kBatch * tm.n) {
    uint32_t wv[kBatch][5];  // the loaded words a window chunk is cut from
    bool vec[kBatch];
#pragma unroll
    for (int m = 0; m < kBatch; m++) {
      const int k = k0 + m * tm.n;
      vec[m] = false;
      if (k >= ntask) continue;
      const int r = int((uint32_t(k) * inv) >> 22), q = k - r * nq;
      const uint8_t* row = rows[r];
      const int gx = x0 - 8 + 8 * q;  // first sample of the left chunk
      if (gx < 0 || gx + 16 > pex + 1 || (reinterpret_cast<uintptr_t>(row) & 15) != 0) continue;
      vec[m] = true;
      if (sb == 2) {
        // samples 4..7 of the left chunk and 0..5 of the right one
        const uint2 a = *reinterpret_cast<const uint2*>(row + int64_t(gx) * 2 + 8);
        const uint4 b = *reinterpret_cast<const uint4*>(row + int64_t(gx) * 2 + 16);
        wv[m][0] = a.x; wv[m][1] = a.y; wv[m][2] = b.x; wv[m][3] = b.y; wv[m][4] = b.z;
      } else {
        // bytes 4..15 of the 16 samples
        const uint4 a = *reinterpret_cast<const uint4*>(row + gx);
        wv[m][0] = a.y; wv[m][1] = a.z; wv[m][2] = a.w;
      }
    }
#pragma unroll
    for (int m = 0; m < kBatch; m++) {
      const int k = k0 + m * tm.n;
      if (k >= ntask) continue;
      const int r = int((uint32_t(k) * inv) >> 22), q = k - r * nq;
      uint16_t* wp = &win[r * ws + 8 * q];
      if (vec[m]) {
        uint4 o;
        if (sb == 2) {
          // window sample 2j of the chunk is sample 5 + 2j of the 16 from gx
          o.x = __funnelshift_r(wv[m][0], wv[m][1], 16);
          o.y = __funnelshift_r(wv[m][1], wv[m][2], 16);
          o.z = __funnelshift_r(wv[m][2], wv[m][3], 16);
          o.w = __funnelshift_r(wv[m][3], wv[m][4], 16);
        } else {
          const uint32_t lo = __funnelshift_r(wv[m][0], wv[m][1], 8);  // bytes 5..8
          const uint32_t hi = __funnelshift_r(wv[m][1], wv[m][2], 8);  // bytes 9..12
          o.x = __byte_perm(lo, 0, 0x4140);
          o.y = __byte_perm(lo, 0, 0x4342);
          o.z = __byte_perm(hi, 0, 0x4140);
          o.w = __byte_perm(hi, 0, 0x4342);
        }
        // (slim rows are 8-byte aligned)
        reinterpret_cast<uint2*>(wp)[0] = make_uint2(o.x, o.y);
        if (8 * q + 4 < ws) reinterpret_cast<uint2*>(wp)[1] = make_uint2(o.z, o.w);
      } else {
        const uint8_t* row = rows[r];
#pragma unroll
        for (int e = 0; e < 8; e++) {
          const int c = 8 * q + e;
          if (c < ww) wp[e] = uint16_t(ld_row(row, sb, max(min(x0 - 3 + c, pex), 0)));
        }
      }
    }
  }
}

// Four 8-bit coefficients in a word.
__device__ __forceinline__ int bytes4(int a, int b, int c, int d) {
  return int((uint32_t(a) & 255u) | ((uint32_t(b) & 255u) << 8) | ((uint32_t(c) & 255u) << 16) | (uint32_t(d) << 24));
}

// The Wiener filter (postfilter.rs:795-822) with vertical taps v0 v1 v2 (and
// the middle one that makes their sum 128) and horizontal ones h0 h1 h2: two
// columns a lane, rows i0 .. i0 + per - 1, four a step (per is rounded up to
// fours, and the window has those rows). `win` is window row 0 at the first
// column. begin(i) is called before rows i .. i + 3 (from 0), emit(i, a, b) takes
// row i's outputs.
template <class Begin, class Emit>
__device__ __forceinline__ void wiener_walk(const uint16_t* win, int ws, int i0, int per, int v0, int v1, int v2, int h0,
                                            int h1, int h2, int bd, Begin begin, Emit emit) {
  const int round0 = bd == 12 ? 5 : 3, round1 = bd == 12 ? 9 : 11;
  const int offset = 1 << (bd + 7 - round0 - 1);
  const int limit = (1 << (bd + 1 + 7 - round0)) - 1;
  const int maxv = (1 << bd) - 1;
  const int h3 = 128 - 2 * (h0 + h1 + h2), v3 = 128 - 2 * (v0 + v1 + v2);
  // the taps but the middle one (which can exceed 8 bits) against the samples
  // c .. c + 7, for the first column and the second
  const int e0 = bytes4(h0, h1, h2, 0), e1 = bytes4(h2, h1, h0, 0);
  const int o0 = bytes4(0, h0, h1, h2), o1 = bytes4(0, h2, h1, h0);
  const int rnd0 = 1 << (round0 - 1), rnd1 = 1 << (round1 - 1);
  const uint16_t* row = win + i0 * ws;
  auto across = [&](int& a, int& b) {
    const uint32_t* q = reinterpret_cast<const uint32_t*>(row);
    row += ws;
    const int q0 = int(q[0]), q1 = int(q[1]), q2 = int(q[2]), q3 = int(q[3]);
    int x = int(uint32_t(q1) >> 16) * h3 + rnd0, y = (q2 & 0xffff) * h3 + rnd0;
    x = __dp2a_hi(q3, e1, __dp2a_lo(q2, e1, __dp2a_hi(q1, e0, __dp2a_lo(q0, e0, x))));
    y = __dp2a_hi(q3, o1, __dp2a_lo(q2, o1, __dp2a_hi(q1, o0, __dp2a_lo(q0, o0, y))));
    a = clip3(-offset, limit - offset, x >> round0);
    b = clip3(-offset, limit - offset, y >> round0);
  };
  // the last six rows' results and four new ones a step
  int a[10], b[10];
#pragma unroll
  for (int k = 0; k < 6; k++) across(a[k], b[k]);
  auto down = [&](const int* t) {
    const int acc = v0 * (t[0] + t[6]) + v1 * (t[1] + t[5]) + v2 * (t[2] + t[4]) + v3 * t[3] + rnd1;
    return uint32_t(clip3(0, maxv, acc >> round1));
  };
#pragma unroll 1
  for (int i = 0; i < per; i += 4) {
    begin(i);
#pragma unroll
    for (int k = 0; k < 4; k++) {
      across(a[6 + k], b[6 + k]);
      emit(i + k, down(a + k), down(b + k));
    }
#pragma unroll
    for (int k = 0; k < 6; k++) {
      a[k] = a[k + 4];
      b[k] = b[k + 4];
    }
  }
}

// A and B of box_filter_rect (postfilter.rs:935-959) packed in a word, A above
// B, from the sum and the sum of squares over a box of radius R. B is at most
// (255 * ((4096 + n / 2) / n) * n * (2^bitdepth - 1) + 2^11) >> 12 < 2^20 for 12
// bits, and all products fit 32 bits but p * s.
constexpr int kAB = 21;  // bits of B: room for the sum of two at 12 bits, of five at 10
template <int R>
__device__ __forceinline__ uint32_t sgr_word(uint32_t sum, uint32_t sq, uint32_t s12, int sh) {
  constexpr uint32_t n = (2 * R + 1) * (2 * R + 1), one_over_n = ((1u << 12) + n / 2) / n;
  const uint32_t half = (1u << sh) >> 1;
  const uint32_t a = (sq + ((1u << (2 * sh)) >> 1)) >> (2 * sh), d = (sum + half) >> sh;
  const int pp = max(int(a * n - d * d), 0);
  // (p * s + 2^19) >> 20, as the high word of p * (s << 12) + 2^31
  const uint32_t z = uint32_t((uint64_t(uint32_t(pp)) * s12 + (1u << 31)) >> 32);
  const uint32_t a2 = uint32_t(__ldg(&g_sgr_a2.v[min(z, 255u)]));
  const uint32_t b = ((256u - a2) * one_over_n * sum + (1u << 11)) >> 12;
  return (a2 << kAB) | b;
}

// The outputs of a parameter set's two filters (box_filter_rect,
// postfilter.rs:901-991) at every sample of a group: the lanes across a
// rectangle, two columns (c and c + 1) a lane, and rows i0 .. i0 + per - 1 (i0
// and per even, and the rectangle's first row even in the plane). `win` is
// window row 0 at column c, rows ws apart: window row i + 3, columns c + 3 and
// c + 4 are the lane's samples of row i. emit(ca, cb, f0a, f0b, f1a, f1b) takes a
// row's samples and both filters' outputs, row by row; a filter of radius 0
// (r0, r1) puts out 0. sa, sb: c_lr.s12 of the filters; sh: bitdepth - 8. DEEP:
// 12 bits, where sums of more than two B's leave their field and the sum over a
// 5x5 box its 16 bits. All lanes of a warp call, with the same `per`.
template <bool DEEP, class Emit>
__device__ __forceinline__ void sgr_walk(const uint16_t* win, int ws, int c, int i0, int per, int r0, int r1, uint32_t sa,
                                         uint32_t sb, int sh, GroupEdges& edges, int gl, int gn, Emit emit) {
  // --- the words of the columns at either side of the group: one at a time, a
  // lane a (row, side). Row j of `second` is output row i0 - 1 + j, of `first`
  // i0 - 1 + 2j ---
  {
    const uint16_t* base = win - c + i0 * ws;  // window row i0, the group's first column
    const int width = 2 * gn;
    if (r1)
#pragma unroll 1
      for (int k = gl; k < 2 * (per + 2); k += gn) {
        const int j = k >> 1, side = k & 1;
        const uint16_t* at = base + (j + 2) * ws + (side ? width : -1) + 3;
        uint32_t s = 0, q = 0;
#pragma unroll
        for (int y = -1; y <= 1; y++)
#pragma unroll
          for (int x = -1; x <= 1; x++) {
            const uint32_t v = at[y * ws + x];
            s += v;
            q += v * v;
          }
        edges.second[j][side] = sgr_word<1>(s, q, sb, sh);
      }
    if (r0)
#pragma unroll 1
      for (int k = gl; k < per + 2; k += gn) {
        const int j = k >> 1, side = k & 1;
        const uint16_t* at = base + (2 * j + 2) * ws + (side ? width : -1) + 3;
        uint32_t s = 0, q = 0;
#pragma unroll
        for (int y = -2; y <= 2; y++)
#pragma unroll
          for (int x = -2; x <= 2; x++) {
            const uint32_t v = at[y * ws + x];
            s += v;
            q += v * v;
          }
        edges.first[j][side] = sgr_word<2>(s, q, sa, sh);
      }
    __syncwarp();
  }
  const bool at_left = gl == 0, at_right = gl == gn - 1;
  // A word's two columns in x, and the sums of each one's neighbours in y
  struct Words {
    uint32_t x0, x1, y0, y1;
  };
  auto with_neighbours = [&](uint32_t x0, uint32_t x1, const uint32_t (&edge)[2]) {
    uint32_t l = __shfl_up_sync(0xffffffffu, x1, 1), r = __shfl_down_sync(0xffffffffu, x0, 1);
    if (at_left) l = edge[0];
    if (at_right) r = edge[1];
    return Words{x0, x1, l + x1, x0 + r};
  };
  // Horizontal sums of a window row around the lane's two columns: the samples
  // (both columns' in the halves of a word) and their squares, radius 2 and 1.
  struct Rows {
    uint32_t s5, s3, q5a, q5b, q3a, q3b;
  };
  const uint16_t* row = win + i0 * ws;
  auto across = [&]() {
    const uint32_t* q = reinterpret_cast<const uint32_t*>(row);
    row += ws;
    // window columns c .. c + 7; the lane's columns are 3 and 4 of them
    const uint32_t k0 = q[0], k1 = q[1], k2 = q[2], k3 = q[3];
    const uint32_t m1 = __byte_perm(k0, k1, 0x5432), m2 = __byte_perm(k1, k2, 0x5432), m3 = __byte_perm(k2, k3, 0x5432);
    Rows t;
    t.s3 = k1 + m2 + k2;                 // (2,3) + (3,4) + (4,5)
    t.s5 = t.s3 + m1 + m3;               // + (1,2) + (5,6)
    const uint32_t p1 = k0 >> 16, p2 = k1 & 0xffffu, p3 = k1 >> 16, p4 = k2 & 0xffffu, p5 = k2 >> 16, p6 = k3 & 0xffffu;
    const uint32_t m = p3 * p3 + p4 * p4;
    t.q3a = p2 * p2 + m;
    t.q3b = p5 * p5 + m;
    t.q5a = p1 * p1 + (p5 * p5 + t.q3a);
    t.q5b = p6 * p6 + (p2 * p2 + t.q3b);
    return t;
  };
  auto lo = [](uint32_t v) { return v & 0xffffu; };
  auto hi = [](uint32_t v) { return v >> 16; };
  // The sums of the rows so far, of step row i: radius 2, row i - 1 (p), rows i
  // and i + 1 together (g) and row i + 1 (o); radius 1, rows i and i + 1 together
  // (g3) and row i + 1 (o3). Samples of both columns in a word, squares apart.
  struct Sums {
    uint32_t s, a, b;
    __device__ __forceinline__ Sums operator+(const Sums& t) const { return Sums{s + t.s, a + t.a, b + t.b}; }
  };
  auto of5 = [](const Rows& t) { return Sums{t.s5, t.q5a, t.q5b}; };
  auto of3 = [](const Rows& t) { return Sums{t.s3, t.q3a, t.q3b}; };
  auto words1 = [&](const Sums& t, const uint32_t (&edge)[2]) {
    return with_neighbours(sgr_word<1>(lo(t.s), t.a, sb, sh), sgr_word<1>(hi(t.s), t.b, sb, sh), edge);
  };
  // (DEEP: the five rows' sample sums leave 16 bits; x is the sum of three rows' at most, y of two)
  auto words2 = [&](const Sums& x, const Sums& y, const uint32_t (&edge)[2]) {
    const uint32_t s = x.s + y.s;
    return with_neighbours(sgr_word<2>(DEEP ? lo(x.s) + lo(y.s) : lo(s), x.a + y.a, sa, sh),
                           sgr_word<2>(DEEP ? hi(x.s) + hi(y.s) : hi(s), x.b + y.b, sa, sh), edge);
  };
  Sums p{}, g5{}, o{}, g3{}, o3{};
  Words f0{}, b0{}, b1{};  // first filter: row i - 1; second: rows i - 1 and i
  {
    const Rows t0 = across(), t1 = across(), t2 = across(), t3 = across(), t4 = across();  // rows i0 - 3 .. i0 + 1
    p = of5(t2);
    o = of5(t4);
    g5 = of5(t3) + o;
    o3 = of3(t4);
    g3 = of3(t3) + o3;
    if (r0) f0 = words2(of5(t0) + of5(t1) + p, g5, edges.first[0]);
    if (r1) {
      b0 = words1(of3(t1) + of3(t2) + of3(t3), edges.second[0]);
      b1 = words1(of3(t2) + g3, edges.second[1]);
    }
  }
  constexpr uint32_t kB = (1u << kAB) - 1;
  // (wa * A's + wb * B's) of words x and y weighed wx and wy, times the sample
  auto blend = [&](uint32_t x, uint32_t y, int wx, int wy, uint32_t cd) {
    return int((wx * (x >> kAB) + wy * (y >> kAB)) * cd + (wx * (x & kB) + wy * (y & kB)));
  };
  auto blend2 = [&](uint32_t x, uint32_t x2, uint32_t y, uint32_t y2, int wx, int wy, uint32_t cd) {
    return DEEP ? int((wx * ((x >> kAB) + (x2 >> kAB)) + wy * ((y >> kAB) + (y2 >> kAB))) * cd +
                      (wx * ((x & kB) + (x2 & kB)) + wy * ((y & kB) + (y2 & kB))))
                : blend(x + x2, y + y2, wx, wy, cd);
  };
  auto blend5 = [&](uint32_t x, uint32_t y, uint32_t x0, uint32_t x2, uint32_t y0, uint32_t y2, uint32_t cd) {
    return DEEP ? int((4 * ((x >> kAB) + (y >> kAB) + (x0 >> kAB) + (x2 >> kAB)) + 3 * ((y0 >> kAB) + (y2 >> kAB))) * cd +
                      (4 * ((x & kB) + (y & kB) + (x0 & kB) + (x2 & kB)) + 3 * ((y0 & kB) + (y2 & kB))))
                : blend(x + y + x0 + x2, y0 + y2, 4, 3, cd);
  };
#pragma unroll 1  // (and the loops below and above: unrolled, they take more registers than a CTA has)
  for (int step = 0; step < per / 2; step++) {
    // row i + 2 completes the second filter's row i + 1, and its output row i
    Rows t = across();
    Words b2{};
    Sums n5 = of5(t);
    const Sums n3 = of3(t);
    if (r1) b2 = words1(g3 + n3, edges.second[2 * step + 2]);
    const uint16_t* mid = row - 3 * ws + 2;  // samples (c - 1, c) and (c + 1, ..) of row i
    uint32_t ca = hi(*reinterpret_cast<const uint32_t*>(mid)), cb = lo(*reinterpret_cast<const uint32_t*>(mid + 2));
    const int sa1 = (blend5(b1.x0, b1.y0, b0.x0, b2.x0, b0.y0, b2.y0, ca) + 256) >> 9;
    const int sb1 = (blend5(b1.x1, b1.y1, b0.x1, b2.x1, b0.y1, b2.y1, cb) + 256) >> 9;
    // row i + 3 completes the first filter's row i + 1: the even output row takes
    // it and row i - 1
    t = across();
    Words f1{};
    const Sums m5 = of5(t);
    if (r0) f1 = words2(p + g5, n5 + m5, edges.first[step + 1]);
    emit(ca, cb, (blend2(f0.x0, f1.x0, f0.y0, f1.y0, 6, 5, ca) + 256) >> 9,
         (blend2(f0.x1, f1.x1, f0.y1, f1.y1, 6, 5, cb) + 256) >> 9, sa1, sb1);
    f0 = f1;
    b0 = b1;
    b1 = b2;
    // and the second filter's row i + 2: the odd row
    if (r1) b2 = words1(o3 + n3 + of3(t), edges.second[2 * step + 3]);
    mid += ws;
    ca = hi(*reinterpret_cast<const uint32_t*>(mid));
    cb = lo(*reinterpret_cast<const uint32_t*>(mid + 2));
    emit(ca, cb, (blend(f0.x0, f0.y0, 6, 5, ca) + 128) >> 8, (blend(f0.x1, f0.y1, 6, 5, cb) + 128) >> 8,
         (blend5(b1.x0, b1.y0, b0.x0, b2.x0, b0.y0, b2.y0, ca) + 256) >> 9,
         (blend5(b1.x1, b1.y1, b0.x1, b2.x1, b0.y1, b2.y1, cb) + 256) >> 9);
    b0 = b1;
    b1 = b2;
    p = o;
    o = m5;
    g5 = n5 + m5;
    o3 = of3(t);
    g3 = n3 + o3;
  }
}

}  // namespace av1pf

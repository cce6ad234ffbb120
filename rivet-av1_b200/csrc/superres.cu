// superres.cu — super-resolution upscaling (7.16).
//
// Reference: rivet-av1 src/decoder/postfilter.rs:515-566 (`upscale`).
//
// The reference upscales the whole CDEF frame and the whole pre-CDEF frame;
// loop restoration reads the latter only at the 4 rows around each stripe
// boundary (LrCtx::sample, postfilter.rs:581-597), so here the pre-CDEF
// frame is upscaled only at those rows, into a small line buffer.
// Item kind 0: rows [y0, y1) of cdef -> up. Kind 1: line rows [y0, y1) of the
// line buffer (4 per stripe boundary: rows B-2 .. B+1 of the boundary at B).
// An item's (at most 4) source rows are staged together in shared memory
// (16-byte loads, the edge samples repeated beyond both ends), behind one barrier.
// What bounds it is instruction issue and the shared-memory reads, so a thread
// makes two neighbouring columns of all the rows: their places, phases and
// coefficients once, and of a row five words that hold the taps of both, which
// dp2a weighs by the 8-bit coefficients, shifted to where each column's taps
// start in the words. A 3840x2160 10-bit 4:2:0 frame from 2363
// columns: 42.7 us with an output a thread and step and 16-bit products, 28.5 now.
// The row buffers are sized per launch to the widest source row among the
// launch's frames.
#include "av1_tables.h"
#include "common.cuh"
#include "kernels.h"

namespace av1pf {

namespace {
constexpr int kMaxRow = 16384 + 16;  // source samples staged per row, at most
constexpr int kRows = 4;             // rows per item
constexpr int kPadL = 8, kPadR = 10;  // edge samples repeated beside a staged row
// row stride of the staged rows (u16): 16-byte aligned
__host__ __device__ constexpr int sr_stride(int n) { return (kPadL + n + kPadR + 7) & ~7; }

// The 8-tap filters (7.16) as bytes, for dp2a: a tap of 128 is held as 127, and
// the sample that it weighs is added once more (phases 0, 1 and 63: it is the
// tap nearer to the output).
struct UpTable {
  uint2 v[64];
};
constexpr UpTable make_up_table() {
  constexpr int16_t f[64][8] = AV1T_UPSCALE_FILTER;
  UpTable t{};
  for (int p = 0; p < 64; p++) {
    uint32_t w[2] = {0, 0};
    for (int k = 0; k < 8; k++) w[k / 4] |= uint32_t(uint8_t(f[p][k] == 128 ? 127 : f[p][k])) << (8 * (k % 4));
    t.v[p] = uint2{w[0], w[1]};
  }
  return t;
}
__device__ const UpTable g_up_table = make_up_table();

// A column's taps against the words that hold them: where in the row's words they
// start (0 .. 2 samples in) is in the coefficients.
struct UpTaps {
  uint32_t k0, k1, k2;
  int near;   // the sample that the largest tap weighs
  int again;  // 1: its weight is 128
  __device__ __forceinline__ UpTaps(int phase, int px, int shift) {
    const uint2 c = __ldg(&g_up_table.v[phase]);
    k0 = c.x << (8 * shift);
    k1 = __funnelshift_l(c.x, c.y, 8 * shift);
    k2 = __funnelshift_l(c.y, 0, 8 * shift);
    near = px + (phase > 31 ? 1 : 0);
    again = phase < 2 || phase == 63 ? 1 : 0;
  }
  __device__ __forceinline__ int of(const uint32_t (&w)[5], int nearest, int maxv) const {
    int sum = nearest * again + 64;
    sum = __dp2a_lo(int(w[0]), int(k0), sum);
    sum = __dp2a_hi(int(w[1]), int(k0), sum);
    sum = __dp2a_lo(int(w[2]), int(k1), sum);
    sum = __dp2a_hi(int(w[3]), int(k1), sum);
    sum = __dp2a_lo(int(w[4]), int(k2), sum);
    return min(max(sum >> 7, 0), maxv);
  }
};

// The item's output rows (postfilter.rs:547-561), two columns of every row a
// thread and step; ALL: all four rows are inside the plane, else those of `have`.
template <int SB, bool ALL>
__device__ __forceinline__ void upscale(const uint16_t* rows, int rs, uint8_t* out, int64_t pitch, int w, int step,
                                        int init, int max_x, int maxv, uint32_t have) {
  // (a caller's plane may start, or have its rows, anywhere)
  const bool pairs = ((reinterpret_cast<uintptr_t>(out) | uintptr_t(pitch)) & uintptr_t(2 * SB - 1)) == 0;
  for (int x = 2 * threadIdx.x; x < w; x += 2 * blockDim.x) {
    // (x * step is about the source column times 2^14: below 2^29. Beyond the
    // pads all taps are the same sample.)
    const int at0 = init - (1 << 14) + x * step, at1 = at0 + step;
    const int px0 = min(max(at0 >> 14, -5), max_x + 4), px1 = min(max(at1 >> 14, -5), max_x + 4);
    const int first = px0 - 3 + kPadL, shift = first & 1;
    const UpTaps u0((at0 & 0x3fff) >> 8, px0, shift), u1((at1 & 0x3fff) >> 8, px1, shift + px1 - px0);
    const uint16_t* row = rows + (first - shift);
    const int n0 = u0.near + kPadL - (first - shift), n1 = u1.near + kPadL - (first - shift);
    const bool both = pairs && x + 1 < w;
    uint8_t* to = out + x * SB;
#pragma unroll
    for (int k = 0; k < kRows; k++) {
      if (ALL || (have >> k & 1)) {
        uint32_t t[5];
#pragma unroll
        for (int q = 0; q < 5; q++) t[q] = reinterpret_cast<const uint32_t*>(row)[q];
        const uint32_t a = uint32_t(u0.of(t, row[n0], maxv)), b = uint32_t(u1.of(t, row[n1], maxv));
        if (both) {
          if (SB == 2)
            *reinterpret_cast<uint32_t*>(to) = a | (b << 16);
          else
            *reinterpret_cast<uint16_t*>(to) = uint16_t(a | (b << 8));
        } else if (SB == 2) {
          reinterpret_cast<uint16_t*>(to)[0] = uint16_t(a);
          if (x + 1 < w) reinterpret_cast<uint16_t*>(to)[1] = uint16_t(b);
        } else {
          to[0] = uint8_t(a);
          if (x + 1 < w) to[1] = uint8_t(b);
        }
      }
      row += rs;
      to += pitch;
    }
  }
}
}  // namespace

template <class F>
__global__ void __launch_bounds__(256, 5) superres_kernel(const __grid_constant__ F one, const FrameDesc* __restrict__ frames,
                                                     const Item* __restrict__ items, int n_items, int rs) {
  AV1PF_TRACE_BEGIN();
  extern __shared__ __align__(16) uint8_t sr_smem[];
  uint16_t* rows = reinterpret_cast<uint16_t*>(sr_smem);  // kRows staged source rows, rs apart
  pdl_wait();  // the previous stage's output is complete past this point
  FOR_EACH_ITEM(it, n_items) {
    const Item item = items[it];
    int p, sy, sb, maxv, step, init, max_x, w, plane_h, kind;
    bool prelf;
    DPlane src, dst;
    {
      const FrameDesc& f = frame_of(one, frames, item.frame);
      p = item.plane;
      kind = item.kind;
      sy = plane_ssy(f, p);
      sb = f.sb;
      maxv = (1 << f.bd) - 1;
      step = f.sr_step[p];
      init = f.sr_init[p];
      max_x = f.sr_maxx[p];
      w = f.sr_w[p];
      plane_h = (f.fh + sy) >> sy;
      // kind 1 reads the loop filter's boundary rows: from the plane, or
      // from f.prelf when the CDEF kernel ran the horizontal LF pass
      prelf = kind == 1 && f.prelf[p].p != nullptr;
      src = kind == 0 ? f.cdef[p] : (prelf ? f.prelf[p] : f.cur[p]);
      dst = kind == 0 ? f.up[p] : f.lines[p];
    }
    const int n_src = max_x + 1;
    const int nr = min(int(item.y1) - int(item.y0), kRows);
    // the source row of output row y0 + k, or -1 outside the plane (uniform across the CTA)
    auto src_row_of = [&](int k) {
      const int r = item.y0 + k;
      int sr = r;
      if (kind == 1) {
        const int s = r / 4 + 1, j = r % 4;
        sr = ((64 * s - 8) >> sy) - 2 + j;
      }
      return sr >= 0 && sr < plane_h ? (prelf ? r : sr) : -1;
    };
    // --- stage the rows ---
    for (int k = 0; k < nr; k++) {
      const int sr = src_row_of(k);
      if (sr < 0) continue;
      const uint8_t* sp = src.p + int64_t(sr) * src.stride * sb;
      uint16_t* rp = rows + k * rs + kPadL;
      const int edge = int(threadIdx.x) < kPadL ? 0 : max_x;
      if (threadIdx.x < kPadL + kPadR)
        rp[int(threadIdx.x) >= kPadL ? n_src + int(threadIdx.x) - kPadL : int(threadIdx.x) - kPadL] =
            uint16_t(sb == 2 ? reinterpret_cast<const uint16_t*>(sp)[edge] : sp[edge]);
      if (sb == 2) {
        const int nv = n_src >> 3;
        for (int q = threadIdx.x; q < nv; q += blockDim.x)
          reinterpret_cast<uint4*>(rp)[q] = reinterpret_cast<const uint4*>(sp)[q];
        for (int q = nv * 8 + threadIdx.x; q < n_src; q += blockDim.x) rp[q] = reinterpret_cast<const uint16_t*>(sp)[q];
      } else {
        const int nv = n_src >> 4;
        for (int q = threadIdx.x; q < nv; q += blockDim.x) {
          const uint4 v = reinterpret_cast<const uint4*>(sp)[q];
          uint4* d = reinterpret_cast<uint4*>(rp + q * 16);
          d[0] = make_uint4(__byte_perm(v.x, 0, 0x4140), __byte_perm(v.x, 0, 0x4342), __byte_perm(v.y, 0, 0x4140),
                            __byte_perm(v.y, 0, 0x4342));
          d[1] = make_uint4(__byte_perm(v.z, 0, 0x4140), __byte_perm(v.z, 0, 0x4342), __byte_perm(v.w, 0, 0x4140),
                            __byte_perm(v.w, 0, 0x4342));
        }
        for (int q = nv * 16 + threadIdx.x; q < n_src; q += blockDim.x) rp[q] = sp[q];
      }
    }
    __syncthreads();
    uint32_t have = 0;  // the item's rows that are inside the plane
#pragma unroll
    for (int k = 0; k < kRows; k++)
      if (k < nr && src_row_of(k) >= 0) have |= 1u << k;
    uint8_t* out = dst.p + int64_t(item.y0) * dst.stride * sb;
    const int64_t pitch = dst.stride * sb;
    if (sb == 2)
      have == 15 ? upscale<2, true>(rows, rs, out, pitch, w, step, init, max_x, maxv, have)
                 : upscale<2, false>(rows, rs, out, pitch, w, step, init, max_x, maxv, have);
    else
      have == 15 ? upscale<1, true>(rows, rs, out, pitch, w, step, init, max_x, maxv, have)
                 : upscale<1, false>(rows, rs, out, pitch, w, step, init, max_x, maxv, have);
    __syncthreads();  // the rows are free for the next item
  }
  AV1PF_TRACE_END(5);
}

cudaError_t superres_init() {
  const int bytes = kRows * sr_stride(kMaxRow) * 2;
  cudaError_t e = cudaFuncSetAttribute(superres_kernel<NoFrame>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(superres_kernel<OneFrame>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  return e;
}

void launch_superres(const FrameSet& frames, const Item* items, int n_items, int row_max, cudaStream_t s) {
  if (n_items <= 0) return;
  const int rs = sr_stride(min(max(row_max, 8), kMaxRow));
  launch_frames(frames, superres_kernel<NoFrame>, superres_kernel<OneFrame>, min(n_items, kItemGrid), 256,
                size_t(kRows * rs * 2), s, items, n_items, rs);
}

}  // namespace av1pf

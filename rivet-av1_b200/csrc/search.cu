// search.cu — the greedy choice of the encoder's CDEF search on the device:
// strength pairs (encoder/cdef.rs:195-250) over the error tables that
// cdef_search_packed_kernel (cdef_packed.cu; up to 10 bits) and
// cdef_search_kernel (cdef.cu; 12 bits) fill, and those tables turned for the
// caller.
//
// The reference sums block errors into an f64 in block order
// (`total += best as f64`). Every block error is an integer far below 2^53,
// so while a total stays below 2^53 each of those additions is exact and the
// f64 total equals the exact integer sum: the kernels sum in u64 (in any
// order) and convert. A total at or above 2^53 (frames of more than ~45,000
// 64x64 blocks at 12 bits) is summed again in f64, in block order, as the
// reference does. The cost of a choice, t + lambda * bits * nb, is evaluated
// with round-to-nearest multiplies and adds in the reference's order (no
// fused multiply-add).
#include <cooperative_groups.h>

#include <cfloat>
#include <utility>

#include "common.cuh"
#include "kernels.h"

namespace av1pf {

namespace {

constexpr uint64_t kExact = uint64_t(1) << 53;

__device__ __forceinline__ uint64_t warp_sum_u64(uint64_t v) {
#pragma unroll
  for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// The reference's f64 total, in block order, of min(best[b], last pair,
// pair (Y, U)) over the blocks (blocks that code no index hold 0 everywhere
// and add nothing). L / Y may be null (no last pair / no candidate).
__device__ double ordered_total(const uint64_t* best, const uint64_t* YL, const uint64_t* UL, const uint64_t* Y,
                                const uint64_t* U, int nfb) {
  double t = 0.0;
  for (int b = 0; b < nfb; b++) {
    uint64_t v = __ldcg(&best[b]);
    if (YL) v = min(v, YL[b] + UL[b]);
    if (Y) v = min(v, Y[b] + U[b]);
    t = __dadd_rn(t, double(v));
  }
  return t;
}

// (total, candidate) of the smaller, the first candidate on equal totals;
// candidate -1 is none.
__device__ __forceinline__ void argmin_pair(double& t, int& c, double t2, int c2) {
  if (c2 >= 0 && (c < 0 || t2 < t || (t2 == t && c2 < c))) {
    t = t2;
    c = c2;
  }
}

// Step k of the greedy (encoder/cdef.rs:215-232). A warp per candidate pair
// scores sum_b min(best[b], last[b], Y[yk][b] + UV[uk][b]) — the reference's
// best_for(set + pair): best[b] holds the minimum over the set but for its
// newest pair `last`, which every scorer folds in (and CTA 0 writes back;
// the min is idempotent, so readers that see either value agree). Lanes
// stride over the blocks (candidate-major table: coalesced, four blocks in
// flight per lane). The last CTA to finish (a fenced arrival count; no CTA
// waits) takes the smallest total, first in (yk, uk) order on ties, and adds
// its pair to the set. Its total is the new set's total, so at set sizes 1,
// 2, 4 and 8 it prices the set from it (encoder/cdef.rs:233-239). The
// candidate lists hold at least 420 pairs, so a pair always remains.
// Launched with programmatic dependent launch: the state is read after
// pdl_wait(). A batch of frames runs side by side: `cpf` CTAs per frame,
// each frame with its own state and arrival count.
__global__ void __launch_bounds__(256) cdef_greedy_step_kernel(const CdefSearchDesc* __restrict__ ds, int cpf) {
  const int fi = blockIdx.x / cpf, lb = blockIdx.x - fi * cpf;
  const CdefSearchDesc& d = ds[fi];
  CdefGreedy* g = d.g;
  uint64_t* tot = d.tot;
  const double lambda = d.lambda;
  const int nfb = d.fb_rows * d.fb_cols, ncand = d.ny * d.nuv;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  pdl_wait();
  const int n = g->n;
  const uint64_t* YL = n ? d.sse + int64_t(g->set_y[n - 1]) * nfb : nullptr;
  const uint64_t* UL = n ? d.sse + int64_t(d.ny + g->set_uv[n - 1]) * nfb : nullptr;
  if (n && lb == 0)
    for (int b = tid; b < nfb; b += blockDim.x) d.best[b] = min(d.best[b], YL[b] + UL[b]);
  const int c = lb * 8 + warp;
  if (c < ncand) {
    const int yk = c / d.nuv, uk = c - yk * d.nuv;
    bool in_set = false;
    for (int i = 0; i < n; i++) in_set |= g->set_y[i] == yk && g->set_uv[i] == uk;
    uint64_t acc = 0;
    if (!in_set) {
      const uint64_t* Y = d.sse + int64_t(yk) * nfb;
      const uint64_t* U = d.sse + int64_t(d.ny + uk) * nfb;
      const uint64_t* B = d.best;
      uint64_t a1 = 0, a2 = 0, a3 = 0;
      int b = lane;
      if (n) {
        for (; b + 96 < nfb; b += 128) {
          acc += min(min(B[b], YL[b] + UL[b]), Y[b] + U[b]);
          a1 += min(min(B[b + 32], YL[b + 32] + UL[b + 32]), Y[b + 32] + U[b + 32]);
          a2 += min(min(B[b + 64], YL[b + 64] + UL[b + 64]), Y[b + 64] + U[b + 64]);
          a3 += min(min(B[b + 96], YL[b + 96] + UL[b + 96]), Y[b + 96] + U[b + 96]);
        }
        for (; b < nfb; b += 32) acc += min(min(B[b], YL[b] + UL[b]), Y[b] + U[b]);
      } else {
        for (; b + 96 < nfb; b += 128) {
          acc += min(B[b], Y[b] + U[b]);
          a1 += min(B[b + 32], Y[b + 32] + U[b + 32]);
          a2 += min(B[b + 64], Y[b + 64] + U[b + 64]);
          a3 += min(B[b + 96], Y[b + 96] + U[b + 96]);
        }
        for (; b < nfb; b += 32) acc += min(B[b], Y[b] + U[b]);
      }
      acc = warp_sum_u64(acc + a1 + a2 + a3);
    }
    if (lane == 0) tot[c] = in_set ? ~uint64_t(0) : acc;
  }
  __shared__ bool s_last;
  __syncthreads();
  if (tid == 0) {
    __threadfence();
    s_last = atomicAdd(&g->arrived, 1u) == unsigned(cpf) - 1;
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  // --- argmin over (total, candidate): per thread, per warp, then all ---
  __shared__ double s_t[8];
  __shared__ int s_c[8];
  double bt = DBL_MAX;
  int bc = -1;
  for (int k = tid; k < ncand; k += blockDim.x) {
    const uint64_t u = __ldcg(&tot[k]);
    if (u == ~uint64_t(0)) continue;  // in the set
    const double t = u < kExact ? double(u)
                                 : ordered_total(d.best, YL, UL, d.sse + int64_t(k / d.nuv) * nfb,
                                                 d.sse + int64_t(d.ny + k % d.nuv) * nfb, nfb);
    argmin_pair(bt, bc, t, k);
  }
#pragma unroll
  for (int o = 16; o; o >>= 1) {
    const double t2 = __shfl_xor_sync(0xffffffffu, bt, o);
    const int c2 = __shfl_xor_sync(0xffffffffu, bc, o);
    argmin_pair(bt, bc, t2, c2);
  }
  if (lane == 0) {
    s_t[warp] = bt;
    s_c[warp] = bc;
  }
  __syncthreads();
  if (tid != 0) return;
  bt = s_t[0];
  bc = s_c[0];
  for (int w = 1; w < 8; w++) argmin_pair(bt, bc, s_t[w], s_c[w]);
  g->set_y[n] = bc / d.nuv;
  g->set_uv[n] = bc % d.nuv;
  g->n = n + 1;
  g->arrived = 0;
  const int size = n + 1;
  if ((size & (size - 1)) != 0) return;  // not a power of two: the level is not complete
  const int bits = __ffs(size) - 1;
  const double pen = __dmul_rn(__dmul_rn(lambda, double(bits)), double(g->nb));
  const double cost = __dadd_rn(bt, pen);
  const double prev = bits == 0 ? DBL_MAX : g->best_cost;
  if (cost < prev) {
    g->best_cost = cost;
    g->best_bits = bits;
  } else if (bits == 0) {
    g->best_cost = DBL_MAX;
  }
}

// All of the greedy in one kernel: a cluster of 8 CTAs per frame, an eighth of
// the pairs a CTA. A CTA holds the errors its pairs need (all chroma candidates'
// rows, and those of its few luma candidates) and best[] in shared memory, in 32
// bits; a step's scores are sums over them, a warp a pair, four blocks a lane and
// load. Every CTA's best pair goes to all eight by distributed shared memory, and
// one cluster barrier later each knows the pair chosen and folds it into its own
// copy of best[]. Then the outcome, as cdef_greedy_finish_kernel. Frames whose
// errors are too large for a lane's 32-bit sum score from the table in global
// memory, in 64 bits. No total reaches 2^53: a block's error is below
// 3 * 4096 * 4095^2, and there are at most kClusterBlocks.
//
// What bounds it: the latency of eight dependent steps. As eight kernels a step
// took 9 us (its launch, the descriptors, the errors' loads from L2, the arrival
// count), 72 us in all for 1080p with the fast lists; now 45 us, half of a step
// its barriers.
constexpr int kClusterCtas = 8, kClusterThreads = 1024, kClusterBlocks = 4096;
constexpr size_t kClusterSmem = 220 * 1024;
__host__ __device__ constexpr int cluster_pairs(int ncand) { return (ncand + kClusterCtas - 1) / kClusterCtas; }
// luma rows of a CTA's run of pairs, at most; blocks rounded up to a lane's four
__host__ __device__ constexpr int cluster_rows(int ncand, int nuv) { return (cluster_pairs(ncand) + nuv - 2) / nuv + 1; }
__host__ __device__ constexpr int cluster_pitch(int nfb) { return (nfb + 127) / 128 * 128; }
size_t cluster_bytes(int ncand, int nuv, int nfb) {
  return size_t(cluster_pitch(nfb)) * (8 + 4 + 4 * size_t(cluster_rows(ncand, nuv) + nuv));
}

__global__ void __launch_bounds__(kClusterThreads) cdef_greedy_cluster_kernel(const CdefSearchDesc* __restrict__ ds) {
  namespace cg = cooperative_groups;
  const cg::cluster_group cluster = cg::this_cluster();
  extern __shared__ __align__(16) uint8_t greedy_smem[];
  constexpr int kWarps = kClusterThreads / 32;
  __shared__ double s_t[kWarps];
  __shared__ int s_c[kWarps];
  __shared__ double x_t[2][kClusterCtas];  // every CTA's best, this step's and the other's
  __shared__ int x_c[2][kClusterCtas];
  const int rank = int(cluster.block_rank());
  const CdefSearchDesc& d = ds[blockIdx.x / kClusterCtas];
  const int nfb = d.fb_rows * d.fb_cols, nuv = d.nuv, ncand = d.ny * nuv;
  const int cpc = cluster_pairs(ncand), c0 = rank * cpc, nc = max(min(cpc, ncand - c0), 0);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int pitch = cluster_pitch(nfb), y_first = c0 / nuv, ny = nc ? (c0 + nc - 1) / nuv - y_first + 1 : 0;
  uint64_t* const best = reinterpret_cast<uint64_t*>(greedy_smem);
  uint32_t* const best32 = reinterpret_cast<uint32_t*>(best + pitch);
  uint32_t* const rows = best32 + pitch;  // the chroma rows, then the luma rows from y_first
  const uint64_t* const sse = d.sse;
  // The first store to a peer's shared memory must find the peer started: every
  // CTA arrives here and waits before its first step, the staging in between.
  cg::cluster_group::arrival_token started = cluster.barrier_arrive();
  pdl_wait();
  bool large = false;  // some error too large for a lane's sum of pitch / 32 pairs of them
  const uint64_t limit = (uint64_t(1) << 31) / unsigned(pitch / 32);
  for (int b = tid; b < pitch; b += kClusterThreads) {
    const uint64_t v = b < nfb ? d.best[b] : 0;
    best[b] = v;
    best32[b] = uint32_t(min(v, uint64_t(0xffffffffu)));
  }
  for (int r = warp; r < nuv + ny; r += kWarps) {
    const uint64_t* from = sse + int64_t(r < nuv ? d.ny + r : y_first + r - nuv) * nfb;
    for (int b = lane; b < pitch; b += 32) {
      const uint64_t v = b < nfb ? from[b] : 0;
      large |= v >= limit;
      rows[r * pitch + b] = uint32_t(v);
    }
  }
  large = __syncthreads_or(large);
  cluster.barrier_wait(std::move(started));
  const double nb = double(d.g->nb), lambda = d.lambda;
  int set[8];  // the pairs chosen
  int best_bits = 0;
  double best_cost = DBL_MAX;
#pragma unroll
  for (int n = 0; n < 8; n++) {
    double bt = DBL_MAX;
    int bc = -1;
    int yk = (c0 + warp) / nuv, uk = c0 + warp - yk * nuv;
    for (int k = warp; k < nc; k += kWarps, uk += kWarps) {
      while (uk >= nuv) {
        uk -= nuv;
        yk++;
      }
      const int c = c0 + k;
      bool in_set = false;
#pragma unroll
      for (int i = 0; i < n; i++) in_set |= set[i] == c;
      if (in_set) continue;
      uint64_t total;
      if (!large) {
        const uint4* Y = reinterpret_cast<const uint4*>(rows + (nuv + yk - y_first) * pitch) + lane;
        const uint4* U = reinterpret_cast<const uint4*>(rows + uk * pitch) + lane;
        const uint4* B = reinterpret_cast<const uint4*>(best32) + lane;
        uint32_t a0 = 0, a1 = 0;
        for (int q = 0; q < pitch / 4; q += 32) {
          const uint4 y = Y[q], u = U[q], m = B[q];
          a0 += min(m.x, y.x + u.x) + min(m.y, y.y + u.y);
          a1 += min(m.z, y.z + u.z) + min(m.w, y.w + u.w);
        }
        const uint32_t acc = a0 + a1;
        total = (uint64_t(__reduce_add_sync(0xffffffffu, acc >> 16)) << 16) + __reduce_add_sync(0xffffffffu, acc & 0xffffu);
      } else {
        const uint64_t* Y = sse + int64_t(yk) * nfb;
        const uint64_t* U = sse + int64_t(d.ny + uk) * nfb;
        uint64_t acc = 0;
        for (int b = lane; b < nfb; b += 32) acc += min(best[b], Y[b] + U[b]);
        total = warp_sum_u64(acc);
      }
      argmin_pair(bt, bc, double(total), c);
    }
    if (lane == 0) {
      s_t[warp] = bt;
      s_c[warp] = bc;
    }
    __syncthreads();
    // (total, pair) of the least over lanes 0 .. m - 1, in all of them
    auto least = [&](int m) {
      for (int o = m / 2; o; o >>= 1) {
        const double t2 = __shfl_xor_sync(0xffffffffu, bt, o);
        const int c2 = __shfl_xor_sync(0xffffffffu, bc, o);
        argmin_pair(bt, bc, t2, c2);
      }
    };
    if (warp == 0) {
      bt = s_t[lane % kWarps];
      bc = s_c[lane % kWarps];
      least(kWarps);
      if (lane < kClusterCtas) {
        *cluster.map_shared_rank(&x_t[n & 1][rank], lane) = bt;
        *cluster.map_shared_rank(&x_c[n & 1][rank], lane) = bc;
      }
    }
    cluster.sync();
    bt = x_t[n & 1][lane % kClusterCtas];
    bc = x_c[n & 1][lane % kClusterCtas];
    least(kClusterCtas);
    set[n] = bc;
    const int size = n + 1;
    if ((size & (size - 1)) == 0) {  // the cost of 1, 2, 4 and 8 pairs (encoder/cdef.rs:233-239)
      const int bits = size == 1 ? 0 : size == 2 ? 1 : size == 4 ? 2 : 3;
      const double cost = __dadd_rn(bt, __dmul_rn(__dmul_rn(lambda, double(bits)), nb));
      if (cost < best_cost) {
        best_cost = cost;
        best_bits = bits;
      }
    }
    {
      const uint64_t* Y = sse + int64_t(bc / nuv) * nfb;
      const uint64_t* U = sse + int64_t(d.ny + bc % nuv) * nfb;
      for (int b = tid; b < nfb; b += kClusterThreads) {
        const uint64_t v = min(best[b], Y[b] + U[b]);
        best[b] = v;
        best32[b] = uint32_t(min(v, uint64_t(0xffffffffu)));
      }
      __syncthreads();
    }
  }
  const int m = 1 << best_bits;
  if (rank == 0 && tid == 0) {
    d.res[0] = int32_t(d.g->nb);
    d.res[1] = best_bits;
#pragma unroll
    for (int i = 0; i < 8; i++) {
      d.res[2 + i] = i < m ? set[i] / nuv : 0;
      d.res[10 + i] = i < m ? set[i] % nuv : 0;
    }
  }
  // --- each coding block's index (encoder/cdef.rs:241-250) ---
  const int stride = d.cdef_stride;
  for (int e = rank * kClusterThreads + tid; e < d.fb_rows * stride; e += kClusterCtas * kClusterThreads) {
    const int r = e / stride, c = e - r * stride;
    int8_t v = d.cdef_idx[e];
    if (c < d.fb_cols && v >= 0) {
      const int b = r * d.fb_cols + c;
      uint64_t least = ~uint64_t(0);
      int pick = 0;
#pragma unroll
      for (int i = 0; i < 8; i++) {
        if (i >= m) continue;
        const uint64_t x = sse[int64_t(set[i] / nuv) * nfb + b] + sse[int64_t(d.ny + set[i] % nuv) * nfb + b];
        if (x < least) {
          least = x;
          pick = i;
        }
      }
      v = int8_t(pick);
    }
    d.table[e] = v;
  }
  cluster.sync();  // no CTA leaves while another may still write to it
}

// The error table block-major, as the caller has it: [block][candidate] from
// [candidate][block], 32 x 32 at a time. Frame blockIdx.z.
__global__ void __launch_bounds__(256) sse_transpose_kernel(const CdefSearchDesc* __restrict__ ds) {
  __shared__ uint64_t tile[32][33];
  const CdefSearchDesc& d = ds[blockIdx.z];
  if (!d.sse_out) return;
  const int nfb = d.fb_rows * d.fb_cols, nc = d.ny + d.nuv;
  const int b0 = blockIdx.x * 32, k0 = blockIdx.y * 32, x = threadIdx.x & 31, y = threadIdx.x >> 5;
  for (int r = y; r < 32; r += 8)
    if (k0 + r < nc && b0 + x < nfb) tile[r][x] = d.sse[int64_t(k0 + r) * nfb + b0 + x];
  __syncthreads();
  for (int r = y; r < 32; r += 8)
    if (b0 + r < nfb && k0 + x < nc) d.sse_out[int64_t(b0 + r) * nc + k0 + x] = tile[x][r];
}

// The outcome (encoder/cdef.rs:241-250): each coding block's index is the
// first of the chosen 1 << best_bits pairs with its least error; the other
// table entries are copied.
__global__ void cdef_greedy_finish_kernel(const CdefSearchDesc* __restrict__ ds, int n, int total) {
  const int eg = blockIdx.x * blockDim.x + threadIdx.x;
  pdl_wait();
  if (eg >= total) return;
  int fi = 0;
  for (int hi = n - 1; fi < hi;) {  // the last frame whose table starts at or before eg
    const int mid = (fi + hi + 1) >> 1;
    if (ds[mid].table0 <= eg)
      fi = mid;
    else
      hi = mid - 1;
  }
  const CdefSearchDesc& d = ds[fi];
  const CdefGreedy* g = d.g;
  const int nfb = d.fb_rows * d.fb_cols, stride = d.cdef_stride;
  const int m = 1 << g->best_bits;
  const int e = eg - d.table0;
  if (e == 0) {
    d.res[0] = int32_t(g->nb);
    d.res[1] = g->best_bits;
    for (int i = 0; i < 8; i++) {
      d.res[2 + i] = i < m ? g->set_y[i] : 0;
      d.res[10 + i] = i < m ? g->set_uv[i] : 0;
    }
  }
  const int r = e / stride, c = e - r * stride;
  int8_t v = d.cdef_idx[e];
  if (c < d.fb_cols && v >= 0) {
    const int b = r * d.fb_cols + c;
    uint64_t best = ~uint64_t(0);
    int pick = 0;
    for (int i = 0; i < m; i++) {
      const uint64_t x = d.sse[int64_t(g->set_y[i]) * nfb + b] + d.sse[int64_t(d.ny + g->set_uv[i]) * nfb + b];
      if (x < best) {
        best = x;
        pick = i;
      }
    }
    v = int8_t(pick);
  }
  d.table[e] = v;
}

}  // namespace

cudaError_t search_init() {
  return cudaFuncSetAttribute(cdef_greedy_cluster_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kClusterSmem));
}

void launch_cdef_greedy(const CdefSearchDesc* ds, int n, int ny, int nuv, int nfb_max, int entries, cudaStream_t s) {
  const int ncand = ny * nuv;
  const size_t bytes = cluster_bytes(ncand, nuv, nfb_max);
  if (bytes <= kClusterSmem && nfb_max <= kClusterBlocks) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(unsigned(n * kClusterCtas));
    cfg.blockDim = dim3(kClusterThreads);
    cfg.dynamicSmemBytes = bytes;
    cfg.stream = s;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = kClusterCtas;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    cudaLaunchKernelEx(&cfg, cdef_greedy_cluster_kernel, ds);
    note_launch();
    return;
  }
  // larger tables: a kernel a step
  const int cpf = (ncand + 7) / 8;
  for (int step = 0; step < 8; step++) launch_pdl(cdef_greedy_step_kernel, n * cpf, 256, 0, s, ds, cpf);
  launch_pdl(cdef_greedy_finish_kernel, (entries + 255) / 256, 256, 0, s, ds, n, entries);
}

void launch_sse_transpose(const CdefSearchDesc* ds, int n, int nfb_max, int nc, cudaStream_t s) {
  sse_transpose_kernel<<<dim3(unsigned((nfb_max + 31) / 32), unsigned((nc + 31) / 32), unsigned(n)), 256, 0, s>>>(ds);
  note_launch();
}

}  // namespace av1pf

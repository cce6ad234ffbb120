// kernels.h — host-side launchers of the stage kernels (internal interface
// between the C ABI implementation and the .cu files).
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "av1pf.h"
#include "desc.h"

namespace av1pf {

struct Item;
struct CdefSearchDesc;
struct CdefGreedy;
struct LrSearchDesc;

// Grid cap of the grid-stride stage kernels: 8 resident CTAs on each of the
// B200's 148 SMs.
constexpr int kNumSMs = 148;
constexpr int kMaxGrid = kNumSMs * 8;
// Grid cap of the item kernels, which launch one CTA per item: the block
// scheduler then hands items of uneven cost to SMs as slots free up.
constexpr int kItemGrid = 1 << 20;

// Counts every kernel launch this library issues (av1pf_launch_count).
void note_launch(uint64_t n = 1);

// Launches a stage kernel with programmatic stream serialization: it may be
// scheduled while the previous kernel on `s` drains (the kernel waits for
// it in pdl_wait() before reading its output). Counts the launch.
template <typename... KArgs, typename... Args>
inline void launch_pdl(void (*kernel)(KArgs...), int grid, int block, size_t smem, cudaStream_t s, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(unsigned(grid));
  cfg.blockDim = dim3(unsigned(block));
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
  note_launch();
}

// The frames of a launch, as the stage kernels' first two parameters:
// descriptors in device memory (after a NoFrame), or the descriptor of a
// launch's only frame in the parameter itself (OneFrame, and null). A
// parameter lives in the constant bank and travels with the launch: a single
// call uploads nothing, its host thread waits for nothing, and the kernels
// read the fields without the two dependent global loads (item, then
// descriptor) that began every CTA.
struct NoFrame {};
struct OneFrame {
  FrameDesc d;
};
static_assert(sizeof(OneFrame) <= 3584, "fits the 4 KB of kernel parameters with the others");
#ifdef __CUDACC__
__device__ __forceinline__ const FrameDesc& frame_of(const NoFrame&, const FrameDesc* p, int i) { return p[i]; }
__device__ __forceinline__ const FrameDesc& frame_of(const OneFrame& f, const FrameDesc*, int) { return f.d; }
#endif

// What the launchers take: `one` (host memory) when not null, else `dev`.
struct FrameSet {
  const FrameDesc* dev = nullptr;
  const FrameDesc* one = nullptr;
};
// How a call's kernels wait for one another, and for the calls before it,
// short of whole grids. A flag is set once it holds the call's epoch or a later
// value, so calls with rising epochs share flags without clearing them. The
// default is none of it: each kernel waits for the whole kernel before it.
//
// p: the readiness flags between the stages (FrameDesc::lf_flag_base ...), or
// null.
//
// complete: a word that holds the epoch of the last call known to be complete,
// or null. A call's first kernel raises it to epoch - 1 from one thread that
// waits for the kernel before it on the stream, the previous call's last; the
// kernels that must not write before an earlier call is done wait for the word
// instead of for that kernel. Calls of small frames (`ahead`) run on two
// scratches in turn: their loop filter and film-grain templates wait for the
// call before the previous one (lf_wait = epoch - 2), their kernels let the
// next launch as they start, and loop restoration, which writes the caller's
// planes, waits for the previous call.
//
// whole: the fused loop filter waits for the kernel before it ahead of reading
// its inputs (which may be what that kernel, or a call before it, writes);
// otherwise it reads them at once and waits only before it writes.
//
// grain: set to the epoch by the film-grain template kernel, which then runs
// first on the call's own stream, one CTA beside the chain (so it has started
// before the output kernel can wait for it), or null: it runs on another
// stream, joined by an event.
struct SyncFlags {
  uint32_t* p = nullptr;
  uint32_t epoch = 1;
  uint32_t* complete = nullptr;
  uint32_t lf_wait = 0;  // the loop filter waits for this in `complete` before it writes; 0: for the previous kernel
  bool ahead = false;
  bool whole = false;
  uint32_t* grain = nullptr;
};

template <typename... PArgs, typename... OArgs, typename... Args>
inline void launch_frames(const FrameSet& fs, void (*by_ptr)(NoFrame, PArgs...), void (*by_value)(OneFrame, OArgs...),
                          int grid, int block, size_t smem, cudaStream_t s, Args... args) {
  if (fs.one)
    launch_pdl(by_value, grid, block, smem, s, OneFrame{*fs.one}, static_cast<const FrameDesc*>(nullptr), args...);
  else
    launch_pdl(by_ptr, grid, block, smem, s, NoFrame{}, fs.dev, args...);
}

// Loop filter (lf.cu)
void launch_lf_prep(const FrameDesc* frames, const Item* items, int n_items, uint64_t* list_v, uint64_t* list_h,
                    uint32_t* counts, uint32_t cap, cudaStream_t s);
// Vertical edges filtered per 64x64 tile in shared memory (copy in -> cur
// included); horizontal decisions appended to list_h when item kind bit 2.
void launch_lf_tiles(const FrameDesc* frames, const Item* items, int n_items, uint64_t* list_h, uint32_t* counts,
                     uint32_t cap, cudaStream_t s);
// Both directions per 64x64 tile in shared memory (copy in -> cur included).
// `flags`: the readiness flags the kernel sets (see FrameDesc).
void launch_lf_fused(const FrameSet& frames, const Item* items, int n_items, SyncFlags flags, cudaStream_t s);
void launch_lf_edges(int pass, const FrameDesc* frames, const uint64_t* list, const uint32_t* count, uint32_t cap,
                     cudaStream_t s);
void launch_dsp_lf(int32_t* edges, const av1pf_lf_edge_params* prm, int n, cudaStream_t s);

// CDEF (cdef.cu)
// What a launch's frames are, as far as the choice of kernel and its shared
// memory go.
struct CdefShape {
  bool lfh = false;      // some item has the horizontal loop-filter pass fused (item kind 1)
  bool half = false;     // the items are half superblocks (Item::a = 0 top, 1 bottom)
  bool shallow = false;  // some frame has at most 10 bits
  bool deep = false;     // some frame has 12 bits
  bool tall = false;     // some frame's chroma is not vertically subsampled
};
// `flags`: the readiness flags the kernel waits for and sets (null for a launch
// with both shallow and deep frames, or with the fused horizontal pass; the
// latter needs the descriptors in device memory).
void launch_cdef(const FrameSet& frames, const Item* items, int n_items, const CdefShape& c, SyncFlags flags,
                 cudaStream_t s);
// The part of it for launches without the fused horizontal pass (cdef_packed.cu).
void launch_cdef_packed(const FrameSet& frames, const Item* items, int n_items, const CdefShape& c, SyncFlags flags,
                        cudaStream_t s);
cudaError_t cdef_packed_init();
// Sets cdef_kernel's dynamic shared-memory limit on the current device.
cudaError_t cdef_init();
void launch_dsp_cdef(const int32_t* win, const av1pf_cdef_taps* taps, uint16_t* res, int n, cudaStream_t s);
// The encoder's CDEF search: per-block squared errors of every candidate
// (one CTA per 64x64 block of n frames, `blocks` in all); counts each
// frame's coding blocks into its greedy state.
// `shallow`: some frame has at most 10 bits; `deep`: some has 12.
void launch_cdef_search(const CdefSearchDesc* ds, int n, int blocks, bool thorough, bool shallow, bool deep,
                        cudaStream_t s);
// The part of it for frames of up to 10 bits (cdef_packed.cu).
void launch_cdef_search_packed(const CdefSearchDesc* ds, int n, int blocks, bool thorough, cudaStream_t s);

// Encoder searches (search.cu)
// The greedy choice of the CDEF search for n frames side by side (ny x nuv pairs,
// at most nfb_max blocks a frame), and its outcome: each coding block's index into
// each frame's table (a copy of its cdef_idx; `entries` over all frames) and the
// chosen pairs into its result.
void launch_cdef_greedy(const CdefSearchDesc* ds, int n, int ny, int nuv, int nfb_max, int entries, cudaStream_t s);
// The error tables of the frames that ask for them (sse_out), block-major.
void launch_sse_transpose(const CdefSearchDesc* ds, int n, int nfb_max, int nc, cudaStream_t s);
// Sets the cluster kernel's dynamic shared-memory limit on the current device.
cudaError_t search_init();
// The loop-filter level search (lf.cu): the errors of every (frame, scale,
// plane), added to each frame's sse. `tiles`: 64x64 tiles over all frames.
void launch_lf_search(const LfSearchDesc* ds, int n, int tiles, cudaStream_t s);
// The loop-restoration search (lr_search.cu): per unit job, the no-filter
// error and the Wiener passes on `s`, the self-guided fits (one CTA per job
// and d.spc sets) on `side` beside them, then the choice.
// Raises the kernels' dynamic shared-memory limits to the device's maximum
// (the same value on every call) on the current device.
cudaError_t lr_search_init();
void launch_lr_search(const LrSearchDesc& d, int njobs, cudaStream_t s, cudaStream_t side, cudaEvent_t fork,
                      cudaEvent_t join);

// Super-resolution (superres.cu)
// `row_max`: the most source samples in a row among the launch's frames.
void launch_superres(const FrameSet& frames, const Item* items, int n_items, int row_max, cudaStream_t s);
// Sets superres_kernel's dynamic shared-memory limit on the current device.
cudaError_t superres_init();

// Loop restoration (lr.cu)
// `flags`: the readiness flags the kernel waits for.
void launch_lr(const FrameSet& frames, const Item* items, int n_items, SyncFlags flags, cudaStream_t s);
// Opts the output kernel into its dynamic shared memory (once per device).
cudaError_t output_init();

// Film grain + output packing (grain.cu)
void launch_grain_prep(const FrameSet& frames, const Item* items, int n_items, const SyncFlags& sync, cudaStream_t s);
void launch_output(const FrameSet& frames, const Item* items, int n_items, const SyncFlags& sync, cudaStream_t s);
// Uploads the LFSR jump-ahead tables (once per device).
cudaError_t upload_grain_tables();

// Device error flags (g_error_flags): read and clear. This bit of them
// means a kernel's bounded wait gave up (ERRF_STALL in common.cuh).
constexpr uint32_t kErrfStall = 4u;
cudaError_t read_error_flags(uint32_t* flags, cudaStream_t s);

}  // namespace av1pf

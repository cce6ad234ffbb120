"""The post-filter work a user of this framework has it do, as measurable cases.

Every case goes through the public C ABI (include/av1pf.h, by its ctypes
bindings): whole filter chains on device planes, batches, host-buffer calls,
the serving loop, and the encoder's filter searches. Inputs are the seeded
synthetic frames of synth/synth.h: a smooth field with steps on the transform
grid and noise, random partitions and transform trees, loop-filter levels,
CDEF presets, restoration units and film grain over the ranges the format
allows.

All outputs are samples, packed bytes, table entries and integer error sums,
so they are compared as they are; no case has floating-point outputs.
"""
import ctypes as C
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "rivet-av1_b200"))

import av1pf as A  # noqa: E402

# A frame's shape and tools; each case states what differs from this.
FRAME = dict(width=1920, height=1080, bit_depth=10, sample_bytes=2, subsampling_x=1, subsampling_y=1, mono=False,
             superres_denom=8, grain=False, lr_unit_shift=0, segmentation=False, delta_lf=0, min_block_log2=2,
             moving=False)
# The resolution mix of batches and served streams: (name in a case, frame).
MIX = [("n360", dict(width=640, height=360, bit_depth=8, sample_bytes=1)),
       ("n540", dict(width=960, height=540, bit_depth=8, sample_bytes=1)),
       ("n720", dict(width=1280, height=720, bit_depth=8, sample_bytes=1)),
       ("n1080", dict(width=1920, height=1080, bit_depth=10)),
       ("n2160", dict(width=3840, height=2160, bit_depth=10, subsampling_x=0, subsampling_y=0))]
BASE_Q_IDX, CDEF_LAMBDA, LR_LAMBDA = 120, 40.0, 150.0


def listed():
    return [
        # the plain path at its smallest: one CIF 8-bit frame, launch latency
        dict(FRAME, name="chain_352x288_8bit", kind="chain", width=352, height=288, bit_depth=8, sample_bytes=1,
             moving=True),
        # SD of a ragged size with segmentation and per-block loop-filter deltas
        dict(FRAME, name="chain_853x477_8bit", kind="chain", width=853, height=477, bit_depth=8, sample_bytes=1,
             segmentation=True, delta_lf=2),
        # a decoder's ordinary HD frame: deblock, CDEF, loop restoration, packing
        dict(FRAME, name="chain_1080p_10bit", kind="chain"),
        # the same frame with film grain on output
        dict(FRAME, name="chain_1080p_10bit_grain", kind="chain", grain=True),
        # 4K delivery with every tool on
        dict(FRAME, name="chain_4k_10bit_superres_grain", kind="chain", width=3840, height=2160, superres_denom=13,
             grain=True),
        # the largest frame: 4K 12-bit 4:4:4 mastering format, every tool on
        dict(FRAME, name="chain_4k_12bit_444_superres_grain", kind="chain", width=3840, height=2160, bit_depth=12,
             subsampling_x=0, subsampling_y=0, superres_denom=10, grain=True),
        # many streams' frames in one planned batch, replayed from its graph
        dict(name="batch_mixed_16", kind="batch", n360=4, n540=4, n720=4, n1080=3, n2160=1),
        # a CPU decoder's frames from pinned host memory and back
        dict(FRAME, name="host_1080p_10bit_x8", kind="host", frames=8),
        # the serving loop: one group of device-resident requests, one a stream
        dict(name="serve_mixed_16", kind="serve", n360=4, n540=4, n720=4, n1080=3, n2160=1),
        # an encoder's three filter searches on a 1080p frame
        dict(FRAME, name="lf_search_1080p", kind="lf_search", frames=1),
        dict(FRAME, name="cdef_search_1080p", kind="cdef_search", frames=1, thorough=False),
        dict(FRAME, name="lr_search_1080p", kind="lr_search", frames=1, effort=1),
    ]


def _drawn_frame(rng, widest):
    """A frame of any shape and format between 64 samples and `widest` wide."""
    w = int(round(math.exp(rng.uniform(math.log(64), math.log(widest)))))
    h = max(32, int(round(w * 9 / 16 * rng.uniform(0.6, 1.1))))
    if rng.random() < 0.5:  # the usual even sizes
        w, h = (w + 7) & ~7, (h + 7) & ~7
    depth, sample_bytes = rng.choice([(8, 1), (8, 1), (10, 2), (10, 2), (12, 2), (8, 2)])
    ssx, ssy = rng.choice([(1, 1), (1, 1), (1, 1), (1, 0), (0, 0)])
    return dict(FRAME, width=min(w, 3840), height=min(h, 2160), bit_depth=depth, sample_bytes=sample_bytes,
                subsampling_x=ssx, subsampling_y=ssy, mono=rng.random() < 0.08,
                superres_denom=rng.choice([8, 8, 8, rng.randint(9, 16)]) if w >= 256 else 8,
                grain=rng.random() < 0.4, lr_unit_shift=rng.choice([0, 0, 1, 2]),
                segmentation=rng.random() < 0.25, delta_lf=rng.choice([0, 0, 1, 2]),
                min_block_log2=rng.choice([2, 2, 3, 4]), moving=rng.random() < 0.2)


def draw(rng):
    kind = rng.choice(["chain"] * 6 + ["batch", "host", "serve", "lf_search", "cdef_search", "lr_search"])
    if kind == "chain":
        return dict(_drawn_frame(rng, 3840), kind=kind)
    if kind in ("batch", "serve"):
        return dict(kind=kind, n360=rng.randint(1, 4), n540=rng.randint(0, 4), n720=rng.randint(0, 4),
                    n1080=rng.randint(0, 3), n2160=rng.randint(0, 1))
    c = _drawn_frame(rng, 1920)
    c["frames"] = max(1, min(8, int(1920 * 1080 / (c["width"] * c["height"])))) if rng.random() < 0.5 else 1
    if kind != "host":  # the searches look at a coded frame before superres and grain
        c.update(superres_denom=8, grain=False)
    if kind == "cdef_search":
        c["thorough"] = rng.random() < 0.3
    if kind == "lr_search":
        c["effort"] = rng.randint(0, 1)
    return dict(c, kind=kind)


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _synth(frame, seed, index):
    kw = {k: int(v) for k, v in frame.items() if k in FRAME and k not in ("grain", "moving")}
    return A.SynthHandle(**kw, enable_grain=int(frame["grain"]), seed=seed * 64 + index, frame_index=index + 1,
                         content=A.CONTENT_MOVING if frame["moving"] else A.CONTENT_FIELD)


def _host(ptr, nbytes):
    return torch.from_numpy(np.frombuffer((C.c_uint8 * nbytes).from_address(ptr), np.uint8))


class _Planes:
    """Planes over one buffer each, as an av1pf_plane[3] and as tensors of samples."""

    def __init__(self, info, buffers, dims):
        self.buffers = buffers
        self.c = (A.Plane * 3)()
        self.samples = []
        for p, (t, (w, h, stride)) in enumerate(zip(buffers, dims)):
            self.c[p].data, self.c[p].stride, self.c[p].width, self.c[p].height = t.data_ptr(), stride, w, h
            v = t if info.sample_bytes == 1 else t.view(torch.int16)
            self.samples.append(v[:h * stride].view(h, stride)[:, :w])


def _visible(info):
    """Zeroed device planes of the visible (upscaled) area."""
    dims = []
    for p in range(info.num_planes):
        sx, sy = (info.subsampling_x, info.subsampling_y) if p else (0, 0)
        w, h = (info.upscaled_width + sx) >> sx, (info.frame_height + sy) >> sy
        dims.append((w, h, (w + 63) // 64 * 64))
    return _Planes(info, [torch.zeros(s * h * info.sample_bytes, dtype=torch.uint8, device="cuda")
                          for _, h, s in dims], dims)


class _Frame:
    """One synthetic frame's planes and maps, put in place by `put` (a host byte tensor to its home)."""

    def __init__(self, sf, put):
        f = sf.f
        self.sf, self.info, self.params = sf, f.info, f.params
        n = f.info.num_planes
        self.inp = _Planes(f.info, [put(_host(f.planes[p].data, f.plane_bytes[p])) for p in range(n)],
                           [(f.planes[p].width, f.planes[p].height, f.planes[p].stride) for p in range(n)])
        self.maps = m = A.Maps()
        m.mi_stride, m.cdef_stride = f.maps.mi_stride, f.maps.cdef_stride
        self.keep = keep = [put(_host(f.maps.mi, f.mi_count * 8)), put(_host(f.maps.cdef_idx, f.cdef_count))]
        m.mi, m.cdef_idx = keep[0].data_ptr(), keep[1].data_ptr()
        for p in range(n):
            keep.append(put(_host(f.maps.lf_tx_size[p], f.tx_count[p])))
            m.lf_tx_size[p] = keep[-1].data_ptr()
            if f.lr_count[p]:
                keep.append(put(_host(f.maps.lr_units[p], f.lr_count[p] * C.sizeof(A.LrUnit))))
                m.lr_units[p] = keep[-1].data_ptr()

    def outputs(self):
        self.ref = _visible(self.info)
        self.packed = torch.zeros(A.frame_bytes(self.info), dtype=torch.uint8, device="cuda")
        return self

    def fill(self, job):
        """The fields that batch jobs, served requests and host jobs share."""
        job.info, job.params, job.maps = C.pointer(self.info), C.pointer(self.params), C.pointer(self.maps)
        job.inp = C.cast(self.inp.c, C.POINTER(A.Plane))
        job.frame_out = self.packed.data_ptr()

    def noisy(self, gen):
        """The input planes with coding noise: per 4x4 block and per sample."""
        amp = 3 << (self.info.bit_depth - 8)
        out, dims = [], []
        for p, s in enumerate(self.inp.samples):
            h, w = s.shape
            blk = torch.randint(-amp, amp + 1, ((h + 3) // 4, (w + 3) // 4), generator=gen, device="cuda")
            v = blk.repeat_interleave(4, 0).repeat_interleave(4, 1)[:h, :w] + s
            v += torch.randint(-(amp // 2), amp // 2 + 1, (h, w), generator=gen, device="cuda")
            v = v.clamp_(0, (1 << self.info.bit_depth) - 1).to(s.dtype).contiguous()
            out.append(v.view(-1).view(torch.uint8))
            dims.append((w, h, w))
        return _Planes(self.info, out, dims)


def _to_device(t):
    return t.cuda()


def _to_pinned(t):
    return torch.empty_like(t, pin_memory=True).copy_(t)


def _context():
    """The program's one context."""
    if not hasattr(_context, "p"):
        p = C.c_void_p()
        A.check(A.lib().av1pf_ctx_create(0, 0, C.byref(p)), "ctx_create")
        _context.p = p
    return _context.p


def _server():
    """The program's one server: 4 slots a stream, at most 64 frames a tick."""
    if not hasattr(_server, "p"):
        p = C.c_void_p()
        cfg = A.ServeConfig(40 << 30, 64, 2, 50, 4)
        A.check(A.lib().av1pf_serve_open(_context(), C.byref(cfg), C.byref(p)), "serve_open")
        _server.p = p
    return _server.p


class _State:
    """What a program keeps: frames, jobs and a batch or streams, closed with it."""
    batch = None
    streams = ()

    def __init__(self, kind):
        self.kind, self.ctx = kind, _context()

    def __del__(self):
        if self.batch:
            A.lib().av1pf_batch_destroy(self.batch)
        for sid in self.streams:
            A.lib().av1pf_serve_close_stream(_server(), sid)


def _frames_of(case):
    if case["kind"] in ("batch", "serve"):
        return [dict(FRAME, **f) for name, f in MIX for _ in range(case[name])]
    return [case] * case.get("frames", 1)


def prepare(case, seed):
    L, kind = A.lib(), case["kind"]
    st = _State(kind)
    put = _to_pinned if kind == "host" else _to_device
    st.frames = frames = [_Frame(_synth(f, seed, i), put) for i, f in enumerate(_frames_of(case))]
    n = len(frames)
    if kind in ("chain", "batch", "serve"):
        for f in frames:
            f.outputs()
    if kind == "batch":
        st.jobs = (A.Job * n)()
        for j, f in zip(st.jobs, frames):
            f.fill(j)
            j.ref_out = C.cast(f.ref.c, C.POINTER(A.Plane))
        st.batch = C.c_void_p()
        A.check(L.av1pf_batch_create(st.ctx, st.jobs, n, 0, C.byref(st.batch)), "batch_create")
    elif kind == "serve":
        st.jobs, st.tickets, st.streams = (A.Request * n)(), (C.c_uint64 * n)(), []
        for j, f in zip(st.jobs, frames):
            f.fill(j)
            j.device, j.ref_out = 1, C.cast(f.ref.c, C.POINTER(A.Plane))
            sid = C.c_int32()
            A.check(L.av1pf_serve_open_stream(_server(), C.byref(f.info), C.byref(sid)), "open_stream")
            st.streams.append(sid.value)
        st.ids = (C.c_int32 * n)(*st.streams)
    elif kind == "host":
        st.jobs = (A.HostJob * n)()
        for j, f in zip(st.jobs, frames):
            f.packed = torch.zeros(A.frame_bytes(f.info), dtype=torch.uint8, pin_memory=True)
            f.fill(j)
    elif kind != "chain":
        gen = torch.Generator(device="cuda").manual_seed(seed)
        st.jobs = ({"lf_search": A.LfSearchJob, "cdef_search": A.CdefSearchJob, "lr_search": A.LrSearchJob}[kind] * n)()
        for j, f in zip(st.jobs, frames):
            info, params = f.info, f.params
            j.info = C.pointer(info)
            f.cur = f.noisy(gen)
            j.cur, j.src = C.cast(f.cur.c, C.POINTER(A.Plane)), C.cast(f.inp.c, C.POINTER(A.Plane))
            if kind == "lr_search":
                f.cdef = f.noisy(gen)
                f.units = [np.zeros((params.lr_unit_rows[p] * params.lr_unit_cols[p], C.sizeof(A.LrUnit)), np.uint8)
                           for p in range(info.num_planes)]
                j.params, j.lam = C.pointer(params), LR_LAMBDA
                j.cdef = C.cast(f.cdef.c, C.POINTER(A.Plane))
                for p, u in enumerate(f.units):
                    j.units_out[p] = C.cast(u.ctypes.data, C.POINTER(A.LrUnit))
                continue
            j.maps = C.pointer(f.maps)
            if kind == "lf_search":
                f.sse = np.zeros((6, 3), np.int64)
                j.params, j.sse_out = C.pointer(params), f.sse.ctypes.data
            else:
                rows, cols = (info.mi_rows + 15) // 16, (info.mi_cols + 15) // 16
                f.table = np.zeros(rows * f.maps.cdef_stride, np.int8)
                f.sse = np.zeros((rows * cols, sum(A.CDEF_SEARCH_N[bool(case["thorough"])])), np.int64)
                f.result = A.CdefSearchResult()
                j.base_q_idx, j.lam, j.result = BASE_Q_IDX, CDEF_LAMBDA, C.pointer(f.result)
                j.cdef_idx_out, j.block_sse = f.table.ctypes.data, f.sse.ctypes.data
        st.option = int(case.get("thorough", case.get("effort", 0)))
    return st


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def run(st):
    L, kind, frames, n = A.lib(), st.kind, st.frames, len(st.frames)
    if kind == "chain":
        f = frames[0]
        A.check(L.av1pf_chain(st.ctx, C.byref(f.info), C.byref(f.params), C.byref(f.maps), f.inp.c, f.ref.c,
                              f.packed.data_ptr(), None), "chain")
    elif kind == "batch":
        A.check(L.av1pf_batch_run(st.batch, None), "batch_run")
    elif kind == "serve":
        A.check(L.av1pf_serve_submit_many(_server(), n, st.ids, st.jobs, st.tickets), "submit_many")
        for t in st.tickets:
            A.check(L.av1pf_serve_poll(_server(), t, 20000, None, None), "poll")
    elif kind == "host":
        if n > 1:
            A.check(L.av1pf_chain_host_many(st.ctx, n, st.jobs), "chain_host_many")
        else:
            f = frames[0]
            A.check(L.av1pf_chain_host(st.ctx, C.byref(f.info), C.byref(f.params), C.byref(f.maps), f.inp.c, None,
                                       f.packed.data_ptr()), "chain_host")
        return [f.packed for f in frames]
    elif kind == "lf_search":
        A.check(L.av1pf_lf_search_many(st.ctx, n, st.jobs, None), "lf_search")
        return [(np.array(j.levels_out), f.sse) for j, f in zip(st.jobs, frames)]
    elif kind == "cdef_search":
        A.check(L.av1pf_cdef_search_many(st.ctx, n, st.jobs, st.option, None), "cdef_search")
        return [(np.frombuffer(f.result, np.int32), f.table, f.sse) for f in frames]
    else:
        A.check(L.av1pf_lr_search_many(st.ctx, n, st.jobs, st.option, None), "lr_search")
        return [(np.array(j.frame_type_out), f.units) for j, f in zip(st.jobs, frames)]
    return [(f.ref.samples, f.packed) for f in frames]


# ---------------------------------------------------------------------------
# the least a pass has to move and compute
# ---------------------------------------------------------------------------
# Integer operations a sample, from the processes as the format defines them:
# deblocking about 10; CDEF 12 taps of 5 operations, the rounding, and on luma
# the direction search's 8 line sums; superres 8 multiply-adds; restoration
# 14 multiply-adds (Wiener; a self-guided unit costs more); grain a scaled add.
LF_OPS, CDEF_OPS, SUPERRES_OPS, LR_OPS, GRAIN_OPS = 10, 80, 16, 30, 6


def work(case):
    nbytes = flops = 0.0
    kind = case["kind"]
    for c in _frames_of(case):
        w, h, sb = c["width"], c["height"], c["sample_bytes"]
        coded = (w * 8 + c["superres_denom"] // 2) // c["superres_denom"]
        chroma = 0.0 if c["mono"] else 2.0 / ((1 + c["subsampling_x"]) * (1 + c["subsampling_y"]))
        s_in, s_out = coded * h * (1 + chroma), w * h * (1 + chroma)
        maps = coded * h / 16 * (8 + 1 + chroma)
        if kind in ("chain", "batch", "serve", "host"):
            packed = s_out * (2 if c["bit_depth"] > 8 else 1)
            nbytes += s_in * sb + maps + packed + (0 if kind == "host" else s_out * sb)
            flops += s_in * (LF_OPS + CDEF_OPS) + s_out * (LR_OPS + (SUPERRES_OPS if coded != w else 0)
                                                           + (GRAIN_OPS if c["grain"] else 0))
        elif kind == "lf_search":  # 5 filtered scales, 6 errors of 3 operations
            nbytes += 2 * s_in * sb + maps
            flops += s_in * (5 * LF_OPS + 18)
        elif kind == "cdef_search":  # a filtered value and its error for every candidate pair
            ny, nuv = A.CDEF_SEARCH_N[bool(case["thorough"])]
            nbytes += 2 * s_in * sb + maps
            flops += coded * h * (ny + chroma * nuv) * 10
        else:  # Wiener sums (two passes of 10 products) and a self-guided fit of about 40 a parameter set
            nbytes += 3 * s_in * sb
            flops += s_in * (60 + (80, 240, 640)[case["effort"]])
    return {"bytes": nbytes, "flops": flops}

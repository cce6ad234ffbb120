"""The readiness flags between the chain's stages, on the work lists that the
planner makes (plan_lists.cpp prints them) and the waits of the kernels that run
them (cdef_packed.cu packed_wait_lf, lr.cu lr_wait_cdef), restated below: every
flag that is waited for is set by some item; every sample that an item reads of
an earlier stage's output is covered by its waits; and every item of an earlier
stage is waited for, so that nothing of a call runs on when its last kernel is
done."""
import os
import random
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
PKG = os.path.join(os.path.dirname(HERE), "rivet-av1_b200")


@pytest.fixture(scope="module")
def lists(tmp_path_factory):
    exe = tmp_path_factory.mktemp("plan") / "plan_lists"
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", os.path.join(PKG, "..", "include"), "-I", os.path.join(PKG, "csrc"),
                    "-I", "/usr/local/cuda/include", os.path.join(HERE, "plan_lists.cpp"), "-L", PKG, "-lav1pf",
                    "-Wl,-rpath," + PKG, "-o", str(exe)], check=True)

    def run(*args):
        out = subprocess.run([str(exe), *map(str, args)], capture_output=True, text=True, check=True).stdout
        got = {"plane": [], "lf": [], "cdef": [], "lr": []}
        for line in out.splitlines():
            name, *v = line.split()
            if name == "frame":
                got[name] = [int(x) for x in v]
            else:
                got[name].append([int(x) for x in v])
        return got

    return run


def spans(lo, hi, shift):
    return range(lo >> shift, (hi >> shift) + 1) if lo <= hi else range(0)


def check(lists, W, H, sx, sy, np=3, pad=(0, 0), lr_cols=64, unit=64, mask=7):
    what = (W, H, sx, sy, np, pad, lr_cols, unit, mask)
    got = lists(W, H, sx, sy, np, *pad, lr_cols, unit, mask)
    flag_sync, n_flags, half, cdef_base, sbc = got["frame"]
    assert flag_sync
    mi_cols, mi_rows = 2 * ((W + 7) >> 3), 2 * ((H + 7) >> 3)
    ss = [(0, 0), (sx, sy), (sx, sy)][:np]
    lf_base, tiles_x = [p[1] for p in got["plane"]], [p[2] for p in got["plane"]]

    # the loop filter's items: one flag each, the mode-info area once
    lf = {}
    for p, _, x0, y0, x1, y1, _, _ in got["lf"]:
        assert x0 % 64 == 0 and y0 % 64 == 0 and x1 <= x0 + 64 and y1 <= y0 + 64
        flag = lf_base[p] + (y0 // 64) * tiles_x[p] + x0 // 64
        assert flag not in lf and flag < n_flags, what
        lf[flag] = (p, x0, y0, x1, y1)
    for p in range(np):
        area = sum((x1 - x0) * (y1 - y0) for q, x0, y0, x1, y1 in lf.values() if q == p)
        want = ((mi_cols * 4) >> ss[p][0]) * ((mi_rows * 4) >> ss[p][1])
        assert area == (want if tiles_x[p] else 0), what

    # CDEF's items: what they wait for, read and set
    R = 32 if half else 64
    cdef, lf_waited = {}, set()
    for _, _, sc, sr, _, _, a, _ in got["cdef"]:
        y0, waits = sr * 64 + a * R, [set(), set(), set()]
        for p in range(np):
            if not tiles_x[p]:
                continue
            px, py = ss[p]
            w, h = (mi_cols * 4) >> px, (mi_rows * 4) >> py
            r0, r1 = max((y0 >> py) - 2, 0), min(((y0 + R) >> py) + 1, h - 1)
            c0, c1 = max(((sc * 64) >> px) - 8, 0), min(((sc * 64 + 64) >> px) + 7, w - 1)
            ty, tx = spans(r0, r1, 6), spans(c0, c1, 6)
            assert len(ty) <= 4 and len(tx) <= 4, what
            waits[p] = {(y, x) for y in ty for x in tx}
            for y, x in waits[p]:
                flag = lf_base[p] + y * tiles_x[p] + x
                assert flag in lf and lf[flag][:3] == (p, x * 64, y * 64), what
                lf_waited.add(flag)
            # its windows: 2 rows and 8 columns around its part, in the mode-info area
            rows = spans(max((y0 >> py) - 2, 0), min((y0 >> py) + (R >> py) + 1, h - 1), 6)
            cols = spans(max(((sc * 64) >> px) - 8, 0), min(((sc * 64) >> px) + (64 >> px) + 7, w - 1), 6)
            assert {(y, x) for y in rows for x in cols} <= waits[p], what
        for part in ((0, 1) if R == 64 else (a,)):
            flag = cdef_base + 2 * sr * sbc + sc + part * sbc
            assert flag not in cdef and flag < n_flags and flag not in lf, what
            cdef[flag] = (y0, sc, waits)  # (a whole superblock sets two)
    assert lf_waited == set(lf), (what, "a loop-filter tile that no item waits for")

    # loop restoration's items
    cdef_waited, covered = set(), [set() for _ in range(np)]
    for plane, pair, x0, iy0, x1, iy1, s, _ in got["lr"]:
        for p in ((1, 2) if pair else (plane,)):
            px, py = ss[p]
            pex, pey = ((W + px) >> px) - 1, ((H + py) >> py) - 1
            top = (-8 + s * 64) >> py
            end = top + (64 >> py) - 1
            y0 = max(top, 0) + iy0
            y1 = min(end, pey, y0 + iy1 - iy0 - 1)
            assert y0 <= y1 and x0 < x1 <= pex + 1 and x1 - x0 <= 64 and y1 - y0 < (32 if x1 - x0 > 32 else 64), what
            for y in range(y0, y1 + 1):
                assert (y, x0) not in covered[p], what
                covered[p] |= {(y, x) for x in range(x0, x1)}
            xa, xb = max(x0 - 3, 0), min(x1 + 2, pex)
            ya, yb = max(y0 - 3, max(top, 0)), min(y1 + 3, min(end, pey))
            hs = range((ya << py) >> 5, (((yb << py) + py) >> 5) + 1)
            cs = range((xa << px) >> 6, min(((xb << px) + px) >> 6, sbc - 1) + 1)
            assert len(hs) <= 4 and len(cs) <= 4, what
            waits = [cdef_base + r * sbc + c for r in hs for c in cs]
            tiles = set()
            for f in waits:
                assert f in cdef, (what, "a half superblock that no item sets")
                cdef_waited.add(f)
                tiles |= cdef[f][2][p]
            # the stripe's rows come from CDEF's output, two on either side of it from the loop filter's
            for y in range(max(y0 - 3, 0), min(y1 + 3, pey) + 1):
                if top <= y <= end:
                    need = {cdef_base + ((y << py) >> 5) * sbc + ((x << px) >> 6) for x in (xa, (xa + xb) // 2, xb)}
                    assert need <= set(waits), what
                elif tiles_x[p]:
                    yy = max(top - 2, y) if y < top else min(end + 2, y)
                    assert {(yy // 64, x) for x in spans(xa, xb, 6)} <= tiles, what
    items = {(y0, sc) for y0, sc, _ in cdef.values()}
    assert {cdef[f][:2] for f in cdef_waited} == items, (what, "a CDEF item that none waits for")
    for p in range(np):
        assert len(covered[p]) == ((W + ss[p][0]) >> ss[p][0]) * ((H + ss[p][1]) >> ss[p][1]), what


@pytest.mark.parametrize("W,H", [(352, 288), (200, 136), (127, 65), (17, 9), (64, 64), (65, 65), (8, 200), (1920, 120)])
@pytest.mark.parametrize("sx,sy,np", [(1, 1, 3), (0, 0, 3), (1, 0, 3), (1, 1, 1)])
def test_flags_of_a_frame(lists, W, H, sx, sy, np):
    for pad in ((0, 0), (24, 24), (160, 100)):
        check(lists, W, H, sx, sy, np, pad)


def test_whole_superblocks(lists):
    """More than one wave of superblocks: CDEF's items are whole ones."""
    check(lists, 2600, 1100, 1, 1, 3, (24, 24))


def test_planes_without_the_loop_filter(lists):
    for mask in (1, 3, 5):
        check(lists, 200, 136, 1, 1, 3, (24, 24), mask=mask)


def test_random_shapes(lists):
    r = random.Random(11)
    for _ in range(24):
        sx, sy = r.choice(((1, 1), (0, 0), (1, 0)))
        check(lists, r.randrange(8, 500), r.randrange(8, 400), sx, sy, r.choice((1, 3)),
              (r.randrange(0, 140), r.randrange(0, 140)), r.choice((32, 64)), r.choice((32, 64, 128, 256)))

"""A CTA of a cluster may touch another's shared memory only once that CTA has
started and until it leaves: in every kernel that maps a peer's shared memory a
cluster barrier comes before the first use and after the last."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "rivet-av1_b200", "csrc")
BARRIER = r"\.sync\(\)|\.barrier_wait\(|barrier\.cluster\.wait"


def kernels(text):
    """(name, body) of every __global__ function, comments taken out."""
    text = re.sub(r"//[^\n]*", "", text)
    for m in re.finditer(r"__global__ void [^;{]*?(\w+_kernel)\(", text):
        start = text.index("{", text.index(")", m.end()))
        depth, at = 0, start
        while True:
            depth += {"{": 1, "}": -1}.get(text[at], 0)
            at += 1
            if depth == 0:
                break
        yield m.group(1), text[start:at]


def test_cluster_barriers_enclose_remote_accesses():
    seen = []
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        for name, body in kernels(open(path).read()):
            remote = [m.start() for m in re.finditer(r"map_shared_rank|mapa\.", body)]
            if not remote:
                continue
            seen.append(name)
            barriers = [m.start() for m in re.finditer(r"\bcluster(?:%s)|barrier\.cluster\.wait" % BARRIER, body)]
            assert any(b < remote[0] for b in barriers), f"{name}: a peer may not have started at the first access"
            assert any(b > remote[-1] for b in barriers), f"{name}: a peer may have left at the last access"
    assert seen == ["cdef_greedy_cluster_kernel"]

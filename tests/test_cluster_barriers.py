"""Order of cluster barriers and accesses to other CTAs' shared memory in the
sources: such an access is only defined once the accessed CTA has started and
while it has not exited, and both are shown by cluster barriers alone.  A
missing one shows in no output until a CTA starts late, so it is read from the
source."""
import pathlib
import re

import pytest

CSRC = pathlib.Path(__file__).resolve().parents[1] / "renderingengine_b200" / "csrc"
REMOTE = re.compile(r"map_shared_rank|\bmapa\b|shared::cluster")
BARRIER = re.compile(r"cluster\.sync\(\)|cluster\.barrier_wait\(|barrier\.cluster\.wait")


def _kernels(text):
    """(name, body) of the kernels of a source without its comments."""
    text = re.sub(r"//[^\n]*|/\*.*?\*/", "", text, flags=re.S)
    for m in re.finditer(r"__global__", text):
        start = text.find("{", m.end())
        if start < 0 or ";" in text[m.end():start]:
            continue
        depth, end = 0, start
        while True:
            depth += {"{": 1, "}": -1}.get(text[end], 0)
            end += 1
            if depth == 0:
                break
        yield re.findall(r"(\w+)\s*\(", text[m.end():start])[-1], text[start:end]


CLUSTER_KERNELS = [(f.name, name, body) for f in sorted(CSRC.glob("*.cu")) for name, body in _kernels(f.read_text())
                   if REMOTE.search(body)]


def test_cluster_kernels_are_found():
    assert "k_cluster_sort" in [name for _, name, _ in CLUSTER_KERNELS]


@pytest.mark.parametrize("file,name,body", CLUSTER_KERNELS, ids=[k[1] for k in CLUSTER_KERNELS])
def test_remote_shared_memory_is_fenced_by_cluster_barriers(file, name, body):
    remote = [m.start() for m in REMOTE.finditer(body)]
    barriers = [m.start() for m in BARRIER.finditer(body)]
    assert barriers and barriers[0] < remote[0], f"{file}: {name} accesses a CTA that may not have started"
    assert barriers[-1] > remote[-1], f"{file}: {name} may exit while another CTA accesses its shared memory"

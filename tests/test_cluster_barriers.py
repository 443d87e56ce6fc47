"""Kernels that use distributed shared memory: another CTA's shared memory exists once that CTA has
started and until it leaves, so a cluster barrier stands before the first access to it and after the
last one. A missing one cannot be seen by running the kernel (the time from launch to access hides
it), so the sources are read."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "nrrs-code_b200" / "csrc"
REMOTE = re.compile(r"map_shared_rank\(|\bmapa\b|shared::cluster\.[bu]")
BARRIER = re.compile(r"cluster\.(sync|barrier_wait)\(|barrier\.cluster\.wait")


def kernels():
    for path in sorted([*CSRC.glob("*.cu"), *CSRC.glob("*.cuh")]):
        text = re.sub(r"//[^\n]*", "", path.read_text())
        for m in re.finditer(r"__global__", text):
            depth, start = 0, text.index("{", m.end())
            for end in range(start, len(text)):
                depth += {"{": 1, "}": -1}.get(text[end], 0)
                if depth == 0:
                    break
            yield path.name, text[m.start():start].split("(")[-2].split()[-1], text[start:end]


def test_cluster_barriers_around_remote_shared_memory():
    found = 0
    for file, name, body in kernels():
        remote = [m.start() for m in REMOTE.finditer(body)]
        if not remote:
            continue
        found += 1
        waits = [m.start() for m in BARRIER.finditer(body)]
        assert any(w < remote[0] for w in waits), f"{file}: {name} touches a CTA that may not have started"
        assert any(w > remote[-1] for w in waits), f"{file}: {name} touches a CTA that may have left"
    assert found

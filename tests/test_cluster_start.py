"""Kernels of thread-block clusters: no block stores into another block's
shared memory before a cluster barrier says that all of them run.  Read from
the sources, since a store that comes too early seldom shows in a result."""
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "krabmaga_gb300", "csrc")

REMOTE = r"st\.(?:async\.)?(?:\w+\.)*shared::cluster|store_remote\s*\("
WAIT = r"barrier\.cluster\.wait|\bcl\.sync\s*\(\)|cluster\.sync\s*\(\)"


def kernels():
    """(file, kernel, body) of every __global__ function."""
    for fn in sorted(os.listdir(CSRC)):
        if not fn.endswith((".cu", ".cuh")):
            continue
        text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, fn)).read())
        for m in re.finditer(r"__global__", text):
            open_ = text.index("{", m.end())
            depth, end = 0, open_
            for end in range(open_, len(text)):
                depth += {"{": 1, "}": -1}.get(text[end], 0)
                if depth == 0:
                    break
            name = re.search(r"\b(k_\w+)\s*\(", text[m.end():open_])
            yield fn, name.group(1) if name else "?", text[open_:end + 1]


def test_remote_stores_follow_a_cluster_barrier():
    seen = []
    for fn, name, body in kernels():
        store = re.search(REMOTE, body)
        if not store:
            continue
        seen.append(name)
        assert re.search(WAIT, body[:store.start()]), (fn, name)
    assert {"k_scan_cluster", "k_small_steps"} <= set(seen), seen

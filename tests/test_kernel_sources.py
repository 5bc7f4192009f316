"""Rules of the CUDA sources that no run can show to be kept (a race that the timing of today hides passes every test).
Read as text, on the CPU."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(__file__), "..", "ferrum-torrens_b200", "csrc")


def _kernels():
    """(file, name, parameters, body) of every __global__ function, comments taken out."""
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        text = re.sub(r"//[^\n]*|/\*.*?\*/", "", open(path).read(), flags=re.S)
        for m in re.finditer(r"__global__[^;{]*?\b(\w+_kernel)\s*\(", text):
            depth, i = 1, m.end()
            while depth:
                depth += {"(": 1, ")": -1}.get(text[i], 0)
                i += 1
            params = text[m.end():i - 1]
            begin = i = text.index("{", i)
            depth = 0
            while True:
                depth += {"{": 1, "}": -1}.get(text[i], 0)
                i += 1
                if not depth:
                    break
            yield os.path.basename(path), m.group(1), params, text[begin:i]


def test_remote_shared_memory_is_stored_to_after_a_cluster_barrier():
    """Every CTA of a cluster must have started before another one stores into its shared memory."""
    found = 0
    for path, name, _, body in _kernels():
        if "map_shared_rank" not in body:
            continue
        found += 1
        before = body[:body.index("map_shared_rank")]
        assert "barrier.cluster.wait" in before or "cluster.sync()" in before, (path, name)
        assert "barrier.cluster.wait" not in before or "barrier.cluster.arrive" in before[:before.index("barrier.cluster.wait")], (path, name)
    assert found


def test_overlapped_kernels_promise_no_read_only_data_but_weights():
    """A kernel launched programmatically is resident while its predecessor still writes: `const .. __restrict__` on such
    data would let the compiler read it before the dependency wait.  Weights are constant all the same."""
    weights = {"gate_up", "down", "shared_gate", "gate_w"}
    launched = set()
    for path in glob.glob(os.path.join(CSRC, "*.cu")):
        launched |= set(re.findall(r"launch_pdl\(\s*(\w+_kernel)", open(path).read()))
    assert launched
    for path, name, params, body in _kernels():
        if name not in launched:
            continue
        bad = set(re.findall(r"const\s+[\w:]+\s*\*\s*__restrict__\s+(\w+)", params)) - weights
        assert not bad, (path, name, bad)
        assert "pdl_wait()" in body, (path, name)

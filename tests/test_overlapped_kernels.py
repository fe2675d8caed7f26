"""Kernels whose life overlaps that of their predecessor in the stream (launch_overlapped and the other launches
with programmatic stream serialization) may not use the read-only data path for what they read: it asks for
data that nobody writes while the kernel lives.  Read in the sources: neither __ldg nor const __restrict__
pointers, from which the compiler infers such loads."""
import glob
import os
import re


CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "portdnn_b200", "csrc")
WAITS = ("overlap_wait();", "griddepcontrol.wait", "grid_dependency_wait();")


def _sources():
    return {os.path.basename(p): re.sub(r"//[^\n]*", "", open(p).read())
            for p in sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh")))}


def _kernels(text):
    """(name, arguments, body) of every kernel defined in a source."""
    for m in re.finditer(r"__global__ void\b(?:\s*__launch_bounds__\([^{;]*?\))?\s+(\w+)\(", text):
        depth, i = 1, m.end()
        while depth:
            depth += {"(": 1, ")": -1}.get(text[i], 0)
            i += 1
        body = text[text.index("{", i):]
        yield m.group(1), text[m.end():i - 1], body[:body.index("\n}\n")]


def test_overlapped_kernels_load_coherently():
    sources, waiting = _sources(), {}
    for name, text in sources.items():
        for kernel, args, body in _kernels(text):
            if any(w in body for w in WAITS) and not re.search(kernel + r"<[^;{}]*<<<", "".join(sources.values())):
                waiting[kernel] = (name, args)
    assert len(waiting) >= 20 and "pointwise_kernel" in waiting and "batchnorm_moments_kernel" in waiting
    for kernel, (name, args) in waiting.items():
        assert not re.search(r"const [^,]*__restrict__", args), kernel
        assert "__ldg(" not in sources[name], name
    for header in ("common.cuh", "column_sums.cuh", "umma.cuh"):
        assert "__ldg(" not in sources[header], header


def test_what_launch_overlapped_launches_waits_first():
    """The wait is the first statement, ahead of every use of a pointer."""
    text = "".join(_sources().values())
    bodies = {kernel: body for _, t in _sources().items() for kernel, _, body in _kernels(t)}
    launched = set(re.findall(r"launch_overlapped\(\s*(\w+)", text)) - {"void"}
    assert len(launched) >= 20
    for kernel in launched:
        assert bodies[kernel].lstrip("{ \n").startswith("overlap_wait();"), kernel

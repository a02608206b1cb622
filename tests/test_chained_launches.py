"""Kernels that start while their predecessor still runs."""
import pathlib
import re

CSRC = pathlib.Path(__file__).resolve().parent.parent / "3deye_gb300" / "csrc"

# Read-only buffers that no chained predecessor writes: the scaled depth of a
# sweep is complete before the depth tiles, launched plainly, are formed from it.
UNCHANGED = {"integrate_bricks_kernel": {"depth"}}


def _kernels(text):
    text = re.sub(r"//[^\n]*", "", text)
    for m in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\s*\((?:[^()]|\([^()]*\))*\)\s*)?(\w+)\s*\(", text):
        depth, i = 1, m.end()
        while depth:
            depth += {"(": 1, ")": -1}.get(text[i], 0)
            i += 1
        params, j = text[m.end():i - 1], text.index("{", i) + 1
        depth, k = 1, j
        while depth:
            depth += {"{": 1, "}": -1}.get(text[k], 0)
            k += 1
        yield m.group(1), params, text[j:k]


def test_a_waiting_kernel_reads_its_predecessors_buffers_coherently():
    """The read-only path (a const __restrict__ pointer, __ldg) is for memory that
    does not change while the kernel runs.  A kernel that waits for its predecessor
    runs while that one writes, so it takes none of its buffers that way."""
    found, waiting = set(), set()
    for f in sorted(CSRC.glob("*.cu")):
        for name, params, body in _kernels(f.read_text()):
            found.add(name)
            if "wait_previous_kernel();" not in body:
                continue
            waiting.add(name)
            ro = {p.split()[-1].lstrip("*") for p in params.split(",")
                  if re.search(r"\bconst\b[^*]*\*\s*__restrict__", p)}
            ro |= set(re.findall(r"__ldg\(\s*&?([\w.]+)", body)) | set(re.findall(r"\w+_ro\b", body))
            assert ro <= UNCHANGED.get(name, set()), (name, ro)
    assert {"raycast_kernel", "integrate_bricks_kernel", "resize_map_kernel", "bilateral_kernel"} <= found
    assert {"integrate_bricks_kernel", "cull_bricks_kernel", "raycast_kernel", "resize_map_kernel"} <= waiting
    # the records that a sweep writes and a cast behind it reads, inside the functions they call
    for f in ("k_raycast.cu", "k_integrate.cu"):
        assert not re.search(r"\w+_ro\s*\(", (CSRC / f).read_text()), f

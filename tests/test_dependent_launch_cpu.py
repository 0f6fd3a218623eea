"""What a kernel that may start before its predecessor has finished must not promise, read from the sources.

``__restrict__`` and ``__ldg`` say that the data they name do not change while the kernel runs, which lets the compiler move such
loads above the wait for the predecessor and take them through a path that is not coherent with its writes.  In a kernel whose
lifetime overlaps the writes of its inputs the promise is false."""
import re
from pathlib import Path

from autoresearch_b200.ops import kernels as K

CSRC = Path(K.__file__).parent / "csrc"


def _sources():
    for f in sorted(CSRC.glob("*.cu*")):
        yield f.name, re.sub(r"//[^\n]*", "", f.read_text())


def _functions(text):
    """(name, signature, body) of every __global__ and __device__ function."""
    for m in re.finditer(r"__(?:global|device)__[^;{=]*?\b(\w+)\s*\(", text):
        if m.group(1) == "__launch_bounds__":
            m = re.compile(r"__launch_bounds__\s*\([^)]*\)\s*(\w+)\s*\(").search(text, m.start())
        brace = text.find("{", m.end())
        semi = text.find(";", m.end())
        if brace < 0 or (0 <= semi < brace):
            continue
        depth, i = 1, brace + 1
        while depth:
            depth += {"{": 1, "}": -1}.get(text[i], 0)
            i += 1
        yield m.group(1), text[m.start():brace], text[brace:i]


def test_early_started_kernels_promise_nothing_about_their_inputs():
    waits = {}
    for name, text in _sources():
        for fn, sig, body in _functions(text):
            if re.search(r"\bgrid_(enter|wait)\s*\(", body) and fn not in ("grid_enter", "grid_wait"):
                waits[name, fn] = sig
    assert len(waits) > 20, sorted(waits)
    assert not [k for k, sig in waits.items() if "__restrict__" in sig]


def test_no_read_only_loads_where_early_started_kernels_live():
    for name, text in _sources():
        if re.search(r"\bgrid_(enter|wait)\s*\(", text):
            assert not re.findall(r"__ldg\s*\(|\.nc\b", text), name


def test_no_launch_leaves_its_error_for_the_next_entry_point():
    """cudaLaunchKernelEx returns its error and leaves it as the thread's last one: every such launch goes through launch_status(), and
    no entry point asks for the last error after one."""
    for name, text in _sources():
        assert len(re.findall(r"\bcudaLaunchKernelEx\(", text)) == len(re.findall(r"\blaunch_status\(cudaLaunchKernelEx\(", text)), name
        assert not re.findall(r"[;{})]\s*launch_dependent\(", text), name            # its code is used

"""Rules of the kernels' launches that no result shows, read out of the sources (no GPU needed)."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cinnamon_b200", "csrc")
SOURCES = {os.path.basename(f): re.sub(r"//[^\n]*", "", open(f).read()) for f in sorted(glob.glob(os.path.join(CSRC, "*.cu*")))}


def test_shared_memory_limits_are_set_on_every_device():
    """A function's attributes belong to a device: set once per process, a second device's launches of the kernel are refused."""
    for name, text in SOURCES.items():
        for m in re.finditer(r"call_once", text):
            assert "cudaFuncSetAttribute" not in text[m.start():text.index("});", m.start())], name


def _kernels():
    """(file, name, body) of every kernel."""
    for file, text in SOURCES.items():
        for m in re.finditer(r"__global__[^{;]*?(\w+)\(", re.sub(r"__launch_bounds__\([^{;]*?\)\s", lambda b: " " * len(b.group()), text)):
            at = depth = text.index("{", m.end())
            i, depth = at, 0
            while True:
                depth += {"{": 1, "}": -1}.get(text[i], 0)
                if depth == 0:
                    break
                i += 1
            yield file, m.group(1), text[at:i]


def test_kernels_trigger_after_their_wait():
    """What starts behind a kernel that triggers after its wait finds everything before that kernel done; the quantisers that work
    beside the kernel ahead of them, and so before their wait, build on it and wait before they end."""
    seen = 0
    for file, name, body in _kernels():
        if "pdl_trigger()" not in body:
            continue
        seen += 1
        assert "pdl_wait()" in body[:body.index("pdl_trigger()")], (file, name)
        if "if (!beside) pdl_wait();" in body:
            assert body.rstrip().endswith("if (beside) pdl_wait();"), (file, name)
    assert seen >= 30


def test_kernels_trigger_once_they_hold_their_tensor_memory():
    """A kernel behind may allocate tensor memory before its wait: a block that triggered before it has its own could wait for a
    block that waits for its end.  The trigger comes from the warp that allocates, after the allocation."""
    seen = 0
    for file, name, body in _kernels():
        alloc = re.search(r"tc_alloc\(|tcgen05\.alloc", body)
        if alloc is None or "pdl_trigger()" not in body:
            continue
        seen += 1
        assert body.count("pdl_trigger()") == 1 and body.index("pdl_trigger()") > alloc.start(), (file, name)
        guards = list(re.finditer(r"if \(warp == ([^)]+)\)", body))
        by = [[g for g in guards if g.start() < at][-1] for at in (alloc.start(), body.index("pdl_trigger()"))]
        assert by[0].group(1) == by[1].group(1), (file, name)
        inside = body[by[1].end():body.index("pdl_trigger()")]
        assert inside.strip() == "" or (inside.strip().startswith("{") and "}" not in inside), (file, name, inside)
    assert seen >= 9

"""Programmatic dependent launches: a kernel that lets its successor start early must itself wait for its
predecessor on every path, or a launch whose threads all leave at once is over before the step ahead of it."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "openfpm_data_b200", "csrc")


def _kernels():
    """(name, body without comments) of every __global__ function of the library."""
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        text = re.sub(r"//[^\n]*", "", open(path).read())
        for m in re.finditer(r"__global__\s+void\b", text):
            start = text.index("{", text.index(")", text.index("k_", m.end())))
            depth, i = 0, start
            while True:
                depth += {"{": 1, "}": -1}.get(text[i], 0)
                i += 1
                if depth == 0:
                    break
            yield re.search(r"k_\w+", text[m.end():]).group(0), text[start + 1:i - 1]


def _statements(body):
    """(depth, statement) in order; braces end a statement too."""
    depth, cur = 0, ""
    for ch in body:
        if ch in "{};":
            if cur.strip():
                yield depth, cur.strip()
            cur = ""
            depth += {"{": 1, "}": -1}.get(ch, 0)
        else:
            cur += ch


def test_early_launches_wait_on_every_path():
    seen = 0
    for name, body in _kernels():
        if "grid_launch_dependents()" not in body:
            continue
        seen += 1
        waited = False  # by a statement that every thread passes
        prev = (0, "")
        for depth, st in _statements(body):
            if depth == 0 and "grid_dependency_wait()" in st and not st.startswith("if"):
                waited = True
            if re.search(r"\breturn\b", st):
                assert waited or (prev[0] == depth > 0 and "grid_dependency_wait()" in prev[1]), (
                    f"{name}: threads leave without the wait: {st!r}")
            prev = (depth, st)
        assert waited, f"{name} never waits"
    assert seen >= 2

"""CPU: rules the kernel sources keep that no run on a GPU would show reliably."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mixture-of-kittens_b200", "csrc")


def _sources():
    for name in sorted(os.listdir(CSRC)):
        if name.endswith((".cu", ".cuh")):
            with open(os.path.join(CSRC, name)) as f:
                yield name, re.sub(r"//[^\n]*", "", f.read())


def _balanced(text, start, pair):
    """End of the bracketed text whose opening bracket is at or after `start`."""
    at = text.index(pair[0], start)
    depth = 0
    for i in range(at, len(text)):
        depth += (text[i] == pair[0]) - (text[i] == pair[1])
        if depth == 0:
            return at, i + 1
    raise AssertionError("unbalanced")


def kernels():
    """name -> (parameter list, body) of every kernel."""
    found = {}
    for _, text in _sources():
        for m in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\s*)?", text):
            at = m.end()
            if m.group().rstrip().endswith("__launch_bounds__"):
                at = _balanced(text, at, "()")[1]
            name = re.match(r"\s*(\w+)", text[at:]).group(1)
            p0, p1 = _balanced(text, at, "()")
            b0, b1 = _balanced(text, p1, "{}")
            found[name] = (text[p0:p1], text[b0:b1])
    return found


def test_kernels_launched_dependently_wait_and_take_no_restrict_pointers():
    """A kernel that waits for the one ahead of it (pdl_wait) must not load its inputs before the wait: loads through const
    __restrict__ parameters or the read-only path may be moved there."""
    found = kernels()
    assert len(found) >= 14
    waiting = {name for name, (_, body) in found.items() if "pdl_wait()" in body}
    assert waiting >= {"grouped_gemm_kernel", "mx_gemm_kernel", "move_rows_kernel", "epilogue_rows_kernel", "sched_count_kernel"}
    for name in waiting:
        params, body = found[name]
        assert "__restrict__" not in params and "__ldg" not in body and ".nc" not in body, name


def test_kernels_without_the_wait_are_launched_plainly():
    """launch_kernel can let a kernel start before the one ahead has finished; it is for kernels that call pdl_wait only."""
    found = kernels()
    plain = {name for name, (_, body) in found.items() if "pdl_wait()" not in body}
    for _, text in _sources():
        for m in re.finditer(r"\b(%s)\b" % "|".join(sorted(plain)), text):
            statement = text[max(text.rfind(c, 0, m.start()) for c in ";{}") + 1:text.index(";", m.end()) if ";" in text[m.end():] else None]
            assert "launch_kernel" not in statement and not re.match(r"\s*auto\s*\*\s*kern", statement), m.group(1)

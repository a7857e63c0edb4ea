"""Kernels that begin while the kernel before them still runs (step_enter) read what that kernel writes by ordinary
loads: no read-only load anywhere in the sources, and no __restrict__ argument but what no kernel of a step, a sort or
a training pass writes, and what the kernel itself only writes.  Checked in the sources, as the promise is one to the compiler."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "code_mpm_gb300", "csrc")

# written by uploads, reorders and the optimiser's own launches only
CONSTANT = {"mats", "dclist", "sid", "W", "bias", "W4", "b4"}
# written, and not read, by the kernel that has them
OUTPUT = {"C", "gbias", "gW", "y", "d", "gW4", "gb4", "gb3", "loss", "kout", "vout"}


def _sources():
    out = {}
    for name in sorted(os.listdir(CSRC)):
        if name.endswith((".cu", ".cuh")):
            with open(os.path.join(CSRC, name), encoding="utf-8") as f:
                out[name] = re.sub(r"//[^\n]*", "", f.read())
    return out


def _closing(text, at, pair):
    depth = 0
    for i in range(at, len(text)):
        depth += (text[i] == pair[0]) - (text[i] == pair[1])
        if depth == 0:
            return i + 1
    raise AssertionError("unbalanced")


def _functions(text):
    """(name, arguments, body, is a kernel) of the functions defined in a source."""
    for m in re.finditer(r"\b(\w+)\(", text):
        head = text[max(0, text.rfind(";", 0, m.start()), text.rfind("}", 0, m.start())):m.start()]
        if "__global__" not in head and "__device__" not in head or m.group(1) == "__launch_bounds__":
            continue
        end = _closing(text, m.end() - 1, "()")
        rest = re.match(r"\s*(const\s*)?\{", text[end:])
        if rest:
            start = end + rest.end() - 1
            yield m.group(1), text[m.end():end - 1], text[start:_closing(text, start, "{}")], "__global__" in head


def test_no_read_only_loads():
    for name, text in _sources().items():
        assert not re.search(r"ld\.global(\.\w+)*\.nc|__ldg\b", text), name


def test_restrict_only_on_what_no_step_writes():
    entering, kernels = {"step_enter"}, []
    functions = [f for text in _sources().values() for f in _functions(text)]
    for _ in range(3):  # and functions that call one that waits
        entering |= {n for n, _, body, k in functions if not k and any(re.search(rf"\b{e}\b", body) for e in entering)}
    for name, args, body, kernel in functions:
        if kernel and any(re.search(rf"\b{e}\b", body) for e in entering):
            kernels.append(name)
            for arg in re.split(r",(?![^(]*\))", args):
                found = re.search(r"__restrict__\s*(\w+)", arg)
                if found:
                    assert found.group(1) in (CONSTANT if "const" in arg.split("*")[0] else OUTPUT), (name, arg)
    assert {"k_p2g_cells", "k_pass1_cells", "k_node_phase_b", "k_pass2", "k_rs_scatter", "k_step_lists",
            "k_layer"} <= set(kernels), kernels

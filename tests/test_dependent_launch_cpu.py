"""Source rules of kernels that are launched as programmatic dependents (they call griddepcontrol.wait, `pdl_wait()`).

Such a kernel is resident while its predecessor still writes, so nothing it reads is read-only for its whole life, which is what the
non-coherent load path (`__ldg`, and `const T * __restrict__` kernel parameters, which compile to it) asks for; and a load that is known
to be invariant may be moved above the wait."""
import glob
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
# parameters of device functions that only ever point to shared memory
SHARED = {"acts", "dy", "ue_tab", "blk"}


def functions():
    """(file, is kernel, parameter list, body) of every device function and kernel"""
    for path in sorted(glob.glob(os.path.join(ROOT, "edge0_b200", "csrc", "*.cu*"))):
        text = re.sub(r"//[^\n]*", "", open(path).read())
        for m in re.finditer(r"__(global|device)__ (?:__forceinline__ )?(?:(?!__(?:global|device)__)[^;{}=])*?\b(?!__launch_bounds__)\w+\(", text):
            if m.group(0).endswith("__launch_bounds__("):
                continue
            at, depth = m.end(), 1
            while depth:                                   # the parameter list, or what __launch_bounds__ has in its parentheses
                depth += {"(": 1, ")": -1}.get(text[at], 0)
                at += 1
            params = text[m.end():at - 1]
            brace = re.match(r"\s*{", text[at:])
            if not brace:
                continue
            beg = at + brace.end()
            end, depth = beg, 1
            while depth:
                depth += {"{": 1, "}": -1}.get(text[end], 0)
                end += 1
            yield os.path.basename(path), m.group(1) == "global", params, text[beg:end]


def test_every_kernel_is_found():
    kernels = [f for f in functions() if f[1]]
    total = sum(len(re.findall(r"__global__", re.sub(r"//[^\n]*", "", open(p).read())))
                for p in glob.glob(os.path.join(ROOT, "edge0_b200", "csrc", "*.cu*")))
    assert len(kernels) == total


def test_dependents_read_through_the_coherent_path():
    bad = []
    for name, kernel, params, body in functions():
        if kernel and "pdl_wait()" not in body:
            continue                                       # an ordinary launch: its predecessor has finished
        bad += [(name, "__ldg", body[m.start():m.start() + 60]) for m in re.finditer(r"__ldg\(", body)]
        for m in re.finditer(r"const [\w:]+ \* __restrict__ (\w+)", params):
            if kernel or m.group(1) not in SHARED:
                bad.append((name, "const __restrict__", m.group(1)))
    assert not bad, bad


def test_no_dependent_right_behind_a_copy():
    """A kernel behind a copy or a memset is an ordinary launch: a call copies before it sets its launch mode or launches anything, behind
    its last launch, or with copy_out, which says so."""
    text = re.sub(r"//[^\n]*", "", open(os.path.join(ROOT, "edge0_b200", "csrc", "capi.cu")).read())
    bad = []
    for m in re.finditer(r"\n(?:\w[\w ]*)?\bint (\w+)\([^;{}]*\) \{\n(.*?)\n\}", text, re.S):
        marks = [("raw" if "Async" in t.group(0) else "launch", t.group(0)) for t in
                 re.finditer(r"cudaMem(?:cpy|set)Async\(|\blaunch_\w+[<(]|\w+_impl[<(]|\bdense_mat\w+\(|whole_layer_overlap\(", m.group(2))]
        for i, (kind, _) in enumerate(marks):
            before, after = (any(k == "launch" for k, _ in part) for part in (marks[:i], marks[i + 1:]))
            if kind == "raw" and before and after:
                bad.append(m.group(1))
    assert not bad, bad

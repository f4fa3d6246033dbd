"""Kernels that start while the kernel before them still runs (programmatic dependents): every one of them waits for it, and none declares what that
kernel may still be writing as __restrict__, which promises the compiler that nobody writes it while the kernel runs."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "xalm_b200", "csrc")
WEIGHTS = {"table", "positions", "W", "w", "wa", "wb", "a", "b"}  # written before the first step only


def closed(text, at, pair="()"):
    """Index behind the bracket that closes the one at text[at]."""
    depth = 0
    for i in range(at, len(text)):
        depth += (text[i] == pair[0]) - (text[i] == pair[1])
        if not depth:
            return i + 1
    raise AssertionError("unbalanced " + pair)


def kernels():
    """name -> (parameters, body)"""
    out = {}
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        text = re.sub(r"//[^\n]*", "", open(path).read())
        for m in re.finditer(r"__global__\s+void\s+(?:(?:__launch_bounds__|__maxnreg__)\s*(?=\())?", text):
            at = m.end()
            if text[at] == "(":
                at = closed(text, at)
            name = re.match(r"\s*(\w+)\s*", text[at:])
            start = at + name.end()
            end = closed(text, start)
            if text[end:].lstrip().startswith("{"):
                body = text.index("{", end)
                out[name.group(1)] = text[start:end], text[body:closed(text, body, "{}")]
    return out


def test_what_a_step_computes_is_no_restrict_parameter_of_a_programmatic_dependent():
    early = {n: k for n, k in kernels().items() if re.search(r"\bpdl_(enter|wait)\(\)", k[1])}
    assert len(early) > 20
    for name, (params, _) in early.items():
        assert set(re.findall(r"__restrict__\s*(\w+)", params)) <= WEIGHTS, name


def test_every_kernel_of_a_one_token_step_waits_for_the_one_before():
    found, ks = set(), kernels()
    for path in glob.glob(os.path.join(CSRC, "*.cu*")):
        found |= set(re.findall(r"launch_step\((\w+)", open(path).read()))
    found |= {"swa_one_kernel", "hgrn2_cols_kernel"}  # launched with a cluster beside
    found = {n for n in found if n in ks}
    assert len(found) > 15
    for name in found:
        assert "pdl_enter()" in ks[name][1], name


def test_no_two_kernels_share_a_name():
    """The checks above look kernels up by name."""
    names = [n for path in glob.glob(os.path.join(CSRC, "*.cu*")) for n in
             re.findall(r"__global__\s+void\s+(?:__launch_bounds__\s*\((?:[^()]|\([^()]*\))*\)|__maxnreg__\s*\(\d+\))?\s*(\w+)\s*\((?=[^;{]*\)\s*\{)", open(path).read())]
    assert len(names) > 70 and sorted(names) == sorted(set(names))

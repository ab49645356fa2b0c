"""Rules of kernels that start while their predecessor on the stream still runs (csrc/common.cuh), checked in the source:
each of them waits for it, and none reads through a `const __restrict__` pointer, which promises data that does not
change for as long as the kernel runs, the time before its wait included."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "torch-tpu_b200", "csrc")


def _strip(src):
    return re.sub(r"//[^\n]*|/\*.*?\*/", " ", src, flags=re.S)


def _closing(src, i, pair):
    depth = 0
    while True:
        depth += (src[i] == pair[0]) - (src[i] == pair[1])
        if depth == 0:
            return i
        i += 1


def _functions(src):
    """(is a kernel, name, parameters, body) of every device function."""
    for m in re.finditer(r"__(global|device)__", src):
        head = re.compile(r"(\w+)\s*\(").search(src, m.end())
        if head.group(1) == "__launch_bounds__":
            head = re.compile(r"(\w+)\s*\(").search(src, _closing(src, head.end() - 1, "()"))
        end = _closing(src, head.end() - 1, "()")
        body = re.compile(r"\s*([{;])").match(src, end + 1)
        if body and body.group(1) == "{":
            yield m.group(1) == "global", head.group(1), src[head.end():end], src[body.end() - 1:_closing(src, body.end() - 1, "{}")]


def test_overlapped_kernels_keep_the_rules():
    seen = 0
    for f in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        src = _strip(open(f).read())
        functions = list(_functions(src))
        kernels = {n: (p, b) for is_kernel, n, p, b in functions if is_kernel}
        launched = set()
        for m in re.finditer(r"moe_launch(?:_as)?\s*\(", src):
            call = src[m.end():_closing(src, m.end() - 1, "()")]
            launched |= {n for n in kernels if re.search(r"\b%s\b" % n, call)}
        overlapped = {n for n, (p, b) in kernels.items() if "pdl_" in b}
        assert launched <= overlapped, (f, "no wait for the predecessor", launched - overlapped)
        seen += len(launched)
        called = {n for is_kernel, n, p, b in functions if not is_kernel for k in overlapped if re.search(r"\b%s\b" % n, kernels[k][1])}
        for is_kernel, n, params, body in functions:
            if n in overlapped or n in called:
                bad = [p.strip() for p in params.split(",") if "const" in p.split("*")[0] and "__restrict__" in p]
                assert not bad, (f, n, bad)
    assert seen >= 20, seen

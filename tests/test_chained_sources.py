"""Chained kernels (csrc/launch.h) may be resident while the kernel before them still writes.  A
__restrict__ pointer parameter promises the compiler that nobody else writes the array during
the kernel, so that it may read it early, past grid_dependency(), or through the read-only
path.  Only arrays that are constant between calls may carry it: const ones, none of them an
array that some chained kernel writes, and no vector of the caller."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "clspmv_b200", "csrc")
VECTORS = {"x", "xg", "y", "yin", "yout", "ybar", "xbar", "abar"}


def _kernels(text):
    """(name, parameter list, body) of every __global__ function defined in `text`."""
    text = re.sub(r"//[^\n]*", "", text)
    for m in re.finditer(r"__global__\s+void\b", text):
        i = m.end()
        bounds = re.compile(r"\s*__launch_bounds__\s*\(").match(text, i)
        if bounds:
            i = _closing(text, bounds.end() - 1, "()")
        head = re.compile(r"\s*(\w+)\s*\(").match(text, i)
        end = _closing(text, head.end() - 1, "()")
        brace = re.compile(r"\s*\{").match(text, end)
        if not brace:
            continue   # a declaration
        yield head.group(1), text[head.end():end - 1], text[brace.end():_closing(text, brace.end() - 1, "{}")]


def _closing(text, at, pair):
    """Index past the bracket that closes the one at `at`."""
    depth = 0
    for i in range(at, len(text)):
        depth += (text[i] == pair[0]) - (text[i] == pair[1])
        if not depth:
            return i + 1
    raise AssertionError("unbalanced source")


def _chained():
    found = {}
    for path in sorted(glob.glob(os.path.join(CSRC, "kernels", "*.cuh")) + glob.glob(os.path.join(CSRC, "*.cu"))):
        with open(path) as f:
            for name, params, body in _kernels(f.read()):
                if re.search(r"grid_dependency\w*\(|gradient_begin\(", body):
                    found[name] = [p.strip() for p in params.split(",") if "*" in p]
    return found


def test_restrict_only_on_constant_arrays():
    kernels = _chained()
    assert len(kernels) >= 14, sorted(kernels)
    written = VECTORS | {re.search(r"(\w+)$", p).group(1) for ps in kernels.values() for p in ps if not p.startswith("const")}
    bad = [f"{k}: {p}" for k, ps in kernels.items() for p in ps
           if "__restrict__" in p and (not p.startswith("const") or re.search(r"(\w+)$", p).group(1) in written)]
    assert not bad, "\n".join(bad)

"""Kernels that are launched before the kernel in front of them ends (launch_early)
are resident while it still writes.  Read from the sources: such a kernel waits
for it, and the arrays that a predecessor writes don't come through the read-only
path (const __restrict__ parameters, __ldg)."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "streamsim_gb300", "csrc")
# parameters that the kernel in front may write: optics, panels and columns, what
# is summed from them, and the lists and counts of a sort or raster
WRITTEN = ("optics", "Bin", "in", "B", "partial", "stats", "done", "keys", "values", "hist", "offsets",
           "totals", "jobs", "jobs_end", "job_count")


def _sources():
    for name in sorted(os.listdir(CSRC)):
        if name.endswith(".cu"):
            with open(os.path.join(CSRC, name)) as f:
                yield name, f.read()


def _kernel(text, name):
    """Parameter list and body of a __global__ function."""
    at = re.search(r"__global__[^;{]*?\b%s\(" % name, text, re.S)
    assert at, name
    depth, i = 1, at.end()
    while depth:
        depth += {"(": 1, ")": -1}.get(text[i], 0)
        i += 1
    params, start = text[at.end():i - 1], text.index("{", i)
    depth, j = 1, start + 1
    while depth:
        depth += {"{": 1, "}": -1}.get(text[j], 0)
        j += 1
    return params, text[start:j]


def _early_kernels():
    for name, text in _sources():
        found = set(re.findall(r"launch_early\(\s*(k_\w+)", text))
        if name == "solve.cu":  # launched through a generic lambda
            found.add("k_jacobi_rows")
        if name == "batched.cu":
            found.add("k_sweep_wide")
        for kernel in sorted(found):
            yield name, kernel


@pytest.mark.parametrize("source,kernel", list(_early_kernels()))
def test_early_kernel(source, kernel):
    text = dict(_sources())[source]
    params, body = _kernel(text, kernel)
    assert "wait_for_previous()" in body
    written = WRITTEN
    if kernel == "k_jacobi_rows":  # see test_first_sweep
        written = tuple(w for w in WRITTEN if w != "optics")
    if kernel == "k_sweep_wide":  # see test_wide_sweeps
        written = tuple(w for w in WRITTEN if w != "Bin")
    for p in params.split(","):
        words = p.replace("*", " ").split()
        if words and words[-1].split("=")[0] in written and "*" in p:
            assert not ("const" in words and "__restrict__" in p), p
    # before the wait only the graph's and the plan's arrays are read
    before = body[:body.index("wait_for_previous()")]
    assert not re.search(r"\b(%s)\s*\[" % "|".join(written), before)
    for arg in re.findall(r"__ldg\(\s*(?:reinterpret_cast<[^>]*>\()?(\w+)", body):
        assert arg not in WRITTEN + ("X4",)


def test_first_sweep():
    """k_jacobi_rows reads optics before it waits, so only a sweep behind another
    sweep of the same call may start early."""
    with open(os.path.join(CSRC, "api.cpp")) as f:
        api = f.read()
    call = re.search(r"jacobi_sweep\(ctx->graph[^;]*;", api).group(0)
    assert re.search(r",\s*i > 0,\s*ctx->stream\)", call)
    solve = dict(_sources())["solve.cu"]
    assert re.search(r"follows \? sweep_rows<true> : sweep_rows<false>", solve)
    assert len(re.findall(r"sweep_rows<true>", solve)) == 1


def test_wide_sweeps():
    """k_sweep_wide gathers its panel through the read-only path.  It starts early
    only behind a k_check that lets it start after its own wait, when the sweep that
    wrote the panel has ended."""
    text = dict(_sources())["batched.cu"]
    _, check = _kernel(text, "k_check")
    early, wait, late = (check.index(x) for x in (
        "if (!late) start_next();", "wait_for_previous();", "if (late) start_next();"))
    assert early < wait < late
    assert check.count("start_next") == 2
    assert re.search(r"if \(follows\)\s*launch_early\(kernel,", text)
    # the only call with follows other than false: behind a k_check of the same loop
    calls = re.findall(r"launch_sweep<(?:float|double)>\([^;]*;", text)
    assert [c.split(",")[-2].strip() for c in calls].count("false") == len(calls) - 1
    loop = text[text.index("const bool wide = !column && !fp64 && (P >= 32 || !g.packed);"):]
    assert re.search(r"flag, k > 0, s\);.*?launch_early\(k_check,[^;]*, wide\);", loop, re.S)

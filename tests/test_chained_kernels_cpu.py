"""Kernels that are launched while their predecessor runs (``launch_chained`` of csrc/common.cuh), looked over in the source.

The compiler may move a load through a ``const __restrict__`` pointer in front of ``grid_wait()`` unless its address comes out of
``after_wait()`` or of a pointer that ``grid_wait()`` was given.  No result shows such a load reliably, the order in the source does."""
import re
from pathlib import Path

import pytest

import llmq_b200

CSRC = Path(llmq_b200.__file__).resolve().parent / "csrc"
FILES = sorted([*CSRC.glob("*.cu"), *CSRC.glob("*.cuh")])
RAW_INDEX = r"\b(?:blockIdx|threadIdx)\.x\b"


def _source(path):
    return re.sub(r"/\*.*?\*/|//[^\n]*", "", path.read_text(), flags=re.S)


def _closing(s, i, pair="()"):
    """Index behind the bracket that closes the one at i."""
    depth = 0
    for j in range(i, len(s)):
        depth += (s[j] == pair[0]) - (s[j] == pair[1])
        if depth == 0:
            return j + 1
    raise ValueError("unbalanced")


def _functions(s):
    """name -> (parameters, body) of the device functions and kernels that are defined in s."""
    s = re.sub(r"__(?:launch_bounds|cluster_dims)__\((?:[^()]|\([^()]*\))*\)", "", s)
    found = {}
    for m in re.finditer(r"__(?:global|device)__\b[^;{}()=]*?\b(\w+)\s*\(", s):
        end = _closing(s, m.end() - 1)
        body = re.match(r"\s*\{", s[end:])
        if body:
            start = end + body.end() - 1
            found[m.group(1)] = (s[m.end():end - 1], s[start:_closing(s, start, "{}")])
    return found


def _chained(s):
    return set(re.findall(r"launch_chained(?:_cluster)?\(\s*(\w+_kernel)\b", s))


def early_loads(sources):
    """'kernel: why' for every chained kernel whose source does not order its read-only loads behind the wait."""
    functions = {}
    for s in sources:
        functions.update(_functions(s))
    problems = []
    for kernel in sorted(set().union(*map(_chained, sources))):
        params, body = functions[kernel]
        wait = re.search(r"\bgrid_wait(?:_only)?\(([^)]*)\)", body)
        if not wait:
            problems.append(f"{kernel}: never waits")
            continue
        read_only = set(re.findall(r"\bconst\b[^,]*\*\s*__restrict__\s+(\w+)", params)) - {p.strip() for p in wait.group(1).split(",")}
        after = re.sub(r"after_wait\([^()]*\)", "", body[wait.end():])
        if "__ldg(" in after:
            problems.append(f"{kernel}: __ldg")
        for p in read_only:                                   # p[0], *p: an address that is known before the wait
            if re.search(rf"\b{p}\[\d+\]|[?=(,]\s*\*{p}\b", after):
                problems.append(f"{kernel}: {p} is read at a constant address")
        if not read_only:
            continue
        if re.search(RAW_INDEX, after):
            problems.append(f"{kernel}: plain index beside {sorted(read_only)}")
        for call in re.finditer(r"\b(\w+)(?:<[\w\s,]*>)?\(", after):
            if call.group(1) in functions and re.search(RAW_INDEX, functions[call.group(1)][1]):
                args = after[call.end():_closing(after, call.end() - 1) - 1]
                for p in read_only & set(re.findall(r"(\w+)\s*(?:,|$)", args)):              # handed over as it is
                    problems.append(f"{kernel}: {p} goes to {call.group(1)}(), which has plain indices")
    return problems


def test_loads_of_chained_kernels_come_after_the_wait():
    sources = [_source(f) for f in FILES]
    assert len(set().union(*map(_chained, sources))) >= 20
    assert early_loads(sources) == []


def test_every_chained_launch_clears_its_status():
    """The status of a launch is taken with LLMQ_LAUNCH_CHECK() or cudaGetLastError(): the launch's own result would leave it recorded, and the next
    kernel's check would report it once more."""
    for f in FILES:
        s = _source(f)
        assert not re.findall(r"(?:=|\breturn\b|\()\s*launch_chained(?:_cluster)?\(.*", s), f.name
        for m in re.finditer(r"\blaunch_chained(?:_cluster)?\(\s*\w+_kernel\b", s):
            assert re.search(r"LLMQ_LAUNCH_CHECK\(\)|cudaGetLastError\(\)", s[m.end():s.index("\n}", m.end())]), (f.name, m.group())


@pytest.mark.parametrize("wait,load,found", [
    ("grid_wait();", "x[after_wait(threadIdx.x)]", False), ("grid_wait(x);", "x[threadIdx.x]", False), ("grid_wait(x);", "sum(x)", False),
    ("grid_wait();", "x[threadIdx.x]", True), ("grid_wait();", "x[0]", True), ("grid_wait(x);", "x[0]", False),
    ("grid_wait();", "sum(x)", True), ("", "x[after_wait(threadIdx.x)]", True)])
def test_early_loads_are_found(wait, load, found):
    s = ("__device__ __forceinline__ float sum(const float* __restrict__ x) { return x[threadIdx.x]; }\n"
         "__global__ void __launch_bounds__(512, 4) a_kernel(float* __restrict__ out, const float* __restrict__ x) { %s out[0] = %s; }\n"
         "int go() { return launch_chained(a_kernel, 1, 512, 0, s, out, x); }\n" % (wait, load))
    assert bool(early_loads([s])) == found

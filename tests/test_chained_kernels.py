"""Rules of the kernels that launch_chained starts before the kernel in front of
them has ended (chain.cuh), read from the sources: each waits in chain_begin()
before it touches memory or returns, and none takes what that kernel may have
written through a const __restrict__ parameter, which would allow the compiler
to read it early and through the non-coherent cache."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "sparse-voxel-octrees_gb300", "csrc")
# explicit read-only loads: of data that was complete before the chain began
COMPLETE = ("a.tris", "a.acc", "g.grid", "bits", "from")


def _sources():
    return {os.path.basename(f): re.sub(r"//[^\n]*", "", open(f).read()) for f in glob.glob(os.path.join(CSRC, "*.cu"))}


def _closing(s, i, pair):
    depth = 1
    while depth:
        depth += (s[i] == pair[0]) - (s[i] == pair[1])
        i += 1
    return i


def _kernels(s):
    for m in re.finditer(r"__global__[^{;]*?\b(k_\w+)\s*\(", s):
        end = _closing(s, m.end(), "()")
        if not re.match(r"\s*\{", s[end:]):
            continue
        body = s.index("{", end) + 1
        yield m.group(1), s[m.end():end - 1], s[body:_closing(s, body, "{}") - 1]


def _chained():
    out = []
    for f, s in sorted(_sources().items()):
        names = set()
        for m in re.finditer(r"\blaunch_chained\(", s):
            call = s[m.end():_closing(s, m.end(), "()")]
            names |= set(re.findall(r"\bk_\w+", call))
        for name, params, body in _kernels(s):
            if name in names or "chain_begin()" in body:
                out.append(pytest.param(params, body, id="%s:%s" % (f, name)))
    return out


@pytest.mark.parametrize("params,body", _chained())
def test_chained_kernel(params, body):
    head, waits, _ = body.partition("chain_begin();")
    assert waits and "return" not in head and "[" not in re.sub(r"__shared__[^;]*;", "", head)
    for p in params.split(","):
        assert not ("__restrict__" in p and re.search(r"\bconst\b", p)), p.strip()
    for m in re.finditer(r"__ldg\(", body):
        arg = body[m.end():_closing(body, m.end(), "()") - 1]
        arg = re.sub(r"reinterpret_cast<[^>]*>\(", "", arg).lstrip("( \n")
        assert arg.startswith(COMPLETE), arg


def test_every_chained_kernel_is_found():
    assert len(_chained()) >= 15

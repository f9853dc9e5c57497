"""CPU check of the CUDA sources: a kernel launched with programmatic stream
serialization (launch_pdl, launch_coop) may start while the kernel before it
still runs, so it waits for that kernel (pdl_wait) before it reads anything
its arguments lead to."""
import glob
import os
import re

import pytest

from conftest import PKG_DIR


def _sources():
    out = {}
    for p in glob.glob(os.path.join(PKG_DIR, "csrc", "*.cu*")) + glob.glob(os.path.join(PKG_DIR, "csrc", "*.h")):
        src = re.sub(r"/\*.*?\*/", " ", open(p).read(), flags=re.S)
        out[p] = re.sub(r"//[^\n]*", " ", src)
    return out


def _balanced(s, i, pair):
    depth = 0
    for j in range(i, len(s)):
        depth += (s[j] == pair[0]) - (s[j] == pair[1])
        if depth == 0:
            return j
    raise AssertionError("unbalanced source")


def _launched():
    names = set()
    for src in _sources().values():
        names |= set(re.findall(r"\blaunch_(?:pdl|coop)\(\s*(k_\w+)", src))
    return sorted(names)


def _kernel(name):
    """(parameter names, body) of the kernel's definition."""
    for src in _sources().values():
        for m in re.finditer(r"\b" + name + r"\s*\(", src):
            if "__global__" not in src[max(0, m.start() - 160):m.start()].rsplit(";", 1)[-1].rsplit("}", 1)[-1]:
                continue
            close = _balanced(src, m.end() - 1, "()")
            params = [re.findall(r"\w+", p)[-1] for p in src[m.end():close].split(",")]
            body = src.index("{", close)
            return params, src[body:_balanced(src, body, "{}")]
    raise AssertionError(f"{name}: no definition")


@pytest.mark.parametrize("name", _launched())
def test_dependent_launches_wait(name):
    params, body = _kernel(name)
    assert "pdl_wait();" in body, f"{name} never waits for the kernel before it"
    before = body[:body.index("pdl_wait();")]
    used = [p for p in params if re.search(r"\b" + p + r"\b", before)]
    assert not used, f"{name} uses {used} before it waits"


def test_some_kernels_are_checked():
    assert len(_launched()) >= 5

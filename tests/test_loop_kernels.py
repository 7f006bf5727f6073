"""The CG loop's kernels run as programmatic dependents: each is resident while
the kernel before it still writes.  What that asks of their source, checked on
the source: the wait is the first statement of every kernel that is launched so,
and no vector that the loop writes is read through the read-only data path."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "fem_b200", "csrc")
HEADERS = ["kernels.cuh", "stencil.cuh", "tail.cuh"]
# written before the loop (set-up and prepare_operator), constant in it
CONSTANT = {"invd", "invdc", "binv", "binvc", "fine", "coarse", "units", "cells"}


def _read(name):
    with open(os.path.join(CSRC, name)) as f:
        return re.sub(r"//[^\n]*", "", f.read())


def _kernels():
    """name -> (parameter list, body) of every __global__ function."""
    out = {}
    for name in HEADERS:
        src = _read(name)
        for m in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\([^;{]*?\)\s*)?(\w+)\s*\(", src):
            i, depth = m.end(), 1
            while depth:
                depth += {"(": 1, ")": -1}.get(src[i], 0)
                i += 1
            params = src[m.end(): i - 1]
            j = src.index("{", i)
            k, depth = j + 1, 1
            while depth:
                depth += {"{": 1, "}": -1}.get(src[k], 0)
                k += 1
            out[m.group(1)] = (params, src[j + 1: k - 1])
    return out


KERNELS = _kernels()
LAUNCHED = set()
for _f in ("engine.cu", "stencil_launch.cuh"):
    _s = _read(_f)
    LAUNCHED |= set(re.findall(r"\blaunch\(H,[^;]*?\b(k_\w+|stencil\w*_kernel)\b", _s))
    LAUNCHED |= set(re.findall(r"auto fn\d* =[^;]*?\b(k_\w+|stencil\w*_kernel)\b", _s))
LAUNCHED -= {"k_coarse_assemble"}   # before the loop, launched plainly


def test_the_kernels_are_found():
    assert {"k_cg_update", "k_cg_dir", "k_bgram", "k_bupdate", "k_bdir", "k_tail", "k_restrict", "k_prolong_add",
            "stencil_kernel", "stencil2b_kernel", "stencil1b_kernel", "k_while_cond"} <= LAUNCHED <= set(KERNELS)


@pytest.mark.parametrize("name", sorted(LAUNCHED))
def test_the_wait_comes_first(name):
    assert KERNELS[name][1].lstrip().startswith("griddep_sync();")


@pytest.mark.parametrize("name", sorted(n for n, k in KERNELS.items() if "griddep_sync" in k[1]))
def test_no_read_only_path_to_loop_vectors(name):
    params, body = KERNELS[name]
    assert "__ldg" not in body
    for p in re.findall(r"const\s+\w+\s*\*\s*__restrict__\s+(\w+)", params):
        if p not in CONSTANT:   # such a parameter is read by ld_val and ld_pair alone
            assert not re.search(rf"\b{p}\s*\[|\*\s*{p}\b", body), p


def test_loads_are_coherent():
    common, kernels = _read("femh_common.cuh"), _read("kernels.cuh")
    for src in (common, kernels):
        assert "__ldg" not in src and ".nc" not in src
    assert len(re.findall(r'asm volatile\("ld\.global\.', common)) == 5

"""Rules of the kernels that may start before the one ahead of them on the stream
has ended, read from the sources: each waits before its first use of a pointer, and
none reads what that one writes through the read-only path (__ldg, or a const
__restrict__ parameter, whose loads may also be moved above the wait)."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "pmpp_b200", "csrc")


def _kernels():
    """name -> (parameter list, body) of every __global__ function."""
    out = {}
    for f in sorted(os.listdir(CSRC)):
        if not f.endswith((".cu", ".cuh")):
            continue
        s = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, f)).read())
        for m in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\((?:[^()]|\([^()]*\))*\)\s*)?(\w+)\s*\(", s):
            a = s.index("{", m.end())
            depth, b = 1, a + 1
            while depth:
                depth += {"{": 1, "}": -1}.get(s[b], 0)
                b += 1
            out[m.group(1)] = (s[m.end():a], s[a:b])
    return out


def _launched_early():
    names = set()
    for f in sorted(os.listdir(CSRC)):
        s = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, f)).read())
        for m in re.finditer(r"launch_dependent\(([^;]*);", s):
            found = re.findall(r"\b(\w*kernel\w*)\b", m.group(1))
            if not found:  # auto k = ...;
                found = re.findall(r"\b(\w*kernel\w*)\b", s[s.rindex("auto k =", 0, m.start()):m.start()].split(";")[0])
            names.update(n for n in found if n != "kernel")
    return names


KERNELS = _kernels()


def test_the_early_kernels_are_found():
    early = _launched_early()
    assert {"bin_count_kernel", "bin_place_kernel", "scan_one_kernel", "scatter_rows_kernel", "gather_kernel_x2",
            "col_pass_kernel", "z_r2c_kernel", "z_c2r_kernel"} <= early
    assert early <= set(KERNELS)
    assert early == {n for n, (_, b) in KERNELS.items() if "wait_for_previous()" in b}


@pytest.mark.parametrize("name", sorted(_launched_early()))
def test_early_kernel_reads_coherently_after_its_wait(name):
    params, body = KERNELS[name]
    assert not re.search(r"const\s+\w+\s*\*\s*__restrict__", params)
    assert "__ldg" not in body
    pointers = re.findall(r"\*\s*(?:__restrict__\s+)?(\w+)\s*[,)]", params)
    before = body[:body.index("wait_for_previous()")]
    for p in pointers:
        assert not re.search(r"\b%s\b" % p, before), p

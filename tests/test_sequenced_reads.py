"""Kernels launched behind one another without a gap (seq_begin) and what they read.

Such a kernel may be resident while its predecessors still write. Data of theirs is read after the
wait by plain loads or by ld_seq. A `__restrict__` parameter lets the compiler take the read-only
path, or move the load above the wait, and a non-volatile load instruction (__ldg, __ldcg) may be
moved too; both are left to data that no sequenced kernel writes. What is checked
is the source: on the device such a read goes wrong only when the timing allows it."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "nanomagmc_gb300", "csrc")

# Written by the host, or by kernels that are launched plainly (whose successors begin after their end).
STATIC = {
    "nmmc_kernels.cu": {"fill", "fill_n", "fill_zoff", "bh", "chains", "tab", "Hd"},
    "nmmc_general.cu": {"mask", "bh", "chains"},
    "nmmc_ising.cu": {"bh", "chains", "tab"},
    "nmmc_gen.cu": {"snaps", "idx", "sig", "cnd"},
}


def sequenced_kernels():
    out = []
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        src = open(path).read()
        for m in re.finditer(r"__global__[^{;]*?\b(k_\w+)\s*\(([^{;]*?)\)\s*\{", src, re.S):
            i, depth = m.end(), 1
            while depth:
                depth += {"{": 1, "}": -1}.get(src[i], 0)
                i += 1
            if re.search(r"seq_(begin|wait)\(\)", src[m.end():i]):
                out.append((os.path.basename(path), m.group(1), m.group(2), src[m.end():i]))
    return out


KERNELS = sequenced_kernels()


def test_every_sequenced_launch_is_of_a_sequenced_kernel():
    names = {k[1] for k in KERNELS}
    assert len(names) > 20
    for path in glob.glob(os.path.join(CSRC, "*.cu")):
        for name in re.findall(r"launch_seq\([^;]*?\b(k_\w+)", open(path).read()):
            assert name in names, name


@pytest.mark.parametrize("file,name,params,body", KERNELS, ids=["%s-%s" % k[:2] for k in KERNELS])
def test_reads_of_a_predecessors_data(file, name, params, body):
    for p in params.split(","):
        p = " ".join(p.split())
        if "__restrict__" in p:
            assert re.search(r"(\w+)$", p).group(1) in STATIC[file], p
    assert "__ldcg" not in body
    for arg in re.findall(r"__ldg\(\s*([^)]*)", body):
        assert re.match(r"&?(\w+)", arg).group(1) in STATIC[file], arg
    # the wait comes before anything is read: only declarations and index arithmetic ahead of it
    ahead = body[:re.search(r"seq_(begin|wait)\(\)", body).start()]
    assert not re.search(r"\b(chains|spins|sweep|planes|bh|in|dout)\s*\[", ahead), ahead

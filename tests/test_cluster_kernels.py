"""Kernels of thread-block clusters write into the shared memory of their peers
only after a cluster barrier: until then a peer may not have started, and its
shared memory may not be accessed. No run can show the order (a peer has mostly
started by then), so the sources are read: in each cluster kernel the first
barrier stands before the first access to a peer.
"""

import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(__file__), "..", "dftax_b200", "csrc")
# instructions that reach into another CTA of the cluster
REMOTE = re.compile(r"(?:st|ld|atom|red)\.(?:async\.)?shared::cluster|multicast::cluster"
                    r"|cta_group::2\.shared::cluster")
BARRIER = re.compile(r"barrier\.cluster\.wait")
FUNCTION = re.compile(r"(\w+)\([^;{}]*\)\s*\{")


def _functions(text):
    """(name, text between the last body and the name, body) of each function."""
    pos = 0
    while (m := FUNCTION.search(text, pos)):
        depth, i = 1, m.end()
        while depth:
            depth += {"{": 1, "}": -1}.get(text[i], 0)
            i += 1
        yield m.group(1), text[pos:m.start()], text[m.end():i]
        pos = i


def _kernels():
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        with open(path) as f:
            text = re.sub(r"//[^\n]*", "", f.read())
        text = re.sub(r"__(?:cluster_dims|launch_bounds)__\([^()]*\)", "", text)
        text = re.sub(r"\bnamespace\s*\w*\s*\{|extern \"C\"\s*\{", "", text)
        funcs = list(_functions(text))
        helpers = [(n, b) for n, head, b in funcs if "__global__" not in head]
        remote = [n for n, b in helpers if REMOTE.search(b)]
        barrier = [n for n, b in helpers if BARRIER.search(b)]
        for name, head, body in funcs:
            if "__global__" not in head:
                continue
            calls = lambda names: [m.start() for n in names  # noqa: E731
                                   for m in re.finditer(rf"\b{n}\b\s*(?:<[^;()]*>)?\(", body)]
            at_remote = calls(remote) + [m.start() for m in REMOTE.finditer(body)]
            at_barrier = calls(barrier) + [m.start() for m in BARRIER.finditer(body)]
            if at_remote:
                yield os.path.basename(path), name, min(at_remote), min(at_barrier, default=None)


KERNELS = list(_kernels())


def test_the_cluster_kernels_are_found():
    assert {(f, n) for f, n, _, _ in KERNELS} == {
        ("lowrank.cu", "pivoted_cholesky_kernel"), ("sp2.cu", "sp2_cluster_kernel"),
        ("ozaki_gemm.cu", "ozaki_gemm_i8_pair")}


@pytest.mark.parametrize("file,kernel,remote,barrier", KERNELS, ids=[k[1] for k in KERNELS])
def test_barrier_before_the_first_remote_access(file, kernel, remote, barrier):
    assert barrier is not None and barrier < remote, (file, kernel)

"""Distributed shared memory is accessed only after a cluster barrier.

A CTA of a cluster may be accessed through shared::cluster once it is known to
have started, which a barrier of the cluster shows; being scheduled together
does not.  A kernel without one may lose a store, or fault, on a run in a
million, so this is checked in the sources.
"""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "tinker-gpu_gb300", "csrc")
REMOTE = re.compile(r"\b(?:ld|st|red|atom)\.(?:\w+\.)*shared::cluster")
WAIT = re.compile(r"barrier\.cluster\.wait")


def _kernels():
    """(file:kernel, text) of every kernel with a remote access, comments left out."""
    out = []
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        text = re.sub(r"//[^\n]*|/\*.*?\*/", "", open(path).read(), flags=re.S)
        for part in text.split("__global__")[1:]:
            if REMOTE.search(part):
                name = re.search(r"\bk_\w+", part).group(0)
                out.append((f"{os.path.basename(path)}:{name}", part))
    return out


def test_kernels_with_remote_accesses_are_found():
    assert {n for n, _ in _kernels()} >= {"pcg.cu:k_pcg_step", "pme.cu:k_fft_small"}


@pytest.mark.parametrize("name, text", _kernels(), ids=lambda v: v if ":" in v and len(v) < 60 else "")
def test_cluster_barrier_before_remote_access(name, text):
    wait = WAIT.search(text)
    assert wait and wait.start() < REMOTE.search(text).start(), name

"""What kernels of several CTAs owe each other.  One that issues tcgen05 instructions for a CTA pair (cta_group::2) issues no other
form: PTX wants one value of .cta_group for all of them, allocation and release of tensor memory among them.  And one that is launched in
clusters touches a peer's shared memory only behind a cluster barrier, which says that the peer runs."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "gevva_b200", "csrc")


def code(path):
    return re.sub(r"//[^\n]*|/\*.*?\*/", "", open(path).read(), flags=re.S)


def one_cta_helpers():
    """Functions of the shared headers that hold a cta_group::1 instruction."""
    names = set()
    for path in glob.glob(os.path.join(CSRC, "*.cuh")):
        for function in re.finditer(r"__device__ __forceinline__ \w+ (\w+)\(.*?\n}\n", code(path), flags=re.S):
            if "cta_group::1" in function[0]:
                names.add(function[1])
    return names


PAIR_SOURCES = sorted(os.path.basename(p) for p in glob.glob(os.path.join(CSRC, "*.cu")) if re.search(r"cta_group::2|gv_cta_pair\.cuh", code(p)))


def test_helpers_are_found():
    assert {"tmem_alloc", "tmem_relinquish", "tmem_dealloc", "tc_commit", "issue_mmas", "issue_sf_copies"} <= one_cta_helpers()
    assert len(PAIR_SOURCES) == 4


@pytest.mark.parametrize("source", PAIR_SOURCES)
def test_pair_kernels_use_the_pair_forms_alone(source):
    text = code(os.path.join(CSRC, source))
    assert "cta_group::1" not in text
    assert [name for name in sorted(one_cta_helpers()) if re.search(rf"\b{name}\s*[<(]", text)] == []


CLUSTER_SOURCES = sorted(os.path.basename(p) for p in glob.glob(os.path.join(CSRC, "*.cu")) if "cudaLaunchAttributeClusterDimension" in code(p))
REMOTE = r"\b(?:cluster_map_shared|cluster_store_uint4|pair_arrive_remote|mbar_arrive_remote|wp_arrive|release_accumulator|pair_tmem_alloc|pair_commit_both|pair_mma)\s*\("


def test_cluster_kernels_are_found():
    assert "router_project.cu" in CLUSTER_SOURCES and len(CLUSTER_SOURCES) == 5


@pytest.mark.parametrize("source", CLUSTER_SOURCES)
def test_peers_are_touched_behind_a_cluster_barrier(source):
    """From the first line of each cluster kernel: the first wait for the cluster comes before the first access to a peer."""
    kernels = [k for k in code(os.path.join(CSRC, source)).split("__global__")[1:] if re.search(r"cluster_cta_rank\(\)", k)]
    assert kernels
    for kernel in kernels:
        body = kernel.split("\n}\n")[0]
        barrier, remote = re.search(r"\bcluster_(?:sync_all|wait)\(\)", body), re.search(REMOTE, body)
        assert barrier and remote and barrier.start() < remote.start()
        # every thread waits as often as it arrives
        assert bool(re.search(r"\bcluster_arrive(?:_relaxed)?\(\)", body)) == bool(re.search(r"\bcluster_wait\(\)", body))

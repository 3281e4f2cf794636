"""Order of steps inside kernels that no run on a GPU would show reliably, read from their source (no GPU).

Tensor memory: a launch lets its successors start once every block of it has said so, and a successor's block keeps its tensor memory until
this launch has ended. A kernel that allocates must therefore hold its columns before it says so: otherwise a successor's block on the
same SM can take them first, and the two wait for one another in tcgen05.alloc and the dependency wait, which no bounded wait covers."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "libinferbit_b200", "csrc")
SOURCES = [p for p in sorted(glob.glob(os.path.join(CSRC, "*.cu"))) if "tcgen05.alloc" in open(p).read()]


def _code(path):
    return re.sub(r"//[^\n]*", "", open(path).read())


@pytest.mark.parametrize("path", SOURCES, ids=[os.path.basename(p) for p in SOURCES])
def test_successors_start_after_the_allocation(path):
    kernels = [k for k in _code(path).split("__global__")[1:] if "tcgen05.alloc" in k]
    assert kernels
    for k in kernels:
        starts = [m.start() for m in re.finditer(r"pdl_launch_dependents\(\)", k)]
        assert starts and k.index("tcgen05.alloc") < starts[0], "successors may start before this kernel's blocks hold their tensor memory"


def test_digit_sums_of_two_activations_are_kept_apart():
    """A block may convert several activations one after the other through the same shared scratch. Each warp leaves its digit sums there
    and threads 0 to 3 add them up: a barrier has to stand between that adding and the next activation's writes, so every
    conversion needs one before it writes."""
    code = _code(os.path.join(CSRC, "xconvert.cuh"))
    bodies = [b for b in re.split(r"\n(?:template|__device__)", code) if "sc.sred[threadIdx.x >> 5][l] = v" in b]
    assert len(bodies) == 3                                  # in registers, in a loop, with a known maximum
    for b in bodies:
        assert "__syncthreads()" in b[:b.index("sc.sred[threadIdx.x >> 5][l] = v")], b.strip().splitlines()[1]


@pytest.mark.parametrize("kernel,arrays", [("assign_exact_kernel", ["C"]), ("assign_filter_kernel", ["C"]), ("accumulate_kernel", ["idx", "dist"]),
                                           ("accumulate_finish_kernel", ["part_sums", "part_counts", "part_inertia"]), ("update_kernel", ["counts", "sums"])])
def test_kmeans_kernels_read_the_launch_ahead_past_l1(kernel, arrays):
    """Arrays that the launch just ahead may have written, in kernels that start before it has ended: no plain or read-only load."""
    code = _code(os.path.join(CSRC, "kmeans.cu"))
    body = next(k for k in code.split("__global__")[1:] if re.search(rf"\b{kernel}\(", k[:200]))
    end = re.search(r"\n}\n", body).start()
    for a in arrays:
        assert not re.search(rf"\b{a}\[", body[:end]), a
        assert re.search(rf"__ldcg\({a} \+", body[:end]), a


def test_no_access_to_a_peers_shared_memory_before_it_has_started():
    """Shared memory of another block of the cluster may be used once that block is known to run, which only a barrier of the cluster says: an
    arrival and a wait stand before the first use. (A block's own barrier and the wait for the launch ahead say nothing about a peer.)"""
    seen = []
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        for k in _code(path).split("__global__")[1:]:
            body = k.split("\n}\n")[0]
            use = re.search(r"st\.shared::cluster\.[uv]|map_shared_rank", body)
            if not use:
                continue
            kernel, ahead = re.search(r"(\w+_kernel)\(", body).group(1), body[:use.start()]
            seen.append(kernel)
            assert "cluster.sync()" in ahead or re.search(r"cluster_arrive(_relaxed)?\(\).*cluster_wait\(\)", ahead, re.S), kernel
    assert seen == ["xprep_tc_cluster_kernel", "linear_tc_kernel", "pq_topk_select_cluster_kernel"]

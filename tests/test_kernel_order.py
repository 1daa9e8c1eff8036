"""Orders in the kernels' sources that no run can show: a fault in them is a matter of timing."""

import re

import pytest

from paged_attention_engine_b200.kernels import build

# What reaches another block of the cluster (its shared memory, or a barrier there), and what shows that all
# of its blocks have started: a completed cluster barrier.
REMOTE = re.compile(r"\.shared::cluster\.(?:f32|b32|u32|b64|v4)|load_from_block\(|mbar_arrive_remote\(|tma_load_2d_pair\(|umma_bf16_pair\(|tcgen05_commit_pair\(")
BARRIER = re.compile(r"barrier\.cluster\.wait|cluster_wait\(\)|cluster_sync\(\)")


def _kernels():
    """(file, name, body) of every kernel."""
    for path in sorted(build.CSRC.glob("*.cu*")):
        text = re.sub(r"//[^\n]*", "", path.read_text())
        for start in re.finditer(r"__global__", text):
            at = text.index("{", start.end())
            head = re.sub(r"__\w+__\s*\([^()]*\)", "", text[start.end() : at])
            name = re.search(r"void\s+(\w+)\s*\(", head).group(1)
            depth, end = 0, at
            while True:
                depth += {"{": 1, "}": -1}.get(text[end], 0)
                end += 1
                if depth == 0:
                    break
            yield path.name, name, text[at:end]


def test_the_kernels_are_found():
    names = {name for _, name, _ in _kernels()}
    assert {"splitk_rms_norm_cluster_kernel", "gemm_tcgen05_pair_kernel", "prefill_tcgen05_kernel"} <= names


@pytest.mark.parametrize("kernel", [n for _, n, body in _kernels() if REMOTE.search(body)])
def test_no_block_of_a_cluster_reaches_another_before_a_cluster_barrier(kernel):
    """Distributed shared memory may be used once every block of the cluster has started."""
    for _, name, body in _kernels():
        if name == kernel and (first := REMOTE.search(body)):
            barrier = BARRIER.search(body)
            assert barrier and barrier.start() < first.start(), f"{name}: {first.group(0)} comes first"


@pytest.mark.parametrize("kernel", ["gemm_tcgen05_persistent_kernel", "gemm_tcgen05_pair_kernel"])
def test_a_many_token_product_loads_nothing_before_the_kernel_before_has_completed(kernel):
    """Its weights may have been written by the kernel before."""
    (body,) = [body for _, name, body in _kernels() if name == kernel]
    assert 0 < body.index("dependent_launch_wait()") < body.index("tma_load_2d")


@pytest.mark.parametrize("kernel", [n for _, n, body in _kernels() if re.search(r"tmem_alloc\(|tcgen05\.alloc", body)])
def test_the_next_kernel_is_let_go_when_tensor_memory_is_held(kernel):
    """A block of the next kernel that took columns first would hold them until this kernel has completed, which then waits for them."""
    for _, name, body in _kernels():
        if name == kernel:
            held = body.index("__syncthreads()", re.search(r"tmem_alloc\(|tcgen05\.alloc", body).start())
            lets_go = [m.start() for m in re.finditer(r"dependent_launch_(?:trigger|prologue)\(\)|launch_dependents", body)]
            assert lets_go and min(lets_go) > held, name

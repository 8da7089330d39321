"""Orders inside the kernels that no run can check safely (a wrong one shows as a hang, and only with blocks of several
launches on one SM), read from the sources."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "lex_gpu_b200" / "csrc"


def code(name):
    return re.sub(r"//[^\n]*", "", (CSRC / name).read_text())


@pytest.mark.parametrize("name,barrier", [("gemm_fp4_sm100.cuh", "__syncthreads()"), ("gemm_fp4_sm100_pair.cuh", "cluster_sync_all()"), ("gemm_fp4_few_sm100.cuh", "__syncthreads()"),
                                          ("matmul_q_fp4_sm100.cuh", "bar.sync 2"), ("matmul_q_chain_sm100.cuh", "__syncthreads()")])
def test_dependents_go_only_once_the_block_holds_its_tensor_memory(name, barrier):
    """A block that let the next launch start while it still waits for its columns could lose them to that launch, which
    then waits for this one."""
    text = code(name)
    kernels = [k for k in re.split(r"(?=__global__)", text) if "tmem_alloc" in k.split("tmem_dealloc")[0]]
    assert kernels
    for k in kernels:
        alloc = k.index("tmem_alloc")
        held = k.index(barrier, alloc)
        assert "allow_dependents" not in k[:alloc] and "allow_dependents" in k[alloc:]
        if "allow_dependents" in k[:held]:                       # then it is the allocating warp itself that does it
            assert "}" not in k[alloc:k.index("allow_dependents")]
    # the warp that does not meet that barrier (the block-scaled kernel's copy warp) leaves it to the others
    if name == "matmul_q_fp4_sm100.cuh":
        copy_warp = kernels[0][kernels[0].index("tma_load_2d"):kernels[0].index("umma_idesc")]
        assert "allow_dependents" not in copy_warp


def test_the_cluster_barrier_brings_the_warp_together_first():
    """barrier.cluster.*.aligned must be executed by all lanes of a warp at once; the matvec meets it behind code whose lanes
    part (tokens that do not exist, outputs that do not divide by the threads), the kernels that sum within a cluster behind loops over
    tokens: every barrier stands behind a __syncwarp of its own, or in cluster_sync_all, which has one."""
    found = [path.name for path in sorted(CSRC.glob("*.cuh")) if "barrier.cluster" in code(path.name)]
    assert "sm100_ptx.cuh" in found
    for name in found:
        for at in re.finditer(r"barrier\.cluster\.(?:arrive|wait)[\w.]*\.aligned", code(name)):
            ahead = code(name)[:at.start()]
            last = max(ahead.rfind("__syncwarp()"), ahead.rfind("barrier.cluster"))
            assert last > ahead.rfind("__device__"), name


@pytest.mark.parametrize("name", ["gemm_fp4_few_sm100.cuh", "matmul_q_fp4_sm100.cuh", "gemm_fp4_sm100_pair.cuh"])
def test_a_block_whose_sums_others_read_waits_for_them(name):
    """Sums in shared memory are read by the other blocks of a cluster: a barrier of the whole cluster before the first read and
    one behind the last, before the block can end."""
    text = code(name)
    reads = [m.start() for m in re.finditer(r"ld_shared_cluster_f32x4\(", text)]
    assert reads
    before, behind = text.rfind("cluster_sync_all()", 0, reads[0]), text.find("cluster_sync_all()", reads[-1])
    assert 0 < before and "tmem_ld_32x32b" not in text[before:reads[-1]]          # (all sums are stored by then)
    assert reads[-1] < behind < text.index("tmem_dealloc", reads[-1])

"""Orders inside the kernels that no run can check safely (a wrong one shows as a hang, and only with blocks of several
launches on one SM), read from the sources."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "lex_gpu_b200" / "csrc"


def code(name):
    return re.sub(r"//[^\n]*", "", (CSRC / name).read_text())


@pytest.mark.parametrize("name,barrier", [("gemm_fp4_sm100.cuh", "__syncthreads()"), ("gemm_fp4_sm100_pair.cuh", "cluster_sync_all()"),
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
    part (tokens that do not exist, outputs that do not divide by the threads)."""
    for name in ("sm100_ptx.cuh", "matvec_fp4_sm100.cuh", "gemm_fp4_sm100_pair.cuh"):
        for at in re.finditer(r"barrier\.cluster\.(?:arrive|wait)[\w.]*\.aligned", code(name)):
            ahead = code(name)[:at.start()]
            last = max(ahead.rfind("__syncwarp()"), ahead.rfind("barrier.cluster"))
            assert last > ahead.rfind("__device__"), name

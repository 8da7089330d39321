"""K split over blocks whose parts are summed within a cluster: the bits of the same split through the workspace."""
import numpy as np
import pytest

import lex_gpu_b200 as L
from lex_gpu_b200 import inputs
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gpu():
    g = L.Gpu(0)
    yield g
    g.close()


def both_ways(gpu, plan, m, n, k, residual):
    """The planner's own split (in a cluster where the device holds them all) and the same split asked for (through the workspace)."""
    x, wq, ws, wg = inputs.make_case(m, n, k, seed_base=800)
    r = inputs.make_residual(m, n, seed_base=801) if residual else None
    q, xb, rb = L.QBuf(gpu, wq, ws, wg), gpu.upload(x), gpu.upload(r) if residual else None
    own = plan(m, n, k, residual=residual)
    splits = own.describe().k_splits
    out = []
    for pipe in (own, plan(m, n, k, residual=residual, k_splits=splits)):
        y = gpu.alloc(4 * m * n)
        gpu.memset(y, 0xFF)
        gpu.run(pipe, q.bind(xb, rb, y))
        out.append(gpu.download(y, np.float32, (m, n)))
    assert gpu.status_word() == 0
    return splits, out, (x, wq, ws, wg, r)


@pytest.mark.parametrize("m,n,k,residual", [(65, 256, 1024, True), (100, 384, 2048, False), (130, 512, 2048, True), (257, 256, 2048, False),
                                            (1024, 2048, 4096, True), (200, 640, 1280, False)])
def test_two_cta_gemm(gpu, m, n, k, residual):
    """Tiles of 64 to 256 tokens, a last tile of few tokens, an odd last pair of rows, parts of unequal length."""
    plan = lambda *a, **kw: gpu.plan_gemm_fp4(*a, kernel=3, **kw)
    splits, (cluster, workspace), (x, wq, ws, wg, r) = both_ways(gpu, plan, m, n, k, residual)
    assert splits > 1
    if np.array_equal(cluster, workspace):
        return
    err, scale, _ = O.err_of_scale(cluster, O.gemm_fp4(x, wq, ws, wg, r=r))      # (asked for, the split may come with another tile)
    assert scale > 1e-3 and err <= 2e-5


@pytest.mark.parametrize("m,n,k,residual", [(1, 128, 8192, True), (3, 640, 8192, False), (4, 5120, 17408, True), (8, 1024, 4096, True),
                                            (17, 256, 5120, False), (32, 896, 7168, True)])
def test_block_scaled_kernel(gpu, m, n, k, residual):
    splits, (cluster, workspace), (x, wq, ws, wg, r) = both_ways(gpu, gpu.plan_matmul_fp4, m, n, k, residual)
    assert splits > 1 and np.array_equal(cluster, workspace)
    err, scale, _ = O.err_of_scale(cluster, O.matmul_q_x(x, wq, ws, wg, r=r))
    assert scale > 1e-3 and err <= 1e-4

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


def both_ways(gpu, plan, m, n, k, residual, tile=False):
    """The planner's own split, summed in clusters, and the same split (`tile`: and tile of tokens) asked for, through the workspace."""
    x, wq, ws, wg = inputs.make_case(m, n, k, seed_base=800)
    r = inputs.make_residual(m, n, seed_base=801) if residual else None
    q, xb, rb = L.QBuf(gpu, wq, ws, wg), gpu.upload(x), gpu.upload(r) if residual else None
    own = plan(m, n, k, residual=residual)
    splits = own.describe().k_splits
    asked = plan(m, n, k, residual=residual, k_splits=splits, **({"tm": own.describe().bm} if tile else {}))
    assert splits > 1 and own.route().cluster == splits and asked.route().cluster == 1 and asked.describe().k_splits == splits
    out = []
    for pipe in (own, asked):
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
    splits, (cluster, workspace), (x, wq, ws, wg, r) = both_ways(gpu, plan, m, n, k, residual, tile=True)
    assert np.array_equal(cluster, workspace)
    err, scale, _ = O.err_of_scale(cluster, O.gemm_fp4(x, wq, ws, wg, r=r))
    assert scale > 1e-3 and err <= 2e-5


@pytest.mark.parametrize("m,ffn,hidden", [(100, 192, 2048), (257, 128, 2048), (200, 320, 1280)])
def test_two_cta_gemm_with_silu_mul(gpu, m, ffn, hidden):
    """silu(gate) * up of the sums within a cluster: the bits of the same split's reduction launch."""
    x, wq, ws, wg = inputs.make_case(m, 2 * ffn, hidden, seed_base=810)
    q, xb = L.QBuf(gpu, wq, ws, (wg * np.float32(0.02)).astype(np.float32)), gpu.upload(x)
    own = gpu.plan_gemm_fp4(m, 2 * ffn, hidden, kernel=3)
    splits = own.describe().k_splits
    asked = gpu.plan_gemm_fp4(m, 2 * ffn, hidden, kernel=3, tm=own.describe().bm, k_splits=splits)
    assert splits > 1 and own.route().cluster == splits and asked.route().cluster == 1
    got = []
    for pipe in (own, asked):
        act = gpu.alloc(2 * m * ffn)
        gpu.memset(act, 0xFF)
        gpu.run_silu(pipe, xb, q.wq, q.ws, q.wg, act)
        got.append(gpu.download(act, np.float16, (m, ffn)))
    assert np.isfinite(got[0]).all() and np.array_equal(got[0].view(np.uint16), got[1].view(np.uint16))
    assert gpu.status_word() == 0


@pytest.mark.parametrize("m,n,k,residual", [(1, 128, 8192, True), (3, 640, 8192, False), (4, 5120, 17408, True), (8, 1024, 4096, True),
                                            (17, 256, 5120, False), (32, 896, 7168, True)])
def test_block_scaled_kernel(gpu, m, n, k, residual):
    splits, (cluster, workspace), (x, wq, ws, wg, r) = both_ways(gpu, gpu.plan_matmul_fp4, m, n, k, residual)
    assert splits > 1 and np.array_equal(cluster, workspace)
    err, scale, _ = O.err_of_scale(cluster, O.matmul_q_x(x, wq, ws, wg, r=r))
    assert scale > 1e-3 and err <= 1e-4

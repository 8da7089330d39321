"""gemm_fp4 of few tokens as one stream of weights per SM (gemm_fp4_few_kernel): shapes where its shares, clusters and token
counts have their edges."""
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


def check(got, want):
    err, scale, rel = O.err_of_scale(got, want)
    assert scale > 1e-3 and err <= 2e-5 and rel <= 2e-3, (err, rel)       # (the bound of the tensor path against the oracle)


@pytest.mark.parametrize("cluster", [1, 2, 3, 5, 6, 8])
@pytest.mark.parametrize("m", [1, 8, 9, 16, 17, 32, 33, 64])
def test_shares_that_cut_tiles(gpu, monkeypatch, m, cluster):
    """Every cluster size: shares that hold whole tiles and parts of two, that lie inside one tile, and tiles of one to several
    shares; one block of weights and odd numbers of them; with a residual."""
    monkeypatch.setenv("LEXB_FEW_C", str(cluster))
    for n, k in ((128, 256 * cluster), (640, 1280), (384, 256 * 17), (256, 512 * cluster)):
        x, wq, ws, wg = inputs.make_case(m, n, k, seed_base=700 + m)
        r = inputs.make_residual(m, n, seed_base=701)
        pipe = gpu.plan_gemm_fp4(m, n, k, residual=True)
        q = L.QBuf(gpu, wq, ws, wg)
        y = gpu.alloc(4 * m * n)
        gpu.memset(y, 0xFF)
        gpu.run(pipe, q.bind(gpu.upload(x), gpu.upload(r), y))
        check(gpu.download(y, np.float32, (m, n)), O.gemm_fp4(x, wq, ws, wg, r=r))
    assert gpu.status_word() == 0


def test_what_is_reported_is_what_runs(gpu):
    """The route is the launch's own; with the phase timers on, the two-CTA GEMM that has them runs instead, and its decode
    loops, of two K steps a turn too, leave their times."""
    m, n, k = 32, 4096, 4096
    x, wq, ws, wg = inputs.make_case(m, n, k, seed_base=720)
    want = O.gemm_fp4(x, wq, ws, wg)
    pipe, q, xb, y = gpu.plan_gemm_fp4(m, n, k), L.QBuf(gpu, wq, ws, wg), gpu.upload(x), gpu.alloc(4 * m * n)
    d, route = pipe.describe(), pipe.route()
    assert d.kernel == 3 and route.threads == 736 and route.blocks % route.cluster == 0 and route.blocks <= 148
    pair = gpu.plan_gemm_fp4(m, n, k, kernel=3)
    assert pair.route().threads == 608 and pair.route().blocks == pair.describe().grid
    whole = gpu.plan_gemm_fp4(512, 17408, 5120).route()
    split = gpu.plan_gemm_fp4(1024, 2048, 4096)
    assert whole.cluster == 1 and split.describe().k_splits > 1 and split.route().cluster == split.describe().k_splits
    try:
        for traced in (True, False):
            gpu.trace_enable(d.grid if traced else 0)
            gpu.memset(y, 0xFF)
            gpu.run(pipe, q.bind(xb, None, y))
            check(gpu.download(y, np.float32, (m, n)), want)
            if traced:
                records = gpu.trace_read(d.grid)
                assert (records[:, 6] > records[:, 0]).all() and (records[:, 15] > 0).all()
                assert (records[:, 8] > 0).all() and (records[:, 9] + records[:, 10] > 0).all()       # decode loop, its waits
    finally:
        gpu.trace_enable(0)
    assert gpu.status_word() == 0

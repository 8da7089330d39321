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
    """Every cluster size, a tile a cluster: shares that lie inside it, of one block of weights and odd numbers of them; with a
    residual."""
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


# (clusters, row tiles, blocks of weights a tile): up to four tiles a cluster, so that a share holds whole tiles and parts of
# others, its last segment another's first, and the sets of accumulators come round again
MANY_TILES = [(1, 449, 1), (1, 449, 3), (2, 225, 3), (3, 131, 5), (6, 77, 3), (8, 50, 3), (8, 50, 7)]


@pytest.mark.parametrize("cluster,tiles,blocks", MANY_TILES)
@pytest.mark.parametrize("m", [9, 17, 33, 64])
def test_clusters_with_several_tiles(gpu, monkeypatch, m, cluster, tiles, blocks):
    """... with and without a residual, and with constant weights: decoded ahead of the stream's order, launch behind launch."""
    monkeypatch.setenv("LEXB_FEW_C", str(cluster))
    n, k = 128 * tiles, 256 * blocks
    x, wq, ws, wg = inputs.make_case(m, n, k, seed_base=730 + m)
    r = inputs.make_residual(m, n, seed_base=731)
    q, xb, rb = L.QBuf(gpu, wq, ws, wg), gpu.upload(x), gpu.upload(r)
    want = O.gemm_fp4(x, wq, ws, wg)
    pipes = {(res, const): gpu.plan_gemm_fp4(m, n, k, residual=res, weights_constant=const) for res in (False, True) for const in (False, True)}
    route = pipes[False, False].route()
    assert route.threads == 736 and route.cluster == cluster and route.blocks < cluster * tiles      # some cluster has several tiles
    ys = {key: gpu.alloc(4 * m * n) for key in pipes}
    for y in ys.values():
        gpu.memset(y, 0xFF)
    for _ in range(2):
        for (res, const), pipe in pipes.items():
            gpu.run(pipe, q.bind(xb, rb if res else None, ys[res, const]))
    got = {key: gpu.download(y, np.float32, (m, n)) for key, y in ys.items()}
    check(got[False, False], want)
    check(got[True, False], O.gemm_fp4(x, wq, ws, wg, r=r))
    assert all(np.array_equal(got[res, True], got[res, False]) for res in (False, True))
    gpu.memset(ys[False, False], 0xFF)
    gpu.memset(ys[True, False], 0xFF)
    gpu.run_launches([(pipes[key], q.bind(xb, rb if key[0] else None, ys[key])) for key in ((False, False), (True, False))])
    assert all(np.array_equal(gpu.download(ys[res, False], np.float32, (m, n)), got[res, False]) for res in (False, True))
    assert gpu.status_word() == 0


@pytest.mark.parametrize("m,cluster,tiles,blocks", [(9, 1, 225, 2), (16, 3, 131, 5), (33, 8, 50, 7), (64, 6, 77, 3), (32, 0, 64, 16), (64, 0, 136, 20)])
def test_silu_mul_fused(gpu, monkeypatch, m, cluster, tiles, blocks):
    """silu(gate) * up of whole segments (lanes exchange the tokens) and of tiles cut by a share's end (summed over the cluster), with
    clusters given and as planned: one f16 step from the formula on the same launch's own gate and up."""
    if cluster:
        monkeypatch.setenv("LEXB_FEW_C", str(cluster))
    n, k = 128 * tiles, 256 * blocks
    x, wq, ws, wg = inputs.make_case(m, n, k, seed_base=740)
    q, xb = L.QBuf(gpu, wq, ws, (wg * np.float32(0.02)).astype(np.float32)), gpu.upload(x)
    pipe = gpu.plan_gemm_fp4(m, n, k)
    assert pipe.route().threads == 736 and (not cluster or pipe.route().cluster == cluster)
    act, y = gpu.alloc(m * n), gpu.alloc(4 * m * n)
    gpu.memset(act, 0xFF)
    gpu.run_silu(pipe, xb, q.wq, q.ws, q.wg, act)
    gpu.run(pipe, q.bind(xb, None, y))
    got, both = gpu.download(act, np.float16, (m, n // 2)).astype(np.float32), gpu.download(y, np.float32, (m, n))
    want = O.np_silu_mul(both[:, 0::2], both[:, 1::2], out_f16=True).astype(np.float32)
    assert np.isfinite(got).all() and np.all(np.abs(got - want) <= np.abs(want) * 2.0 ** -10 + 1e-7)
    check(both, O.gemm_fp4(x, wq, ws, (wg * np.float32(0.02)).astype(np.float32)))
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

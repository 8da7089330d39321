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

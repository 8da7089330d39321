"""Runs of matmul_q steps of several K, and of plans that split K, as one persistent launch."""
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


@pytest.fixture(autouse=True)
def every_run_is_taken(monkeypatch):
    """These lists are too narrow to pay as a run where plans split K; what a run computes is tested here, not when one is chosen."""
    monkeypatch.setenv("LEXB_CHAIN_SPLITS", "1")


@pytest.mark.parametrize("m,xf32", [(1, False), (2, True), (4, False), (5, True), (8, False)])
def test_steps_of_several_k_share_a_launch(gpu, m, xf32):
    """K of 2 to 68 stages (groups of scale bytes that end inside), plans with 1, 2 and 8 parts of K, more tiles than SMs, a
    residual, one activation buffer read with two K: each step's bits are those of its own launch."""
    shapes = [(4096, 1024), (640, 17408), (1024, 512), (640, 8192), (2048, 2048), (8192, 1024), (128, 1536)]
    ks = sorted({k for _, k in shapes})
    xs = {k: inputs.make_x(m, k, seed_base=600 + k) for k in ks}
    if xf32:
        xs = {k: v.astype(np.float32) * np.float32(1.0009765625) for k, v in xs.items()}
    xb = {k: gpu.upload(v) for k, v in xs.items()}
    sets = [inputs.make_weights(n, k, seed_base=601, copy=i) for i, (n, k) in enumerate(shapes)]
    r = np.random.Generator(np.random.PCG64(602)).standard_normal((m, 640)).astype(np.float32)
    rb = gpu.upload(r)
    xb[512] = xb[1024]                                            # the same buffer, its first half read as [m, 512]
    xs[512] = xs[1024].reshape(-1)[:m * 512].reshape(m, 512)
    pipes = [gpu.plan_matmul_fp4(m, n, k, residual=(i == 1), x_half=not xf32) for i, (n, k) in enumerate(shapes)]
    assert {p.describe().k_splits for p in pipes} >= {1, 2, 8}
    ys = [gpu.alloc(4 * m * n) for n, _ in shapes]
    binds = [L.QBuf(gpu, *w).bind(xb[k], rb if i == 1 else None, ys[i]) for i, (w, (n, k)) in enumerate(zip(sets, shapes))]
    alone = []
    for i, (n, k) in enumerate(shapes):
        gpu.run(pipes[i], binds[i])
        gpu.sync()
        alone.append(gpu.download(ys[i], np.float32, (m, n)))
        err, scale, _ = O.err_of_scale(alone[i], O.matmul_q_x(xs[k], *sets[i], r=r if i == 1 else None))
        assert scale > 1e-3 and err <= 1e-4
    steps = L.StepList(list(zip(pipes, binds)))
    assert gpu.list_runs(steps) == [len(shapes)] * len(shapes)
    for _ in range(2):
        for y in ys:
            gpu.memset(y, 0xEE)
        gpu.run_launches(steps)
        for i, (n, _) in enumerate(shapes):
            assert np.array_equal(gpu.download(ys[i], np.float32, (m, n)), alone[i]), shapes[i]
    assert gpu.status_word() == 0


def test_bad_scale_bytes_in_one_part_of_k(gpu):
    """NaN scale bytes and negative ones in different parts of a split K: that row is NaN, no other is."""
    m, n, k = 3, 640, 8192
    x = inputs.make_x(m, k, seed_base=610)
    wq, ws, wg = inputs.make_weights(n, k, seed_base=611)
    ws = ws.copy()
    for row, col, byte in ((3, 5, 0x7F), (200, k // 16 - 1, 0xFF), (639, 300, 0x7F)):
        ws[row, col] = byte
    ws[7, ::3] |= 0x80
    other = inputs.make_weights(4096, 1024, seed_base=612)
    pipe, first = gpu.plan_matmul_fp4(m, n, k), gpu.plan_matmul_fp4(m, 4096, 1024)
    assert pipe.describe().k_splits > 1
    y, ya = gpu.alloc(4 * m * n), gpu.alloc(4 * m * 4096)
    xb, x1 = gpu.upload(x), gpu.upload(inputs.make_x(m, 1024, seed_base=613))
    q = L.QBuf(gpu, wq, ws, wg)
    gpu.run(pipe, q.bind(xb, None, y))
    gpu.sync()
    alone = gpu.download(y, np.float32, (m, n))
    gpu.memset(y, 0)
    steps = [(first, L.QBuf(gpu, *other).bind(x1, None, ya)), (pipe, q.bind(xb, None, y))]
    assert gpu.list_runs(steps) == [2, 2]
    gpu.run_launches(steps)
    got = gpu.download(y, np.float32, (m, n))
    assert np.array_equal(got, alone, equal_nan=True)
    bad = np.isnan(got).any(axis=0)
    assert set(np.flatnonzero(bad)) == {3, 200, 639} and np.isnan(got[:, bad]).all()
    assert gpu.status_word() == 0


@pytest.mark.parametrize("m,k,mixed", [(4, 512, True), (3, 512, True), (8, 512, True), (4, 512, False), (1, 512, True)])
def test_bad_scale_bytes_in_later_tiles_of_few_stages(gpu, m, k, mixed):
    """Tiles of two stages, five and more of them a block: the scale warps are several tiles ahead of the epilogue, and a
    NaN scale byte still reaches its own row of its own tile and no other."""
    shapes = ([(640, 17408)] if mixed else []) + [(16384, k)] * 6
    xs = {kk: inputs.make_x(m, kk, seed_base=630) for _, kk in shapes}
    xb = {kk: gpu.upload(x) for kk, x in xs.items()}
    rng = np.random.Generator(np.random.PCG64(631))
    sets, rows = [], []
    for i, (n, kk) in enumerate(shapes):
        wq, ws, wg = inputs.make_weights(n, kk, seed_base=632, copy=i)
        bad = rng.choice(n, size=n // 100, replace=False)          # one row in a hundred: most tiles have one
        ws = ws.copy()
        ws[bad, rng.integers(0, kk // 16, size=bad.size)] = rng.choice(np.array([0x7F, 0xFF], dtype=np.uint8), size=bad.size)
        sets.append((wq, ws, wg))
        rows.append(set(bad.tolist()))
    pipes = [gpu.plan_matmul_fp4(m, n, kk) for n, kk in shapes]
    ys = [gpu.alloc(4 * m * n) for n, _ in shapes]
    binds = [L.QBuf(gpu, *w).bind(xb[kk], None, y) for w, (_, kk), y in zip(sets, shapes, ys)]
    alone = []
    for pipe, bind, y, (n, _) in zip(pipes, binds, ys, shapes):
        gpu.run(pipe, bind)
        gpu.sync()
        alone.append(gpu.download(y, np.float32, (m, n)))
    steps = L.StepList(list(zip(pipes, binds)))
    assert gpu.list_runs(steps) == [len(shapes)] * len(shapes)
    for _ in range(3):
        for y in ys:
            gpu.memset(y, 0)
        gpu.run_launches(steps)
        for i, (n, _) in enumerate(shapes):
            got = gpu.download(ys[i], np.float32, (m, n))
            assert set(np.flatnonzero(np.isnan(got).any(axis=0)).tolist()) == rows[i]
            assert np.array_equal(got, alone[i], equal_nan=True)
    assert gpu.status_word() == 0


@pytest.mark.parametrize("m,ks", [(4, (768,)), (8, (768,)), (3, (1536, 768)), (4, (1792,)), (1, (1536, 512)), (6, (1792, 768, 512))])
def test_negative_scale_bytes_in_tiles_of_few_stages(gpu, m, ks):
    """Tiles of 2, 3, 6 and 7 stages: their groups of scale bytes fill the ring before the first stages' digit rows are due, and a
    negative scale byte waits for its stage.  Signs and NaN bytes in every tile; each step's bits are those of its own launch."""
    shapes = [(16384, k) for k in ks for _ in range(3)]
    xb = {k: gpu.upload(inputs.make_x(m, k, seed_base=640)) for k in ks}
    rng = np.random.Generator(np.random.PCG64(641))
    pipes, binds, ys, rows = [], [], [], []
    for i, (n, k) in enumerate(shapes):
        wq, ws, wg = inputs.make_weights(n, k, seed_base=642, copy=i)
        ws = np.where(rng.random(ws.shape) < 0.1, ws | 0x80, ws).astype(np.uint8)
        bad = rng.choice(n, size=n // 100, replace=False)
        ws[bad, rng.integers(0, k // 16, size=bad.size)] = rng.choice(np.array([0x7F, 0xFF], dtype=np.uint8), size=bad.size)
        y = gpu.alloc(4 * m * n)
        pipes.append(gpu.plan_matmul_fp4(m, n, k))
        binds.append(L.QBuf(gpu, wq, ws, wg).bind(xb[k], None, y))
        ys.append(y)
        rows.append(set(bad.tolist()))
    alone = []
    for pipe, bind, y, (n, _) in zip(pipes, binds, ys, shapes):
        gpu.run(pipe, bind)
        gpu.sync()
        alone.append(gpu.download(y, np.float32, (m, n)))
    steps = L.StepList(list(zip(pipes, binds)))
    assert gpu.list_runs(steps) == [len(shapes)] * len(shapes)
    for y in ys:
        gpu.memset(y, 0)
    gpu.run_launches(steps)
    for i, (n, _) in enumerate(shapes):
        got = gpu.download(ys[i], np.float32, (m, n))
        assert np.array_equal(got, alone[i], equal_nan=True)
        assert set(np.flatnonzero(np.isnan(got).any(axis=0)).tolist()) == rows[i]
    assert gpu.status_word() == 0


@pytest.mark.parametrize("m", [1, 4])
def test_plans_of_other_splits_over_the_same_buffers(gpu, m):
    """A list planned with K whole and one with the planner's split, over the same buffers and in either order: each is summed as its
    own launches are."""
    shapes = [(640, 17408), (384, 8192)]
    xb = {k: gpu.upload(inputs.make_x(m, k, seed_base=650)) for _, k in shapes}
    plans = {which: [gpu.plan_matmul_fp4(m, n, k, k_splits=which) for n, k in shapes] for which in (0, 1)}
    assert all(p.describe().k_splits > 1 for p in plans[0]) and all(p.describe().k_splits == 1 for p in plans[1])
    for order in ((1, 0), (0, 1)):
        sets = [L.QBuf(gpu, *inputs.make_weights(n, k, seed_base=651, copy=i + 2 * order[0])) for i, (n, k) in enumerate(shapes)]
        ys = [gpu.alloc(4 * m * n) for n, _ in shapes]
        binds = [q.bind(xb[k], None, y) for q, (_, k), y in zip(sets, shapes, ys)]

        def results():
            return [gpu.download(y, np.float32, (m, n)) for y, (n, _) in zip(ys, shapes)]

        alone = {}
        for which in order:
            for pipe, bind in zip(plans[which], binds):
                gpu.run(pipe, bind)
            gpu.sync()
            alone[which] = results()
        assert not np.array_equal(alone[0][0], alone[1][0])        # (or the test tells nothing)
        for which in order:
            for y in ys:
                gpu.memset(y, 0xEE)
            gpu.run_launches(list(zip(plans[which], binds)))
            assert all(np.array_equal(a, b) for a, b in zip(results(), alone[which])), (order, which)


def test_lists_of_growing_activations_on_two_streams(gpu):
    """The digit rows of a run live in an arena per stream that grows with the lists: results stay right when a later list needs
    more of it, an earlier one comes again, and another stream has its own."""
    import torch
    m = 4
    lists = []
    for ks in ((1024, 2048), (1024, 2048, 8192, 512), (4096, 1024, 17408, 2048, 512)):
        steps, want = [], []
        for i, k in enumerate(ks):
            x, (wq, ws, wg) = inputs.make_x(m, k, seed_base=620 + i), inputs.make_weights(256, k, seed_base=621, copy=i)
            y = gpu.alloc(4 * m * 256)
            steps.append((gpu.plan_matmul_fp4(m, 256, k), L.QBuf(gpu, wq, ws, wg).bind(gpu.upload(x), None, y)))
            want.append((y, O.matmul_q_x(x, wq, ws, wg)))
        lists.append((steps, L.StepList(steps), want))
    other = torch.cuda.Stream()
    try:
        for stream in (None, other.cuda_stream, None):
            gpu.set_stream(stream)
            for which in (0, 1, 0, 2, 1):
                _, steps, want = lists[which]
                for y, _ in want:
                    gpu.memset(y, 0xEE)
                gpu.sync()
                gpu.run_launches(steps)
                for y, w in want:
                    err, scale, _ = O.err_of_scale(gpu.download(y, np.float32, w.shape), w)
                    assert scale > 1e-3 and err <= 1e-4
    finally:
        gpu.set_stream(None)
    assert gpu.status_word() == 0


@pytest.mark.parametrize("t,shapes,runs", [
    (4, [(640, 17408)] * 2, [1, 1]),                                               # 10 blocks of 68 stages against 40 of 9
    (1, [(512, 12800), (8704, 2816)], [1, 1]),
    (1, [(19456, 2816), (19456, 2816), (640, 17408)], [2, 2, 1]),                  # the pair goes without the long narrow one
    (1, [(640, 17408), (19456, 2816), (19456, 2816)], [1, 2, 2]),
    (2, [(1024, 4096)] * 5 + [(256, 17408)], [5] * 5 + [1]),
    (4, [(1024, 4096)] * 4, [4] * 4),
    (4, [(17408, 5120), (17408, 5120), (5120, 17408)] * 3, [9] * 9)])
def test_a_run_of_split_plans_is_taken_where_it_pays(gpu, monkeypatch, t, shapes, runs):
    """... and the results are those of the steps' own launches either way."""
    monkeypatch.delenv("LEXB_CHAIN_SPLITS")
    gen = np.random.Generator(np.random.PCG64(660))
    weights = {}
    for n, k in set(shapes):
        weights[n, k] = L.QBuf(gpu, gen.integers(0, 256, (n, k // 2), dtype=np.uint8), gen.integers(0x30, 0x48, (n, k // 16), dtype=np.uint8),
                               np.ones(n, np.float32))
    xb = {k: gpu.upload(inputs.make_x(t, k, seed_base=662)) for _, k in set(shapes)}
    ys = [gpu.alloc(4 * t * n) for n, _ in shapes]
    steps = [(gpu.plan_matmul_fp4(t, n, k), weights[n, k].bind(xb[k], None, y)) for (n, k), y in zip(shapes, ys)]
    assert gpu.list_runs(steps) == runs
    for pipe, bind in steps:
        gpu.run(pipe, bind)
    gpu.sync()
    alone = [gpu.download(y, np.float32, (t, n)) for y, (n, _) in zip(ys, shapes)]
    for y in ys:
        gpu.memset(y, 0xEE)
    gpu.run_launches(steps)
    assert all(np.array_equal(gpu.download(y, np.float32, a.shape), a) for y, a in zip(ys, alone))
    assert gpu.status_word() == 0

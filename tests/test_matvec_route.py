"""How the matvec lays a shape out over the SMs: host arithmetic, checked without a GPU."""
import random

import pytest

import lex_gpu_b200 as L
from lex_gpu_b200 import build, device


@pytest.fixture(scope="module", autouse=True)
def lib():
    build.build()


def at_once(r):
    """Row blocks of 16 that a block (a cluster) works on at a time."""
    return r.threads // 32 * r.cluster // r.parts


@pytest.mark.parametrize("m", [1, 4, 8])
@pytest.mark.parametrize("k", [64, 128, 256, 384, 512])
def test_a_short_k_keeps_its_blocks(m, k):
    """With few parts of K a block takes several row blocks at once; on a matrix of few rows that must not leave it to a
    handful of SMs, each with its whole share in a row."""
    for n in (1024, 2048, 4096, 8192):
        r = device.matvec_route(m, n, k)
        assert r.cluster == 1 and at_once(r) <= 4, (n, r.blocks)
        assert r.blocks * 4 >= min(148, n // 16) and r.groups == 1


def test_every_shape_is_covered_once():
    rng = random.Random(1)
    shapes = [(rng.randint(1, 16), 16 * rng.randint(1, 1792), 32 * rng.randint(1, 544), rng.choice([0, 0, 0, 1024, 4096])) for _ in range(400)]
    for m, n, k, kc in shapes + [(1, 16, 32, 0), (16, 16, 17408, 0), (8, 28672, 17408, 0), (16, 28672, 17408, 1024)]:
        r = device.matvec_route(m, n, k, kc)
        warps, row_blocks, slices = r.threads // 32, n // 16, -(-k // 128)
        assert r.threads in (128, 256) and r.cluster in (1, 2, 4, 8) and r.blocks % r.cluster == 0
        assert r.parts == min(8, 1 << (slices - 1).bit_length()) and r.cluster <= r.parts <= warps * r.cluster
        groups, clusters = -(-row_blocks // at_once(r)), r.blocks // r.cluster
        assert clusters * r.groups >= groups and clusters <= groups and (clusters - 1) * r.groups < groups
        assert r.kc >= k or (r.kc % 1024 == 0 and r.groups == 1)


def test_shapes_it_refuses():
    for bad in [(17, 16, 32, 0), (1, 24, 32, 0), (1, 16, 48, 0), (0, 16, 32, 0), (1, 16, 32, 512)]:
        with pytest.raises(L.LexbError):
            device.matvec_route(*bad)

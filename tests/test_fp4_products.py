"""The identity the product decode rests on (lex_gpu_b200/csrc/fp4_decode.cuh), restated in numpy: one f16 fused multiply-add
with two factors of the group gives every weight f16(f32(f32(e * s) * wg)) exactly."""
import numpy as np

F16, F32, F64 = np.float16, np.float32, np.float64


def weights(e, s, wg):
    """As the operator defines them: two roundings."""
    return ((F32(e) * s).astype(F32) * wg).astype(F32).astype(F16)


def products(e, s, wg):
    """As the kernels form them.  Every f16 step is exact or rounded once: the arithmetic here is in f64, rounded to f16."""
    A = (s * wg).astype(F32).astype(F16)
    B = ((s * F32(1.5)).astype(F32) * wg).astype(F32).astype(F16)
    pow2 = (A.view(np.uint16) & 0x7C00).view(F16)                          # u * 2^10
    diff = (A.astype(F64) * -1.5 + B.astype(F64)).astype(F16)              # one fused multiply-add
    limit = (pow2.astype(F64) * 2.0 ** -10 * 0.375).astype(F16)
    d = np.clip(diff, -limit, limit)
    base = (A.astype(F64) - pow2.astype(F64) * 2.0 ** -10).astype(F16)
    extra = (pow2.astype(F64) * 2.0 ** -10 + d.astype(F64)).astype(F16)
    low = (e * extra.astype(F64)).astype(F16)
    return (e * base.astype(F64) + low.astype(F64)).astype(F16)


def test_products_are_the_weights():
    rng = np.random.Generator(np.random.PCG64(1))
    # mantissas of the row scale: a spread of all, and those whose products fall beside a tie of the rounding to f16
    ties = (np.arange(1 << 10, dtype=np.uint32) << 13 | 0x1000)[:, None] + np.arange(-2, 3, dtype=np.int32)[None, :].astype(np.uint32)
    spread = np.arange(0, 1 << 23, 131, dtype=np.uint32)
    mantissas = np.concatenate([ties.ravel() & 0x7FFFFF, spread, rng.integers(0, 1 << 23, 20000, dtype=np.uint32)])
    edges = np.array([0, 1, 2, 0x7FFFFE, 0x7FFFFF], dtype=np.uint32)
    mantissas = np.concatenate([mantissas, edges])
    for sm in range(8):                                                    # mantissas of the block scale
        s = F32(1 + sm / 8)
        # (beside a tie of s * wg too)
        near = ((np.arange(1 << 10) + 0.5) / 1024 + 1) / float(s)
        near = near[(near >= 1) & (near < 2)].astype(F32).view(np.uint32) & 0x7FFFFF
        m = np.concatenate([mantissas, near, near - 1, near + 1]) & np.uint32(0x7FFFFF)
        for exp in (-10, -9, -1, 0, 10, 11):                               # 2^-10 <= s * wg < 2^12
            wg = (m | np.uint32((127 + exp) << 23)).view(F32)
            prod = (s * wg).astype(F32)
            wg = wg[(prod >= 2.0 ** -10) & (prod < 2.0 ** 12)]
            for e in (0.5, 1.0, 1.5, 2.0, 3.0, 4.0, 6.0):
                want, got = weights(e, s, wg), products(e, s, wg)
                assert np.array_equal(want.view(np.uint16), got.view(np.uint16)), (sm, exp, e)
                neg = products(-e, s, wg)
                assert np.array_equal(neg.view(np.uint16), want.view(np.uint16) ^ 0x8000)


def test_code_8_gives_minus_zero():
    wg = np.array([0.0, 1.0, 1.75, 3.9], dtype=F32)
    assert (products(-0.0, F32(1.0), wg).view(np.uint16) == 0x8000).all()
    assert (products(0.0, F32(1.0), wg).view(np.uint16) == 0).all()

"""The FP64 kernels' branch-free arithmetic (phys/math_fast64.cuh) against
pmp_math.h and IEEE division, bit for bit, and droplets whose arguments leave
its range (the whole sub-cycle again with the plain functions) against the
oracle."""
import numpy as np
import pytest

from pelemp_b200 import capi, spray
from pelemp_b200 import workloads as W
from tests.gpu_util import assert_bitwise, gpu_run, oracle_run

pytestmark = pytest.mark.gpu

N = 2_000_000
EXP, LOG, POW, CBRT, LOG1P, POW07, DIV, INV, NEAR1, DIVK = range(10)


def evaluate(fn, x, y=None):
    x = np.ascontiguousarray(x, np.float64)
    y = np.ones_like(x) if y is None else np.ascontiguousarray(y, np.float64)
    fast, plain, odd = np.empty_like(x), np.empty_like(x), np.empty(x.size, np.int32)
    rc = spray.lib().pmp_debug_math(fn, x.ctypes.data, y.ctypes.data, x.size, fast.ctypes.data, plain.ctypes.data,
                                    odd.ctypes.data)
    assert rc == capi.PMP_OK
    return fast, plain, odd.astype(bool)


def same(fast, plain, odd):
    return np.array_equal(fast[~odd].view(np.int64), plain[~odd].view(np.int64))


def bits(rng, n, lo, hi):
    """Doubles with random significands (often nearly all zeros or ones) and exponents in [lo, hi]."""
    m = rng.integers(0, 1 << 52, n, dtype=np.int64)
    kind = rng.integers(0, 8, n)
    few = rng.integers(0, 4, n)
    m = np.where(kind == 0, few, np.where(kind == 1, (1 << 52) - 1 - few, m))
    e = rng.integers(lo + 1023, hi + 1024, n, dtype=np.int64)
    return ((e << 52) | m).view(np.float64)


@pytest.mark.parametrize("fn,lo,hi", [(LOG, -1022, 1023), (CBRT, -100, 100), (LOG1P, -60, 60), (POW07, -60, 60),
                                      (INV, -299, 299)])
def test_functions(fn, lo, hi):
    rng = np.random.default_rng(fn)
    x = bits(rng, N, lo, hi)
    fast, plain, odd = evaluate(fn, x)
    assert same(fast, plain, odd)
    # all-ones significands, in double (INV) or single precision (the rest), are handed over
    assert odd.mean() < 0.13


def test_exp():
    rng = np.random.default_rng(1)
    x = np.concatenate([rng.uniform(-255.9, 255.9, N), rng.uniform(-1e-3, 1e-3, N), [0.0, -0.0]])
    fast, plain, odd = evaluate(EXP, x)
    assert same(fast, plain, odd) and not odd.any()
    assert evaluate(EXP, [256.0, -256.0, 1e9, np.inf, np.nan])[2].all()


def test_pow_and_zeros():
    rng = np.random.default_rng(2)
    x = np.concatenate([bits(rng, N, -60, 60), np.zeros(4)])
    for y in (0.077, 3.0):
        fast, plain, odd = evaluate(POW, x, np.full_like(x, y))
        assert same(fast, plain, odd) and not odd[-4:].any() and odd.mean() < 1e-3
    fast, plain, odd = evaluate(CBRT, np.zeros(4))
    assert same(fast, plain, odd) and not odd.any()
    assert evaluate(LOG, [0.0, -1.0, 5e-324, np.inf, np.nan])[2].all()


@pytest.mark.parametrize("fn", [DIV, NEAR1, DIVK])
def test_division(fn):
    rng = np.random.default_rng(10 + fn)
    for lo, hi in ((-1, 1), (-290, 290)):
        x, y = bits(rng, N, lo, hi), bits(rng, N, lo, hi)
        x[::97] = 0.0
        x[1::3] *= -1.0
        fast, plain, odd = evaluate(fn, x, y)
        assert np.array_equal(fast[~odd], plain[~odd])
        assert not odd.any() if fn != DIV else odd.mean() < 0.05
    if fn != DIVK:
        assert evaluate(fn, [1.0] * 6, [0.0, 5e-324, np.inf, np.nan, -1.0, 1e200])[2].all()


def test_rare_states_match_the_oracle(oracle):
    """Droplets at rest in a gas at rest, on cell planes, near the vapour
    pressure fit's pole, nearly evaporated, in vapour-rich gas."""
    prob = W.config1(n=6000, steps=2)
    st = prob.state[0]
    st[0:3] = 0.0
    st[4 + 2, :, :, 20:] = 0.3 * st[3, :, :, 20:]  # fuel vapour in part of the box
    st[4, :, :, 20:] *= 0.7
    st[5, :, :, 20:] *= 0.7
    p = prob.parts[0]
    p["rdata"][0:3, 0:1000] = 0.0
    cells = np.floor(p["pos"][:, 500:2000] / prob.dx[0])
    p["pos"][:, 500:2000] = (cells + 0.5) * prob.dx[0]
    p["rdata"][3, 2000:2200] = 56.3
    p["rdata"][4, 2200:2400] = 3e-8
    pg, _, _ = gpu_run(prob, 2)
    po, _ = oracle_run(oracle, prob, 2)
    assert_bitwise(pg, po)


@pytest.mark.parametrize("mode", [capi.PMP_MODE_FP64, capi.PMP_MODE_MIXED])
def test_gas_records_of_unusual_cells(mode, oracle):
    """Boxes whose grown cells fill no whole CTA, a third of the cells with a density whose significand
    is all ones (the division itself instead of the reciprocal), zeros among the species."""
    prob = W.config2(n=3000, steps=1, ncells=(26, 18, 14), box=(13, 18, 14))
    rng = np.random.default_rng(4)
    shape = prob.state[0].shape[1:]
    odd = rng.random((14 + 6, 18 + 6, 26 + 6)) < 1 / 3
    for (lo, _), st in zip(prob.boxes, prob.state):
        i = lo[0]  # the same cells in the overlap of the grown boxes
        m = odd[:shape[0], :shape[1], i:i + shape[2]]
        Y = st[4:9] / st[3]
        st[3] = np.where(m, np.nextafter(0.5, 0.0), st[3])
        st[4:9] = Y * st[3]
    pg, _, _ = gpu_run(prob, 1, mode=mode)
    po, _ = oracle_run(oracle, prob, 1)
    if mode == capi.PMP_MODE_FP64:
        assert_bitwise(pg, po)
    else:  # the mixed form's bound
        for a, b in zip(pg, po):
            for row in (capi.PSTATE_T, capi.PSTATE_DIA):
                assert np.max(np.abs(a["rdata"][row] / b["rdata"][row] - 1)) <= 1e-4


@pytest.mark.parametrize("fn", [DIV, NEAR1, DIVK])
def test_dividends(fn):
    """Bits of quotients over the dividends' stated range; zeros of either sign give +0."""
    rng = np.random.default_rng(20 + fn)
    for lo, hi in ((-600, -300), (300, 600)):
        x, y = bits(rng, N, lo, hi), bits(rng, N, -290, 290)
        x[1::3] *= -1.0
        assert same(*evaluate(fn, x, y))
    fast, plain, odd = evaluate(fn, [0.0, -0.0] * 64, bits(rng, 128, -290, 290))
    assert np.array_equal(fast[~odd], plain[~odd]) and not np.signbit(fast[~odd]).any()


TINY = np.array([1e-100, 1e-181, 1e-200, 1e-290, 1e-300, 1e-310, 5e-324, 0.0, -0.0])


@pytest.mark.parametrize("where", ["liquid", "gas"])
def test_tiny_fractions_match_the_oracle(where, oracle):
    """Mass fractions far below the dividends' range, subnormal, zero and -0: the droplets' bits, the
    zeros' signs among them."""
    prob = W.config2(n=6000, steps=2, ncells=(32, 16, 16), box=(16, 16, 16))
    rng = np.random.default_rng(1)
    if where == "liquid":
        for p in prob.parts:
            n = p["id"].size
            v, first = rng.choice(TINY, n), rng.integers(0, 2, n) == 0
            p["rdata"][5:7] = np.where(first, v, 1.0 - v), np.where(first, 1.0 - v, v)
    else:
        shape = prob.state[0].shape[1:]
        for s in range(5):
            tiny = rng.choice(TINY, (shape[0], shape[1], 32 + 6))
            m = rng.random(tiny.shape) < 0.3
            for (lo, _), st in zip(prob.boxes, prob.state):  # the same cells in the overlap of the grown boxes
                part = (slice(None), slice(None), slice(lo[0], lo[0] + shape[2]))
                st[4 + s] = np.where(m[part], tiny[part], st[4 + s])
    pg, _, _ = gpu_run(prob, 2)
    po, _ = oracle_run(oracle, prob, 2)
    assert_bitwise(pg, po)
    for a, b in zip(pg, po):
        assert np.array_equal(np.signbit(a["rdata"]), np.signbit(b["rdata"]))

"""The bounds that the integer-pipe quotient and root (csrc/swgpu_soft64.cuh) rest
on, in a host model of their steps (no GPU): every remainder stays in the range
that its next digit is taken from, with the hardware's estimates pushed to either
end of their error, and the result is the correctly rounded one."""
import numpy as np
import pytest

U = np.uint64
F = np.float32
SHRINK = F(0.99999952316284)  # 1 - 2^-21, as the source has it


def _lead(m):
    """The leading 24 bits of a 53-bit significand as a float in [1, 2)."""
    return (m >> U(29)).astype(np.float64).astype(F) * F(2.0 ** -23)


def _floor23(x):
    x = x.astype(np.float64)
    assert (x >= 0).all() and (x < 2 ** 23).all()
    return np.floor(x).astype(U)


def _bits23(v, at):
    assert (v >> U(at + 23) == 0).all()  # else the float loses its leading bits
    return (v >> U(at)).astype(F)


def _significands(rng, n, kind):
    m = rng.integers(1 << 52, 1 << 53, n, dtype=U)
    few = rng.integers(0, 1 << 12, n, dtype=U)
    if kind == "low":
        m = U(1 << 52) + few
    elif kind == "high":
        m = U((1 << 53) - 1) - few
    elif kind == "cut":  # the bits below the leading 24 all ones
        m = m | U((1 << 29) - 1)
    return m


@pytest.mark.parametrize("push", [-1.0, 0.0, 1.0])
@pytest.mark.parametrize("of_b", ["any", "low", "high", "cut"])
@pytest.mark.parametrize("of_a", ["any", "low", "high", "cut", "near"])
def test_quotient(of_a, of_b, push):
    rng = np.random.default_rng(3)
    n = 1 << 17
    B = _significands(rng, n, of_b)
    if of_a == "near":  # A just below B (2A near 2B: a quotient near 2) and just above
        A0 = np.clip(B.astype(np.int64) + rng.integers(-9, 9, n), 1 << 52, (1 << 53) - 1).astype(U)
    else:
        A0 = _significands(rng, n, of_a)
    # rcp.approx is within 2^-23 for an operand in [1, 2)
    r = (1.0 / _lead(B).astype(np.float64) + push * 2.0 ** -23).astype(F) * SHRINK
    small = A0 < B
    A = np.where(small, A0 + A0, A0)
    af = np.where(small, _lead(A0) * F(2), _lead(A0))
    q1 = _floor23((af * r) * F(2097152.0))
    R1 = (A << U(21)) - q1 * B
    assert (R1.astype(np.float64) < 5.0 * B.astype(np.float64)).all()
    q2 = _floor23(_bits23(R1, 33) * (r * F(2.0)))
    R2 = (R1 << U(20)) - q2 * B
    assert (R2.astype(np.float64) < 6.375 * B.astype(np.float64)).all()
    q3 = _floor23(_bits23(R2, 33) * (r * F(0.00390625)))
    R3 = (R2 << U(11)) - q3 * B
    assert (R3.astype(np.float64) < 1.02 * B.astype(np.float64)).all()
    N = (q1 << U(31)) + (q2 << U(11)) + q3
    N = N + (R3 + R3 > B).astype(U)
    # 2^52 A / B rounded: the quotient of the two as FP64 numbers, in [1, 2]
    want = A0.astype(np.float64) * np.where(small, 2.0, 1.0) / B.astype(np.float64)
    assert np.array_equal(N, (want * 2.0 ** 52).astype(U))


@pytest.mark.parametrize("push", [-1.0, 0.0, 1.0])
@pytest.mark.parametrize("odd", [False, True])
@pytest.mark.parametrize("of_x", ["any", "low", "high", "cut"])
def test_root(of_x, odd, push):
    rng = np.random.default_rng(4)
    X0 = _significands(rng, 1 << 17, of_x)
    X = X0 + X0 if odd else X0
    xf = _lead(X0) * F(2 if odd else 1)
    # rsqrt.approx is within 2^-22.9 relative
    y = (1.0 / np.sqrt(xf.astype(np.float64)) * (1.0 + push * 2.0 ** -22.9)).astype(F) * SHRINK
    s1 = _floor23((xf * y) * F(2097152.0))
    R1 = X - (s1 * s1 << U(10))
    est = _bits23(R1, 13) * (y + y)
    # (fmaf: one rounding)
    e = est.astype(np.float64)
    s2 = _floor23((e + (est * est).astype(np.float64) * float(F(-2.2737368e-13))).astype(F))
    R2 = (R1 << U(30)) - (s1 * s2 << U(21)) - s2 * s2
    s3 = _floor23(_bits23(R2, 26) * (y * F(0.03125)))
    R3 = (R2 << U(22)) - (s1 * s3 << U(32)) - (s2 * s3 << U(12)) - s3 * s3
    S = (s1 << U(31)) + (s2 << U(11)) + s3
    signed = R3.view(np.int64)
    N = S + (signed > S.view(np.int64)).astype(U) + (signed > (3 * S + U(2)).view(np.int64)).astype(U)
    want = np.sqrt(X0.astype(np.float64) * (2.0 if odd else 1.0) * 2.0 ** -52)
    assert np.array_equal(N, (want * 2.0 ** 52).astype(U))

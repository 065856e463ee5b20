"""The normalisation that the GPU's kernels call (three quotients of one
reciprocal) against correctly rounded division, bit for bit: random
significands, the pairs whose quotient lies closest to a rounding boundary,
components and lengths on either side of the limits where it divides plainly,
signed zeros, tiny components, no length. Needs a B200."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _bits(a):
    return np.ascontiguousarray(a, np.float32).view(np.uint32)


def _check_quotients(ctx, xyz, s):
    xyz, s = np.asarray(xyz, np.float32).reshape(-1, 3), np.asarray(s, np.float32)
    _, q = ctx.normalize(xyz, s)
    want = xyz / s[:, None]  # IEEE division: correctly rounded
    bad = np.nonzero((_bits(q) != _bits(want)).any(1))[0]
    assert bad.size == 0, (bad.size, xyz[bad[:4]], s[bad[:4]], q[bad[:4]], want[bad[:4]])


def test_random_significands(ctx):
    rng = np.random.default_rng(1)
    n = 4_000_000
    s = np.ldexp(rng.integers(1 << 23, 1 << 24, n).astype(np.float64), rng.integers(-60 - 23, 60 - 23, n)).astype(np.float32)
    m = rng.integers(1 << 23, 1 << 24, (n, 3)) * rng.choice([-1, 1], (n, 3))
    x = np.ldexp(m.astype(np.float64), np.log2(s).astype(int)[:, None] - 25 - rng.integers(0, 30, (n, 3)))
    _check_quotients(ctx, x, s)


def _next_to_midpoints(d, below_one):
    """(m, s): m / s, in [1/2, 1) or [1, 2), within d / s of a midpoint K / 2^b of
    two floats (K odd, 25 bits): m 2^b = K s + d. An odd s has one K modulo 2^b for
    odd d; d = +-2 takes an even s and halves the equation."""
    bits = 25 if below_one else 24
    s = np.arange((1 << 23) + 1, 1 << 24, 2, dtype=np.int64)
    if d % 2 == 0:
        s, d, bits = np.arange((1 << 22) + 1, 1 << 23, 2, dtype=np.int64), d // 2, bits - 1
    mod = (1 << bits) - 1
    inv = s.copy()  # Newton's iteration for 1 / s modulo 2^bits
    for _ in range(5):
        inv = (inv * (2 - (s * inv & mod))) & mod
    ms, ss = [], []
    for base in range(0, 1 << 25, 1 << bits):
        k = (-d * inv & mod) + base
        m = (k * s + d) >> bits
        ok = (k % 2 == 1) & (k >= 1 << 24) & (m < 1 << 24)
        ms.append(m[ok])
        ss.append(s[ok] << (0 if s[0] > 1 << 23 else 1))
    return np.concatenate(ms), np.concatenate(ss)


@pytest.mark.parametrize("below_one", [False, True])
@pytest.mark.parametrize("d", [-3, -2, -1, 1, 2, 3])
def test_quotients_next_to_a_rounding_boundary(ctx, d, below_one):
    m, s = _next_to_midpoints(d, below_one)
    assert m.size > 1_000_000
    x = m.astype(np.float64) / 4  # powers of two keep significands; no component above the length
    _check_quotients(ctx, np.stack([x, -x, x / 4096], 1), s)


def test_limits_zeros_and_tiny_components(ctx):
    rng = np.random.default_rng(2)
    x, s = [], []
    for e in list(range(-126, 128)):
        for _ in range(40):
            sl = np.float32(np.ldexp(rng.uniform(0.5, 1.0), e))
            # components from the length down to the smallest subnormal
            f = np.ldexp(rng.uniform(-1, 1, 3), -rng.integers(0, 160, 3))
            c = (sl.astype(np.float64) * f).astype(np.float32)
            c[rng.integers(0, 3)] = rng.choice([0.0, -0.0, c[0]])
            x.append(c)
            s.append(sl)
    edge = [2.0 ** -60, 2.0 ** 60, 2.0 ** -100, 2.0 ** -126, 2.0 ** -149]
    for a in edge:
        for up in (np.float32(a), np.nextafter(np.float32(a), np.float32(np.inf)), np.nextafter(np.float32(a), np.float32(0))):
            for b in edge + [1.0, 2.0 ** 100]:
                if np.float32(b) >= up and up > 0:
                    x.append(np.float32([up, -up, 0.0]))
                    s.append(np.float32(b))
    _check_quotients(ctx, np.stack(x), np.array(s))


def test_normalised_vectors(ctx):
    rng = np.random.default_rng(3)
    v = (rng.normal(size=(200_000, 3)) * np.exp(rng.uniform(-20, 20, (200_000, 1)))).astype(np.float32)
    v[::7, 0], v[::11, 1], v[::13, 2] = 0.0, -0.0, 1e-25
    u, _ = ctx.normalize(v, np.abs(v).max(1) * 2)
    w = v.astype(np.float64)
    length = np.sqrt((w * w).sum(1, keepdims=True))
    far = length[:, 0] > 2.0 ** -60  # its square is a normal number
    assert far.sum() > 199_000
    # three roundings in the sum (halved by the root), one each of root and quotient
    assert (np.abs(u - w / length) <= (0.5 * 1.5 + 0.5 + 0.5) * 2.0 ** -23 * np.abs(w / length) * 1.01)[far].all()
    assert np.array_equal(np.signbit(u)[far], np.signbit(v)[far])
    none, _ = ctx.normalize(np.zeros((1, 3)), np.ones(1))
    assert np.isnan(none).all()  # 0 / 0, as the reference's division

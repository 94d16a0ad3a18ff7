"""The zero counts of the panel expansions' blocks (panel.cu), on the CPU against
the row recurrence.

n2, the sign changes in a block of the solution that starts with u = 0, is
counted at the panel's centre and corrected by one where the sign of the entry
T12 asks for it.  That is right while at most one level of the block (a zero of
T12) lies on either side of the centre, and a block is counted by its rows
unless this is certain: the rows vary by at most 16 / B^2 over the block, or the
sign variations of T12's Taylor coefficients (Budan's theorem) leave it no
second root, or the counts at the panel's ends differ from the centre's by at
most one.  Two wells with a barrier between them have levels in pairs."""
import numpy as np
import pytest

RHO, FLAT, D = 10.0, 16.0, 14


def _zeros(s, x):
    """sign changes and whether T12 is negative, for shifts x"""
    x = np.atleast_1d(x)
    u, e, n, prev = np.zeros_like(x), np.ones_like(x), np.zeros(len(x), int), np.zeros(len(x), bool)
    for v in s:
        e = e - (v + 2.0 - x) * u
        u = u + e
        n += (u < 0) != prev
        prev = u < 0
    return n, prev


def _t12(s, xc, r):
    u, e = np.zeros(D + 1), np.zeros(D + 1)
    e[0] = 1.0
    for v in s:
        f = e - (v + 2.0 - xc) * u
        f[1:] += r * u[:-1]
        e, u = f, u + f
    return u


def _variations(c):
    return int(np.sum((c[1:] < 0) != (c[:-1] < 0)))


def _shifted(c, h):
    c = c.copy()
    for i in range(D):
        for j in range(D - 1, i - 1, -1):
            c[j] += h * c[j + 1]
    return c


def _by_rows(s, xc, r):
    B = len(s)
    if (s.max() - s.min()) * B * B <= FLAT:
        return False
    c = _t12(s, xc, r)
    v = _variations(c)
    if _variations(_shifted(c, -1.0)) - v <= 1 and v - _variations(_shifted(c, 1.0)) <= 1:
        return False
    n = _zeros(s, [xc - r, xc, xc + r])[0]
    return n[0] > n[1] + 1 or n[2] < n[1] - 1


def _centre_rule(s, xc, r, t):
    """n2 at xc + r t from that at the centre and the sign of T12 there"""
    n2 = _zeros(s, xc)[0][0]
    odd = _zeros(s, xc + r * t)[1]
    return np.where(odd != bool(n2 & 1), n2 + np.where(t > 0, -1, 1), n2)


def _blocks(B):
    i = np.arange(B)
    yield "even", np.full(B, -2.0 + 0.3)
    yield "ramp", -2.0 + 0.02 * i / B
    for a in (0.0005, 0.02, 0.2):
        for waves in (1, 2, 3, 5):
            yield "waves %g %d" % (a, waves), -2.0 + a * np.cos(2 * np.pi * waves * (i - 0.25 * B) / B)
    rng = np.random.default_rng(B)
    for a in (1e-3, 0.05):
        yield "layers %g" % a, -2.0 + a * np.repeat(rng.uniform(-1, 1, B // 8), 8)


@pytest.mark.parametrize("B", [16, 32, 64, 128])
def test_counts_within_a_panel(B):
    r = RHO / B ** 2
    t = np.linspace(-1.0, 1.0, 41)
    for name, s in _blocks(B):
        for xc in np.linspace(-0.5 * r, (s.max() + 2.0) + 2 * r, 60):
            if not _by_rows(s, xc, r):
                want, got = _zeros(s, xc + r * t)[0], _centre_rule(s, xc, r, t)
                assert np.array_equal(got, want), (name, xc, got - want)


def test_two_wells():
    """128 rows, a barrier in their middle: the centre's rule is wrong by two in
    panels that hold a pair of levels on one side of the centre, and each of
    them is counted by its rows"""
    i = np.arange(128)
    s = -2.0 + 0.02 * np.cos(2 * np.pi * (i - 32) / 64)
    r = RHO / 128 ** 2
    t = np.linspace(-1.0, 1.0, 41)
    wrong = 0
    for xc in np.linspace(-0.02, 0.03, 200):
        off = _centre_rule(s, xc, r, t) - _zeros(s, xc + r * t)[0]
        if np.any(off):
            wrong += 1
            assert set(np.abs(off)) <= {0, 2} and _by_rows(s, xc, r)
    assert wrong > 0

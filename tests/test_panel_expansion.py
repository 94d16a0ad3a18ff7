"""The identities behind the panel expansions of the eigen-solve (panel.cu), on
the CPU against the row recurrence.

For rows sigma_i = s_i + 2 - x the state (u, e) obeys e_i = e_{i-1} - sigma_i
u_{i-1}, u_i = u_{i-1} + e_i.  The 2 x 2 matrix of a block of B rows is expanded
in x = xc + r t to degree 14 with r B^2 <= 10, and

- the product of the block matrices gives the determinant u_{n-1} and its
  derivatives as the rows do;
- nz minus the sign changes counted per block (the zeros n2 of the solution that
  starts with u = 0, counted at the centre and corrected by the sign of the
  entry T12, plus the parity of the block's ends) is the Sturm count;
- the derivative chains give the weighted sums of squares through u e_eps - e
  u_eps = -sum W_i u_{i-1}^2.

Tolerances: the term left out is at most rho^15 / 30! = 4e-18 of an entry; over
n rows the recurrences themselves round to about n eps = 2e-13 for n = 1000."""
import numpy as np
import pytest

D, DW, RHO = 14, 11, 10.0


def _expand(s, w, a, b, xc, r):
    T, V, n2 = np.zeros((D + 1, 2, 2)), np.zeros((DW + 1, 2, 2)), 0
    for col in (0, 1):
        u, e = np.zeros(D + 1), np.zeros(D + 1)
        v, f = np.zeros(DW + 1), np.zeros(DW + 1)
        (u if col == 0 else e)[0] = 1.0
        prev = False
        for i in range(a, b):
            sg = s[i] + 2.0 - xc
            f = f - sg * v - w[i] * u[:DW + 1]
            f[1:] += r * v[:-1]
            e = e - sg * u
            e[1:] += r * u[:-1]
            u, v = u + e, v + f
            if col:
                n2 += (u[0] < 0) != prev
                prev = u[0] < 0
        T[:, 0, col], T[:, 1, col], V[:, 0, col], V[:, 1, col] = u, e, v, f
    return T, V, n2


def _at(c, t):
    return np.polynomial.polynomial.polyval(t, c.transpose(0, 1, 2))


@pytest.mark.parametrize("n", [5, 127, 128, 129, 255, 512, 1000])
@pytest.mark.parametrize("amp", [2e-4, 3e-2, 0.4])
def test_block_matrices_against_rows(n, amp):
    rng = np.random.default_rng(n)
    z = np.linspace(0.0, 1.0, n)
    s = -2.0 + amp * (0.6 + 0.4 * np.cos(7.0 * z + rng.uniform(0, 6)) + 0.1 * np.sin(31.0 * z))
    w = np.exp(8.0 * z)
    lo, hi = 0.1 * amp, 1.1 * amp
    xc, r = 0.5 * (lo + hi), 0.5 * (hi - lo)
    B = 128
    while B > 1 and r * B * B > RHO:
        B //= 2
    assert r * B * B <= RHO
    blocks = [_expand(s, w, a, min(n, a + B), xc, r) for a in range(0, n, B)]
    for t in (-1.0, -0.7, -0.01, 0.0, 0.3, 0.999, 1.0):
        x = xc + r * t
        # rows, with d/dx, the sign changes and the sum of w u^2; blocks beside
        # them; both rescaled by the same powers of two after every block
        u, e, u1, e1, zeros, acc = 1.0, 1.0, 0.0, 0.0, 0, 0.0
        y, y1, yw, zb = np.array([1.0, 1.0]), np.zeros(2), np.zeros(2), 0
        for k, (T, V, n2) in enumerate(blocks):
            for i in range(k * B, min(n, (k + 1) * B)):
                sg = s[i] + 2.0 - x
                acc += w[i] * u * u
                e1, e = e1 - sg * u1 + u, e - sg * u
                un, u1 = u + e, u1 + e1
                zeros += (un < 0) != (u < 0)
                u = un
            m, d, v = _at(T, t), _at(np.arange(1, D + 1)[:, None, None] * T[1:], t) / r, _at(V, t)
            yn = m @ y
            y1, yw = m @ y1 + d @ y, m @ yw + v @ y
            if (m[0, 1] < 0) != bool(n2 & 1):
                n2 += -1 if t > 0 else 1
            zb += n2 + ((n2 & 1) != ((y[0] < 0) != (yn[0] < 0)))
            y = yn
            sc = 2.0 ** -np.floor(np.log2(max(abs(u), abs(e), abs(u1), abs(e1))))
            u, e, u1, e1, acc = u * sc, e * sc, u1 * sc, e1 * sc, acc * sc * sc
            y, y1, yw = y * sc, y1 * sc, yw * sc
        big = max(abs(u), abs(e))
        assert abs(y[0] - u) <= 1e-11 * big and abs(y[1] - e) <= 1e-11 * big, (t, y, u, e)
        assert np.max(np.abs(y1 - [u1, e1])) <= 1e-10 * max(abs(u1), abs(e1)), (t, y1, u1, e1)
        assert zb == zeros, (t, zb, zeros)
        got = y[1] * yw[0] - y[0] * yw[1]
        assert abs(got - acc) <= 1e-8 * abs(acc), (t, got, acc)

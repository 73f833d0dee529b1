"""Coefficients of the P and Q functions of H_0 and H_1 (Abramowitz & Stegun 9.2.5-9.2.6) at
x >= 8, as polynomials in z = (8/x)^2, for pytential_b200/csrc/helmholtz.cuh:

    python tests/golden/make_hankel_pq.py

From the integral that defines them, with u = v^2 in Poisson's integral for H_nu,
    P_nu + i Q_nu = (2 / sqrt(pi)) int_0^inf e^(-v^2) g_nu(1 + i v^2 / (2 x)) dv * (1 or 2 v^2),
    g_0(s) = s^(-1/2), g_1(s) = s^(1/2),
by the midpoint rule (exponentially convergent: the nearest singularity is 2.8 off the real
axis) in extended precision, then Chebyshev interpolation in z (Clenshaw, Chebyshev Series
for Mathematical Functions, 1962, tabulates the same expansions) cut at degree 12, where the
next term is below 2e-17, as powers of z.
"""

import numpy as np

TERMS = 13
L = np.longdouble
PI = L(4) * np.arctan(L(1))


def pq(nu, x):
    """(P_nu, Q_nu) at an array x >= 8, extended precision."""
    x = np.asarray(x, L)
    h = L(1) / 16
    v = (np.arange(128, dtype=L) + L(1) / 2) * h
    root = np.sqrt(1 + 1j * ((v ** 2)[None] / (2 * x[:, None])).astype(np.clongdouble))
    f = 1 / root if nu == 0 else root * (2 * v ** 2)
    s = (2 / np.sqrt(PI)) * (f * (np.exp(-v ** 2) * h)).sum(1)
    return s.real, s.imag


def coefficients():
    """{"P0", "Q0", "P1", "Q1": TERMS powers of z}; Q_nu = (8 / x) times its polynomial."""
    n = 24
    k = np.arange(n, dtype=L) + L(1) / 2
    t = np.cos(PI * k / n)
    x = 8 / np.sqrt((t + 1) / 2)
    out = {}
    for nu in (0, 1):
        P, Q = pq(nu, x)
        for name, f in ((f"P{nu}", P), (f"Q{nu}", Q * x / 8)):
            c = [(2 / L(n)) * (f * np.cos(PI * j * k / n)).sum() for j in range(TERMS)]
            c[0] /= 2
            # T_j(2 z - 1) by their recurrence in powers of z
            line = np.array([L(-1), L(2)])
            T = [np.array([L(1)]), line]
            while len(T) < TERMS:
                a = 2 * np.convolve(line, T[-1])
                a[:len(T[-2])] -= T[-2]
                T.append(a)
            m = np.zeros(TERMS, L)
            for cj, Tj in zip(c, T):
                m[:len(Tj)] += cj * Tj
            out[name] = m.astype(np.float64)
    return out


if __name__ == "__main__":
    for name, c in coefficients().items():
        print(f"    {{  // {name}")
        for i in range(0, TERMS, 4):
            print("     " + " ".join(f"{v:.17g}," for v in c[i:i + 4]))
        print("    },")

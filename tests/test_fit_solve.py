"""The offset fit's normal equations, solved by the device code compiled for the CPU, against rational arithmetic:
well spread points, points near a line, and points in a corner with a few far ones.  Where the cofactor form answers,
twelve roundings of values up to the largest offset (5), divided by the smallest determinant it takes (0.3 of the
diagonal's product), bound what it may add to elimination's error: 12 * 2^-53 * 5 / 0.3 = 2.2e-14."""
import os
import subprocess
from fractions import Fraction

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "gmtsar-gpu_gb300", "csrc")
MAIN = r"""
#include <stdio.h>
#include "fit_solve.cuh"
int main() {
    double S[9], c[3], q[3];
    int np;
    while (scanf("%d", &np) == 1) {
        for (int k = 0; k < 9; k++) if (scanf("%la", &S[k]) != 1) return 1;
        xcg::fit_solve(S, np, c);
        xcg::fit_solve_regular(S, np, q);
        printf("%a %a %a %a %a %a\n", c[0], c[1], c[2], q[0], q[1], q[2]);
    }
}
"""


def _exact(S, npar):
    M = [[S[0], S[1], S[2]], [S[1], S[3], S[4]], [S[2], S[4], S[5]]]
    A = [[Fraction(M[i][j]) for j in range(npar)] + [Fraction(S[6 + i])] for i in range(npar)]
    for k in range(npar):
        p = max(range(k, npar), key=lambda i: abs(A[i][k]))
        A[k], A[p] = A[p], A[k]
        for i in range(k + 1, npar):
            f = A[i][k] / A[k][k]
            A[i] = [a - f * b for a, b in zip(A[i], A[k])]
    c = [Fraction(0)] * 3
    for k in range(npar - 1, -1, -1):
        c[k] = (A[k][npar] - sum(A[k][j] * c[j] for j in range(k + 1, npar))) / A[k][k]
    return c


@pytest.mark.parametrize("npar,kind", [(3, "spread"), (3, "diagonal"), (3, "corner"), (2, "spread"), (2, "corner")])
def test_no_less_accurate_than_elimination(tmp_path, npar, kind):
    (tmp_path / "m.cpp").write_text(MAIN)
    exe = str(tmp_path / "m")
    subprocess.run(["g++", "-O2", "-ffp-contract=off", "-I" + CSRC, str(tmp_path / "m.cpp"), "-o", exe], check=True)
    r = np.random.default_rng(npar * 100 + len(kind))
    systems = []
    for t in range(120):
        n, width = int(r.integers(20, 400)), 10.0 ** r.uniform(-6.5, 0)
        u, v = r.uniform(-1, 1, (2, n))
        if kind == "diagonal":
            v = np.clip(u + width * v, -1, 1)
        if kind == "corner":
            far = r.random(n) < 0.03
            u, v = np.where(far, u, 0.9 + 0.1 * width * u), np.where(far, v, -0.9 + 0.1 * width * v)
        w = r.uniform(0, 1, n) if t % 2 else np.ones(n)
        o = 3 + 0.5 * u - 0.7 * v + 0.1 * r.standard_normal(n)
        S = [float(x) for x in (w.sum(), (w * u).sum(), (w * v).sum(), (w * u * u).sum(), (w * u * v).sum(),
                                (w * v * v).sum(), (w * o).sum(), (w * u * o).sum(), (w * v * o).sum())]
        systems.append((S, u, v))
    text = "\n".join(f"{npar} " + " ".join(x.hex() for x in S) for S, _, _ in systems)
    out = subprocess.run([exe], input=text, capture_output=True, text=True, check=True).stdout.split("\n")
    for (S, u, v), line in zip(systems, out):
        got, want = [float.fromhex(x) for x in line.split()], _exact(S, npar)

        def off(c):                           # the worst fitted offset's error
            d = [float(Fraction(c[k]) - want[k]) for k in range(3)]
            return np.abs(d[0] + d[1] * u + d[2] * v).max()
        assert off(got[3:]) <= off(got[:3]) + 2.2e-14

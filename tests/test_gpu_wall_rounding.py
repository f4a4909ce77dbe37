"""The wall pressure of a moving wall, bit for bit.

With a wall at rest the products of its velocity vanish and its pressure is the same however they
are rounded; with a wall that moves (F != 0, time-accurate) the roundings show, and the pressure
solve amplifies them. They are part of the step's definition: the formula is evaluated here from the
planes of the finished step, every product rounded or melted into a sum (one exact rounding, by
rational arithmetic) as the kernels do. The device's sine may differ from the host's by an ulp;
all columns must agree for the same one.
"""
import math
from fractions import Fraction

import numpy as np
import pytest

from cfd_solver_b200.grid import ogrid

pytestmark = pytest.mark.gpu


def fma(a, b, c):
    return float(Fraction(a) * Fraction(b) + Fraction(c))


def wall_pressure(g, Re, Ri, F, swall, U, V, T, P):
    W, d0, d1 = g.n0 - 1, 1.0 / (g.n0 - 1), 1.0 / (g.n1 - 1)
    speed = math.pi / 12.0 * 2.0 * math.pi * F
    acc = 2.0 * math.pi * F * speed * swall
    out = np.empty(W)
    for i in range(W):
        e, w = (i + 1) % W, (i - 1) % W
        x, y, J = float(g.xix[0, i]), float(g.xiy[0, i]), float(g.jac[0, i])
        u, v = float(U[0, i]), float(V[0, i])
        uxi = fma(x, u, y * v)
        uet = fma(float(g.etx[0, i]), u, float(g.ety[0, i]) * v)
        t = []
        for f in (U, V):
            fe, fw, f0, f1, f2 = (float(f[0, e]), float(f[0, w]), float(f[0, i]), float(f[1, i]), float(f[2, i]))
            aa = float(g.alph[0, i]) * ((fe + fw) - 2 * f0) / (d0 * d0)
            gg = float(g.gam[0, i]) * ((f0 + f2) - 2 * f1) / (d1 * d1)
            bb = float(g.beta[0, i]) * (((float(f[1, e]) + fw) - float(f[1, w])) - fe) / (2 * d0 * d1)
            cv = uxi * 0.5 * (fe - fw) / d0 + uet * (f1 - f0) / d1
            t.append(((aa + gg) - 2 * bb) / Re - cv)
        fu = t[0] - acc * float(g.y[0, i])
        fv = fma(Ri, float(T[0, i]), fma(acc, float(g.x[0, i]), t[1]))
        s = fma(fv, x * J, fu * (-y * J))
        out[i] = fma(-s, d1, float(P[1, i]))
    return out


@pytest.mark.parametrize("host", [False, True])
@pytest.mark.parametrize("n0,n1,skew,F,Re", [(33, 25, 0.1, 0.7, 100.0), (65, 49, 0.2, 5.0, 100.0), (24, 9, 0.0, 5.0, 1.0),
                                             (90, 40, 0.2, 5.0, 1000.0), (113, 70, 0.1, 0.7, 1.0)])
def test_wall_pressure_of_a_moving_wall(n0, n1, skew, F, Re, host):
    from cfd_solver_b200.solver import Batch, case_params
    g = ogrid(n0, n1, skew=skew)
    with Batch([g], [case_params(g, Re=Re, Ri=1.0, dt=1e-2, F=F, time_accurate=1)]) as b:
        b.profile(host)
        for _ in range(3):
            b.step(1)
            U, V, T, P = (b.plane(0, k) for k in ("u", "v", "T", "p"))
            s = math.sin(2.0 * math.pi * F * b.stats(0)["time"])
            wrong = [np.count_nonzero(wall_pressure(g, Re, 1.0, F, q, U, V, T, P) != P[0, :n0 - 1])
                     for q in (s, np.nextafter(s, 2.0), np.nextafter(s, -2.0))]
            assert min(wrong) == 0, wrong

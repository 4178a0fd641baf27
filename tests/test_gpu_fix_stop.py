"""The iteration at which a gauge fixing stops: the first one whose theta is at
or below the limit, whether the check is made by the next iteration's first
half-step (up to 512 theta partials) or by a kernel of its own, and wherever
in a batch of 8, 16, ... iterations that iteration lies."""
import ctypes as C

import numpy as np
import pytest

from lceqcd_b200 import Lattice, _lib
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu

COUP = dict(beta=12.0, x=0.09, y=0.3, lam=1.7, seed=4, precision="f64")
ITGF = _lib.LCE_ITGF_FIX_COMPONENT | _lib.LCE_ITGF_ASCEND
# in the first batch (1-8), on its last iteration, in the second (9-24), on its last, in the third
STOPS = (1, 2, 7, 8, 9, 16, 23, 24, 25)


def fix(g, form, cap):
    """theta and iterations of a fixing, converged or not."""
    th, it = C.c_double(), C.c_int()
    if form == "plain":
        rc = g.lib.lce_landau_gauge(g.h, 0, C.byref(th), C.byref(it), cap)
    elif form == "tracked":
        rc = g.lib.lce_landau_gauge_from(g.h, 0, _lib.LCE_GF_START_IDENTITY, None, C.byref(th), C.byref(it), cap)
    else:
        rc = g.lib.lce_it_landau_gauge(g.h, 0, 0.2, ITGF, C.byref(th), C.byref(it), cap)
    assert rc in (0, _lib.LCE_ERR_GF_NOT_CONVERGED)
    return th.value, it.value, rc == 0


def configuration(L):
    g = Lattice(L, **COUP)
    g.init_hot(2)
    g.sweeps(3, 0)
    u, a = g.download()
    g.close()
    return u, a


# sites per parity: 480; 8448 (blocks of 256); 131072 (512 partials); 135168 (528: a check kernel); 262144; 266240
@pytest.mark.parametrize("L", [(12, 10, 8), (32, 44, 12), (64, 64, 64), (64, 64, 66), (64, 64, 128), (64, 64, 130)])
@pytest.mark.parametrize("form", ["plain", "tracked", "iterative"])
def test_stops_at_the_first_theta_within_the_limit(L, form):
    u, a = configuration(L)
    g = Lattice(L, limit_or=1e-30, **COUP)
    g.upload(u, a)
    theta = []  # after 1, 2, ... iterations
    for n in range(1, max(STOPS) + 4):
        th, it, ok = fix(g, form, n)
        assert not ok and it == n
        theta.append(th)
    g.close()
    for k in STOPS:
        for limit in (theta[k - 1] * (1 + 1e-9), theta[k - 1] * (1 - 1e-9)):
            want = next((j for j, th in enumerate(theta, 1) if th <= limit), None)
            assert want != k if limit < theta[k - 1] else want is not None and want <= k
            if want is None:
                continue
            h = Lattice(L, limit_or=limit, **COUP)
            h.upload(u, a)
            assert fix(h, form, 1000) == (theta[want - 1], want, True), (k, limit)
            h.close()


@pytest.mark.parametrize("form", ["plain", "iterative"])
def test_thetas_and_stops_are_the_oracles(form):
    """Iteration by iteration against the oracle's own loop (FP64 on both sides:
    theta within the tolerance of the converged comparisons, 1e-8)."""
    L = (12, 10, 8)
    u, a = configuration(L)
    g = Lattice(L, limit_or=1e-30, **COUP)
    g.upload(u, a)
    o = Oracle(L, COUP["beta"], COUP["x"], COUP["y"], lam=COUP["lam"], limit_or=1e-30)
    theta = []
    for n in range(1, 28):
        o.set_fields(np.asarray(u, np.float64), np.asarray(a, np.float64))
        da1, it = o.landau_gauge(max_iters=n) if form == "plain" else o.it_landau_gauge(0.2, 3, max_iters=n)
        th, itg, _ = fix(g, form, n)
        assert it == itg == n and abs(th - da1) <= 1e-8 * da1
        theta.append(da1)
    g.close()
    for k in STOPS:
        want = next(j for j, th in enumerate(theta, 1) if th <= theta[k - 1])
        h = Lattice(L, limit_or=theta[k - 1] * (1 + 1e-7), **COUP)
        h.upload(u, a)
        assert fix(h, form, 1000)[1:] == (want, True), k
        h.close()

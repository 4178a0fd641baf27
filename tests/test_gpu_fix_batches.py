"""Gauge fixings whose iterations are checked by the next one's first half-step
(up to 1024 theta partials), by a check kernel of their own, and with blocks of
128 and 256 threads: batches of 8, 16, ... iterations must count and stop as
single ones do."""
import numpy as np
import pytest

from lceqcd_b200 import Lattice, LceError

pytestmark = pytest.mark.gpu

COUP = dict(beta=12.0, x=0.09, y=0.3, lam=1.7, seed=4)


# sites per parity: 4; 480; 8192 and 8448 (block edge); 262144 and 264192 (partials edge)
@pytest.mark.parametrize("L", [(2, 2, 2), (12, 10, 8), (32, 32, 16), (32, 44, 12), (64, 64, 128), (64, 64, 130)])
@pytest.mark.parametrize("form", ["plain", "tracked", "iterative"])
def test_cap_and_stop_between_batches(L, form):
    def fix(g, n):
        f = {"plain": lambda: g.landau_gauge(max_iters=n), "tracked": lambda: g.landau_gauge_from("identity", max_iters=n),
             "iterative": lambda: g.it_landau_gauge(0.2, fix_component=True, ascend=True, max_iters=n)}[form]
        try:
            return f()[-1], True
        except LceError:
            return n, False
    g = Lattice(L, limit_or=1e-30, precision="f64", **COUP)
    g.init_hot(2)
    g.sweeps(3, 0)
    u, a = g.download()
    for n in (1, 7, 8, 9, 25):  # within, at and after the first batches' ends
        it, ok = fix(g, n)
        assert not ok and it == n
        if form == "plain" and n == 9:
            # 8 iterations and one more give the same field
            g2 = g.download(which=1)
            fix(g, 8)
            with pytest.raises(LceError):
                g.gauge_fix_continue(max_iters=1)
            g3 = g.download(which=1)
            assert np.array_equal(g2[0], g3[0]) and np.array_equal(g2[1], g3[1])
    theta = g.theta()
    g.close()
    # the count at a limit: the first iteration whose theta is at or below it,
    # whichever batch it falls in (the check takes theta before the iteration's
    # last half-step, theta() after it, so the count is not 25's)
    h = Lattice(L, limit_or=float(theta), precision="f64", **COUP)
    h.upload(u, a)
    it, ok = fix(h, 400)
    assert ok and it >= 1
    hu, ha = h.download(which=1)
    h.close()
    k = Lattice(L, limit_or=1e-30, precision="f64", **COUP)
    k.upload(u, a)
    assert fix(k, it) == (it, False)
    ku, ka = k.download(which=1)
    assert np.array_equal(hu, ku) and np.array_equal(ha, ka)
    k.close()

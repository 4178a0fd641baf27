"""Runs of sweeps with up to 64 reduction slots each (the most a composition may
have) through graphs of 8 sweeps, whose finalizes but the last run in a block of
the next sweep's first pass: every slot of every sweep must count, so fields,
step, measurements and status equal those of single sweeps bit for bit."""
import numpy as np
import pytest

from lceqcd_b200 import Lattice

pytestmark = pytest.mark.gpu


# slots: 34 (the first count past 32 of a block of 128 threads), 36, 50 and 64;
# the ahiggs1 slots of 20 and 27 calls reach past the 32nd, so that the step of
# the next sweep depends on them; lattices of one chunk and of several
@pytest.mark.parametrize("n_link_or,n_higgs_metro", [(4, 0), (4, 1), (0, 20), (0, 27), (9, 0)])
@pytest.mark.parametrize("L,precision,threads", [
    ((8, 8, 8), "f32", 128), ((40, 32, 30), "f32", 128), ((40, 32, 30), "f32", 256), ((64, 40, 32), "f32", 448),
    ((64, 40, 32), "f32", 512), ((8, 8, 8), "f64", 0), ((24, 24, 24), "f64", 0), ((32, 24, 30), "f64", 0)])
def test_graphs_of_sweeps_equal_single_sweeps(L, precision, threads, n_link_or, n_higgs_metro):
    par = dict(beta=9.0, x=0.1, y=0.45, seed=31, precision=precision, n_link_or=n_link_or, n_higgs_metro=n_higgs_metro,
               delta0=2.0, tile_threads=threads)
    # FP64: the tuned shapes include 128 threads; the single sweeps pin 256
    g = Lattice(L, sweep_mode="passes" if threads else "auto", **par)
    r = Lattice(L, sweep_mode="passes", **par)
    for h in (g, r):
        h.init_hot(2)
        h.sweeps(40, 0)  # past the tuning
    for measflag in (1, 0, 1):
        g.sweeps(24, measflag)
        for _ in range(24):
            r.sweeps(1, measflag)
        m0, m1 = g.meas1(), r.meas1()
        for k in m0:
            x, y = np.asarray(m0[k]), np.asarray(m1[k])
            # tuned FP64: sums grouped by its own tiles
            assert np.all(np.abs(x - y) <= (0.0 if threads else 1e-12) * np.maximum(1.0, np.abs(y))), (k, x, y)
        (u0, a0), (u1, a1) = g.download(), r.download()
        assert np.array_equal(u0, u1) and np.array_equal(a0, a1)
    for h in (g, r):
        h.close()

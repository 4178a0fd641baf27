"""The FP64 update kernels in tiles of 128 sites: a candidate of the autotuner,
whose first sweep of a context it always is."""
import numpy as np
import pytest

from lceqcd_b200 import Ensemble, Lattice, Params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L", [(2, 4, 2), (6, 10, 6), (16, 16, 16), (24, 20, 28)])
@pytest.mark.parametrize("kw", [dict(), dict(imode=1, agauge_hits=3), dict(n_link_or=2, n_higgs_metro=1)])
def test_f64_tuned_tiles_match_fixed_tiles(L, kw):
    """Sweep by sweep through the tuning (the four forms in turn) and through
    graphs of 8 sweeps in the chosen one: the fields are those of the 256-site
    tiles bit for bit, the measurements (sums grouped per tile) to 1e-12."""
    par = dict(beta=9.0, x=0.1, y=0.45, seed=23, precision="f64", delta0=2.0, **kw)
    g, r = Lattice(L, sweep_mode="auto", **par), Lattice(L, sweep_mode="passes", **par)
    assert r.tile_shape()[0] == 256
    for h in (g, r):
        h.init_hot(2)
    for n in [1] * 16 + [19]:
        for h in (g, r):
            h.sweeps(n, 1)
        (u0, a0), (u1, a1) = g.download(), r.download()
        np.testing.assert_array_equal(u0, u1)
        np.testing.assert_array_equal(a0, a1)
        m0, m1 = g.meas1(), r.meas1()
        for k in m0:
            x, y = np.asarray(m0[k]), np.asarray(m1[k])
            assert np.all(np.abs(x - y) <= 1e-12 * np.maximum(1.0, np.abs(y))), k
    assert g.sweep_mode() != "auto" and g.tile_shape()[0] in (128, 256)
    assert g.rng_position() == r.rng_position()
    for h in (g, r):
        h.close()


def test_f64_batch_tuned_tiles_match_fixed_tiles():
    specs = [Params(L=L, beta=6.0 + i, x=0.1, y=0.2, seed=40 + i, precision="f64")
             for i, L in enumerate([(2, 2, 2), (8, 12, 6), (16, 16, 16)])]
    out = []
    for mode in ("auto", "passes"):
        e = Ensemble([Params(**{**s.__dict__, "sweep_mode": mode}) for s in specs])
        e.init_hot(3)
        e.sweeps(1, 1)
        out.append(([e.download(chain=i) for i in range(len(specs))], e.meas_batch()))
        e.close()
    for (u0, a0), (u1, a1) in zip(out[0][0], out[1][0]):
        np.testing.assert_array_equal(u0, u1)
        np.testing.assert_array_equal(a0, a1)
    for m0, m1 in zip(out[0][1], out[1][1]):
        for k in m0:
            x, y = np.asarray(m0[k]), np.asarray(m1[k])
            assert np.all(np.abs(x - y) <= 1e-12 * np.maximum(1.0, np.abs(y))), k

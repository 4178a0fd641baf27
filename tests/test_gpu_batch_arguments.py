"""Batches whose passes have at least 512 tiles find their chains in the kernels'
arguments: every tile shape, both precisions and the 3-hit link update, each
chain against the same chain run alone, bit for bit in the fields."""
import numpy as np
import pytest

from lceqcd_b200 import Ensemble, Lattice, Params

pytestmark = pytest.mark.gpu

# chains of 34 tiles of 512 sites or more, and two small ones between
EXTENTS = [(34, 32, 32)] * 8 + [(10, 6, 8), (2, 4, 2)] + [(36, 30, 34)] * 8


@pytest.mark.parametrize("mode,threads,precision", [
    ("passes", 128, "f32"), ("passes", 256, "f32"), ("passes", 448, "f32"), ("passes", 512, "f32"),
    ("passes2", 128, "f32"), ("passes2", 256, "f32"), ("passes", 0, "f64"), ("passes2", 0, "f64"), ("auto", 0, "f64")])
@pytest.mark.parametrize("hits", [1, 3])
def test_large_batch_equals_single_chains(mode, threads, precision, hits):
    sites = (threads or 256) * (2 if mode == "passes2" else 1)
    assert sum(-(-l1 * l2 * l3 // 2 // sites) for l1, l2, l3 in EXTENTS) >= 512 and len(EXTENTS) <= 128

    def par(i, m):
        return Params(L=EXTENTS[i], beta=6.0 + i % 5, x=0.08 + 0.01 * (i % 3), y=0.1 + 0.1 * (i % 4), imode=i % 2,
                      seed=40 + i, precision=precision, sweep_mode=m, tile_threads=threads, agauge_hits=hits,
                      n_link_or=1, n_higgs_metro=1)
    ens = Ensemble([par(i, mode) for i in range(len(EXTENTS))])
    ens.init_hot(3)
    start = [ens.download(chain=i) for i in range(len(EXTENTS))]
    n = 21 if mode == "auto" else 2  # through the tuning, all its forms
    ens.sweeps(n, 1)
    meas = ens.meas_batch()
    for i in (0, 7, 8, 9, 10, 17):
        p = par(i, "passes" if mode == "auto" else mode)
        lat = Lattice(p.L, **{k: v for k, v in p.__dict__.items() if k != "L"})
        lat.upload(*start[i])
        lat.sweeps(n, 1)
        u, a = lat.download()
        ub, ab = ens.download(chain=i)
        assert np.array_equal(u, ub) and np.array_equal(a, ab), i
        m, one = lat.meas1(), ens.meas1(i)
        assert one == meas[i]
        for k in m:
            x, y = np.asarray(m[k]), np.asarray(one[k])
            # the tuned form's sums are grouped by its own tiles
            assert np.all(np.abs(x - y) <= (1e-12 if mode == "auto" else 0.0) * np.maximum(1.0, np.abs(y))), (i, k)
        lat.close()
    ens.close()

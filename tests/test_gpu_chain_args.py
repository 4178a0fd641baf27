"""Where the update kernels find their chains: the parameter bank (one chain; a
batch of up to 128 chains and 512 tiles or more) or the table in memory.  Each
chain of a batch must come out as it does alone, bit for bit."""
import numpy as np
import pytest

from lceqcd_b200 import Ensemble, Lattice, Params

pytestmark = pytest.mark.gpu


# tiles of 128 sites: 60 chains x 8^3 = 120 (table); 24 of 8^3-24^3 cross 512 in
# the parameter bank; 129 chains are past the table's place there; ragged extents
@pytest.mark.parametrize("extents", [[(8, 8, 8)] * 60, [(8, 8, 8), (16, 16, 16), (24, 24, 24)] * 8,
                                     [(8, 6, 10), (14, 10, 22)] * 64 + [(4, 4, 4)], [(34, 20, 16)] * 16])
@pytest.mark.parametrize("mode,threads", [("passes", 128), ("passes", 448), ("passes2", 256)])
def test_batch_equals_single_chains(extents, mode, threads):
    def par(i, L):
        return Params(L=L, beta=6.0 + i % 5, x=0.08 + 0.01 * (i % 3), y=0.1 + 0.1 * (i % 4), imode=i % 2, seed=40 + i,
                      sweep_mode=mode, tile_threads=threads, n_link_or=1, n_higgs_metro=1)
    ens = Ensemble([par(i, L) for i, L in enumerate(extents)])
    ens.init_hot(3)
    start = [ens.download(chain=i) for i in range(len(extents))]
    ens.sweeps(2, 1)
    meas = ens.meas_batch()
    for i in sorted({0, 1, len(extents) // 2, len(extents) - 1}):
        p = par(i, extents[i])
        lat = Lattice(p.L, beta=p.beta, x=p.x, y=p.y, imode=p.imode, seed=p.seed, sweep_mode=mode, tile_threads=threads,
                      n_link_or=1, n_higgs_metro=1)
        lat.upload(*start[i])
        lat.sweeps(2, 1)
        u, a = lat.download()
        ub, ab = ens.download(chain=i)
        assert np.array_equal(u, ub) and np.array_equal(a, ab), i
        m = lat.meas1()
        assert all(m[k] == meas[i][k] for k in m), (i, m, meas[i])
        lat.close()
    ens.close()

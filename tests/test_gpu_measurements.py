"""The measurements' block splits against plain NumPy sums: slices of one and of
several segments, ragged last segments, slices above the 128 x 128 limit of the
small segments, and lattices whose tiles do not divide the parities.

Tolerance: the sums are FP64 over at most 1.4e5 terms of one sign or of random
sign bounded by 1, so their relative rounding is below 1e-11 of the sum of
magnitudes; FP64 fields enter exactly, and the transform's products add a few
1e-16 per link."""
import numpy as np
import pytest

from lceqcd_b200 import Lattice

pytestmark = pytest.mark.gpu


def natural(f, L):
    """[2, V/2, c] -> [z, y, x, c] (parity 0: x + y + z even)."""
    L1, L2, L3 = L
    h = f.reshape(2, L3, L2, L1 // 2, -1)
    out = np.empty((L3, L2, L1, h.shape[-1]))
    for z in range(L3):
        for y in range(L2):
            for p in range(2):
                out[z, y, (p + y + z) % 2::2] = h[p, z, y]
    return out


def mul(p, q):
    a, b, c, d = p[..., 0] + 1j * p[..., 1], p[..., 2] + 1j * p[..., 3], q[..., 0] + 1j * q[..., 1], \
        q[..., 2] + 1j * q[..., 3]
    x, y = a * c - b * d.conj(), a * d + b * c.conj()
    return np.stack([x.real, x.imag, y.real, y.imag], -1)


def inv(p):
    return p * np.array([1, -1, -1, -1])


def zcorr(s, w):
    return np.array([(s * np.roll(s, -z, 0)).sum() for z in range(len(s))]) / (len(s) * w)


@pytest.mark.parametrize("L", [(2, 2, 2), (16, 16, 6), (34, 32, 4), (66, 50, 34), (130, 128, 4), (128, 128, 2),
                               (200, 170, 2)])
def test_measurements_match_numpy(L):
    rng = np.random.default_rng(sum(L))
    V = L[0] * L[1] * L[2]
    u = rng.normal(size=(3, 2, V // 2, 4))
    u /= np.linalg.norm(u, axis=-1, keepdims=True)
    g = rng.normal(size=(2, V // 2, 4)).astype(np.float32)
    g /= np.linalg.norm(g, axis=-1, keepdims=True)
    a = rng.normal(size=(2, V // 2, 3))
    lat = Lattice(L, precision="f64", alpha=0.8)
    lat.upload(u, a)
    lat.set_transform(g)
    lat.apply_transform()
    U, A, G = [natural(u[m], L) for m in range(3)], natural(a, L), natural(g.astype(np.float64), L)
    up = lambda f, mu: np.roll(f, -1, 2 - mu)  # noqa: E731
    uf = [mul(mul(G, U[m]), inv(up(G, m))) for m in range(3)]
    uf = [f / np.linalg.norm(f, axis=-1, keepdims=True) for f in uf]
    iA = np.stack([0 * A[..., 0], A[..., 2], A[..., 1], A[..., 0]], -1)
    t = mul(mul(G, iA), inv(G))
    af = t[..., [3, 2, 1]]
    udl, adl = lat.download(which=1)
    assert np.abs(natural(udl[1], L) - uf[1]).max() < 1e-12
    # a tracked transform is FP32-uploaded, so |G| differs from 1 by ~1e-7: A_f scales with it exactly
    assert np.abs(natural(adl, L) - af).max() < 1e-12 * np.abs(af).max()

    c = (1.0, 1.0, 0.8)
    tol = dict(rtol=1e-11, atol=1e-13)
    np.testing.assert_allclose(lat.gauge_functional(), sum(c[m] * uf[m][..., 0].sum() for m in range(3)) / (2.8 * V),
                               **tol)
    div = sum(c[m] * (uf[m][..., 1:] - np.roll(uf[m][..., 1:], 1, 2 - m)) for m in range(3))
    odd = np.indices((L[2], L[1], L[0])).sum(0) % 2 == 1
    np.testing.assert_allclose(lat.theta(), (div ** 2).sum(-1)[odd].sum() / (V // 2), **tol)
    plaq = sum(mul(mul(U[m], up(U[n], m)), inv(mul(U[n], up(U[m], n))))[..., 0].sum()
               for m in range(3) for n in range(m + 1, 3)) / (3 * V)
    np.testing.assert_allclose(lat.plaquette(), plaq, rtol=1e-11, atol=1e-12)
    ca, cu, c3, am = lat.correlator()
    sa = af.mean((1, 2))
    sl = [f.mean((1, 2))[:, [1, 3, 2]] * np.array([1, 1, -1]) for f in uf]
    np.testing.assert_allclose(ca, zcorr(sa, 1), **tol)
    np.testing.assert_allclose(cu, zcorr(np.concatenate(sl[:2], 1), 2), **tol)
    np.testing.assert_allclose(c3, zcorr(sl[2], 1), **tol)
    np.testing.assert_allclose(am, sa.mean(0), **tol)
    r2 = (A ** 2).sum(-1)
    for got, f in ((lat.polyakov(), np.cos(4 * np.sqrt(r2))), (lat.scalarcorr(), r2)):
        s = f.mean((1, 2))
        np.testing.assert_allclose(got[0], s, **tol)
        np.testing.assert_allclose(got[1], zcorr(s[:, None], 1), **tol)
    np.testing.assert_allclose(lat.polyakov()[2], np.cos(4 * np.sqrt(r2)).mean() ** 2, **tol)
    np.testing.assert_allclose(lat.scalarcorr()[2], r2.mean(), **tol)
    lat.close()

"""Performance cases: the work a lattice user has this package do, through its
public entry points (`lceqcd_b200`), with the inputs made on the spot.

    listed()            the fixed cases, from one 16^3 FP64 chain to 256^3
    draw(rng)           one more case of the same ranges
    prepare(case, seed) the handle and the fields a program holds before the call
    run(state)          one pass, and what it computed
    work(case)          bytes and floating-point operations of one pass
    exact(case, seed)   the same results in 64 bits, where they are defined

Kinds of cases:

    sweeps     a production run between two saved configurations: n sweeps
               queued by `sweeps`, the last measured values, and the fields
               brought to (pinned) host memory
    loop       the loop of f/main.f: `sweep` with its measured values read back
               after every sweep, then the configuration
    routines   the update routines called one by one with their acceptances, as
               the reference's driver calls them, and the un-fixed measurements
    ensemble   many chains of uneven volume and couplings in one batch
    fix_or     the reference's overrelaxed Landau gauge fixing and correlators
    fix_cg     the conjugate-gradient Fourier-accelerated fixing and correlators
    measure    every measurement on a configuration with a known transform
    train      training of the warm-start network on recorded pairs

A Monte Carlo update accepts or rejects on a comparison, and a gauge fixing
stops on one, so their results have no value "in 64 bits" for a given 32-bit
run (`exact` gives None); the measurements have.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from lceqcd_b200 import lattice as lq

LINK, HIGGS = 4, 3  # reals per link, per site's A


def _vol(L):
    return L[0] * L[1] * L[2]


def _case(kind, L, **kw):
    c = {"kind": kind, "L1": L[0], "L2": L[1], "L3": L[2], "precision": "f32", "beta": 12.0, "x": 0.09, "y": 0.3}
    c.update(kw)
    return c


def listed():
    return [
        # the smallest production chain: the reference's plain method in FP64 at
        # 16^3, heatbath + 4 overrelaxations + Metropolis, read after every sweep
        _case("loop", (16, 16, 16), name="loop_16_f64", precision="f64", beta=9.0, x=0.1, y=0.45, n=10,
              n_link_or=4, n_higgs_metro=1),
        # the driver's own loop over routines on a small ragged lattice: every
        # option off its default (3-hit link update, Higgs mode 1, Metropolis)
        _case("routines", (24, 20, 28), name="routines_24x20x28", beta=9.0, x=0.1, y=0.45, imode=1),
        # a small FP32 chain, where a pass is shorter than a wave
        _case("sweeps", (32, 32, 32), name="sweeps_32", n=40, measflag=1),
        # the headline chain: 64^3, measured on every sweep
        _case("sweeps", (64, 64, 64), name="sweeps_64", n=80, measflag=1),
        # the same chain on the plain FP64 path
        _case("sweeps", (64, 64, 64), name="sweeps_64_f64", precision="f64", n=20, measflag=1),
        # heatbath + 4 overrelaxations at 128^3, ten sweeps between configurations
        _case("sweeps", (128, 128, 128), name="sweeps_128_or4", n=10, measflag=1, n_link_or=4),
        # the full-scale chain: 256^3, HB + 4 OR + Higgs Metropolis, 20 sweeps
        # between gauge-fixed measurements
        _case("sweeps", (256, 256, 256), name="sweeps_256_pipeline", beta=16.0, x=0.08, y=0.2, n=20, measflag=1,
              n_link_or=4, n_higgs_metro=1),
        # 96 chains of 16^3, 32^3 and 48^3 over a grid of couplings in one batch
        _case("ensemble", (16, 32, 48), name="ensemble_96", chains=96, n=20, measflag=1),
        # the reference's gauge fixing on extents that are not powers of two
        _case("fix_or", (48, 40, 36), name="fix_or_48x40x36", lam=1.7, limit_or=1e-10),
        # the gauge-fixed measurement at 128^3
        _case("fix_cg", (128, 128, 128), name="fix_cg_128", limit_or=1e-10),
        # all measurements of a 256^3 configuration
        _case("measure", (256, 256, 256), name="measure_256"),
        # the warm-start network at 128^3, one epoch over two pairs
        _case("train", (128, 128, 128), name="train_128", pairs=2, lr=1e-3),
    ]


def _even(v):
    return max(4, 2 * int(round(v / 2)))


def _extents(rng, lo, hi):
    """Even extents around an edge spread over its logarithm, unlike one another."""
    edge = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return tuple(_even(edge * rng.uniform(0.8, 1.25)) for _ in range(3))


def draw(rng):
    coup = {"beta": round(rng.uniform(6.0, 16.0), 3), "x": round(rng.uniform(0.08, 0.1), 4),
            "y": round(rng.uniform(0.1, 0.5), 3)}
    kind = rng.choice(["loop", "routines", "sweeps", "sweeps", "sweeps", "ensemble", "fix_or", "fix_cg", "measure",
                       "train"])
    if kind == "loop":
        return _case(kind, _extents(rng, 8, 64), precision=rng.choice(["f32", "f64"]), n=rng.randint(2, 20),
                     n_link_or=rng.randint(0, 4), n_higgs_metro=rng.randint(0, 1), **coup)
    if kind == "routines":
        return _case(kind, _extents(rng, 8, 64), precision=rng.choice(["f32", "f64"]), imode=rng.randint(0, 1), **coup)
    if kind == "sweeps":
        f64 = rng.random() < 0.25
        L = _extents(rng, 12, 64 if f64 else 200)
        return _case(kind, L, precision="f64" if f64 else "f32", n=max(4, min(80, int(4e7 / _vol(L)))),
                     measflag=rng.randint(0, 1), n_link_or=rng.choice([0, 0, 1, 4]), n_higgs_metro=rng.randint(0, 1),
                     agauge_hits=rng.choice([1, 1, 3]), imode=rng.randint(0, 1), **coup)
    if kind == "ensemble":
        return _case(kind, tuple(sorted(_even(math.exp(rng.uniform(math.log(8), math.log(48)))) for _ in range(3))),
                     precision=rng.choice(["f32", "f32", "f64"]), chains=rng.randint(3, 64), n=rng.randint(4, 20),
                     measflag=rng.randint(0, 1))
    if kind == "fix_or":
        return _case(kind, _extents(rng, 10, 56), precision=rng.choice(["f32", "f32", "f64"]), lam=1.7,
                     limit_or=rng.choice([1e-8, 1e-9, 1e-10]), **coup)
    if kind == "fix_cg":
        L = tuple(1 << rng.randint(4, 7) for _ in range(3))
        return _case(kind, L, precision=rng.choice(["f32", "f32", "f64"]), limit_or=rng.choice([1e-8, 1e-9, 1e-10]),
                     **coup)
    if kind == "measure":
        return _case(kind, _extents(rng, 12, 180), precision=rng.choice(["f32", "f64"]), **coup)
    return _case("train", (rng.choice([16, 32, 128]), _even(rng.uniform(16, 64)), _even(rng.uniform(16, 64))),
                 pairs=rng.randint(1, 4), lr=1e-3, **coup)


# ---------------------------------------------------------------- preparation
OPTIONS = ("beta", "x", "y", "precision", "imode", "n_link_or", "n_higgs_metro", "agauge_hits", "lam", "limit_or")


def _lattice(case, seed):
    kw = {k: case[k] for k in OPTIONS if k in case}
    return lq.Lattice(L=(case["L1"], case["L2"], case["L3"]), seed=seed, **kw)


def _pinned(case, nsites):
    """Host buffers of a configuration in the reference's layout, and their arrays."""
    t = torch.float64 if case["precision"] == "f64" else torch.float32
    u = torch.empty(3 * nsites * LINK, dtype=t, pin_memory=True)
    a = torch.empty(nsites * HIGGS, dtype=t, pin_memory=True)
    return u, a, u.numpy(), a.numpy()


def _warm(lat, seed, n, measflag=1):
    """A hot start brought near equilibrium; the first sweeps also choose the
    context's sweep form, as in any run."""
    lat.init_hot(seed)
    lat.sweeps(n, measflag)
    lat.synchronize()


def _ensemble_params(case, seed):
    """Chains of the three edges in equal parts over a grid of couplings."""
    out, n = [], case["chains"]
    edges = (case["L1"], case["L2"], case["L3"])
    for i in range(n):
        e = edges[i * 3 // n]
        out.append(lq.Params(L=(e, e, e), beta=(6.0, 9.0, 12.0, 16.0)[i % 4], y=(0.1, 0.3, 0.5)[(i // 4) % 3],
                             x=(0.08, 0.1)[(i // 12) % 2], precision=case["precision"], seed=seed * 1000 + i + 1))
    return out


def _random_su2(n, spread, gen, dtype):
    """Unit quaternions around 1 with Gaussian vector parts."""
    v = torch.randn(n, 3, generator=gen, device="cuda", dtype=torch.float64) * spread
    r = v.norm(dim=1, keepdim=True)
    return torch.cat([torch.cos(r), torch.sin(r) * v / r.clamp_min(1e-300)], dim=1).to(dtype)


def _measure_fields(case, seed):
    """Links scattered around 1 by a tenth, a transform of larger angles and a
    Gaussian Higgs field, in the package's site order [.., parity, site]."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    V = case["L1"] * case["L2"] * case["L3"]
    t = torch.float64 if case["precision"] == "f64" else torch.float32
    u = _random_su2(3 * V, 0.3, gen, t).reshape(3, 2, V // 2, LINK)
    g = _random_su2(V, 0.8, gen, torch.float32).reshape(2, V // 2, LINK)
    a = (0.6 * torch.randn(2, V // 2, HIGGS, generator=gen, device="cuda", dtype=torch.float64)).to(t)
    return u, g, a


def prepare(case, seed):
    kind = case["kind"]
    if kind == "ensemble":
        ens = lq.Ensemble(_ensemble_params(case, seed))
        _warm(ens, seed, 40, case["measflag"])
        sites = [_vol(p.L) for p in ens.params]
        u, a, un, an = _pinned(case, sum(sites))
        at = np.concatenate([[0], np.cumsum(sites)])
        views = [(un[3 * LINK * b:3 * LINK * e], an[HIGGS * b:HIGGS * e]) for b, e in zip(at[:-1], at[1:])]
        return {"case": case, "lat": ens, "u": u, "a": a, "views": views}
    lat = _lattice(case, seed)
    state = {"case": case, "lat": lat}
    V = case["L1"] * case["L2"] * case["L3"]
    if kind == "measure":
        u, g, a = _measure_fields(case, seed)
        lat.upload(u.cpu().numpy(), a.cpu().numpy())
        lat.set_transform(g.cpu().numpy())
        return state
    _warm(lat, seed, 40 if V > 1 << 20 else 100, case.get("measflag", 1))
    if kind == "train":
        net = lq.GaugeNet(seed=seed)
        lat.landau_gauge_from("identity", max_iters=0) if not _fourier_ok(case) else lat.landau_gauge_fourier_cg()
        for _ in range(case["pairs"]):
            lat.sweeps(10, 0)
            ok = _fourier_ok(case)
            lat.landau_gauge_warm(net=net, use_net=False, record=True, fourier=ok, cg=ok)
        net.train(epochs=1, lr=case["lr"])
        state["net"] = net
        return state
    state["delta"] = 1.0
    state["u"], state["a"], state["un"], state["an"] = _pinned(case, V)
    return state


def _fourier_ok(case):
    return all(n & (n - 1) == 0 for n in (case["L1"], case["L2"], case["L3"]))


# ---------------------------------------------------------------- one pass
MEAS = ("plaq", "akin", "a2", "a4", "acc_gauge", "acc_hb", "acc_or", "acc_metro", "acc_link_or", "delta")


def _row(m):
    return [m[k] for k in MEAS]


def run(state):
    case, lat = state["case"], state["lat"]
    kind = case["kind"]
    if kind == "sweeps":
        lat.sweeps(case["n"], case["measflag"])
        m = lat.meas1()
        lat.download_into(state["un"], state["an"])
        return {"meas": np.array(_row(m)), "u": state["u"], "a": state["a"]}
    if kind == "loop":
        rows = [_row(lat.sweep(1)) for _ in range(case["n"])]
        lat.download_into(state["un"], state["an"])
        return {"meas": np.array(rows), "u": state["u"], "a": state["a"]}
    if kind == "routines":
        acc = [lat.ahiggs2(1), lat.ahiggs3(1)]
        metro, state["delta"] = lat.ahiggs1(state["delta"], 1)
        acc += [metro, state["delta"], lat.agauge1(1), lat.link_or(1)]
        lat.renorm()
        m = lat.meas1()
        pol, sca = lat.polyakov(), lat.scalarcorr()
        lat.download_into(state["un"], state["an"])
        return {"acc": np.array(acc, np.float32), "meas": np.array(_row(m)), "polyakov": pol, "scalar": sca,
                "u": state["u"], "a": state["a"]}
    if kind == "ensemble":
        lat.sweeps(case["n"], case["measflag"])
        rows = [_row(m) for m in lat.meas_batch()]
        for k, (un, an) in enumerate(state["views"]):
            lat.download_into(un, an, chain=k)
        return {"meas": np.array(rows), "u": state["u"], "a": state["a"]}
    if kind == "fix_or":
        theta, iters = lat.landau_gauge()
        corr = lat.correlator()
        lat.download_into(state["un"], state["an"], which=1)
        return {"theta": theta, "iters": iters, "corr": corr, "u": state["u"], "a": state["a"]}
    if kind == "fix_cg":
        theta, iters, plain = lat.landau_gauge_fourier_cg("identity")
        functional = lat.gauge_functional()
        corr, pol, sca = lat.correlator(), lat.polyakov(), lat.scalarcorr()
        lat.download_into(state["un"], state["an"], which=1)
        return {"theta": theta, "iters": [iters, plain], "functional": functional, "corr": corr, "polyakov": pol,
                "scalar": sca, "u": state["u"], "a": state["a"]}
    if kind == "measure":
        lat.apply_transform()
        return {"functional": lat.gauge_functional(), "theta": lat.theta(), "plaq": lat.plaquette(),
                "corr": lat.correlator(), "polyakov": lat.polyakov(), "scalar": lat.scalarcorr()}
    loss = state["net"].train(epochs=1, lr=case["lr"])
    return {"loss": loss, "params": state["net"].params()}


# ---------------------------------------------------------------- work of a pass
# Floating-point operations per site: a link update is four SU(2) products per
# staple plane (2 x 4 x 28), the proposal (~80) and the hopping term (~130); a
# Higgs update rotates A by six links (6 x 45) and proposes (~40).
FLOP_LINK, FLOP_HIGGS = 450, 320


def _sweep_work(V, case, n):
    """A sweep reads the fields once and writes them once."""
    w = 8 if case["precision"] == "f64" else 4
    links = 3 * (case.get("agauge_hits", 1) + case.get("n_link_or", 0))
    higgs = 2 + case.get("n_higgs_metro", 0)
    return n * 2 * 15 * w * V, n * V * (links * FLOP_LINK + higgs * FLOP_HIGGS)


def work(case):
    kind, L = case["kind"], (case["L1"], case["L2"], case["L3"])
    w, V = 8 if case["precision"] == "f64" else 4, _vol(L)
    fields = 15 * w * V  # a configuration: 12 + 3 reals per site
    if kind in ("sweeps", "loop"):
        b, f = _sweep_work(V, case, case["n"])
        return {"bytes": b + fields, "flops": f}
    if kind == "routines":
        return {"bytes": 3 * fields, "flops": V * (3 * 4 * FLOP_LINK + 3 * FLOP_HIGGS)}
    if kind == "ensemble":
        V = sum(_vol(p.L) for p in _ensemble_params(case, 1))
        b, f = _sweep_work(V, case, case["n"])
        return {"bytes": b + 15 * w * V, "flops": f}
    if kind == "fix_or":
        # an iteration reads and writes U_f and A_f once; their number grows
        # like the longest edge (about 40 per site of it at theta < 1e-10)
        n = 40 * max(L)
        return {"bytes": n * 2 * fields, "flops": n * V * 400}
    if kind == "fix_cg":
        # an iteration reads U_f for the gradient, and reads and writes U_f,
        # A_f and the transform; about 1.3 iterations per site of the longest edge
        n = 1.3 * max(L)
        lg = math.log2(V)
        return {"bytes": n * (12 * w * V + 2 * 19 * w * V), "flops": n * V * (2 * 2 * 5 * lg + 600)}
    if kind == "measure":
        # transform the fields, then each measurement reads what it needs
        fixed = fields
        return {"bytes": fields + 16 * V + fixed + 2 * 12 * w * V + 12 * w * V + fixed + 2 * 3 * w * V,
                "flops": V * (6 * 28 + 3 * 3 * 28 + 60)}
    # forward, input gradient and weight gradient of 4 layers of 27 x 16 x 16
    n = case["pairs"]
    return {"bytes": n * V * (4 * 2 * 32 + 4 * 2 * 32), "flops": n * V * (4 + 3 + 4) * 2 * 27 * 16 * 16}


# ---------------------------------------------------------------- 64-bit results
def _natural(f, L):
    """Parity-split [2, V/2, c] -> [z, y, x, c]: parity 0 holds x + y + z even,
    sites in the order z, y, x / 2."""
    L1, L2, L3 = L
    h = f.reshape(2, L3, L2, L1 // 2, -1).to(torch.float64)
    out = torch.empty(L3, L2, L1, h.shape[-1], dtype=torch.float64, device=f.device)
    odd = (torch.arange(L3, device=f.device)[:, None] + torch.arange(L2, device=f.device)[None, :]) % 2 == 1
    for p in (0, 1):
        first = odd if p == 0 else ~odd  # rows whose parity-p sites start at x = 1
        out[:, :, 0::2][~first] = h[p][~first]
        out[:, :, 1::2][first] = h[p][first]
    return out


def _mul(p, q):
    """Product of first rows (a, b), U = {{a, b}, {-b*, a*}}, as (Re a, Im a, Re b, Im b)."""
    a = torch.complex(p[..., 0], p[..., 1])
    b = torch.complex(p[..., 2], p[..., 3])
    c = torch.complex(q[..., 0], q[..., 1])
    d = torch.complex(q[..., 2], q[..., 3])
    x, y = a * c - b * d.conj(), a * d + b * c.conj()
    return torch.stack([x.real, x.imag, y.real, y.imag], dim=-1)


def _inv(p):
    return torch.stack([p[..., 0], -p[..., 1], -p[..., 2], -p[..., 3]], dim=-1)


def _shift(f, mu, n):
    """The field at x + n mu (mu = 0, 1, 2: x, y, z of [z, y, x, ..])."""
    return torch.roll(f, -n, dims=2 - mu)


def _zcorr(s, weight):
    """sum over the columns of the periodic autocorrelation over z of slice means s [L3, c]."""
    L3 = s.shape[0]
    return torch.stack([(s * torch.roll(s, -z, dims=0)).sum() for z in range(L3)]) / (L3 * weight)


def exact(case, seed):
    if case["kind"] != "measure":
        return None
    L = (case["L1"], case["L2"], case["L3"])
    u, g, a = _measure_fields(case, seed)
    G = _natural(g, L)
    A = _natural(a, L)
    U = [_natural(u[mu], L) for mu in range(3)]
    del u, g, a
    V = _vol(L)
    plaq = 0.0
    for mu in range(3):
        for nu in range(mu + 1, 3):
            p = _mul(_mul(U[mu], _shift(U[nu], mu, 1)), _inv(_mul(U[nu], _shift(U[mu], nu, 1))))
            plaq += float(p[..., 0].sum())
    plaq /= 3.0 * V
    # iA has the first row (i a3, a2 + i a1); the transform acts as G iA G^+
    iA = torch.stack([torch.zeros_like(A[..., 0]), A[..., 2], A[..., 1], A[..., 0]], dim=-1)
    t = _mul(_mul(G, iA), _inv(G))
    Af = torch.stack([t[..., 3], t[..., 2], t[..., 1]], dim=-1)
    del iA, t
    functional, div, slices = 0.0, None, []
    for mu in range(3):
        f = _mul(_mul(G, U[mu]), _inv(_shift(G, mu, 1)))
        f = f / f.norm(dim=-1, keepdim=True)
        functional += float(f[..., 0].sum()) / (3.0 * V)
        d = f[..., 1:] - _shift(f[..., 1:], mu, -1)
        div = d if div is None else div + d
        s = f.mean(dim=(1, 2))
        slices.append(torch.stack([s[:, 1], s[:, 3], -s[:, 2]], dim=-1))
        U[mu] = None
        del f
    z, y, x = (torch.arange(n, device=A.device) for n in (L[2], L[1], L[0]))
    odd = (z[:, None, None] + y[None, :, None] + x[None, None, :]) % 2 == 1
    theta = float((div.square().sum(-1) * odd).sum()) / (V // 2)
    sa = Af.mean(dim=(1, 2))
    r2 = A.square().sum(-1)
    pol = torch.cos(4.0 * r2.sqrt()).mean(dim=(1, 2))
    sca = r2.mean(dim=(1, 2))
    host = lambda v: v.cpu().numpy()  # noqa: E731
    corr = (host(_zcorr(sa, 1.0)), host(_zcorr(torch.cat(slices[:2], dim=-1), 2.0)), host(_zcorr(slices[2], 1.0)),
            host(sa.mean(0)))
    polyakov = (host(pol), host(_zcorr(pol[:, None], 1.0)), float(pol.mean()) ** 2)
    scalar = (host(sca), host(_zcorr(sca[:, None], 1.0)), float(sca.mean()))
    return {"functional": functional, "theta": theta, "plaq": plaq, "corr": corr, "polyakov": polyakov,
            "scalar": scalar}

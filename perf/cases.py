"""Timed cases of the propagators, the eigensolver, the spectrum stage and the
warm start's network, each through the entry point a program calls.

A pass of a propagation case loads new inputs into a plan that the program
keeps, propagates them and reads C(t) and the final state back, which is what
a scan over potentials or initial conditions does per job.  Sizes are those of
the repository's workloads and tests: the uneven 1D Morse scan (256..2048
points), 1D packets of any even size, the 256 x 256 coupled Morse grid, the
128^3 anharmonic oscillator, the 128 x 128 eigensolver with its MLP.
"""
import math

import numpy as np
import torch

import espec_b200 as E
from espec_b200 import _native as N
from espec_b200 import eig as EG
from espec_b200 import spectrum as SP
from espec_b200 import warmstart as WS

SHFS = N.SHFS
SCAN = "256,384,512,768,1024,1536,2048"
TWOPI_DIGT = 6.283185307  # the reference's 2 pi in the kinetic table (dkeft.f:38)


def listed():
    return [
        # the batched Morse scan over packet sizes and parameters, FP64 and mixed: the headline use
        dict(name="scan_fp64", kind="batch", sizes=SCAN, npk=2048, steps=800, precision="fp64"),
        dict(name="scan_mixed", kind="batch", sizes=SCAN, npk=2048, steps=800, precision="mixed"),
        # a scan on grids outside the power-of-two plans (decks use 200, 201, 250, 560 points)
        dict(name="scan_any_size", kind="batch", sizes="200,250,300,490,560,1000,1500", npk=592,
             steps=400, precision="fp64"),
        # one packet with the printed rows of a deck: 16 steps, then E, norm and C(t) of the row
        dict(name="rows_1d", kind="rows", n=512, rows=8, lc=16),
        # the 256 x 256 coupled Morse grid with its absorbing potential, split operator
        dict(name="spo_2d", kind="fftgrid", method="spo", np="256,256", steps=1000,
             precision="fp64"),
        # the 128^3 anharmonic oscillator, mixed precision
        dict(name="spo_3d_mixed", kind="fftgrid", method="spo", np="128,128,128", steps=1000,
             precision="mixed"),
        # second-order differences with the FFT kinetic term on a ragged 3D grid
        dict(name="sod_3d", kind="fftgrid", method="sod", np="64,32,128", steps=500,
             precision="fp64"),
        # short-iterative Lanczos of order 12 on the 256 x 256 coupled Morse grid, mask absorber
        dict(name="sil_2d", kind="sil", np="256,256", order=12, steps=100),
        # second-order differences, finite-difference H, on a grid of odd sides
        dict(name="psod_2d", kind="psod", np="1023,769", steps=400),
        # initial states: lowest two of 64 coupled Morse potentials on 128 x 128, cold start
        dict(name="eigen_2d", kind="eigen", np="128,128", npk=64, states=2),
        # spectra of a scan's C(t): assembly, lifetime damping, window, transform
        dict(name="spectra", kind="spectra", npk=1024, mf=12),
        # one gradient of the warm start's network (5 -> 3 x 256 -> 4 x 1024), minibatch of 256
        dict(name="mlp_gradient", kind="mlp", rows=256, out=4096),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["batch", "batch", "any", "rows", "fftgrid", "fftgrid", "sil", "psod",
                       "eigen", "spectra", "mlp"])
    if kind == "batch":
        sizes = sorted(rng.sample([256, 384, 512, 768, 1024, 1536, 2048], rng.randint(1, 7)))
        return dict(kind="batch", sizes=",".join(map(str, sizes)), npk=_log(rng, 8, 1800),
                    steps=rng.randint(100, 500), precision=rng.choice(["fp64", "fp64", "mixed"]))
    if kind == "any":
        sizes = sorted({2 * _log(rng, 40, 900) for _ in range(rng.randint(1, 6))})
        return dict(kind="batch", sizes=",".join(map(str, sizes)), npk=_log(rng, 4, 400),
                    steps=rng.randint(50, 300), precision="fp64")
    if kind == "rows":
        return dict(kind="rows", n=2 * _log(rng, 64, 1024), rows=rng.randint(2, 12),
                    lc=_log(rng, 4, 32))
    if kind == "fftgrid":
        ndim = rng.choice([2, 2, 3])
        while True:
            np_ = [rng.choice([32, 64, 128, 256, 512]) for _ in range(ndim)]
            if math.prod(np_) <= (1 << 18 if ndim == 2 else 1 << 20):
                break
        method = rng.choice(["spo", "spo", "sod"])
        return dict(kind="fftgrid", method=method, np=",".join(map(str, np_)),
                    steps=rng.randint(50, 500),
                    precision=rng.choice(["fp64", "mixed"]) if method == "spo" else "fp64")
    if kind == "sil":
        ndim = rng.choice([1, 2, 2, 3])
        lo, hi = {1: (64, 2000), 2: (32, 256), 3: (12, 40)}[ndim]
        return dict(kind="sil", np=",".join(str(_log(rng, lo, hi)) for _ in range(ndim)),
                    order=rng.randint(4, 16), steps=rng.randint(10, 100))
    if kind == "psod":
        ndim = rng.choice([1, 2, 2, 3])
        lo, hi = {1: (64, 4000), 2: (40, 880), 3: (16, 80)}[ndim]
        return dict(kind="psod", np=",".join(str(_log(rng, lo, hi)) for _ in range(ndim)),
                    steps=rng.randint(50, 400))
    if kind == "eigen":
        return dict(kind="eigen", np="%d,%d" % (_log(rng, 32, 112), _log(rng, 32, 112)),
                    npk=_log(rng, 1, 64), states=rng.randint(1, 2))
    if kind == "spectra":
        mf = rng.randint(8, 14)
        return dict(kind="spectra", npk=_log(rng, 1, 1 << (21 - mf)), mf=mf)
    return dict(kind="mlp", rows=_log(rng, 32, 512), out=rng.choice([1024, 2048, 4096]))


def _ints(text):
    return [int(x) for x in text.split(",")]


# -- inputs -----------------------------------------------------------------

def _morse(x, de, a, re):
    return de * (1.0 - np.exp(-a * (x - re))) ** 2


def _batch_inputs(case, seed):
    """Morse packets of uneven sizes on [0.5, 8] bohr, parameters of the scan."""
    rng = np.random.default_rng(seed)
    k = case["npk"]
    # which packet has which size belongs to the plan, not to its inputs
    n = np.random.default_rng(k).choice(np.asarray(_ints(case["sizes"])), size=k)
    p = [rng.uniform(*r, k) for r in ((0.05, 0.25), (0.6, 1.6), (1.0, 2.5), (900.0, 30000.0),
                                      (-0.3, 0.5), (0.1, 0.3))]
    off = np.concatenate([[0], np.cumsum(n)])
    sh = 7.5 / (n - 1)
    x = 0.5 + (np.arange(off[-1]) - np.repeat(off[:-1], n)) * np.repeat(sh, n)
    de, a, re, mass, c, s = p
    r = [np.repeat(q, n) for q in (de, a, re, re + c, s)]
    v = _morse(x, r[0], r[1], r[2])
    psi = np.exp(-((x - r[3]) ** 2) / (2.0 * r[4] ** 2))
    psi /= np.repeat(np.sqrt(np.add.reduceat(psi * psi, off[:-1])), n)
    return dict(n=n, off=off, sh=sh, sm=mass, v=v, psi=psi, dt=0.5 * SHFS)


def _rows_inputs(case, seed):
    rng = np.random.default_rng(seed)
    x = np.linspace(0.5, 8.0, case["n"])
    v = _morse(x, rng.uniform(0.1, 0.2), rng.uniform(0.9, 1.1), 1.4)
    psi = np.exp(-((x - rng.uniform(1.6, 2.0)) ** 2) / 0.08).astype(complex)
    psi /= np.sqrt(np.sum(np.abs(psi) ** 2))
    return dict(v=v, psi=psi, sh=x[1] - x[0], sm=918.0, dt=0.5 * SHFS)


def _cap(q):
    """Quadratic absorber of 0.01 Eh on the outer 15 % of an axis."""
    w = 0.15 * (q[-1] - q[0])
    return 0.01 * (np.maximum(np.maximum(q[0] + w - q, q - q[-1] + w), 0.0) / w) ** 2


def _grid_inputs(case, seed):
    """Coupled Morse modes (1D/2D) or an anharmonic oscillator (3D) with a
    displaced, moving Gaussian; arrays flattened x fastest."""
    rng = np.random.default_rng(seed)
    np_ = _ints(case["np"])
    nd = len(np_)
    if nd == 3:
        ax = [np.linspace(-2.5, 2.5, n) for n in np_]
        om, m = [0.01, 0.012, 0.015], [1836.0] * 3
        v = [0.5 * m[a] * (om[a] * rng.uniform(0.9, 1.1)) ** 2 * ax[a] ** 2 for a in range(3)]
        c = [rng.uniform(-0.3, 0.3) for _ in range(3)]
        s = [1.0 / math.sqrt(m[a] * om[a]) for a in range(3)]
    else:
        ax = [np.linspace(0.5, 8.0, n) for n in np_]
        m = [918.0, 1500.0][:nd]
        par = [(0.17, 1.0, 1.4), (0.12, 1.2, 1.8)][:nd]
        v = [_morse(ax[a], d * rng.uniform(0.9, 1.1), al, re)
             for a, (d, al, re) in enumerate(par)]
        c = [(1.6, 2.0)[a] + rng.uniform(-0.1, 0.1) for a in range(nd)]
        s = [0.15] * nd
    sh = [q[1] - q[0] for q in ax]
    g = [q.reshape([-1 if a == i else 1 for i in reversed(range(nd))]) for a, q in enumerate(ax)]

    def total(parts):  # sum of one function per axis, x fastest
        return sum(f.reshape(q.shape) for f, q in zip(parts, g)) + np.zeros(np_[::-1])

    V = total(v)
    if nd == 2:
        V = V + 0.01 * (g[0] - 1.4) * (g[1] - 1.8)
    if nd == 3:
        V = V + 1e-4 * (g[0] ** 2 * g[1] - g[1] ** 3 / 3)
    k0 = [rng.uniform(-1.0, 1.0) for _ in range(nd)]
    psi = np.exp(total([-((ax[a] - c[a]) ** 2) / (2 * s[a] ** 2) for a in range(nd)])
                 + 1j * total([k0[a] * ax[a] for a in range(nd)]))
    psi /= np.sqrt(np.sum(np.abs(psi) ** 2))
    W = total([_cap(q) for q in ax])
    shm = [1.0 / (((24.0 * m[a]) * sh[a]) * sh[a]) for a in range(nd)]
    emax_fd = 64.0 * sum(shm) + V.max()
    emax_fft = sum((math.pi / sh[a]) ** 2 / (2 * m[a]) for a in range(nd)) + V.max()
    if case["kind"] == "sil":
        dt = min(1.0, 6.0 / emax_fd)
    elif case["kind"] == "psod":
        dt = min(0.1, 0.4 / emax_fd)  # stable for dt E_max < 1
    elif case["method"] == "sod":
        dt = min(0.1, 0.4 / emax_fft)
    else:
        dt = 1.0 if nd == 2 else 2.0
    return dict(np=np_, sh=sh, sm=m, shm=shm, v=V.ravel(), psi=psi.ravel(), w=W.ravel(),
                dt=dt * SHFS, dt_au=dt)


def _spectra_inputs(case, seed):
    """C(t) of packets: a few levels with random populations, weakly damped."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    k, nt = case["npk"], 1 << (case["mf"] - 1)
    dt = 0.5 * SHFS
    t = torch.arange(nt, dtype=torch.float64, device="cuda") * 0.5
    pop = torch.rand((k, 6), dtype=torch.float64, device="cuda", generator=gen)
    pop /= pop.sum(1, keepdim=True)
    e = torch.rand((k, 6), dtype=torch.float64, device="cuda", generator=gen) * 0.2
    c = torch.zeros((k, nt), dtype=torch.complex128, device="cuda")
    for j in range(6):
        c += torch.polar(pop[:, j:j + 1] * torch.exp(-1e-4 * t), -e[:, j:j + 1] * t)
    return dict(c=c, dt=dt, tf=nt * dt, tal=0.01, de=2.0)


def _eigen_inputs(case, seed):
    g = EG.Grid2D(_ints(case["np"]))
    q = torch.tensor(WS.sample_params(case["npk"], seed), dtype=torch.float64, device="cuda")
    st = EG.lcg_start(g.n, case["states"], q.device)
    return dict(grid=g, v=EG.morse2d_potentials(g, q),
                start=st.expand(case["npk"], case["states"], g.n).contiguous())


def _mlp_inputs(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.rand((case["rows"], 5), device="cuda", generator=gen) * 2 - 1
    return dict(x=x.to(torch.bfloat16),
                t=torch.randn((case["rows"], case["out"]), device="cuda", generator=gen))


# -- what a program holds before the call, and the call ---------------------

def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        i = _batch_inputs(case, seed)
        b = E.SpoBatch(i["n"], i["sh"], i["sm"], i["dt"], precision=case["precision"])
        nc = case["npk"] * (case["steps"] + 1)
        out = [torch.empty(m, dtype=torch.float64, pin_memory=True).numpy()
               for m in (nc, nc, b.total, b.total)]
        psi = torch.from_numpy(i["psi"]).cuda()
        return dict(case=case, plan=b, v=torch.from_numpy(i["v"]).cuda(),
                    psi=(psi, torch.zeros_like(psi)), out=out)
    if kind == "rows":
        i = _rows_inputs(case, seed)
        return dict(case=case, plan=E.SpoBatch([case["n"]], [i["sh"]], [i["sm"]], i["dt"]), i=i)
    if kind == "fftgrid":
        i = _grid_inputs(case, seed)
        if case["method"] == "sod":
            g = E.SodGrid(i["np"], i["sh"], i["sm"], i["dt"])
        else:
            g = E.SpoGrid(i["np"], i["sh"], i["sm"], i["dt"], precision=case["precision"],
                          absorb=N.ABS_VOPTIC)
        return dict(case=case, plan=g, i=i, ab=None if case["method"] == "sod" else -i["w"])
    if kind in ("sil", "psod"):
        i = _grid_inputs(case, seed)
        g = (E.SilGrid(i["np"], i["shm"], i["dt"], case["order"], absorb=N.ABS_SMOOTHW)
             if kind == "sil" else E.PsodGrid(i["np"], i["shm"], i["dt"], absorb=N.ABS_SMOOTHW))
        return dict(case=case, plan=g, i=i, ab=np.exp(-i["w"] * i["dt_au"]))
    if kind == "spectra":
        return dict(case=case, **_spectra_inputs(case, seed))
    if kind == "eigen":
        return dict(case=case, **_eigen_inputs(case, seed))
    return dict(case=case, net=WS.MLP([5, 256, 256, 256, case["out"]], seed=seed),
                **_mlp_inputs(case, seed))


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "batch":
        b, o = s["plan"], s["out"]
        b.load(s["v"], s["psi"])
        b.run(case["steps"])
        b.results_into(*o)
        return o
    if kind == "rows":
        b, lc = s["plan"], case["lc"]
        b.load(s["i"]["v"], s["i"]["psi"])
        table = []
        for k in range(case["rows"]):
            (b.run if k == 0 else b.advance)(lc)
            cr, ci = np.empty(lc + 1), np.empty(lc + 1)
            b.results_into(cr, ci, None, None)
            e, norm = b.energies()
            # a continued segment writes samples 1..lc
            table.append([e, norm, cr[1:], ci[1:]])
        return table, b.results()[1]
    if kind in ("fftgrid", "sil", "psod"):
        g = s["plan"]
        g.load(s["i"]["v"], s["i"]["psi"], vabc=s.get("ab"))
        g.run(case["steps"])
        c, psi = g.results()
        return [c, psi]
    if kind == "spectra":
        return SP.spectra(s["c"], case["mf"], s["dt"], s["tf"], tal=s["tal"], de=s["de"])
    if kind == "eigen":
        r = EG.solve(s["grid"], s["v"], s["start"], nstates=case["states"])
        # the residual is read as a program reads it: reached or not
        return r["eval"], r["vec"], r["matvecs"], r["resid"] <= 1e-9
    net = s["net"]
    hs, zs = net.forward(s["x"])
    rows, dy = net.loss_grad(zs[-1], s["t"])
    return zs[-1], rows, net.backward(hs, zs, dy)


# -- what a pass cannot do without -------------------------------------------

def work(case):
    kind = case["kind"]
    if kind == "batch":
        sizes = _ints(case["sizes"])
        n = sum(sizes) / len(sizes) * case["npk"]
        lg = sum(x * math.log2(x) for x in sizes) / sum(sizes)
        return dict(bytes=8 * (3 * n + 2 * n + 2 * case["npk"] * (case["steps"] + 1)),
                    flops=n * case["steps"] * (10 * lg + 20))
    if kind == "rows":
        n, st = case["n"], case["rows"] * case["lc"]
        return dict(bytes=8 * (5 * n + 2 * st), flops=n * (st * (10 * math.log2(n) + 20)))
    if kind in ("fftgrid", "sil", "psod"):
        n, st = math.prod(_ints(case["np"])), case["steps"]
        if kind == "fftgrid":
            per = 10 * math.log2(n) + 20
        elif kind == "psod":
            per = 2 * 9 * len(_ints(case["np"])) + 20
        else:  # m stencils, Gram-Schmidt (dots and updates) and the expansion, two chains
            m = case["order"]
            per = 2 * (m * (9 * len(_ints(case["np"])) + 8) + 2 * m * (m + 1) + 4 * m)
        ins = 4 if kind != "fftgrid" or case["method"] == "spo" else 3
        return dict(bytes=8 * ((ins + 2) * n + 2 * (st + 1)), flops=n * st * per)
    if kind == "spectra":
        n = case["npk"] << case["mf"]
        return dict(bytes=16 * (n + n // 2), flops=n * (5 * case["mf"] + 40))
    if kind == "eigen":
        # about 500 applications of H per state at 128 x 128 (fewer on coarser grids), each
        # with its share of the reorthogonalisation against up to 40 vectors
        np_ = _ints(case["np"])
        n, k, s = math.prod(np_), case["npk"], case["states"]
        return dict(bytes=8 * n * k * (1 + 2 * s), flops=4 * n * k * s * max(np_) * (18 + 84 + 40))
    r, o = case["rows"], case["out"]
    w = 5 * 256 + 2 * 256 * 256 + 256 * o
    return dict(bytes=2 * w + 4 * w + 10 * r + 8 * r * o, flops=6 * r * w)


# -- the same in 64 bits, without the repository's code -----------------------

def _tc(n, sh, sm):
    k = np.fft.fftfreq(n) * n
    return (k * TWOPI_DIGT / (n * sh)) ** 2 / (2.0 * sm)


def _cuda(x):
    return torch.from_numpy(np.ascontiguousarray(x)).cuda()


def _spo(v, psi, tc, dt, steps, vabc=None, dims=(-1,)):
    """Strang steps; C(t) of every step over the trailing axes `dims`."""
    h = torch.polar(torch.ones_like(v) if vabc is None else torch.exp(0.5 * dt * vabc),
                    -0.5 * dt * v)
    k = torch.polar(torch.ones_like(tc), -dt * tc)
    p, bra, c = psi, psi.conj(), [(psi.abs() ** 2).sum(dims).to(psi.dtype)]
    for _ in range(steps):
        p = h * torch.fft.ifftn(k * torch.fft.fftn(h * p, dim=dims), dim=dims)
        c.append((bra * p).sum(dims))
    return torch.stack(c, -1), p


def _exact_batch(case, seed):
    i = _batch_inputs(case, seed)
    n, off, steps = i["n"], i["off"], case["steps"]
    c = np.zeros((len(n), steps + 1), complex)
    psi = np.zeros(off[-1], complex)
    for m in np.unique(n):
        ks = np.nonzero(n == m)[0]
        pick = off[ks][:, None] + np.arange(m)
        tc = np.stack([_tc(m, i["sh"][k], i["sm"][k]) for k in ks])
        cc, pp = _spo(_cuda(i["v"][pick]), _cuda(i["psi"][pick].astype(complex)), _cuda(tc),
                      i["dt"] / SHFS, steps)
        c[ks], psi[pick] = cc.cpu().numpy(), pp.cpu().numpy()
    return [c.real.ravel(), c.imag.ravel(), psi.real, psi.imag]


def _exact_rows(case, seed):
    i = _rows_inputs(case, seed)
    n, lc = case["n"], case["lc"]
    v, tc = _cuda(i["v"]), _cuda(_tc(n, i["sh"], i["sm"]))
    p = psi0 = _cuda(i["psi"])
    table = []
    for _ in range(case["rows"]):
        _, p1 = _spo(v, p, tc, i["dt"] / SHFS, 0)
        cs = []
        for _ in range(lc):
            _, p1 = _spo(v, p1, tc, i["dt"] / SHFS, 1)
            cs.append((psi0.conj() * p1).sum())
        p = p1
        c = torch.stack(cs).cpu().numpy()
        e = (v * p.abs() ** 2).sum() + (tc * torch.fft.fft(p).abs() ** 2).sum() / n
        table.append([np.array([float(e)]), np.array([float((p.abs() ** 2).sum())]),
                      c.real.copy(), c.imag.copy()])
    return table, p.cpu().numpy()


def _exact_fftgrid(case, seed):
    i = _grid_inputs(case, seed)
    shape = i["np"][::-1]
    dims = tuple(range(-len(shape), 0))
    tc = sum(_tc(n, i["sh"][a], i["sm"][a]).reshape([-1 if k == len(shape) - 1 - a else 1
                                                     for k in range(len(shape))])
             for a, n in enumerate(i["np"]))
    v, psi, tc = _cuda(i["v"].reshape(shape)), _cuda(i["psi"].reshape(shape)), _cuda(tc)
    dt, steps = i["dt"] / SHFS, case["steps"]
    if case["method"] == "spo":
        c, p = _spo(v, psi, tc, dt, steps, _cuda(-i["w"].reshape(shape)), dims)
    else:
        def h(x):
            return v * x + torch.fft.ifftn(tc * torch.fft.fftn(x, dim=dims), dim=dims)

        c, p = _leapfrog(h, psi, dt, steps, 0.5, None)
    return [c.cpu().numpy(), p.reshape(-1).cpu().numpy()]


def _leapfrog(h, psi0, dt, steps, first, mask):
    """psi(t+dt) = psi(t-dt) - 2 i dt H psi(t) from psi0, started by an Euler
    step of `first` dt (psodfft.f: 1, psod.f: 1/2) and a step of dt from it."""
    def upd(old, src, f):
        x = old - 2j * dt * f * h(src)
        return x if mask is None else mask * x

    c = [(psi0.conj() * psi0).sum()]
    prev, cur = psi0, psi0
    if steps >= 1:
        cur = upd(psi0, upd(psi0, psi0, first), 0.5)
        c.append((psi0.conj() * cur).sum())
    for _ in range(2, steps + 1):
        prev, cur = cur, upd(prev, cur, 1.0)
        c.append((psi0.conj() * cur).sum())
    return torch.stack(c), cur


def _fd(i, x, lead):
    """The 4th-order finite-difference H on the trailing grid axes of x."""
    shape = i["np"][::-1]
    out = (30.0 * sum(i["shm"]) + _cuda(i["v"].reshape(shape))) * x
    for a, s in enumerate(i["shm"]):
        ax = lead + len(shape) - 1 - a
        n = x.shape[ax]
        for d, f in ((1, -16.0), (2, 1.0)):
            if n > d:
                out.narrow(ax, d, n - d).add_(x.narrow(ax, 0, n - d), alpha=f * s)
                out.narrow(ax, 0, n - d).add_(x.narrow(ax, d, n - d), alpha=f * s)
    return out


def _exact_psod(case, seed):
    i = _grid_inputs(case, seed)
    shape = i["np"][::-1]
    mask = _cuda(np.exp(-i["w"] * i["dt_au"]).reshape(shape))
    c, p = _leapfrog(lambda x: _fd(i, x, 0), _cuda(i["psi"].reshape(shape)), i["dt"] / SHFS,
                     case["steps"], 0.25, mask)
    return [c.cpu().numpy(), p.reshape(-1).cpu().numpy()]


def _exact_sil(case, seed):
    i = _grid_inputs(case, seed)
    shape, m, dt = i["np"][::-1], case["order"], i["dt"] / SHFS
    mask = _cuda(np.exp(-i["w"] * i["dt_au"]).reshape(shape)).reshape(-1)
    psi0 = _cuda(i["psi"])
    x = torch.stack([psi0.real, psi0.imag])  # the two real chains
    c = [(psi0.conj() * psi0).sum()]
    for _ in range(case["steps"]):
        nrm = x.norm(dim=1, keepdim=True)
        L = torch.zeros((2, m, x.shape[1]), dtype=torch.float64, device="cuda")
        T = torch.zeros((2, m, m), dtype=torch.float64, device="cuda")
        w = x / nrm
        for j in range(m):
            L[:, j] = w
            hv = _fd(i, w.reshape([2] + shape), 1).reshape(2, -1)
            T[:, j, j] = (w * hv).sum(1)
            for _ in range(2):
                hv = hv - (L[:, :j + 1].transpose(1, 2) @ (L[:, :j + 1] @ hv[:, :, None]))[..., 0]
            b = hv.norm(dim=1)
            if j + 1 < m:
                T[:, j, j + 1] = T[:, j + 1, j] = b
                w = hv / b[:, None]
        e, z = torch.linalg.eigh(T)
        y = torch.polar(torch.ones_like(e), -dt * e).unsqueeze(1) * z.to(torch.complex128)
        coef = (y @ z.transpose(1, 2).to(torch.complex128))[:, :, 0] * nrm
        out = (coef[:, :, None] * L).sum(1)
        psi = mask * (out[0] + 1j * out[1])
        x = torch.stack([psi.real, psi.imag])
        c.append((psi0.conj() * psi).sum())
    return [torch.stack(c).cpu().numpy(), psi.cpu().numpy()]


def _exact_spectra(case, seed):
    i = _spectra_inputs(case, seed)
    c, mc = i["c"], 1 << (case["mf"] - 1)
    j = torch.arange(2 * mc, dtype=torch.float64, device="cuda")
    x = torch.cat([c[:, mc - 1:mc].conj(), c.flip(1)[:, :mc].conj(), c[:, 1:]], 1)
    t = -i["tf"] + j * i["dt"]
    damp = torch.exp(-t.abs() * i["tal"] * 1.5192676)
    shift = torch.polar(damp, -i["de"] * 1.5192676 * t)
    tau = (2 * mc * i["dt"]) ** 2 / math.log(1e3) ** 2
    return torch.fft.ifft(torch.roll(x * shift * torch.exp(-t * t / tau), mc, 1))


def _exact_eigen(case, seed):
    """Eigenvalues from one long Lanczos run with full reorthogonalisation."""
    s = _eigen_inputs(case, seed)
    g, k = s["grid"], case["npk"]
    i = dict(np=g.np, shm=g.shm, v=np.zeros(g.n))
    V = s["v"]
    m = min(g.n, 480)
    gen = torch.Generator(device="cuda").manual_seed(1)
    w = torch.randn((k, g.n), dtype=torch.float64, device="cuda", generator=gen)
    w /= w.norm(dim=1, keepdim=True)
    L = torch.zeros((k, m, g.n), dtype=torch.float64, device="cuda")
    T = torch.zeros((k, m, m), dtype=torch.float64, device="cuda")
    zero = torch.zeros(1, device="cuda")
    for j in range(m):
        L[:, j] = w
        hv = _fd(i, w.reshape([k] + g.np[::-1]), 1).reshape(k, -1) + V * w + zero
        T[:, j, j] = (w * hv).sum(1)
        for _ in range(2):
            hv = hv - (L[:, :j + 1].transpose(1, 2) @ (L[:, :j + 1] @ hv[:, :, None]))[..., 0]
        b = hv.norm(dim=1)
        if j + 1 < m:
            T[:, j, j + 1] = T[:, j + 1, j] = b
            w = hv / b[:, None]
    return torch.linalg.eigvalsh(T)[:, :case["states"]].contiguous(), None, None, None


def _exact_mlp(case, seed):
    s = prepare(case, seed)
    W, b = [w.double() for w in s["net"].W], [x.double() for x in s["net"].b]
    hs, zs = [s["x"].double()], []
    for i, (w, x) in enumerate(zip(W, b)):
        z = hs[-1] @ w + x
        zs.append(z)
        if i + 1 < len(W):
            hs.append(0.5 * z * (1.0 + torch.erf(z / math.sqrt(2.0))))
    y = zs[-1].clone().requires_grad_()
    d = y - s["t"].double()
    rows = (d * d).sum(1) / d.numel()
    dy, = torch.autograd.grad(rows.sum(), y)
    grads = []
    for i in reversed(range(len(W))):
        grads[:0] = [hs[i].T @ dy, dy.sum(0)]
        if i:
            z = zs[i - 1]
            pdf = torch.exp(-0.5 * z * z) / math.sqrt(2.0 * math.pi)
            dy = (dy @ W[i].T) * (0.5 * (1.0 + torch.erf(z / math.sqrt(2.0))) + z * pdf)
    return zs[-1], rows.detach(), grads


def exact(case, seed):
    return {"batch": _exact_batch, "rows": _exact_rows, "fftgrid": _exact_fftgrid,
            "sil": _exact_sil, "psod": _exact_psod, "spectra": _exact_spectra,
            "eigen": _exact_eigen, "mlp": _exact_mlp}[case["kind"]](case, seed)

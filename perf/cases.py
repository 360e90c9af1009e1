"""Timed cases: what a user of this framework has it do, through its public
entry points, from the smallest calls to the largest.

Mechanisms: the three synthetic ones of the configurations (10 species / 27
reactions, 53 / 325, 561 / 2539).  States: T ~ U[800, 2800] K, P log-uniform
in [1, 50] atm, Y ~ Dirichlet(0.5), as everywhere else in this repository;
a third of the cases' states have a few species absent (mass fraction zero),
as initial mixtures do.

    listed()            the cases
    draw(rng)           one more case of the same ranges
    prepare(case, seed) inputs on the device and the handle a program keeps
    run(state)          one pass
    work(case)          bytes and operations a pass cannot do without
    exact(case, seed)   the outputs in 64 bits by plain torch
"""
import math
import tempfile

import torch

from create_rate_subs_gb300 import synth
from create_rate_subs_gb300 import work as crs_work
from create_rate_subs_gb300.mechanism import Mechanism
from create_rate_subs_gb300.rates import RateSubs
from create_rate_subs_gb300.surrogate import MLP

ATM = 101325.0
RU = 8314.4621
# the learned surrogate's network (inputs T, ln P, 53 mass fractions) and
# its training batch
NET = (55, 256, 256, 256, 53)

# kind "wdot": RateSubs.wdot; "host": RateSubs.wdot_host on pinned arrays;
# "dydt": RateSubs.dydt; "functions": the four reference functions in turn;
# "infer" / "train": the surrogate's network.
_SPAN = {  # (kind, mech, mode) -> range of n
    ("wdot", "small", "fp64"): (64, 1 << 18),
    ("wdot", "gri53", "fp64"): (16, 1 << 20),
    ("wdot", "gri53", "mixed"): (1 << 10, 1 << 22),
    ("wdot", "large561", "fp64"): (1 << 9, 1 << 17),
    ("wdot", "large561", "mixed"): (1 << 9, 1 << 17),
    ("wdot", "large561", "gemm"): (1 << 12, 1 << 18),
    ("host", "gri53", "fp64"): (1 << 12, 1 << 19),
    ("dydt", "gri53", "fp64"): (1 << 8, 1 << 19),
    ("functions", "gri53", "fp64"): (1 << 8, 1 << 16),
    ("infer", "", ""): (1 << 10, 1 << 20),
    ("train", "", ""): (1 << 12, 1 << 15),
}


def _case(kind, mech, mode, n, absent=False, conv=False, name=None):
    c = {"kind": kind, "mech": mech, "mode": mode, "n": int(n), "absent": absent, "conv": conv}
    return dict(c, name=name) if name else c


def listed():
    return [
        # the smallest configuration: a validation batch, one launch
        _case("wdot", "small", "fp64", 1024, name="small fp64 1024"),
        # a handful of reactors advanced together: latency of one call
        _case("wdot", "gri53", "fp64", 97, absent=True, name="gri53 fp64 97"),
        # the plain FP64 configuration at its size
        _case("wdot", "gri53", "fp64", 1 << 20, name="gri53 fp64 2^20"),
        # the mixed-precision configuration at its size
        _case("wdot", "gri53", "mixed", 1 << 22, name="gri53 mixed 2^22"),
        # a host solver's cells: pinned arrays in, pinned arrays out
        _case("host", "gri53", "fp64", 200003, name="gri53 host 200003"),
        # the right-hand side of a reactor integrator, odd number of cells
        _case("dydt", "gri53", "fp64", 50021, absent=True, name="gri53 dydt 50021"),
        # the drop-in functions one after another, every intermediate kept
        _case("functions", "gri53", "fp64", 20000, name="gri53 functions 20000"),
        # the large mechanism: sums in FP64, mixed rates, the contraction
        _case("wdot", "large561", "fp64", 20011, name="large561 fp64 20011"),
        _case("wdot", "large561", "mixed", 65536, absent=True, name="large561 mixed 65536"),
        _case("wdot", "large561", "gemm", 1 << 18, name="large561 gemm 2^18"),
        # the surrogate's network: serving and one training step
        _case("infer", "", "", 1 << 20, name="surrogate infer 2^20"),
        _case("train", "", "", 16384, name="surrogate train 16384"),
    ]


def draw(rng):
    kind, mech, mode = rng.choice(sorted(_SPAN))
    lo, hi = _SPAN[kind, mech, mode]
    n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    if kind == "train":  # batches are multiples of 128
        n = max(128, n // 128 * 128)
    return _case(kind, mech, mode, n, absent=kind in ("wdot", "dydt") and rng.random() < 0.35,
                 conv=kind == "dydt" and rng.random() < 0.5)


_handles = {}


def _mechanism(name):
    """The parsed mechanism and its device handle, made once per process."""
    if name not in _handles:
        mp, tp = synth.write_mechanism(name, tempfile.mkdtemp(prefix="crs_cases_"))
        mech = Mechanism.from_chemkin(mp, tp)
        _handles[name] = (mech, RateSubs(mech))
    return _handles[name]


def _states(N, n, seed, absent):
    """(T, P, Y) on the device; Y holds all N rows."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    f64 = dict(dtype=torch.float64, device="cuda")
    T = 800.0 + 2000.0 * torch.rand(n, generator=g, **f64)
    P = ATM * torch.exp(math.log(50.0) * torch.rand(n, generator=g, **f64))
    Y = torch._standard_gamma(torch.full((N, n), 0.5, **f64), generator=g)
    if absent:
        Y[torch.rand((N, n), generator=g, device="cuda") < 0.2] = 0.0
        Y[N - 1] += 1e-3
    Y /= Y.sum(dim=0)
    return T, P, Y


def _rows(n, seed):
    """Feature rows (bf16, padded to 64 columns and 128 rows) and targets of
    n states for the network."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    M = (n + 127) // 128 * 128
    X = torch.zeros((M, 64), dtype=torch.bfloat16, device="cuda")
    X[:n, : NET[0]] = torch.randn((n, NET[0]), generator=g, device="cuda").clamp(-4, 4)
    Tg = torch.randn((n, NET[-1]), generator=g, device="cuda")
    return X, torch.sign(Tg) * torch.log1p(Tg.abs())


def prepare(case, seed):
    kind, n = case["kind"], case["n"]
    s = dict(case)
    if kind in ("infer", "train"):
        s["net"] = MLP(list(NET), seed=seed)
        s["X"], s["Tg"] = _rows(n, seed + 1)
        if kind == "infer":
            # rows a multiple of 4 floats apart, as Surrogate allocates them
            s["Y"] = torch.empty((n, 64), dtype=torch.float32, device="cuda")
        else:
            s["XT"] = s["X"].t().contiguous()
            s["loss"] = torch.zeros(1, device="cuda")
        return s
    mech, rs = _mechanism(case["mech"])
    N = mech.n_species
    T, P, Y = _states(N, n, seed, case["absent"])
    s["rs"] = rs
    if kind == "dydt":
        y = torch.cat([T[None], Y[: N - 1]])
        if case["conv"]:
            inv = torch.tensor(1.0 / mech.tables["sp_mw"], device="cuda")
            P = P / (RU * T * (Y * inv[:, None]).sum(0))  # density
        s["p"], s["y"] = P, y
    elif kind == "host":
        s["T"], s["P"], s["Y"] = (a.cpu().pin_memory() for a in (T, P, Y[: N - 1].contiguous()))
        s["out"] = torch.empty((N, n), dtype=torch.float64).pin_memory()
    else:
        s["T"], s["P"], s["Y"] = T, P, Y[: N - 1].contiguous()
    return s


def run(s):
    kind = s["kind"]
    if kind == "wdot":
        return s["rs"].wdot(s["T"], s["P"], s["Y"], mode=s["mode"])
    if kind == "host":
        return s["rs"].wdot_host(s["T"], s["P"], s["Y"], mode=s["mode"], out=s["out"])
    if kind == "dydt":
        return s["rs"].dydt(s["p"], s["y"], conv=s["conv"], mode=s["mode"])
    if kind == "functions":
        rs = s["rs"]
        y_N, mw, rho, conc = rs.eval_conc(s["T"], s["P"], s["Y"])
        fwd, rev = rs.eval_rxn_rates(s["T"], s["P"], conc)
        pm = rs.get_rxn_pres_mod(s["T"], s["P"], conc)
        return y_N, mw, rho, conc, fwd, rev, pm, rs.eval_spec_rates(fwd, rev, pm)
    if kind == "infer":
        return s["net"].infer(s["X"], s["n"], s["Y"])[:, : NET[-1]]
    net = s["net"]
    net.train_step(s["X"], s["XT"], s["Tg"], 1e-3, loss_slot=s["loss"])
    return {"gW": net.gW, "gb": net.gb, "W": net.W32, "b": net.b32, "mW": net.mW, "vW": net.vW,
            "bf16": net.W}


def work(case):
    kind, n = case["kind"], case["n"]
    if kind in ("infer", "train"):
        macs = sum(a * b for a, b in zip(NET, NET[1:]))
        params = macs + sum(NET[1:])
        if kind == "infer":
            return {"bytes": n * (2.0 * NET[0] + 4.0 * NET[-1]) + 2.0 * params,
                    "flops": 2.0 * n * macs}
        # features and targets once; weights and both moments read and
        # written, gradients written; forward, weight and data gradients
        # (no data gradient into the features)
        return {"bytes": n * (2.0 * NET[0] + 4.0 * NET[-1]) + (6 * 4.0 + 4.0 + 2.0) * params,
                "flops": 2.0 * n * (3 * macs - NET[0] * NET[1])}
    t = _mechanism(case["mech"])[0].tables
    N, R, NREV, NPM = (int(x) for x in t["dims"][:4])
    w = crs_work.work(t)
    flops = float(w["flops"] + w["transcendentals"])
    if kind == "functions":  # conc, fwd, rev and pm are written and read again
        b = 8.0 * (2 + N - 1 + 3 + N + N) + 16.0 * (N + R + NREV + NPM)
    elif kind == "dydt":
        b = 8.0 * (1 + N + N)
        flops += 2 * 13.0 * N + 6.0 * N
    else:
        b = float(crs_work.state_bytes(N))
    return {"bytes": n * b, "flops": n * flops}


# ---- the same quantities by plain torch in 64 bits ------------------------
# From the mechanism's numbers (Arrhenius rows, NASA-7 coefficients,
# stoichiometry, third-body and fall-off constants); none of the library's
# evaluation code.


def _mat(t, ptr, idx, val, cols):
    """Dense (rows, cols) matrix of a CSR list."""
    m = torch.zeros((len(ptr) - 1, cols), dtype=torch.float64)
    for r in range(len(ptr) - 1):
        for e in range(ptr[r], ptr[r + 1]):
            m[r, idx[e]] += val[e]
    return m.cuda()


class _Exact(object):
    def __init__(self, t):
        d = lambda a: torch.as_tensor(a, dtype=torch.float64).cuda()
        self.N, self.R, self.NREV, self.NPM = (int(x) for x in t["dims"][:4])
        self.t = t
        self.rows = d(t["rate_par"])
        self.mw, self.tmid = d(t["sp_mw"]), d(t["sp_tmid"])
        self.lo, self.hi = d(t["sp_lo"]), d(t["sp_hi"])
        self.rx, self.px, self.ef = [], [], None
        # factor lists, padded with a species N of concentration one
        for ptr, sp, nint, out in ((t["rx_ptr"], t["rx_sp"], t["rx_nint"], self.rx),
                                   (t["px_ptr"], t["px_sp"], t["px_nint"], self.px)):
            lists = [[int(sp[e]) for e in range(ptr[r], ptr[r + 1]) for _ in range(nint[e])]
                     for r in range(self.R)]
            w = max(len(x) for x in lists)
            out += list(torch.tensor([x + [self.N] * (w - len(x)) for x in lists]).t().cuda())
        self.nu = _mat(t, t["nu_ptr"], t["nu_sp"], t["nu_val"], self.N)
        self.eff = _mat(t, t["pm_eff_ptr"], t["pm_eff_sp"], t["pm_eff_val"], self.N)
        self.rev = torch.tensor([r for r in range(self.R) if t["rev_idx"][r] >= 0]).cuda()
        self.pm = torch.tensor([r for r in range(self.R) if t["pm_idx"][r] >= 0]).cuda()

    def rate(self, rows, T):
        c = self.rows[rows]
        return torch.exp(c[:, 1:2] + c[:, 2:3] * torch.log(T) - c[:, 3:4] / T)

    def conc(self, T, P, Y):
        y_N = 1.0 - Y.sum(0)
        X = torch.cat([Y, y_N[None]]) / self.mw[:, None]
        mw = 1.0 / X.sum(0)
        rho = P * mw / (RU * T)
        return y_N, mw, rho, rho * X

    def thermo(self, T):
        """cp/R, h/R of every species."""
        a = torch.where(T <= self.tmid[:, None, None], self.lo.t()[:, :, None].permute(1, 0, 2),
                        self.hi.t()[:, :, None].permute(1, 0, 2))
        p = [a[:, j] for j in range(7)]
        cp = p[0] + T * (p[1] + T * (p[2] + T * (p[3] + T * p[4])))
        h = p[5] + T * (p[0] + T * (p[1] / 2 + T * (p[2] / 3 + T * (p[3] / 4 + T * p[4] / 5))))
        return cp, h, p

    def pres_mod(self, T, P, C):
        t = self.t
        thd = P / (RU * T) + self.eff @ C
        out = torch.empty_like(thd)
        for p in range(self.NPM):
            if t["pm_kind"][p] == 0:
                out[p] = thd[p]
                continue
            m = C[int(t["pm_sp"][p])] if t["pm_sp"][p] >= 0 else thd[p]
            k = [self.rate([int(t[q][p])], T)[0] for q in ("pm_k0", "pm_kinf")]
            Pr = k[0] * m / k[1]
            lP = torch.log10(Pr.clamp_min(1e-300))
            F = 1.0
            if t["pm_form"][p] == 1:
                c = [float(x) for x in t["pm_troe"][p]]
                f = c[0] * torch.exp(-T / c[1]) + c[2] * torch.exp(-T / c[3])
                if t["pm_troe_t2"][p]:
                    f = f + torch.exp(-c[4] / T)
                lF = torch.log10(f.clamp_min(1e-300))
                A, B = lP - 0.67 * lF - 0.4, 0.806 - 1.1762 * lF - 0.14 * lP
                F = 10.0 ** (lF / (1.0 + (A / B) ** 2))
            elif t["pm_form"][p] == 2:
                c = [float(x) for x in t["pm_sri"][p]]
                F = (c[0] * torch.exp(-c[1] / T) + torch.exp(-T / c[2])) ** (1.0 / (1.0 + lP * lP))
                if t["pm_sri_de"][p]:
                    F = F * c[3] * T ** c[4]
            out[p] = F * (Pr if t["pm_kind"][p] == 1 else 1.0) / (1.0 + Pr)
        return out

    def rates(self, T, P, C):
        C1 = torch.cat([C, torch.ones_like(C[:1])])
        kf = self.rate(slice(0, self.R), T)
        fwd = kf.clone()
        for f in self.rx:
            fwd *= C1[f]
        _, h, p = self.thermo(T)
        s = p[6] + p[0] * torch.log(T) + T * (p[1] + T * (p[2] / 2 + T * (p[3] / 3 + T * p[4] / 4)))
        nu = self.nu[self.rev]
        lkc = nu @ (s - h / T) + nu.sum(1, keepdim=True) * torch.log(ATM / (RU * T))
        # kf / Kc as one exponential: either factor may leave the range
        c = self.rows[self.rev]
        rev = torch.exp(c[:, 1:2] + c[:, 2:3] * torch.log(T) - c[:, 3:4] / T - lkc)
        for f in self.px:
            rev *= C1[f[self.rev]]
        return fwd, rev

    def functions(self, T, P, Y):
        y_N, mw, rho, C = self.conc(T, P, Y)
        fwd, rev = self.rates(T, P, C)
        pm = self.pres_mod(T, P, C)
        q = fwd.clone()
        q[self.rev] -= rev
        q[self.pm] *= pm
        return y_N, mw, rho, C, fwd, rev, pm, self.nu.t() @ q

    def wdot(self, T, P, Y):
        return self.functions(T, P, Y)[-1]

    def dydt(self, p, y, conv):
        T, Y = y[0], y[1:]
        y_N = 1.0 - Y.sum(0)
        mw = 1.0 / (torch.cat([Y, y_N[None]]) / self.mw[:, None]).sum(0)
        P = p * RU * T / mw if conv else p
        rho = p if conv else p * mw / (RU * T)
        W = self.wdot(T, P, Y)
        cp, h, _ = self.thermo(T)
        if conv:
            cp, h = cp - 1.0, h - T
        c = RU / self.mw[:, None]
        dT = -(W * h * RU).sum(0) / (rho * (c * cp * torch.cat([Y, y_N[None]])).sum(0))
        return torch.cat([dT[None], W[:-1] * self.mw[:-1, None] / rho])


_exact = {}


def _silu_grad(z):
    s = torch.sigmoid(z)
    return s * (1.0 + z * (1.0 - s))


def _exact_net(case, seed):
    s = prepare(case, seed)
    net, n, L = s["net"], case["n"], len(NET) - 1
    W = [net.W[l][: NET[l + 1], : NET[l]].double() for l in range(L)]
    b = [v.double() for v in net.b32]
    a, z = [s["X"][:n, : NET[0]].double()], []
    for l in range(L):
        z.append(a[-1] @ W[l].t() + b[l])
        a.append(z[-1] * torch.sigmoid(z[-1]) if l < L - 1 else z[-1])
    if case["kind"] == "infer":
        return a[-1]
    g = 2.0 * (a[-1] - s["Tg"].double()) / (n * NET[-1])
    gW, gb = [None] * L, [None] * L
    for l in range(L - 1, -1, -1):
        gW[l], gb[l] = g.t() @ a[l], g.sum(0)
        if l:
            g = (g @ W[l]) * _silu_grad(z[l - 1])
    # the updates divide each gradient by its own size: no 64-bit value
    # decides the sign of one that rounds to zero
    none = [None] * L
    return {"gW": gW, "gb": gb, "W": none, "b": none, "mW": [0.1 * v for v in gW],
            "vW": [0.001 * v * v for v in gW], "bf16": none}


def exact(case, seed):
    kind, n = case["kind"], case["n"]
    if kind in ("infer", "train"):
        return _exact_net(case, seed)
    mech, _ = _mechanism(case["mech"])
    if case["mech"] not in _exact:
        _exact[case["mech"]] = _Exact(mech.tables)
    e = _exact[case["mech"]]
    s = prepare(case, seed)
    if kind == "host":
        s.update({k: s[k].cuda() for k in ("T", "P", "Y")})
    parts = []
    step = max(256, (1 << 26) // e.R)
    for i in range(0, n, step):
        j = min(n, i + step)
        if kind == "dydt":
            parts.append((e.dydt(s["p"][i:j], s["y"][:, i:j], case["conv"]),))
        elif kind == "functions":
            parts.append(e.functions(s["T"][i:j], s["P"][i:j], s["Y"][:, i:j]))
        else:
            parts.append((e.wdot(s["T"][i:j], s["P"][i:j], s["Y"][:, i:j]),))
    out = [torch.cat(p, dim=-1) for p in zip(*parts)]
    return tuple(out) if kind == "functions" else out[0].cpu() if kind == "host" else out[0]

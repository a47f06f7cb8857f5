"""What this library's users have it do, as measurable cases.

Five families, all through the public entry points: whole HMC trajectories of
one lattice ("traj", Lattice.update_gauge), CG solves on device vectors ("cg",
tg_cg_dev), the operator M and its adjoint on device vectors ("apply",
Lattice.apply_dev), the pseudofermion force from host arrays ("force",
Lattice.pf_force) and a batch of independent chains ("batch", Batch.trajectory).
Molecular-dynamics step sizes are ones at which the integrator is stable, so
trajectories can be compared digit by digit.

exact() restates each in plain torch, complex128, with solves to the rounding
of FP64.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

import thirring2d_gb300 as tg

FP64, MIXED = tg.native.PREC_FP64, tg.native.PREC_MIXED
NF = 2.0  # flavours in the gauge action


def listed():
    base = dict(mu=0.0, bc_t=-1, bc_x=1)
    return [
        # The reference program's own run: 16^2, MT19937 stream, CG to |r|^2 < 1e-30,
        # ten leapfrog steps.  Nothing but latency.
        dict(base, name="traj_16_mt", kind="traj", nt=16, nx=16, m=0.1, g=0.5, sigma=0.1, npf=1, steps=10, tau=0.25,
             prec=FP64, tol=0.0, rng="mt"),
        # The force study: 64^2, two pseudofermions, mixed precision at a tight tolerance.
        dict(base, name="traj_64_pf2", kind="traj", nt=64, nx=64, m=0.1, g=0.5, sigma=0.3, npf=2, steps=10, tau=0.25,
             prec=MIXED, tol=1e-12, rng="philox"),
        # An ordinary production lattice with a chemical potential, neither side a multiple of 32.
        dict(base, name="traj_100x60_mu", kind="traj", nt=100, nx=60, m=0.1, g=0.5, mu=0.1, bc_x=-1, sigma=0.2, npf=1,
             steps=10, tau=0.2, prec=FP64, tol=1e-10, rng="philox"),
        # The large-lattice run (the benchmark's lattice, half its steps), in both precisions.
        dict(base, name="traj_1024_fp64", kind="traj", nt=1024, nx=1024, m=0.05, g=0.6, sigma=0.3, npf=1, steps=10,
             tau=0.015, prec=FP64, tol=1e-10, rng="philox"),
        dict(base, name="traj_1024_mixed", kind="traj", nt=1024, nx=1024, m=0.05, g=0.6, sigma=0.3, npf=1, steps=10,
             tau=0.015, prec=MIXED, tol=1e-10, rng="philox"),
        # A solve on the largest configured lattice, ill-conditioned, beyond L2.
        dict(base, name="cg_2048_mixed", kind="cg", nt=2048, nx=2048, m=0.02, g=0.8, sigma=0.5, prec=MIXED, tol=1e-10),
        # A large lattice whose side is a round number and no multiple of 32.
        dict(base, name="cg_1000_fp64", kind="cg", nt=1000, nx=1000, m=0.05, g=0.6, sigma=0.3, prec=FP64, tol=1e-10),
        # The operator by itself, as a measurement code applies it: M, then M^dagger.
        dict(base, name="apply_1024_fp64", kind="apply", nt=1024, nx=1024, m=0.05, g=0.6, sigma=0.3, prec=FP64),
        dict(base, name="apply_2048_fp32", kind="apply", nt=2048, nx=2048, m=0.02, g=0.8, sigma=0.5, prec=MIXED),
        # The force on caller-owned host arrays (the autograd check's backward pass).
        dict(base, name="force_256_pf2", kind="force", nt=256, nx=256, m=0.1, g=0.5, sigma=0.3, npf=2, prec=FP64,
             tol=1e-10),
        # 512 chains of sides 16 ... 128 with their own couplings, on the instance the
        # autotuner picks for them, and the field of every chain read back.
        dict(name="batch_512_mixed", kind="batch", n=512, side=0, steps=10, tau=0.1, prec=MIXED, tol=1e-10,
             block=1451241),
        # 512 chains of the reference's own lattice size, FP64, on their tuned instance.
        dict(name="batch_512x16_fp64", kind="batch", n=512, side=16, steps=10, tau=0.25, prec=FP64, tol=1e-12,
             block=12808),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["traj", "traj", "cg", "cg", "apply", "force", "batch"])
    prec = rng.choice([FP64, MIXED])
    if kind == "batch":
        # one side for all, or (0) sides of 16 ... 128
        return dict(kind=kind, n=_log_int(rng, 8, 512), side=rng.choice([0, 0, _log_int(rng, 8, 48)]), steps=rng.randint(3, 8),
                    tau=0.05, prec=prec, tol=10.0 ** rng.uniform(-12, -10), block=rng.choice([1451241, 51201, 25604]))
    hi = {"traj": 400, "cg": 1400, "apply": 2048, "force": 400}[kind]
    nt, nx = _log_int(rng, 8, hi), _log_int(rng, 8, hi)
    if rng.random() < 0.4:  # many lattices are chosen round
        nt, nx = 8 * max(1, nt // 8), 32 * max(1, nx // 32)
    c = dict(kind=kind, nt=nt, nx=nx, m=round(math.exp(rng.uniform(math.log(0.05), math.log(0.5))), 4),
             g=round(rng.uniform(0.2, 1.2), 3), mu=rng.choice([0.0, 0.0, round(rng.uniform(0.0, 0.3), 3)]), bc_t=-1,
             bc_x=rng.choice([-1, 1]), sigma=round(rng.uniform(0.1, 0.5), 3), prec=prec)
    if kind != "apply":
        c["tol"] = 10.0 ** rng.uniform(-12, -10)
    if kind in ("traj", "force"):
        c["npf"] = rng.choice([1, 1, 2])
    if kind == "traj":
        c["steps"] = rng.randint(2, 8)
        c["tau"] = c["steps"] * 1.0 / max(math.sqrt(nt * nx), 64.0)
        c["rng"] = rng.choice(["philox", "mt"])
    return c


# ---- inputs -----------------------------------------------------------------------

def _gauge(c, seed):
    return np.random.default_rng([seed, 1]).normal(0, c["sigma"], (c["nt"], c["nx"], 2))


def _vectors(c, seed, n):
    r = np.random.default_rng([seed, 2]).normal(size=(n, c["nt"], c["nx"], 2))
    return r.view(np.complex128)[..., 0]


def _mt_seed(seed):
    return 2 * (seed % 1_000_000) + 1


def _chains(c, seed):
    """n chains: sides uniform in {16 ... 128} (the case's own draw, whatever the
    seed) or all `side`, each with its own mass, coupling, Philox seed and field."""
    r = np.random.default_rng([seed, 3])
    sides = np.random.default_rng(c["n"]).choice([c["side"]] if c["side"] else [16, 24, 32, 48, 64, 96, 128], c["n"])
    chains, fields = [], []
    for L in (int(x) for x in sides):
        k = len(chains)
        chains.append(dict(nt=L, nx=L, m=float(r.uniform(0.05, 0.5)), g=float(r.uniform(0.2, 1.2)), mu=0.0, bc_t=-1,
                           bc_x=1, seed=int(seed * 1000 + k)))
        fields.append(r.normal(0, 0.2, (L, L, 2)))
    return chains, fields


def _cg(c):
    return tg.cg_params(rel_tol=c["tol"], abs_tol2=1e-30 if c["tol"] == 0 else 0.0, precision=c["prec"])


def prepare(case, seed):
    c = case
    s = dict(case=c)
    if c["kind"] == "batch":
        chains, fields = _chains(c, seed)
        s["B"] = tg.Batch(chains)
        for i, A in enumerate(fields):
            s["B"].set_gauge(i, A)
        s["bp"] = tg.batch_params(nsteps=c["steps"], tau=c["tau"], block=c["block"], cg=_cg(c))
        return s
    L = s["L"] = tg.Lattice(c["nt"], c["nx"], c["m"], c["g"], c["mu"], c["bc_t"], c["bc_x"])
    L.set_gauge(_gauge(c, seed))
    L.synchronize()
    if c["kind"] == "traj":
        if c["rng"] == "mt":
            L.seed_mersenne(_mt_seed(seed), 543210)
        s["hp"] = tg.hmc_params(nsteps=c["steps"], tau=c["tau"], npf=c["npf"], seed=seed, cg=_cg(c),
                                rng=tg.native.RNG_MT if c["rng"] == "mt" else tg.native.RNG_PHILOX)
        s["A"] = torch.empty((c["nt"], c["nx"], 2), dtype=torch.float64, pin_memory=True).numpy()
    elif c["kind"] == "force":
        s["phi"] = _vectors(c, seed, c["npf"])
        s["cp"] = _cg(c)
    else:
        dt = torch.complex64 if c["kind"] == "apply" and c["prec"] == MIXED else torch.complex128
        s["v"] = torch.from_numpy(_vectors(c, seed, 1)[0]).to("cuda", dt)
        s["out"] = torch.empty_like(s["v"])
        s["out2"] = torch.empty_like(s["v"])
        if c["kind"] == "cg":
            s["cp"] = _cg(c)
    return s


_ACTIONS = ("Sg0", "Spf0", "Smd0", "Smom0", "Sg1", "Spf1", "Smd1", "Smom1")


def run(state):
    s, c = state, state["case"]
    if c["kind"] == "traj":
        r = s["L"].update_gauge(s["hp"])
        return dict(A=s["L"].get_gauge(s["A"]), accepted=r.accepted, **{k: getattr(r, k) for k in _ACTIONS})
    if c["kind"] == "batch":
        res = s["B"].trajectory(s["bp"])
        return dict(A=np.concatenate([s["B"].get_gauge(i).reshape(-1) for i in range(s["B"].n)]),
                    accepted=np.array([r.accepted for r in res]),
                    **{k: np.array([getattr(r, k) for r in res]) for k in _ACTIONS})
    if c["kind"] == "force":
        F, _ = s["L"].pf_force(s["phi"], s["cp"])
        return F
    if c["kind"] == "cg":
        res = tg.native.CgResult()
        tg.native.check(s["L"].lib.tg_cg_dev(s["L"].h, ctypes.byref(s["cp"]), ctypes.c_void_p(s["v"].data_ptr()),
                                             ctypes.c_void_p(s["out"].data_ptr()), ctypes.byref(res)), True)
        return s["out"]
    for dagger, out in ((False, s["out"]), (True, s["out2"])):
        s["L"].apply_dev(s["v"].data_ptr(), out.data_ptr(), dagger, c["prec"])
    return s["out"], s["out2"]


def _iterations(c):
    """CG iterations of one solve: about 16 / m at 1e-10 on these fields."""
    return 16.0 / c["m"] * (math.log10(1 / c["tol"]) if c.get("tol") else 15.0) / 10.0


def work(case):
    """Bytes: fields in and results out, once.  Flops: 144 per site and CG
    iteration (two applies of 16 complex multiply-adds, three vector updates and
    two norms), 36 per site and lone apply."""
    c = case
    if c["kind"] == "batch":
        sites = c["n"] * (c["side"] ** 2 if c["side"] else 4901)  # the mean of 16^2 ... 128^2
        its = _iterations(dict(c, m=0.195))  # 16 / m over m uniform in [0.05, 0.5]
        return dict(bytes=32.0 * sites, flops=144.0 * sites * its * (c["steps"] + 1))
    V = c["nt"] * c["nx"]
    if c["kind"] == "traj":
        return dict(bytes=32.0 * V, flops=144.0 * V * _iterations(c) * (c["steps"] + 1) * c["npf"])
    if c["kind"] == "force":
        return dict(bytes=(32.0 + 16.0 * c["npf"]) * V, flops=144.0 * V * _iterations(c) * c["npf"])
    if c["kind"] == "cg":
        return dict(bytes=48.0 * V, flops=144.0 * V * _iterations(c))
    # the vector read once by each apply, both links, both results
    return dict(bytes=(128.0 if c["prec"] == FP64 else 64.0) * V, flops=72.0 * V)


# ---- the same in plain torch, 64 bits ------------------------------------------------

class _Field:
    """The operator on one gauge field, or on a stack of them (a leading axis;
    m, g then have shape [n, 1, 1])."""

    def __init__(self, A, m, g, mu, bc_t, bc_x):
        self.A, self.m, self.g, self.ep, self.em = A, m, g, math.exp(mu), math.exp(-mu)
        nt, nx = A.shape[-3], A.shape[-2]
        ft = torch.where(torch.arange(nx, device=A.device) % 2 == 1, -0.5, 0.5).to(A.dtype).expand(nt, nx).clone()
        fx = torch.full((nt, nx), 0.5, dtype=A.dtype, device=A.device)
        ft[-1] *= bc_t
        fx[:, -1] *= bc_x
        self.wt, self.wx = torch.polar(torch.ones_like(A[..., 0]), A[..., 0]) * ft, \
            torch.polar(torch.ones_like(A[..., 1]), A[..., 1]) * fx
        self.wtb, self.wxb = self.wt.conj().roll(1, -2).resolve_conj(), self.wx.conj().roll(1, -1).resolve_conj()

    def apply(self, v, dagger):
        s, cf, cb = (-1, -self.em, self.ep) if dagger else (1, self.ep, -self.em)
        return self.m * v + cf * (self.wt * v.roll(-1, -2)) + cb * (self.wtb * v.roll(1, -2)) \
            + s * (self.wx * v.roll(-1, -1) - self.wxb * v.roll(1, -1))

    def solve(self, b):
        dot = lambda u: (u.real.square() + u.imag.square()).sum((-2, -1), keepdim=True)  # noqa: E731
        x, r, p = torch.zeros_like(b), b.clone(), b.clone()
        rr = dot(r)
        stop = 1e-28 * rr
        for it in range(20000):
            q = self.apply(p, False)
            live = rr > stop  # a stack's finished systems stand still
            a = torch.where(live, rr / dot(q), 0.0)
            x += a * p
            r -= a * self.apply(q, True)
            new = torch.where(live, dot(r), rr)
            p = torch.where(live, r + (new / rr) * p, p)
            rr = new
            if it % 16 == 0 and not bool((rr > stop).any()):
                break
        return x

    def pf_force(self, chi):
        q = self.apply(chi, False)
        nxt = lambda u, ax: u.roll(-1, ax)  # noqa: E731
        ft = self.wt * (self.ep * q.conj() * nxt(chi, -2) - self.em * chi.conj() * nxt(q, -2))
        fx = self.wx * (q.conj() * nxt(chi, -1) - chi.conj() * nxt(q, -1))
        return 2 * torch.stack((ft.imag, fx.imag), -1)

    def gauge_action(self):
        return (NF / self.g * (1 - torch.cos(self.A)).sum(-1)).sum((-2, -1))


def _philox(seed, site, stream):
    """Philox4x32-10 at counter (site, stream, 0, 0): two uniforms of 53 bits."""
    u = np.uint64
    c = [np.asarray(site, u), np.full(np.shape(site), stream, u), np.zeros(np.shape(site), u), np.zeros(np.shape(site), u)]
    k0, k1, low = seed & 0xFFFFFFFF, seed >> 32, u(0xFFFFFFFF)
    for _ in range(10):
        p0, p1 = u(0xD2511F53) * c[0], u(0xCD9E8D57) * c[2]
        c = [(p1 >> u(32)) ^ c[1] ^ u(k0), p1 & low, (p0 >> u(32)) ^ c[3] ^ u(k1), p0 & low]
        k0, k1 = (k0 + 0x9E3779B9) & 0xFFFFFFFF, (k1 + 0xBB67AE85) & 0xFFFFFFFF
    f = lambda hi, lo: (((hi << u(21)) ^ (lo >> u(11))).astype(np.float64) + 0.5) * 2.0 ** -53  # noqa: E731
    return f(c[0], c[1]), f(c[2], c[3])


def _philox_pairs(seed, shape, stream):
    u1, u2 = _philox(seed, np.arange(shape[0] * shape[1]), stream)
    return (np.sqrt(-2 * np.log(u1)) * np.exp(2j * np.pi * u2)).reshape(shape)


class _MT:
    """The reference's stream: MT19937 from the 69069 recurrence, blocks handed out last first."""

    def __init__(self, seed, warmup):
        w = [seed & 0xFFFFFFFF]
        for _ in range(623):
            w.append(69069 * w[-1] & 0xFFFFFFFF)
        self.bits = np.random.MT19937()
        self.bits.state = {"bit_generator": "MT19937", "state": {"key": np.array(w, np.uint32), "pos": 624}}
        self.left = np.empty(0)
        self.take(warmup)

    def take(self, n):
        more = -(-max(0, n - len(self.left)) // 624)
        new = self.bits.random_raw(624 * more).reshape(more, 624)[:, ::-1].reshape(-1) * 2.0 ** -32
        got, self.left = np.split(np.concatenate((self.left, new)), [n])
        return got

    def pairs(self, shape):
        u = self.take(2 * shape[0] * shape[1])
        return (np.sqrt(-2 * np.log(u[0::2])) * np.exp(2j * np.pi * u[1::2])).reshape(shape)


def _trajectory(A, m, g, mu, bc_t, bc_x, etas, mom, noise, u, steps, tau):
    """One leapfrog trajectory (A, momenta and noise may be stacks)."""
    dot = lambda a, b: (a.real * b.real + a.imag * b.imag).sum((-2, -1))  # noqa: E731
    field = lambda a: _Field(a, m, g, mu, bc_t, bc_x)  # noqa: E731
    eps, f = tau / steps, field(A)
    phis = [f.apply(e, True) for e in etas]
    out = dict(Sg0=f.gauge_action(), Spf0=sum(dot(e, e) for e in etas), Smom0=mom.square().sum((-3, -2, -1)),
               Smd0=dot(noise, f.apply(noise, True)))
    old, p = A, mom
    A = A + eps * p
    gi = torch.as_tensor(NF / g)
    for i in range(steps):
        f = field(A)
        F = (gi.unsqueeze(-1) if gi.ndim else gi) * torch.sin(A)
        for phi in phis:
            F = F + f.pf_force(f.solve(phi))
        F[..., 0] -= (f.ep - f.em) * (f.wt * noise.conj() * noise.roll(-1, -2)).imag
        p = p - eps * F
        A = A + eps * p if i == steps - 1 else A + 2 * eps * p
    f = field(A)
    out |= dict(Sg1=f.gauge_action(), Spf1=sum(dot(phi, f.solve(phi)) for phi in phis),
                Smom1=p.square().sum((-3, -2, -1)), Smd1=dot(noise, f.apply(noise, True)))
    dH = sum(out[k + "1"] - out[k + "0"] for k in ("Sg", "Spf", "Smd", "Smom"))
    ok = torch.exp(-dH) > u
    out["A"] = torch.where(ok.reshape(ok.shape + (1, 1, 1)), A, old)
    return out


def _cuda(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _exact_batch(c, seed):
    if c["n"] * (c["side"] ** 2 if c["side"] else 4901) * (c["steps"] + 1) > 3_000_000:
        return None
    chains, fields = _chains(c, seed)
    out = dict(A=[None] * c["n"], **{k: torch.empty(c["n"], dtype=torch.float64) for k in _ACTIONS})
    for L in sorted({k["nt"] for k in chains}):
        who = [i for i, k in enumerate(chains) if k["nt"] == L]
        stack = lambda stream: np.stack([_philox_pairs(chains[i]["seed"], (L, L), stream) for i in who])  # noqa: E731
        col = lambda key: torch.tensor([chains[i][key] for i in who], dtype=torch.float64, device="cuda").reshape(-1, 1, 1)  # noqa: E731
        mom = np.ascontiguousarray(stack(16)).view(np.float64).reshape(len(who), L, L, 2)
        u = _cuda(np.array([_philox(chains[i]["seed"], 0xFFFFFFFF, 18)[0] for i in who]).reshape(-1))
        r = _trajectory(_cuda(np.stack([fields[i] for i in who])), col("m"), col("g"), 0.0, -1, 1, [_cuda(stack(0))],
                        _cuda(mom), _cuda(stack(17)), u, c["steps"], c["tau"])
        for j, i in enumerate(who):
            out["A"][i] = r["A"][j].reshape(-1)
        for k in _ACTIONS:
            out[k][torch.tensor(who)] = r[k].cpu()
    return dict(out, A=torch.cat(out["A"]), accepted=None)


def exact(case, seed):
    c = case
    if c["kind"] == "batch":
        return _exact_batch(c, seed)
    shape = (c["nt"], c["nx"])
    f = _Field(_cuda(_gauge(c, seed)), c["m"], c["g"], c["mu"], c["bc_t"], c["bc_x"])
    if c["kind"] == "traj":
        if shape[0] * shape[1] * (c["steps"] + 1) * _iterations(c) > 6e9:
            return None
        if c["rng"] == "mt":
            mt = _MT(_mt_seed(seed), 543210)
            draws = [mt.pairs(shape) for _ in range(c["npf"] + 2)]
            u = float(mt.take(1)[0])
        else:
            draws = [_philox_pairs(seed, shape, k) for k in [*range(c["npf"]), 16, 17]]
            u = float(_philox(seed, 0xFFFFFFFF, 18)[0])
        mom = np.ascontiguousarray(draws[-2]).view(np.float64).reshape(*shape, 2)
        r = _trajectory(f.A, c["m"], c["g"], c["mu"], c["bc_t"], c["bc_x"], [_cuda(e) for e in draws[:-2]], _cuda(mom),
                        _cuda(draws[-1]), u, c["steps"], c["tau"])
        return dict(A=r["A"], accepted=None, **{k: float(r[k]) for k in _ACTIONS})
    v = _cuda(_vectors(c, seed, c.get("npf", 1)))
    if c["kind"] == "force":
        return sum(f.pf_force(f.solve(phi)) for phi in v)
    if c["kind"] == "cg":
        return f.solve(v[0])
    v = v[0].to(torch.complex64).to(torch.complex128) if c["prec"] == MIXED else v[0]
    return f.apply(v, False), f.apply(v, True)

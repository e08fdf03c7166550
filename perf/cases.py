"""The work that programs built on this package give it, as cases that can be timed and compared.

Each case names a public entry point (``kind``) and its sizes; ``prepare`` makes what the program
holds before the call, ``run`` is one pass, ``exact`` the same result in 64 bits by plain torch and
``work`` the bytes and operations no implementation can do without.

    rhs         Plan.velocity_rhs: one evaluation of the flow's right-hand side
    transforms  Plan.rfft_mpi and Plan.irfft_mpi: both directions in the reference's own layout
    step        ForcedDNS.step: one whole time step, flow and droplets
    ensemble    Ensemble.run: five steps of a batch of small boxes
    gather      Droplets.gather: a field interpolated at the droplets
    collide     Collider.collide: the colliding pairs
    infer       LearnedInterp.infer: the learned interpolation at the droplets
    train       LearnedInterp.train: one epoch of mini-batches
    exact_sum   Plan.exact_sum: the direct Fourier sum that judges an interpolation
"""
import math

import numpy as np
import torch

TWO_PI = 2.0 * math.pi
R_MED = 0.002 * TWO_PI  # median droplet radius of the 256^3 configuration
SETTLING = 0.1          # its settling acceleration
EPS = 0.1               # its forcing power, on shells 1..2
MIXED = (96, 192, 360, 384)


def listed():
    return [
        # the smallest grid the parity tests and golden runs use: six short launches per call
        dict(name="rhs 32 f64", kind="rhs", N=32, precision="f64", nu=0.01, kf=2),
        # the 256^3 configuration's grid
        dict(name="rhs 256 f32", kind="rhs", N=256, precision="f32", nu=2.5e-3, kf=2),
        # the smallest grid on which plain FP64 tricubic meets the interpolation tolerance; 360 is
        # no power of two, so rows and tiles are ragged
        dict(name="rhs 360 f64", kind="rhs", N=360, precision="f64", nu=2.5e-3, kf=2),
        # the precision check's grid, the largest there is
        dict(name="rhs 512 f32", kind="rhs", N=512, precision="f32", nu=1e-3, kf=2),
        # set_velocity, checkpoints and post-processing: the reference's rfft_mpi and irfft_mpi on
        # a vector field, rows of N/2 + 1 coefficients
        dict(name="transforms 192 f32", kind="transforms", N=192, precision="f32", ncomp=3),
        # the 256^3 production step: learned interpolation, 1e6 settling droplets, collisions
        dict(name="step 256 f32 learned", kind="step", N=256, precision="f32", n=1_000_000, method="learned",
             integrator="rk2if", collide=True),
        # a rank's share of the ensemble configuration: 64^3 boxes, trilinear droplets, collisions
        dict(name="ensemble 16 x 64", kind="ensemble", N=64, boxes=16, precision="f32"),
        # droplets set to the fluid velocity at the start and umat of a saved state: positions in
        # no order, an FP64 field of an uneven grid
        dict(name="gather 192 f64 tricubic", kind="gather", N=192, precision="f64", n=500_003, method="tricubic"),
        # the collision search of the 256^3 configuration, on its own
        dict(name="collide 1e6", kind="collide", n=1_000_000),
        # the learned interpolation of the 256^3 configuration, on its own
        dict(name="infer 256 f32", kind="infer", N=256, precision="f32", n=1_000_000),
        # a stretch of the network's training: 64 batches of 4096
        dict(name="train 64 x 4096", kind="train", n=262_144, batch=4096),
        # the judge at an output interval: 1% of 1e6 droplets against the 256^3 spectrum
        dict(name="exact sum 256 f32", kind="exact_sum", N=256, precision="f32", n=10_000),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the same ranges: every grid the package has, droplets over three decades."""
    kind = rng.choice(("rhs", "rhs", "transforms", "step", "step", "ensemble", "gather", "collide", "infer", "train",
                       "exact_sum"))
    prec = rng.choice(("f32", "f64"))
    if kind == "rhs":
        N = rng.choice((16, 32, 64, 96, 128, 192, 256) + ((360, 384) if prec == "f32" else ()))
        return dict(kind=kind, N=N, precision=prec, nu=round(rng.uniform(1e-3, 2e-2), 6), kf=rng.randint(1, 3))
    if kind == "transforms":
        N = rng.choice((16, 32, 64, 96, 128, 192) + ((256,) if prec == "f32" else ()))
        return dict(kind=kind, N=N, precision=prec, ncomp=rng.randint(1, 4))
    if kind == "step":
        N = rng.choice((32, 64, 96, 128))
        if rng.random() < 0.25:
            return dict(kind=kind, N=N, precision=prec, n=0, method="none", integrator="rk4", collide=False)
        method = rng.choice(("trilinear", "tricubic") + (("learned",) if N not in MIXED else ()))
        return dict(kind=kind, N=N, precision=prec, n=_log(rng, 1_000, 200_000), method=method, integrator="rk2if",
                    collide=rng.random() < 0.5)
    if kind == "ensemble":
        return dict(kind=kind, N=rng.choice((32, 64)), boxes=rng.randint(3, 14), precision="f32")
    if kind == "gather":
        N = rng.choice((32, 64, 96, 128, 192, 256))
        return dict(kind=kind, N=N, precision=prec, n=_log(rng, 1_000, 1_000_000),
                    method=rng.choice(("trilinear", "tricubic", "cosine")))
    if kind == "collide":
        return dict(kind=kind, n=_log(rng, 1_000, 1_000_000))
    if kind == "infer":
        return dict(kind=kind, N=rng.choice((64, 128, 256)), precision=prec, n=_log(rng, 1_000, 1_000_000))
    if kind == "train":
        return dict(kind=kind, n=_log(rng, 5_000, 250_000), batch=rng.choice((1000, 2048, 4096, 8192)))
    N = rng.choice((32, 64, 96, 128, 192, 256))
    return dict(kind=kind, N=N, precision=prec, n=min(_log(rng, 100, 20_000), int(1e4 * (256 / N) ** 3)))


# ---- inputs and 64-bit operators, in plain torch --------------------------------------------------
def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


class _Grid:
    """Wave numbers and masks of an N^3 grid in the reference layout (N, N, N/2 + 1)."""

    def __init__(self, N):
        k = torch.fft.fftfreq(N, 1.0 / N, dtype=torch.float64, device="cuda")
        self.N, self.kc = N, N // 3
        self.k = (k[:, None, None], k[None, :, None], k[: N // 2 + 1].abs()[None, None, :])
        self.k2 = self.k[0] ** 2 + self.k[1] ** 2 + self.k[2] ** 2
        self.keep = self.k2 <= self.kc * self.kc + self.kc  # round(|k|) <= N / 3
        self.mzp = (self.kc + 8) // 8 * 8

    def project(self, f):
        kd = (self.k[0] * f[0] + self.k[1] * f[1] + self.k[2] * f[2]) / self.k2.clamp_min(1.0)
        return torch.stack([f[c] - self.k[c] * kd for c in range(3)])

    def inverse(self, f):
        return torch.stack([torch.fft.irfftn(g, s=(self.N,) * 3) for g in f])

    def cube(self, full):
        """The dealiased cube layout (..., 2 kc + 1, 2 kc + 1, kc + 1 padded to a multiple of 8)."""
        rows = torch.cat([torch.arange(self.kc + 1), torch.arange(self.N - self.kc, self.N)]).cuda()
        c = full.index_select(-3, rows).index_select(-2, rows)[..., : self.kc + 1]
        return torch.nn.functional.pad(c, (0, self.mzp - self.kc - 1)).contiguous()


def _flow(N, seed):
    """(grid, solenoidal spectrum of a developed flow): random phases, E(k) rising as k^4 to its
    peak near k = 4, then k^(-5/3) with a viscous tail up to the dealiased edge, mean energy 0.5."""
    g, G = _generator(seed), _Grid(N)
    k = G.k2.sqrt()
    shape = k * (1.0 + (k / 4.0) ** 2) ** (-17.0 / 12.0) * torch.exp(-2.5 * k / (N / 3)) * G.keep
    f = torch.stack([torch.fft.rfftn(torch.randn((N, N, N), dtype=torch.float64, device="cuda", generator=g))
                     for _ in range(3)])
    f = G.project(f) * shape
    w = torch.where(G.k[2] == 0, 1.0, 2.0)
    return G, f * (N ** 3 / (w * f.abs().square()).sum().sqrt())


def _rhs(G, uk, nu, f0, kf, visc):
    """P[(u x w)^ + f] - visc nu k^2 uk on the dealiased modes, f of constant power f0 per shell."""
    i = 1j
    kx, ky, kz = G.k
    u = G.inverse(uk)
    w = G.inverse(torch.stack([i * (ky * uk[2] - kz * uk[1]), i * (kz * uk[0] - kx * uk[2]),
                               i * (kx * uk[1] - ky * uk[0])]))
    nl = torch.stack([torch.fft.rfftn(u[a] * w[b] - u[b] * w[a]) for a, b in ((1, 2), (2, 0), (0, 1))])
    del u, w
    weight = torch.where(kz == 0, 1.0, 2.0).double() * TWO_PI ** 3 / float(G.N) ** 6
    e = (0.5 * weight * uk.abs().square()).sum(0)
    for s in range(1, kf + 1):
        shell = (G.k2 > s * s - s) & (G.k2 <= s * s + s)
        nl = nl + torch.where(shell, f0 / (2.0 * e[shell].sum()), 0.0) * uk
    return torch.where(G.keep, G.project(nl), 0.0) - visc * nu * G.k2 * uk


def _end_of_step(G, uk):
    """The reality round trip (kz = 0 plane made Hermitian) and the projection."""
    p = uk[..., 0]
    uk = uk.clone()
    uk[..., 0] = 0.5 * (p + torch.roll(torch.flip(p, (1, 2)), (1, 1), (1, 2)).conj())
    return torch.where(G.keep, G.project(uk), 0.0)


def _axis(method, s):
    """(offsets, weights (n, W)) of a kernel along one axis at fractional grid offsets s."""
    if method == "trilinear":
        return (0, 1), torch.stack([1 - s, s], 1)
    if method == "cosine":
        return (-1, 0, 1, 2), torch.stack([(1 + torch.cos((s - o) * (math.pi / 2))) / 4 for o in (-1, 0, 1, 2)], 1)
    return (-1, 0, 1, 2), torch.stack([-s * (s - 1) * (s - 2) / 6, (s + 1) * (s - 1) * (s - 2) / 2,
                                       -(s + 1) * s * (s - 2) / 2, (s + 1) * s * (s - 1) / 6], 1)


def _stencil(f, pos, offsets):
    """f (C, N, N, N) at the W^3 grid points around each position: (n, C, W, W, W), and the offsets."""
    N = f.shape[-1]
    q = pos * (N / TWO_PI)
    fl = q.floor()
    j = [(fl[:, d, None].long() + torch.tensor(offsets, device=f.device)) % N for d in range(3)]
    flat = (j[0][:, :, None, None] * N + j[1][:, None, :, None]) * N + j[2][:, None, None, :]
    return f.reshape(f.shape[0], -1)[:, flat].transpose(0, 1), q - fl


def _interp(f, pos, method):
    """f (C, N, N, N) interpolated at pos (n, 3): (n, C)."""
    out = []
    for p in pos.split(1 << 17):
        offsets = _axis(method, p[:, 0])[0]
        s, t = _stencil(f, p, offsets)
        w = [_axis(method, t[:, d])[1] for d in range(3)]
        out.append(torch.einsum("ncabd,na,nb,nd->nc", s, *w))
    return torch.cat(out)


def _poly():
    return torch.tensor([[1, 1, 1, 1], [-3, -1, 1, 3], [1, -1, -1, 1], [-1, 3, -3, 1]], dtype=torch.float64, device="cuda")


def _canonical(f, pos):
    """Stencil of the velocity f in the canonical frame, as polynomial coefficients D (n, 3, 4, 4, 4),
    with the frame's offsets, axis order, per-component sign and the scale of the high orders."""
    s, t = _stencil(f, pos, (-1, 0, 1, 2))
    refl = t > 0.5
    for d in range(3):
        s = torch.where(refl[:, d, None, None, None, None], torch.flip(s, (2 + d,)), s)
    r = torch.where(refl, 1 - t, t)
    order = torch.sort(r, dim=1, descending=True, stable=True).indices
    D = torch.empty_like(s)
    for p in ((0, 1, 2), (0, 2, 1), (1, 0, 2), (1, 2, 0), (2, 0, 1), (2, 1, 0)):
        m = (order == torch.tensor(p, device=order.device)).all(1)
        D[m] = s[m][:, list(p)].permute(0, 1, 2 + p[0], 2 + p[1], 2 + p[2])
    sign = torch.where(refl, -1.0, 1.0).double().gather(1, order)
    D = torch.einsum("ncabd,ia,jb,kd->ncijk", D * sign[:, :, None, None, None], _poly(), _poly(), _poly())
    a = torch.arange(4, device=D.device)
    high = (a[:, None, None] + a[None, :, None] + a[None, None, :]) >= 3
    scale = (D[:, :, high].square().sum((1, 2)) / 162).sqrt()
    return D, r.gather(1, order), order, sign, scale


def _network(f, seed):
    """Weights as training starts them, with the feature scales of this flow and a small output:
    a dict of arrays W1 (195, 128), b1, W2 (128, 128), b2, W3 (128, 3), b3, fs (64), os."""
    rng = np.random.default_rng(seed + 1)

    def lin(i, o):
        lim = math.sqrt(6.0 / i)
        return rng.uniform(-lim, lim, (i, o)).astype(np.float32), (0.1 * rng.standard_normal(o)).astype(np.float32)

    (W1, b1), (W2, b2), (W3, b3) = lin(195, 128), lin(128, 128), lin(128, 3)
    at = torch.rand((4096, 3), dtype=torch.float64, device="cuda", generator=_generator(seed + 2)) * TWO_PI
    D, _, _, _, scale = _canonical(f, at)
    rms = (D / scale[:, None, None, None, None]).square().mean((0, 1)).sqrt().clamp_min(1e-30)
    return dict(W1=W1, b1=b1, W2=W2, b2=b2, W3=0.1 * W3, b3=0.1 * b3,
                fs=(1.0 / rms).reshape(64).float().cpu().numpy(), os=0.02)


def _learned(f, pos, net):
    """tricubic + scale * os * MLP at pos, with the FP32 weights and everything else in 64 bits."""
    w = {k: torch.as_tensor(np.asarray(v, np.float64), device="cuda") for k, v in net.items() if k != "os"}
    out = []
    for p in pos.split(1 << 16):
        D, t, order, sign, scale = _canonical(f, p)
        x = D / scale[:, None, None, None, None] * w["fs"].reshape(4, 4, 4)
        h = torch.cat([x.reshape(len(p), 192), t - 0.5], 1) @ w["W1"] + w["b1"]
        h = torch.nn.functional.silu(h) @ w["W2"] + w["b2"]
        y = torch.nn.functional.silu(h) @ w["W3"] + w["b3"]
        corr = torch.zeros_like(y).scatter(1, order, scale[:, None] * float(np.float32(net["os"])) * sign * y)
        out.append(_interp(f, p, "tricubic") + corr)
    return torch.cat(out)


def _droplets(n, seed, nu):
    """Uniform positions, lognormal radii and the Stokes times they have (tau ~ r^2, median St = 0.5)."""
    g = _generator(seed + 3)
    pos = torch.rand((n, 3), dtype=torch.float64, device="cuda", generator=g) * TWO_PI
    radius = R_MED * torch.exp(0.3 * torch.randn(n, dtype=torch.float64, device="cuda", generator=g))
    return pos, radius, 0.5 * math.sqrt(nu / EPS) * (radius / R_MED).square()


def _cell(n):
    """Collision cells of twice the radius that all but 1e-4 of the droplets stay below, and not
    narrower than a quarter droplet per cell asks for."""
    return min(max(2.0 * R_MED * math.exp(0.3 * 3.719), TWO_PI / max(3, round((4.0 * n) ** (1 / 3)))), TWO_PI / 3)


def _step_parameters(N):
    nu, dt = (2.5e-3, 1e-3) if N >= 256 else (0.01, 2e-3)
    return nu, dt, EPS * TWO_PI ** 3 / 2


def _real(case):
    return torch.float32 if case["precision"] == "f32" else torch.float64


def _complex(case):
    return torch.complex64 if case["precision"] == "f32" else torch.complex128


def _step_inputs(case, seed):
    """What a run has after set-up, rounded to the plan's precision: grid, spectrum, network,
    droplets at (nearly) the fluid velocity."""
    G, uk = _flow(case["N"], seed)
    uk = uk.to(_complex(case))
    if not case["n"]:
        return G, uk, None, None
    u = G.inverse(uk.to(torch.complex128))
    net = _network(u, seed) if case["method"] == "learned" else None
    pos, radius, tau = _droplets(case["n"], seed, _step_parameters(case["N"])[0])
    vel = _interp(u, pos, "trilinear")
    return G, uk, net, (pos, vel.to(_real(case)), tau.to(_real(case)), radius)


def _velocity(case, seed):
    """The planar physical velocity of a flow, in the plan's precision."""
    G, uk = _flow(case["N"], seed)
    return G.inverse(uk).to(_real(case))


# ---- the cases' states and passes ----------------------------------------------------------------
def prepare(case, seed):
    from lucky_droplets_b200.collide import Collider
    from lucky_droplets_b200.dns import Droplets, ForcedDNS
    from lucky_droplets_b200.mlp import LearnedInterp, flat_from_mats
    from lucky_droplets_b200.spectral import Plan

    kind, s = case["kind"], {"case": case}
    if kind == "rhs":
        G, uk = _flow(case["N"], seed)
        s["plan"] = Plan(case["N"], case["precision"])
        s["uk"] = G.cube(uk).to(_complex(case))
        s["ku"] = torch.empty_like(s["uk"])
    elif kind == "transforms":
        N, nc, g = case["N"], case["ncomp"], _generator(seed)
        s["plan"] = Plan(N, case["precision"])
        s["u"] = torch.randn((nc, N, N, N), dtype=_real(case), device="cuda", generator=g)
        s["fk"] = torch.fft.rfftn(torch.randn((nc, N, N, N), dtype=torch.float64, device="cuda", generator=g),
                                  dim=(1, 2, 3)).to(_complex(case))
        s["fu"], s["v"] = torch.empty_like(s["fk"]), torch.empty_like(s["u"])
    elif kind == "step":
        G, uk, net, drops = _step_inputs(case, seed)
        nu, dt, f0 = _step_parameters(case["N"])
        dns = s["dns"] = ForcedDNS(case["N"], nu, dt, f0, shell_no=(1, 2), integrator=case["integrator"],
                                   precision=case["precision"])
        dns.set_uk_full(uk)
        if drops is not None:
            pos, vel, tau, radius = drops
            d = Droplets(dns.plan, pos, vel, tau, method="tricubic" if net else case["method"], g=SETTLING,
                         radius=radius)
            col = Collider(d.n, _cell(d.n)) if case["collide"] else None
            dns.attach(d, collider=col, sort_every=20 if case["collide"] else 0)
            if net:
                d.use_learned(LearnedInterp(dns.plan, params=flat_from_mats(**net)))
    elif kind == "ensemble":
        from lucky_droplets_b200.ensemble import Ensemble
        # the configuration's uneven droplet counts, radii and Stokes times, restarted from flows
        # and droplets of this seed
        ens = s["ens"] = Ensemble(case["boxes"], case["N"], precision=case["precision"], seed=0)
        ens.pos.copy_(_droplets(ens.n, seed, 0.01)[0])
        for j in range(ens.nb):
            G, uk = _flow(case["N"], 1000 * int(seed) + j)
            ens.uk[j].copy_(G.cube(uk))
            m = ens.box == j
            ens.vel[m] = _interp(G.inverse(uk), ens.pos[m], "trilinear").to(ens.vel.dtype)
        ens.sort()
        ens.capture(5)
    elif kind == "gather":
        plan = Plan(case["N"], case["precision"])
        s["u"] = _velocity(case, seed)
        pos, radius, tau = _droplets(case["n"], seed, 0.01)
        s["drops"] = Droplets(plan, pos, torch.zeros_like(pos), tau, method=case["method"])
        s["out"] = torch.empty((case["n"], 3), dtype=_real(case), device="cuda")
    elif kind == "collide":
        s["pos"], s["radius"], _ = _droplets(case["n"], seed, 0.01)
        s["collider"] = Collider(case["n"], _cell(case["n"]))
        s["pairs"] = torch.zeros((max(1024, 4 * case["n"]), 2), dtype=torch.int32, device="cuda")
    elif kind == "infer":
        plan = Plan(case["N"], case["precision"])
        u = _velocity(case, seed)
        s["net"] = LearnedInterp(plan, params=flat_from_mats(**_network(u.double(), seed)))
        s["u4"] = torch.cat([u, torch.zeros_like(u[:1])]).permute(1, 2, 3, 0).contiguous()
        s["pos"] = _sorted_positions(case, seed)
        s["out"] = torch.empty((case["n"], 3), dtype=_real(case), device="cuda")
        s["work"] = s["net"].workspace(case["n"])
    elif kind == "train":
        n, g = case["n"], _generator(seed)
        X = torch.zeros((n, 208), dtype=torch.bfloat16, device="cuda")
        X[:, :195] = torch.randn((n, 195), device="cuda", generator=g)
        T = torch.tanh(X[:, :3].float() * X[:, 64:67].float()) + 0.3 * torch.randn((n, 3), device="cuda", generator=g)
        s["data"] = (X, T, torch.rand(n, device="cuda", generator=g) + 0.5)
        s["net"] = LearnedInterp(Plan(16, "f32"), seed=int(seed))
    else:
        G, uk = _flow(case["N"], seed)
        s["plan"] = Plan(case["N"], case["precision"])
        s["uk"] = G.cube(uk).to(_complex(case))
        s["pos"] = _droplets(case["n"], seed, 0.01)[0]
        s["out"] = torch.empty((case["n"], 3), dtype=torch.float64, device="cuda")
    return s


def _cell_keys(pos, nc):
    c = (pos * (nc / TWO_PI)).long().clamp(max=nc - 1)
    return (c[:, 0] * nc + c[:, 1]) * nc + c[:, 2]


def _sorted_positions(case, seed):
    """Positions in cell order, as a run keeps them for its stencil loads."""
    pos = _droplets(case["n"], seed, 0.01)[0]
    return pos[torch.argsort(_cell_keys(pos, case["N"] // 4), stable=True)].contiguous()


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "rhs":
        f0 = EPS * TWO_PI ** 3 / case["kf"]
        return state["plan"].velocity_rhs(state["uk"], case["nu"], f0, tuple(range(1, case["kf"] + 1)), ku=state["ku"])
    if kind == "transforms":
        plan = state["plan"]
        return {"forward": plan.rfft_mpi(state["u"], state["fu"]), "inverse": plan.irfft_mpi(state["fk"], state["v"])}
    if kind == "step":
        dns = state["dns"]
        dns.step()
        out = {"uk": dns.uk}
        if dns.droplets is not None:
            out.update(pos=dns.droplets.pos, vel=dns.droplets.vel, ids=dns.droplets.ids)
        if dns.collider is not None:
            out["colliding"] = dns.collider.count
        return out
    if kind == "ensemble":
        ens = state["ens"]
        ens.run(5)
        return {"uk": ens.uk, "pos": ens.pos, "vel": ens.vel, "ids": ens.dids, "colliding": ens.collider.box_counts}
    if kind == "gather":
        return state["drops"].gather(state["u"], out=state["out"])
    if kind == "collide":
        found = state["collider"].collide(state["pos"], state["radius"], state["pairs"])
        return {"count": int(found.shape[0]), "pairs": state["pairs"]}
    if kind == "infer":
        return state["net"].infer(state["u4"], state["pos"], out=state["out"], work=state["work"])
    if kind == "train":
        losses = state["net"].train(*state["data"], batch=case["batch"], lr=2e-3)
        return {"losses": losses, "params": state["net"].params}
    return state["plan"].exact_sum(state["uk"], state["pos"], out=state["out"])


# ---- the same in 64 bits ---------------------------------------------------------------------------
def _exact_step(case, seed):
    G, uk, net, drops = _step_inputs(case, seed)
    uk = uk.to(torch.complex128)
    uk = torch.where(G.keep, uk, 0.0)
    nu, h, f0 = _step_parameters(case["N"])
    if case["integrator"] == "rk4":
        k1 = _rhs(G, uk, nu, f0, 2, 1.0)
        k2 = _rhs(G, uk + h / 2 * k1, nu, f0, 2, 1.0)
        k3 = _rhs(G, uk + h / 2 * k2, nu, f0, 2, 1.0)
        k4 = _rhs(G, uk + h * k3, nu, f0, 2, 1.0)
        return {"uk": G.cube(_end_of_step(G, uk + h / 6 * (k1 + 2 * k2 + 2 * k3 + k4)))}
    E = torch.exp(-nu * h * G.k2)
    n1 = _rhs(G, uk, nu, f0, 2, 0.0)
    mid = E * (uk + h * n1)
    new = _end_of_step(G, E * (uk + h / 2 * n1) + h / 2 * _rhs(G, mid, nu, f0, 2, 0.0))
    pos, vel, tau, _ = drops
    if case["collide"]:
        order = torch.argsort(_cell_keys(pos, int(TWO_PI / _cell(case["n"]))), stable=True)
        pos, vel, tau = pos[order], vel[order], tau[order]
    vel, tau = vel.double(), tau.double()[:, None]

    def accel(spec, x, v):
        u = G.inverse(spec)
        a = ((_learned(u, x, net) if net else _interp(u, x, case["method"])) - v) / tau
        a[:, 2] -= SETTLING
        return a

    a1 = accel(uk, pos, vel)
    vs = vel + h * a1
    a2 = accel(mid, pos + h * vel, vs)
    return {"uk": G.cube(new), "pos": pos + h / 2 * (vel + vs), "vel": vel + h / 2 * (a1 + a2), "ids": None,
            "colliding": None}


def _exact_sum(uk, pos):
    """The Fourier sum of cube-layout uk at pos, the three axes as dense contractions."""
    kc = (uk.shape[1] - 1) // 2
    k = torch.cat([torch.arange(kc + 1), torch.arange(-kc, 0)]).double().cuda()
    ex, ey, ez = (torch.exp(1j * k[:, None] * pos[None, :, d]) for d in range(3))
    ez = ez[: kc + 1].clone()
    ez[1:] *= 2.0
    out = torch.zeros((3, pos.shape[0]), dtype=torch.float64, device="cuda")
    for ix in range(uk.shape[1]):
        t = uk[:, ix, :, : kc + 1] @ ez          # (3, ky, n)
        out += ((t * ey).sum(1) * ex[ix]).real
    return out.T


def exact(case, seed):
    kind = case["kind"]
    if kind == "rhs":
        G, uk = _flow(case["N"], seed)
        uk = uk.to(_complex(case)).to(torch.complex128)
        return G.cube(_rhs(G, uk, case["nu"], EPS * TWO_PI ** 3 / case["kf"], case["kf"], 1.0))
    if kind == "transforms":
        N, nc, g = case["N"], case["ncomp"], _generator(seed)
        u = torch.randn((nc, N, N, N), dtype=_real(case), device="cuda", generator=g).double()
        fk = torch.fft.rfftn(torch.randn((nc, N, N, N), dtype=torch.float64, device="cuda", generator=g),
                             dim=(1, 2, 3)).to(_complex(case)).to(torch.complex128)
        return {"forward": torch.fft.rfftn(u, dim=(1, 2, 3)), "inverse": torch.fft.irfftn(fk, s=(N,) * 3, dim=(1, 2, 3))}
    if kind == "step":
        return _exact_step(case, seed)
    if kind == "gather":
        return _interp(_velocity(case, seed).double(), _droplets(case["n"], seed, 0.01)[0], case["method"])
    if kind == "infer":
        u = _velocity(case, seed).double()
        return _learned(u, _sorted_positions(case, seed), _network(u, seed))
    if kind == "exact_sum":
        G, uk = _flow(case["N"], seed)
        uk = G.cube(uk).to(_complex(case)).to(torch.complex128)
        return _exact_sum(uk, _droplets(case["n"], seed, 0.01)[0]) / float(case["N"]) ** 3
    # an ensemble starts from its own construction, pairs are whole numbers, and an epoch's end
    # depends on every rounding before it
    return None


def work(case):
    """Inputs read once and outputs written once; transforms as 2.5 N^3 log2 N^3 each, the network's
    and the sum's multiply-adds as two."""
    kind, N = case["kind"], case.get("N", 0)
    r = 8 if case.get("precision") == "f64" else 4
    kc = N // 3
    cube = 3 * (2 * kc + 1) ** 2 * (kc + 1) * 2 * r
    fft = 2.5 * N ** 3 * 3 * math.log2(N) if N else 0.0
    mlp = 2 * (195 * 128 + 128 * 128 + 128 * 3)
    n = case.get("n", 0)
    if kind == "rhs":
        return {"bytes": 2 * cube, "flops": 9 * fft}
    if kind == "transforms":
        nc = case["ncomp"]
        return {"bytes": 2 * nc * (N ** 3 * r + N * N * (N // 2 + 1) * 2 * r), "flops": 2 * nc * fft}
    if kind == "step":
        stages = 2 if case["integrator"] == "rk2if" else 4
        taps = 0 if not n else {"trilinear": 8, "tricubic": 64, "learned": 64}[case["method"]]
        per = stages * (taps * 6 + (mlp if case["method"] == "learned" else 0))
        return {"bytes": 2 * cube + n * (2 * (24 + 3 * r) + r + (16 if case["collide"] else 0)),
                "flops": stages * 9 * fft + n * per}
    if kind == "ensemble":
        n = 27_500 * case["boxes"]
        return {"bytes": 5 * (case["boxes"] * 2 * cube + n * (2 * (24 + 3 * r) + r + 12)),
                "flops": 5 * (case["boxes"] * 18 * fft + n * 96)}
    if kind == "gather":
        return {"bytes": min(3 * N ** 3, 192 * n) * r + n * (24 + 3 * r), "flops": 384 * n}
    if kind == "collide":
        return {"bytes": 40 * n, "flops": 10 * n}
    if kind == "infer":
        return {"bytes": min(4 * N ** 3, 256 * n) * r + n * (24 + 3 * r), "flops": mlp * n}
    if kind == "train":
        used = n // min(case["batch"], n) * min(case["batch"], n)
        return {"bytes": used * (208 * 2 + 16 + 4), "flops": used * (mlp + 2 * (2 * 128 * 3 + 2 * 128 * 128 + 195 * 128))}
    modes = 2 / 3 * math.pi * (kc + 0.5) ** 3
    return {"bytes": cube + 48 * n, "flops": 12 * modes * n}

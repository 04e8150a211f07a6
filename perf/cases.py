"""Performance cases: what programs have this framework do, through its public entry points.

Kinds:
  kick     cube_gpu_kick on a device-resident state (PM1, PM2, PM3 and PP: nearly all of a
           step), then the velocities read back into the caller's page-locked array
  step     cube_gpu_step (drift and kick) on a device-resident state, then the state read back
  host     cube_gpu_step_host: the loop body of a host that keeps the particles itself
  power    Context.power, the power spectrum of the resident particles
  density  cube_gpu_pm1_density_noalloc on the caller's device arrays
  force    DPM.force and DPM.force_vjp of the differentiable PM step
  grad     Simulate and Density of cube_nu_b200.adjoint, forward and backward

Particle states are drawn here with torch, from the seed alone: a lattice displaced by a
smooth random field (early times), plus haloes (late times), in the checkpoint layout.
"form" is the pair of forms of the step: "chosen" (int64 fixed-point deposit, queue PP, each
step one CUDA graph) or "plain" (the defaults of Params).
"""
import ctypes
import math

import numpy as np
import torch
import torch.utils.checkpoint

from cube_nu_b200 import _lib, adjoint
from cube_nu_b200.params import DEPOSIT_FIXED, DEPOSIT_FP32, Params

# A step's inputs early in a run: a_mid at z = 49, and a dt that moves particles by a few
# thousandths of a cell, so that a state stays what it is over the passes of a measurement.
STEP = {"dt": 0.02, "a_mid": 0.02, "vrms": 0.1}
# A kick's: dv of the order of v, so that an error of the force shows in the velocities.
KICK = {"dt": 0.5, "a_mid": 0.5, "vrms": 0.3}


def _nbody(name, kind, ng, nnt, nns, np_nc, count, izipx, form, halo):
    case = {"name": name} if name else {}
    return case | {"kind": kind, "ng": ng, "nnt": nnt, "nns": nns, "np_nc": np_nc, "np": count, "izipx": izipx,
                   "form": form, "halo": halo}


def listed():
    return [
        # a density field for a caller on a latency-bound path: 32^3 cells, a ragged particle count
        {"name": "density_32", "kind": "density", "nc": 32, "np": 261893, "izipx": 2, "form": "chosen"},
        # one force and its adjoint on a small differentiable mesh
        {"name": "force_64", "kind": "force", "n": 64, "np": 32768},
        # a whole step of the smallest box (the geometry of the tests), in the plain form
        _nbody("step_32_plain", "step", 64, 2, 2, 2, 32768, 1, "plain", 0.0),
        # a step of the 128^3 configuration (200 Mpc/h, mesh 256^3, int8 codes), chosen form
        _nbody("step_128", "step", 256, 4, 4, 2, 2097152, 1, "chosen", 0.0),
        # the same box for a host program that keeps its particles, with its own int16 codes
        _nbody("host_128_plain", "host", 256, 4, 4, 2, 2097152, 2, "plain", 0.0),
        # the default parameters (ng = 128, 64 particles per cell), plain form, mildly clustered
        _nbody("kick_default_plain", "kick", 128, 4, 4, 4, 2093117, 2, "plain", 0.1),
        # three tiles a side and a ragged particle count: sides of 72, 128 and 64
        _nbody("kick_288", "kick", 288, 3, 4, 2, 2901013, 1, "chosen", 0.1),
        # an eighth of the 512^3 box at its mesh sides (PM2 288^3, PM3 144^3), chosen form
        _nbody("kick_256", "kick", 512, 2, 4, 2, 16777216, 2, "chosen", 0.0),
        # one tile of that box in the plain form
        _nbody("kick_tile_plain", "kick", 256, 1, 4, 2, 2097152, 2, "plain", 0.0),
        # an eighth of the clustered 256^3 configuration late in its run: thousands of particles in a cell
        _nbody("kick_late", "kick", 128, 2, 4, 4, 2097152, 2, "chosen", 0.45),
        # P(k) on a grid of twice the mesh, as cicpower measures it
        {"name": "power_512", "kind": "power", "ng": 256, "np": 2097152, "izipx": 2, "form": "chosen", "nw": 512},
        # the differentiable configuration at a quarter of its length: forward and gradient
        {"name": "grad_256", "kind": "grad", "n": 256, "np": 2097152, "steps": 5},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["kick"] * 9 + ["step"] * 3 + ["host"] * 2 + ["power"] * 2 + ["density"] * 2 + ["force", "grad"])
    form = rng.choice(["chosen", "plain"])
    izipx = rng.choice([1, 2])
    if kind == "density":
        nc = rng.choice([16, 24, 32, 48, 64])
        return {"kind": kind, "nc": nc, "np": min(2097152, _log_int(rng, nc ** 3, 16 * nc ** 3)), "izipx": izipx,
                "form": form}
    if kind in ("force", "grad"):
        n = rng.choice([32, 48, 64, 96, 128, 144, 192, 256] if kind == "force" else [32, 48, 64, 96, 128])
        case = {"kind": kind, "n": n, "np": _log_int(rng, n ** 3 // 8, n ** 3 // 4)}
        if kind == "grad":
            case["steps"] = rng.randint(2, 8)
        return case
    if kind == "power":
        return {"kind": kind, "ng": rng.choice([64, 128, 256]), "np": _log_int(rng, 1 << 15, 1 << 22), "izipx": izipx,
                "form": form, "nw": rng.choice([64, 96, 128, 192, 256, 384, 512])}
    # tiles of 32 to 256 fine cells a side; every mesh side of the levels is 2^a 3^b
    ngp, nns = rng.choice([(32, 4), (32, 2), (64, 4), (64, 8), (96, 4), (96, 6), (256, 4)])
    nnt = rng.choice({32: [2, 3, 4, 6, 8], 64: [1, 2, 3, 4], 96: [1, 2, 3], 256: [1]}[ngp])
    ng = ngp * nnt
    np_nc = rng.choice([2, 2, 3, 4]) if ng <= 128 else 2
    n = (ng // 4 * np_nc) ** 3
    n = n if rng.random() < 0.3 else max(1024, int(n * rng.uniform(0.8, 1.0)))
    halo = rng.choice([0.0, 0.0, 0.1, 0.3, 0.5]) if kind == "kick" else 0.0
    return _nbody("", kind, ng, nnt, nns, np_nc, n, izipx, form, halo)


# ------------------------------------------------------------------------------------
# Inputs
# ------------------------------------------------------------------------------------
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _displacement(m, g, rms):
    """Three components of a smooth random displacement field on an m^3 lattice (a
    gradient of a Gaussian field with power on the large scales), (m^3, 3), x fastest."""
    w = torch.randn((m, m, m), generator=g, device="cuda")
    k1 = torch.fft.fftfreq(m, 1.0 / m, device="cuda")
    kx = torch.arange(m // 2 + 1, device="cuda", dtype=torch.float32)
    k2 = kx[None, None, :] ** 2 + k1[None, :, None] ** 2 + k1[:, None, None] ** 2
    k2[0, 0, 0] = 1.0
    wk = torch.fft.rfftn(w) * torch.exp(-k2 * (2.0 / m) ** 2) * k2 ** -1.25
    wk[0, 0, 0] = 0.0
    out = torch.empty((m, m, m, 3), device="cuda")
    for d, k in enumerate((kx[None, None, :], k1[None, :, None], k1[:, None, None])):
        out[..., d] = torch.fft.irfftn(1j * k * wk, s=(m, m, m))
    out = out.reshape(-1, 3)
    return out * (rms / out.square().mean().sqrt())


def _positions(n, nc, g, halo):
    """Positions (n, 3) in coarse cells and a smooth velocity pattern: a displaced lattice
    cut to n points, with a share `halo` of the particles moved into haloes of a power-law
    range of masses."""
    m = max(2, math.ceil(round(n ** (1 / 3), 6)))
    m += m % 2
    disp = _displacement(m, g, 0.15 if halo == 0 else 0.4)
    q = (torch.arange(m, device="cuda") + 0.5) * (nc / m)
    lat = torch.stack(torch.meshgrid(q, q, q, indexing="ij")[::-1], dim=-1).reshape(-1, 3)
    if m ** 3 > n:
        keep = torch.randperm(m ** 3, generator=g, device="cuda")[:n].sort().values
        lat, disp = lat[keep], disp[keep]
    x = lat.double() + disp.double()
    vel = disp / disp.square().mean().sqrt()
    nh = int(n * halo)
    if nh:
        count = max(4, int(nc ** 3 * 0.01))
        mass = torch.rand(count, generator=g, device="cuda", dtype=torch.float64).clamp_min(1e-3) ** -(0.5 + 0.5 * halo)
        centre = torch.rand((count, 3), generator=g, device="cuda", dtype=torch.float64) * nc
        edge = torch.cumsum(mass, 0) / mass.sum()
        who = torch.randperm(n, generator=g, device="cuda")[:nh]
        h = torch.searchsorted(edge, torch.rand(nh, generator=g, device="cuda", dtype=torch.float64)).clamp_max(count - 1)
        r = torch.rand(nh, generator=g, device="cuda", dtype=torch.float64) ** 1.5 * 0.35 * mass[h] ** (1 / 3) + 0.01
        u = torch.randn((nh, 3), generator=g, device="cuda", dtype=torch.float64)
        x[who] = centre[h] + u / u.norm(dim=1, keepdim=True).clamp_min(1e-9) * r[:, None]
        vel[who] = torch.randn((nh, 3), generator=g, device="cuda")
    return torch.remainder(x, float(nc)), vel


def _state(case, seed, nc, nnt, vrms):
    """(xp, vp, pid, rhoc) in the checkpoint layout as CUDA tensors."""
    g = _gen(seed)
    x, vel = _positions(case["np"], nc, g, case.get("halo", 0.0))
    n, bits, nt = case["np"], 8 * case["izipx"], nc // nnt
    cell = x.floor().long().clamp_(0, nc - 1)
    code = ((x - cell) * (1 << bits)).floor().long().clamp_(0, (1 << bits) - 1)
    code = torch.where(code >= 1 << (bits - 1), code - (1 << bits), code)
    t, l = cell // nt, cell % nt
    order = ((((t[:, 2] * nnt + t[:, 1]) * nnt + t[:, 0]) * nt + l[:, 2]) * nt + l[:, 1]) * nt + l[:, 0]
    perm = torch.sort(order, stable=True).indices
    xp = code[perm].to(torch.int8 if bits == 8 else torch.int16)
    vp = (vel[perm] * (vrms / vel.square().mean().sqrt())).float()
    rhoc = torch.bincount(order, minlength=nc ** 3).int()
    return xp.contiguous(), vp.contiguous(), torch.arange(1, n + 1, device="cuda")[perm].contiguous(), rhoc


def _params(case, nnt=None, nns=None):
    p = Params(ng=case["ng"], nnt=nnt or case["nnt"], nns=nns or case["nns"], np_nc=case.get("np_nc", 2),
               izipx=case["izipx"], box=case["ng"] * 200.0 / 256.0)
    if case["form"] == "chosen":
        p.deposit_mode, p.pp_queue, p.step_graph = DEPOSIT_FIXED, True, True
    else:
        p.deposit_mode = DEPOSIT_FP32
    p.mass_p_cdm = float(p.ng) ** 3 / case["np"]
    return p


def _pinned(t):
    h = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
    h.copy_(t)
    return h


def _ptr(t):
    return ctypes.c_void_p(t.data_ptr())


def _mesh_inputs(case, seed):
    """Inputs of the differentiable step: real positions in mesh cells, and a cotangent of
    the force, or velocities, (drift, kick) factors and a target density."""
    g, n = _gen(seed), case["n"]
    x, vel = _positions(case["np"], n, g, 0.0)
    x = torch.remainder(x.float(), float(n)).clamp_max(n * (1 - 2 ** -23)).contiguous()
    s = {"kind": case["kind"], "x": x}
    if case["kind"] == "force":
        s["u"] = torch.randn(x.shape, generator=g, device="cuda")
    else:
        s["x"].requires_grad_(True)
        s["v"] = (0.3 * vel).float().contiguous().requires_grad_(True)
        s["steps"] = [(0.5, 0.01 * (1 + k)) for k in range(case["steps"])]
        s["target"] = 1 + 0.5 * torch.randn((n,) * 3, generator=g, device="cuda")
    return s


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("force", "grad"):
        return _mesh_inputs(case, seed) | {"dpm": adjoint.DPM(case["n"], 3.5, case["n"] ** 3 / case["np"])}
    if kind == "density":
        p = _params({**case, "ng": 4 * case["nc"]}, nnt=2, nns=2)
        xp, _, _, rhoc = _state(case, seed, case["nc"], 2, 0.0)
        return {"kind": kind, "lib": _lib.load(), "cp": p.to_c(), "np": case["np"], "xp": xp, "rhoc": rhoc,
                "rho": torch.empty((case["nc"],) * 3, device="cuda")}
    if kind == "power":
        p = _params(case, nnt=case["ng"] // 64, nns=4)
    else:
        p = _params(case)
    use = KICK if kind == "kick" else STEP
    st = _state(case, seed, p.nc, p.nnt, use["vrms"])
    vz = float(st[1][:, 2].abs().max())
    host = [_pinned(t) for t in st]
    del st
    torch.cuda.empty_cache()  # the context takes what it needs of the free memory
    s = {"kind": kind, "ctx": _lib.Context(p), "host": host, "vz": vz, "dt_old": use["dt"], **use}
    if kind == "power":
        s["nw"] = case["nw"]
    if kind != "host":
        s["ctx"].upload(*[h.numpy() for h in host])
    return s


# ------------------------------------------------------------------------------------
# One pass
# ------------------------------------------------------------------------------------
def _read_back(ctx, *arrays):
    n = ctypes.c_int64()
    _lib._check(ctx._lib.cube_gpu_download(ctx._h, *[None if a is None else _ptr(a) for a in arrays], ctypes.byref(n)),
                "cube_gpu_download")


def _results(so):
    return {"f2max": [so.f2max_pm1, so.f2max_pm2, so.f2max_pm3, so.f2max_pp], "vmax": list(so.vmax),
            "dt": [so.dt_pm1, so.dt_pm2, so.dt_pm3, so.dt_pp, so.dt_vmax],
            "mass": [so.mass_pm1, so.mass_pm2, so.mass_pm3], "pairs": float(so.pp_pairs),
            "candidates": float(so.pp_candidates), "napm": [float(so.napm[i]) for i in range(2, 6)]}


def run(state):
    kind = state["kind"]
    if kind == "force":
        return {"force": state["dpm"].force(state["x"]), "vjp": state["dpm"].force_vjp(state["x"], state["u"])}
    if kind == "grad":
        x, v, target = state["x"], state["v"], state["target"]
        end = adjoint.Simulate.apply(x, v, state["dpm"], state["steps"], 0.25, 5)
        rho = adjoint.Density.apply(end, state["dpm"])
        loss = ((rho - target) ** 2).mean()
        gx, gv = torch.autograd.grad(loss, (x, v))
        return {"rho": rho.detach(), "loss": loss.detach(), "gx": gx, "gv": gv}
    if kind == "density":
        stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
        _lib._check(state["lib"].cube_gpu_pm1_density_noalloc(
            ctypes.byref(state["cp"]), _ptr(state["xp"]), _ptr(state["rhoc"]), ctypes.c_int64(state["np"]),
            _ptr(state["rho"]), stream), "cube_gpu_pm1_density_noalloc")
        return {"rho": state["rho"]}
    ctx = state["ctx"]
    if kind == "power":
        xi, _, out = ctx.power(state["nw"])
        return {"modes": xi[:, 0], "k": xi[:, 1], "raw": xi[:, 2], "power": xi[:, 3], "corrected": xi[:, 4],
                "mean": out.mean}
    xp, vp, pid, rhoc = state["host"]
    dt, a_mid = state["dt"], state["a_mid"]
    if kind == "kick":
        so = ctx.kick(dt, a_mid)
        _read_back(ctx, None, vp, None, None)
        return {"vp": vp, **_results(so)}
    if kind == "step":
        so = ctx.step(dt, state["dt_old"], a_mid, state["vz"])
        _read_back(ctx, xp, vp, pid, rhoc)
    else:
        so = ctx.step_host(xp.numpy(), vp.numpy(), pid.numpy(), rhoc.numpy(), dt, state["dt_old"], a_mid, state["vz"])
    state["vz"] = so.vz_max
    return {"xp": xp, "vp": vp, "pid": pid, "rhoc": rhoc, **_results(so)}


# ------------------------------------------------------------------------------------
# What a pass cannot do without
# ------------------------------------------------------------------------------------
def _fft(n):
    """Flops of one real transform of an n^3 mesh."""
    return 2.5 * n ** 3 * math.log2(n ** 3)


def work(case):
    kind, n = case["kind"], case["np"]
    if kind == "density":
        return {"bytes": n * 3 * case["izipx"] + case["nc"] ** 3 * 8, "flops": n * 27 * 2}
    if kind == "force":
        return {"bytes": n * 12 * 4, "flops": 3 * _fft(case["n"]) + n * 27 * 30}
    if kind == "grad":  # forward kicks, and their recomputation and adjoint in the backward
        s = case["steps"]
        return {"bytes": n * 12 * 4 + case["n"] ** 3 * 8, "flops": s * (5 * _fft(case["n"]) + n * 27 * 40)}
    if kind == "power":
        return {"bytes": n * 3 * case["izipx"] + n * 4, "flops": _fft(case["nw"]) + case["nw"] ** 3 * 10}
    p = _params(case)
    nc, ngt, nft = p.nc, p.ngt, p.nft(2)
    flops = 2 * (_fft(nc) + p.ntiles * _fft(ngt) + p.ns3 * _fft(nft))
    flops += 10 * (nc ** 3 + p.ntiles * ngt ** 3 + p.ns3 * nft ** 3) + n * 3 * 27 * 10
    per = {"kick": 3 * case["izipx"] + 24, "step": 6 * case["izipx"] + 40, "host": 6 * case["izipx"] + 40}[kind]
    return {"bytes": n * per + nc ** 3 * 4, "flops": flops}


def tolerance(case):
    # about four times what two runs of the plain form (FP32 atomics) differ by
    if case["kind"] == "density":
        return {"rel": 1e-6, "max": 1e-5}
    if case["kind"] == "force":
        return {"rel": 5e-6, "max": 5e-5}
    if case["kind"] == "grad":
        return {"rel": 5e-5, "max": 5e-3}
    if case["kind"] == "power":
        return {"rel": 2e-5, "max": 2e-4}
    return {"rel": 1e-5, "max": 2e-4, "differ": 1e-3}


# ------------------------------------------------------------------------------------
# The same in 64 bits with plain torch
# ------------------------------------------------------------------------------------
D = torch.float64
RSF = {1: 1, 2: 2, 3: 4, 4: 6, 5: 8}


def _green(n, soft, cut, size):
    """The force kernel of one mesh level: the optimal influence function for TSC, the
    4-point gradient and an S2 cloud of `soft`, less the one of `cut` (0: none)."""
    def mode(m):
        return (torch.remainder(torch.arange(m, device="cuda", dtype=D) + n // 2, n) - n // 2) * (2 * math.pi / n)

    kz, ky, kx = mode(n)[:, None, None], mode(n)[None, :, None], mode(n // 2 + 1)[None, None, :]

    def cloud(k, a):
        y = a * k / 2
        return 12 / y ** 4 * (2 - 2 * torch.cos(y) - y * torch.sin(y))

    def sinc(k):
        return torch.where(k == 0, 1.0, torch.sin(k / 2) / torch.where(k == 0, 1.0, k / 2))

    grad = [4 / 3 * torch.sin(k) - torch.sin(2 * k) / 6 for k in (kz, ky, kx)]
    num = 0
    for c in range(-2, 3):
        for b in range(-2, 3):
            for a in range(-2, 3):
                k = (kz + 2 * math.pi * c, ky + 2 * math.pi * b, kx + 2 * math.pi * a)
                k2 = k[0] ** 2 + k[1] ** 2 + k[2] ** 2
                k2[k2 == 0] = 1.0
                km = k2.sqrt()
                s = cloud(km, soft) ** 2
                if cut:
                    s = s - cloud(km, cut) ** 2
                s *= sinc(k[0]) ** 6 * sinc(k[1]) ** 6 * sinc(k[2]) ** 6 / k2
                num = num + s * (grad[0] * k[0] + grad[1] * k[1] + grad[2] * k[2])
    u2 = 1
    for k in (kz, ky, kx):
        s2 = torch.sin(k / 2) ** 2
        u2 = u2 * (1 - s2 + 2 / 15 * s2 * s2)
    den = grad[0] ** 2 + grad[1] ** 2 + grad[2] ** 2
    g = 4 * math.pi * num / torch.where(den == 0, 1.0, den) / u2 ** 2 / size ** 2
    h = n // 2
    for z in (0, h):
        for y in (0, h):
            g[z, y, 0] = g[z, y, h] = 0.0
    return g


def _tsc(x):
    fl = x.floor()
    l = x - fl
    return fl.long() - 1, torch.stack([0.5 * (1 - l) ** 2, 0.75 - (l - 0.5) ** 2, 0.5 * l * l], dim=-1)


def _cells27(first, w, n, wrap):
    """Index (np, 27) into an n^3 mesh and the weights, 0 where a cell lies outside it."""
    i = first[:, :, None] + torch.arange(3, device="cuda")
    ok = (i >= 0) & (i < n)
    i = torch.remainder(i, n) if wrap else i.clamp(0, n - 1)
    w = w if wrap else w * ok
    idx = (i[:, 2, :, None, None] * n + i[:, 1, None, :, None]) * n + i[:, 0, None, None, :]
    ww = w[:, 2, :, None, None] * w[:, 1, None, :, None] * w[:, 0, None, None, :]
    return idx.reshape(-1, 27), ww.reshape(-1, 27)


def _spread(rho, base, first, w, n, wrap, values, step=1 << 20):
    for a in range(0, first.shape[0], step):
        idx, ww = _cells27(first[a:a + step], w[a:a + step], n, wrap)
        rho.index_add_(0, (idx + base[a:a + step, None]).reshape(-1), (ww * values).reshape(-1))


def _solve(rho, green, n):
    phi = torch.fft.irfftn(torch.fft.rfftn(rho, dim=(1, 2, 3)) * green, s=(n,) * 3, dim=(1, 2, 3))
    out = []
    for d in (3, 2, 1):
        r = [torch.roll(phi, -o, d) for o in (-2, -1, 1, 2)]
        out.append((2 / 3 * (r[2] - r[1]) + (r[0] - r[3]) / 12).reshape(-1))
    return out


def _gather(force, base, first, w, n, wrap, step=1 << 20):
    out = torch.empty((first.shape[0], 3), device="cuda", dtype=D)
    for a in range(0, first.shape[0], step):
        idx, ww = _cells27(first[a:a + step], w[a:a + step], n, wrap)
        idx = idx + base[a:a + step, None]
        for d in range(3):
            out[a:a + step, d] = (force[d][idx] * ww).sum(1)
    return out


def _boxes(cell, frac, nc, side, halo, pitch, green, n, mass, chosen, dv):
    """Adds the forces of the boxes `chosen` ((nc/side)^3 truth values) to dv: boxes of `side`
    coarse cells with a halo, meshes of `pitch` cells a coarse cell."""
    m = nc // side
    own, loc = cell // side, cell % side
    number = torch.full((m ** 3,), -1, device="cuda")
    number[chosen] = torch.arange(int(chosen.sum()), device="cuda")
    parts = []
    options = []
    for d in range(3):
        o = [(own[:, d], loc[:, d], torch.ones_like(loc[:, d], dtype=torch.bool))]
        o.append(((own[:, d] - 1) % m, loc[:, d] + side, loc[:, d] < halo))
        o.append(((own[:, d] + 1) % m, loc[:, d] - side, loc[:, d] >= side - halo))
        options.append(o)
    for oz in options[2]:
        for oy in options[1]:
            for ox in options[0]:
                ok = ox[2] & oy[2] & oz[2]
                box = number[(oz[0] * m + oy[0]) * m + ox[0]]
                ok &= box >= 0
                at = ok.nonzero()[:, 0]
                k = torch.stack([ox[1][at], oy[1][at], oz[1][at]], dim=1)
                parts.append((box[at], (k + frac[at]) * pitch))
    box, x = torch.cat([p[0] for p in parts]), torch.cat([p[1] for p in parts])
    del parts
    order = torch.sort(box, stable=True)
    box, x = order.values, x[order.indices]
    mine = number[(own[:, 2] * m + own[:, 1]) * m + own[:, 0]]
    morder = torch.sort(mine, stable=True)
    per = max(1, (1 << 27) // n ** 3)
    total = int(chosen.sum())
    for b in range(0, total, per):
        e = min(total, b + per)
        lo, hi = torch.searchsorted(box, torch.tensor([b, e], device="cuda")).tolist()
        rho = torch.zeros((e - b) * n ** 3, device="cuda", dtype=D)
        first, w = _tsc(x[lo:hi])
        _spread(rho, (box[lo:hi] - b) * n ** 3, first + halo * pitch, w, n, False, mass)
        force = _solve(rho.reshape(e - b, n, n, n), green, n)
        lo, hi = torch.searchsorted(morder.values, torch.tensor([b, e], device="cuda")).tolist()
        who = morder.indices[lo:hi]
        first, w = _tsc((loc[who] + frac[who]) * pitch)
        dv[who] += _gather(force, (mine[who] - b) * n ** 3, first + halo * pitch, w, n, False)


def _pair_force(r, a):
    e = 2 * r / a
    near = 224 * e - 224 * e ** 3 + 70 * e ** 4 + 48 * e ** 5 - 21 * e ** 6
    mid = 12 / e ** 2 - 224 + 896 * e - 840 * e ** 2 + 224 * e ** 3 + 70 * e ** 4 - 48 * e ** 5 + 7 * e ** 6
    return torch.where(e > 2, 1 / r ** 2, torch.where(e > 1, mid, near) / 35 / a ** 2)


def _pairs(cell, frac, order, nc, reach, app):
    """Short-range forces (np, 3) per unit mass: the difference of two S2 clouds of `app` and
    of each particle's own `reach` fine cells."""
    n = cell.shape[0]
    start = torch.zeros(nc ** 3 + 1, device="cuda", dtype=torch.long)
    start[1:] = torch.cumsum(torch.bincount(order, minlength=nc ** 3), 0)
    by_cell = torch.sort(order, stable=True).indices
    out = torch.zeros((n, 3), device="cuda", dtype=D)
    off = frac * 4
    for dz in (-1, 0, 1):
        for dy in (-1, 0, 1):
            for dx in (-1, 0, 1):
                need = torch.ones(n, dtype=torch.bool, device="cuda")
                for d, s in enumerate((dx, dy, dz)):
                    need &= (off[:, d] < reach) if s < 0 else (4 - off[:, d] < reach) if s > 0 else need
                who = need.nonzero()[:, 0]
                nb = torch.remainder(cell[who] + torch.tensor([dx, dy, dz], device="cuda"), nc)
                nb = (nb[:, 2] * nc + nb[:, 1]) * nc + nb[:, 0]
                count = start[nb + 1] - start[nb]
                edge = torch.cumsum(count, 0)
                a, total = 0, int(edge[-1]) if len(edge) else 0
                while a < len(who):
                    base = int(edge[a - 1]) if a else 0
                    b = max(a + 1, int(torch.searchsorted(edge, base + (1 << 25), right=True)))
                    c = count[a:b]
                    i = torch.repeat_interleave(who[a:b], c)
                    k = torch.arange(i.shape[0], device="cuda") - torch.repeat_interleave(edge[a:b] - c - base, c)
                    j = by_cell[torch.repeat_interleave(start[nb[a:b]], c) + k]
                    rv = off[j] + 4.0 * torch.tensor([dx, dy, dz], device="cuda", dtype=D) - off[i]
                    r2 = (rv * rv).sum(1)
                    hit = ((r2 > 0) & (r2 < reach[i] ** 2)).nonzero()[:, 0]
                    i, rv, r = i[hit], rv[hit], r2[hit].sqrt()
                    f = (_pair_force(r, app) - _pair_force(r, reach[i])) / r
                    out.index_add_(0, i, rv * f[:, None])
                    a = b
    return out


def _kicked(p, xp, vp, cell, dt, a_mid):
    nc, rcs = p.nc, p.ratio_cs
    bits = 8 * p.izipx
    frac = (torch.remainder(xp.long(), 1 << bits).to(D) + 0.5) / (1 << bits)
    mass = float(np.float32(p.particle_mass()))
    dv = torch.zeros((xp.shape[0], 3), device="cuda", dtype=D)
    # the whole box on its coarse mesh
    first, w = _tsc(cell + frac)
    rho = torch.zeros(nc ** 3, device="cuda", dtype=D)
    zero = torch.zeros(xp.shape[0], device="cuda", dtype=torch.long)
    _spread(rho, zero, first, w, nc, True, mass)
    dv += _gather(_solve(rho.reshape(1, nc, nc, nc), _green(nc, 3.5, 0.0, rcs), nc), zero, first, w, nc, True)
    # tiles
    every = torch.ones(p.nnt ** 3, dtype=torch.bool, device="cuda")
    _boxes(cell, frac, nc, p.nt, p.ncb, rcs, _green(p.ngt, 3.5, 3.5 * rcs, 1.0), p.ngt, mass, every, dv)
    # subtiles, each at the refinement its densest cell asks for
    order = (cell[:, 2] * nc + cell[:, 1]) * nc + cell[:, 0]
    m = nc // p.ntt
    most = torch.bincount(order, minlength=nc ** 3).reshape(m, p.ntt, m, p.ntt, m, p.ntt).amax(dim=(1, 3, 5)).reshape(-1)
    cls = 2 + (most >= 24 * 64).long() + (most >= 114 * 64).long() + (most >= 320 * 64).long()
    for c in range(2, 6):
        chosen = cls == c
        if bool(chosen.any()):
            r = RSF[c]
            _boxes(cell, frac, nc, p.ntt, 1, rcs * r, _green(p.nft(c), 3.5, 3.5 * r, 1.0 / r), p.nft(c), mass, chosen, dv)
    sub = cell // p.ntt
    rsf = torch.tensor([0, 1, 2, 4, 6, 8], device="cuda", dtype=D)[cls[(sub[:, 2] * m + sub[:, 1]) * m + sub[:, 0]]]
    dv += mass * _pairs(cell, frac, order, nc, 3.5 / rsf, 0.06)
    return vp.to(D) + dv * (a_mid * dt / 6 / math.pi)


def _cells_of(p, rhoc):
    """Coarse cell (np, 3) of every particle of a state in the checkpoint layout."""
    c = torch.repeat_interleave(torch.arange(rhoc.numel(), device="cuda"), rhoc.long())
    nt, nnt = p.nt, p.nnt
    t, r = c // nt ** 3, c % nt ** 3
    return torch.stack([t % nnt * nt + r % nt, t // nnt % nnt * nt + r // nt % nt, t // nnt ** 2 * nt + r // nt ** 2], dim=1)


def _drifted(p, st, cell, dt_mid, vz):
    """The state after the drift, in its order: codes, velocities and cells."""
    xp, vp, pid, rhoc = st
    bits, nt, nnt, ncb = 8 * p.izipx, p.nt, p.nnt, p.ncb
    move = torch.tensor(dt_mid, device="cuda", dtype=torch.float32) * vp
    unit = torch.remainder(xp.long(), 1 << bits)
    loc = cell % nt
    to = torch.ceil(loc + (unit.to(D) + 0.5) / (1 << bits) + (move / 4).to(D)).long() - (loc + 1)
    step = move.to(D) * ((1 << bits) / 4)
    code = torch.remainder(unit + (torch.sign(step) * torch.floor(step.abs() + 0.5)).long(), 1 << bits)
    new = torch.remainder(cell + to, p.nc)
    rel = new % nt - to + ncb
    layers = 2 * math.ceil(np.float32(np.float32(dt_mid) * np.float32(vz)) / 4) + 2
    t, l = new // nt, new % nt
    dest = ((((t[:, 2] * nnt + t[:, 1]) * nnt + t[:, 0]) * nt + l[:, 2]) * nt + l[:, 1]) * nt + l[:, 0]
    key = (((rel[:, 2] % layers) * 256 + rel[:, 2]) * 256 + rel[:, 1]) * 256 + rel[:, 0]
    perm = torch.sort(key, stable=True).indices
    perm = perm[torch.sort(dest[perm], stable=True).indices]
    return code[perm], vp[perm], new[perm]


def exact(case, seed):
    kind, n = case["kind"], case["np"]
    if kind in ("force", "grad"):
        if kind == "grad" and n * case["steps"] > 1.2e7:
            return None
        return _exact_dpm(case, seed)
    if kind == "power" and case["nw"] > 512:
        return None
    if kind not in ("density", "power") and (n > 3.2e6 or case["halo"] > 0.4):
        return None
    if kind == "density":
        p = _params({**case, "ng": 4 * case["nc"]}, nnt=2, nns=2)
    elif kind == "power":
        p = _params(case, nnt=case["ng"] // 64, nns=4)
    else:
        p = _params(case)
    use = KICK if kind == "kick" else STEP
    st = _state(case, seed, p.nc, p.nnt, use["vrms"])
    cell = _cells_of(p, st[3])
    bits = 8 * case["izipx"]
    frac = (torch.remainder(st[0].long(), 1 << bits).to(D) + 0.5) / (1 << bits)
    if kind == "density":
        first, w = _tsc(cell + frac)
        rho = torch.zeros(p.nc ** 3, device="cuda", dtype=D)
        _spread(rho, torch.zeros(n, device="cuda", dtype=torch.long), first, w, p.nc, True, float(np.float32(p.particle_mass())))
        return {"rho": rho.reshape((p.nc,) * 3)}
    if kind == "power":
        return _exact_power(case, p, cell + frac)
    none = {k: None for k in ("f2max", "vmax", "dt", "mass", "pairs", "candidates", "napm")}
    if kind == "kick":
        return {"vp": _kicked(p, st[0], st[1], cell, use["dt"], use["a_mid"]), **none}
    vz = float(st[1][:, 2].abs().max())
    xp, vp, cell = _drifted(p, st, cell, use["dt"], vz)
    vp = _kicked(p, xp, vp, cell, use["dt"], use["a_mid"])
    return {"xp": None, "vp": vp, "pid": None, "rhoc": None, **none}


def _exact_power(case, p, x):
    nw, n = case["nw"], case["np"]
    pos = x * (nw / p.nc) - 0.5
    fl = pos.floor()
    rho = torch.zeros(nw ** 3, device="cuda", dtype=D)
    for c in range(2):
        for b in range(2):
            for a in range(2):
                o = torch.tensor([a, b, c], device="cuda")
                w = torch.where(o == 1, pos - fl, 1 - (pos - fl)).prod(1)
                i = torch.remainder(fl.long() + o, nw)
                rho.index_add_(0, (i[:, 2] * nw + i[:, 1]) * nw + i[:, 0], w)
    mean = rho.mean()
    ck = torch.fft.rfftn((rho / mean - 1).reshape(nw, nw, nw)) / nw ** 3
    m = torch.remainder(torch.arange(nw, device="cuda") + nw // 2, nw) - nw // 2
    mx = m[: nw // 2 + 1]
    k = (mx.to(D)[None, None, :] ** 2 + m.to(D)[None, :, None] ** 2 + m.to(D)[:, None, None] ** 2).sqrt()
    c1 = 1 - 2 / 3 * torch.sin(math.pi * m.to(D) / nw) ** 2
    noise = c1[None, None, : nw // 2 + 1] * c1[None, :, None] * c1[:, None, None] / n
    amp = ck.abs() ** 2
    i, h = torch.arange(nw, device="cuda"), nw // 2
    ix, iy, iz = i[None, None, : h + 1], i[None, :, None], i[:, None, None]
    ex, ey = (ix == 0) | (ix == h), (iy == 0) | (iy == h)
    keep = ~(ex & (iy > h)) & ~(ex & ey & (iz > h)) & ~((ix == 0) & (iy == 0) & (iz == 0))
    nbin = int(round(float(np.float32(h) * np.sqrt(np.float32(3)))))
    bins = k[keep].float().round().long()
    def total(v):
        return torch.zeros(nbin + 1, device="cuda", dtype=D).index_add_(0, bins, v)
    count = total(torch.ones_like(k[keep]))
    box = float(np.float32(p.box))
    return {"modes": count, "k": total(k[keep]) / count * (2 * math.pi / box), "raw": total(amp[keep]) / count * box ** 3,
            "power": total((amp - noise)[keep]) / count * box ** 3, "corrected": None, "mean": mean}


def _exact_dpm(case, seed):
    s = _mesh_inputs(case, seed)
    n, mass = case["n"], float(np.float32(case["n"] ** 3 / case["np"]))
    green = _green(n, 3.5, 0.0, 1.0)

    def mesh(x):
        first, w = _tsc(x)
        idx, ww = _cells27(first, w, n, True)
        return idx, ww, torch.zeros(n ** 3, device="cuda", dtype=D).index_add(0, idx.reshape(-1), (mass * ww).reshape(-1))

    def force(x):
        idx, ww, rho = mesh(x)
        f = _solve(rho.reshape(1, n, n, n), green, n)
        return torch.stack([(c[idx] * ww).sum(1) for c in f], dim=1)

    x = s["x"].detach().to(D).requires_grad_(True)
    if case["kind"] == "force":
        f = force(x)
        return {"force": f.detach(), "vjp": torch.autograd.grad((f * s["u"].to(D)).sum(), x)[0]}
    v = s["v"].detach().to(D).requires_grad_(True)
    y, u = x, v
    for a, b in s["steps"]:
        y = torch.remainder(y + float(np.float32(a)) * u, float(n))
        u = u + float(np.float32(b)) * torch.utils.checkpoint.checkpoint(force, y, use_reentrant=False)
    y = torch.remainder(y + 0.25 * u, float(n))
    rho = mesh(y)[2].reshape(n, n, n)
    loss = ((rho - s["target"].to(D)) ** 2).mean()
    gx, gv = torch.autograd.grad(loss, (x, v))
    return {"rho": rho.detach(), "loss": loss.detach(), "gx": gx, "gv": gv}


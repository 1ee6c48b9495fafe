"""The workloads this framework is timed on.

A case is one of four things a user of the library does, at one size, storage
type and set of options:

  cavity      run `steps` iterations of a lattice in hand and read the density
              and velocity fields back (a save interval of the lbmcl program)
  run         the whole job: create the lattice with seeded noise, run it,
              read the fields back, destroy it
  checkpoint  restart from a population file in host memory, run `steps`
              iterations, write the populations back to host memory
  grad        one evaluation of the mid-plane loss and its gradient with
              respect to the lid profile (and tau) through the autograd
              function, as an optimiser calls it every iteration

`exact` evaluates the same physics in 64 bits with plain torch: the D3Q19 BGK
lid-driven cavity in the post-stream form (pull from s - e_i, walls hold the
initial equilibrium), its noise from the documented Philox / Box-Muller recipe.
"""
import math

import numpy as np
import torch
from torch.utils.checkpoint import checkpoint as _recompute

from lbmcl_gb300 import capi
from lbmcl_gb300.adjoint import cavity_loss

NU, LID, SIGMA = 0.0089, 0.05, 1e-4
BYTES = {"fp32": 4, "fp64": 8, "fp16": 2, "bf16": 2}
FLOPS = 220       # additions and multiplications of one FLUID site's update
FLOPS_ADJ = 250   # the same of its transposed update


def listed():
    return [
        # the reference's own test run: 32^3, fields saved every 20 iterations
        dict(name="cavity_32_fp32", kind="cavity", dim=32, precision="fp32", steps=20),
        # a small lattice in the compact storage, one save interval
        dict(name="cavity_64_fp16", kind="cavity", dim=64, precision="fp16", steps=100),
        # the largest lattice of the reference's benchmark sweep, 50 iterations
        dict(name="cavity_128_fp32", kind="cavity", dim=128, precision="fp32", steps=50),
        # a lattice that is no power of two, in the other 16-bit type
        dict(name="cavity_200_bf16", kind="cavity", dim=200, precision="bf16", steps=50),
        # the double-precision run that accuracy is judged by
        dict(name="cavity_256_fp64", kind="cavity", dim=256, precision="fp64", steps=10),
        # the headline: 512^3 in 16-bit storage
        dict(name="cavity_512_fp16", kind="cavity", dim=512, precision="fp16", steps=100),
        # the same lattice in the reference's single precision
        dict(name="cavity_512_fp32", kind="cavity", dim=512, precision="fp32", steps=20),
        # a short job from scratch: noise, iterations, fields
        dict(name="run_256_fp16", kind="run", dim=256, precision="fp16", steps=20),
        # restart and write of a population checkpoint in the reference's layout
        dict(name="checkpoint_136_fp32", kind="checkpoint", dim=136, precision="fp32", steps=20),
        # the gradient of the small optimisation problem, lid profile and tau
        dict(name="grad_64_fp32_tau", kind="grad", dim=64, precision="fp32", steps=100, every=20, tau=True),
        # lid profile only (the sweep over stored linearisation points)
        dict(name="grad_256_fp16", kind="grad", dim=256, precision="fp16", steps=200, every=20, tau=False),
        # 16-bit storage with tau (recomputed full states), mid size
        dict(name="grad_128_fp16_tau", kind="grad", dim=128, precision="fp16", steps=100, every=10, tau=True),
    ]


def draw(rng):
    kind = rng.choice(["cavity"] * 5 + ["run"] + ["checkpoint"] + ["grad"] * 3)
    lo, hi = {"cavity": (16, 512), "run": (32, 256), "checkpoint": (16, 200), "grad": (16, 256)}[kind]
    if kind == "grad":
        prec = rng.choice(["fp32", "fp32", "fp16", "bf16"])
    else:
        prec = rng.choice(["fp32", "fp32", "fp16", "fp16", "bf16", "fp64"])
    step = 8 if prec in ("fp16", "bf16") else 4
    dim = int(math.exp(rng.uniform(math.log(lo), math.log(hi + 1)))) // step * step
    dim = max(16, min(hi, dim))
    case = dict(kind=kind, dim=dim, precision=prec)
    if kind == "grad":
        case["every"] = rng.randrange(4, 21)
        case["steps"] = rng.randrange(case["every"], 201)
        case["tau"] = rng.random() < 0.4
        # no more than the 256^3 case's site updates
        case["steps"] = max(case["every"], min(case["steps"], int(150 * (256 / dim) ** 3)))
    else:
        case["steps"] = int(math.exp(rng.uniform(math.log(10), math.log(201))))
        # no more than the time of the headline case
        cap = 100 * 512.0 ** 3 * {"fp64": 1 / 50, "fp32": 0.4}.get(prec, 0.6)
        case["steps"] = max(1, min(case["steps"], int(cap / dim ** 3)))
    return case


# -- inputs -----------------------------------------------------------------------------------------------------------


def _lid(case, seed):
    """The per-column lid velocity, [y, x]: the nominal value with a tenth of it as noise (float values)."""
    g = np.random.default_rng([seed, case["dim"], 1])
    return (LID + 0.1 * LID * g.standard_normal((case["dim"], case["dim"]))).astype(np.float32)


def _target(case, seed):
    """The wanted u_x on the loss plane, [z, x]."""
    g = np.random.default_rng([seed, case["dim"], 2])
    return (0.02 * g.standard_normal((case["dim"], case["dim"]))).astype(np.float32)


def _stored(case, seed, device):
    """The populations of a checkpoint, [q, z, y, x]: rest equilibrium and a perturbation as large as a developed
    cavity flow's."""
    D = case["dim"]
    dtype = torch.float64 if case["precision"] == "fp64" else torch.float32
    g = torch.Generator(device=device).manual_seed(seed)
    w = torch.tensor(W, dtype=torch.float64, device=device).view(19, 1, 1, 1)
    return (w * (1 + 0.02 * torch.randn(19, D, D, D, generator=g, device=device))).to(dtype)


def _stride(case):
    """The reference's default layout stride for population files, or what the lattice size has of it."""
    return math.gcd(case["dim"] ** 3, 32)


def _csoa(f, stride):
    """[q, z, y, x] -> the reference's layout: blocks of `stride` sites, the 19 populations of a block in turn."""
    return f.reshape(19, -1, stride).transpose(0, 1).reshape(-1)


def _pinned(count, dtype):
    return torch.empty(count, dtype=dtype, pin_memory=True).numpy()


def prepare(case, seed):
    kind, D, prec = case["kind"], case["dim"], case["precision"]
    state = dict(case, seed=seed)
    lid = _lid(case, seed)
    if kind == "grad":
        state["lid"] = torch.from_numpy(lid).requires_grad_(True)
        state["tau"] = torch.tensor(3 * NU + 0.5, requires_grad=bool(case["tau"]))
        state["target"] = _target(case, seed)
        return state
    macro = torch.float64 if prec == "fp64" else torch.float32
    if kind == "checkpoint":
        state["file"] = _pinned(19 * D ** 3, macro)
        state["file"][:] = _csoa(_stored(case, seed, "cuda"), _stride(case)).cpu().numpy()
        state["f"] = _pinned(19 * D ** 3, macro)
        state["lattice"] = capi.Lattice(D, NU, LID, precision=prec, stride=_stride(case), lid=lid)
        return state
    state["rho"], state["u"] = _pinned(D ** 3, macro), _pinned(3 * D ** 3, macro)
    state["lid"] = lid
    if kind == "cavity":
        state["lattice"] = capi.Lattice(D, NU, LID, precision=prec, lid=lid, seed=seed, noise_sigma=SIGMA)
    return state


# -- one pass ---------------------------------------------------------------------------------------------------------


def run(s):
    if s["kind"] == "cavity":
        L = s["lattice"]
        L.step(s["steps"], every=s["steps"])
        return {"rho": L.rho(s["rho"]), "u": L.u(s["u"])}
    if s["kind"] == "run":
        with capi.Lattice(s["dim"], NU, LID, precision=s["precision"], lid=s["lid"], seed=s["seed"],
                          noise_sigma=SIGMA) as L:
            L.step(s["steps"], every=s["steps"])
            return {"rho": L.rho(s["rho"]), "u": L.u(s["u"])}
    if s["kind"] == "checkpoint":
        L = s["lattice"]
        L.load_f(s["file"])
        L.step(s["steps"])
        return {"f": L.f(s["f"])}
    lid = s["lid"].detach().requires_grad_(True)
    tau = s["tau"].detach().requires_grad_(bool(s["tau"].requires_grad))
    loss = cavity_loss(lid, tau, None, dim=s["dim"], iterations=s["steps"], checkpoint_every=s["every"],
                       plane_y=s["dim"] // 2, target=s["target"], precision=s["precision"])
    loss.backward()
    out = {"loss": loss.detach(), "lid": lid.grad}
    if tau.grad is not None:
        out["tau"] = tau.grad
    return out


def work(case):
    """Inputs read once and outputs written once; the updates of all iterations."""
    D, T, b = case["dim"], case["steps"], BYTES[case["precision"]]
    m = 8 if case["precision"] == "fp64" else 4
    sites = (D - 2) ** 3
    flops = T * sites * FLOPS
    if case["kind"] == "cavity":      # state in and out, fields out
        return {"bytes": 2 * 19 * b * D ** 3 + 4 * m * D ** 3, "flops": flops}
    if case["kind"] == "run":         # lid in, fields out
        return {"bytes": 8 * D ** 2 + 4 * m * D ** 3, "flops": flops}
    if case["kind"] == "checkpoint":  # populations in and out
        return {"bytes": 2 * 19 * m * D ** 3, "flops": flops}
    # the linearisation point of every iteration written and read, the profile and its gradient
    return {"bytes": T * sites * 2 * 3 * 4 + 12 * D ** 2, "flops": flops + T * sites * FLOPS_ADJ}


# -- the same in 64 bits ----------------------------------------------------------------------------------------------

E = [(0, 0, 0), (1, 0, 0), (0, 1, 0), (-1, 0, 0), (0, -1, 0), (0, 0, -1), (0, 0, 1), (1, 1, 0), (-1, 1, 0), (-1, -1, 0),
     (1, -1, 0), (1, 0, -1), (0, 1, -1), (-1, 0, -1), (0, -1, -1), (1, 0, 1), (0, 1, 1), (-1, 0, 1), (0, -1, 1)]
W = [1 / 3] + [1 / 18] * 6 + [1 / 36] * 12
OPP = [E.index(tuple(-c for c in e)) for e in E]


def _signed(e, u):
    """e . u for e of -1, 0, 1; None where e is 0."""
    s = None
    for c, v in zip(e, u):
        if c:
            t = v if c > 0 else -v
            s = t if s is None else s + t
    return s


def _equilibrium(i, rho, u, u2):
    eu = _signed(E[i], u)
    return W[i] * rho * ((1 - 1.5 * u2) if eu is None else (1 + 3 * eu + 4.5 * eu * eu - 1.5 * u2))


def _lid_equilibrium(i, lid):
    ex = E[i][0]
    return W[i] * (1 + 3 * ex * lid + 4.5 * ex * ex * lid * lid - 1.5 * lid * lid)


def _walls(f, lid):
    """The slots of sites whose source is a wall: the site's initial equilibrium (moving on the lid's plane)."""
    D = f[0].shape[0]
    for i, (ex, ey, ez) in enumerate(E):
        for axis, e in ((0, ez), (1, ey), (2, ex)):
            if e:
                at = 1 if e > 0 else D - 2
                sl = [slice(1, D - 1)] * 3
                sl[axis] = at
                f[i][tuple(sl)] = W[i]
                sl[0] = D - 2
                if axis == 0:
                    if at == D - 2:
                        f[i][tuple(sl)] = _lid_equilibrium(i, lid)[1:-1, 1:-1]
                else:
                    f[i][tuple(sl)] = _lid_equilibrium(i, lid)[tuple(sl[1:])]
    return f


def _rest(D, lid):
    """The initial populations, [z, y, x] each (NaN on the walls)."""
    f = []
    for i in range(19):
        r = torch.full((D, D, D), math.nan, dtype=torch.float64, device=lid.device)
        r[1:-1, 1:-1, 1:-1] = W[i]
        r[D - 2, 1:-1, 1:-1] = _lid_equilibrium(i, lid)[1:-1, 1:-1]
        f.append(r)
    return f


def _philox(site, block, seed):
    M = 0xFFFFFFFF
    c = [site & M, site >> 32, torch.full_like(site, block), torch.zeros_like(site)]
    k0, k1 = seed & M, (seed >> 32) & M
    for _ in range(10):
        p0, p1 = c[0] * 0xD2511F53, c[2] * 0xCD9E8D57  # modulo 2^64
        c = [((p1 >> 32) & M) ^ c[1] ^ k0, p1 & M, ((p0 >> 32) & M) ^ c[3] ^ k1, p0 & M]
        k0, k1 = (k0 + 0x9E3779B9) & M, (k1 + 0xBB67AE85) & M
    return c


def _noise(f, seed):
    """N(0, SIGMA^2) on every population of the FLUID sites: two Box-Muller pairs per Philox block of four words."""
    D = f[0].shape[0]
    r = torch.arange(2, D - 2, device=f[0].device)
    site = r.view(1, 1, -1) + D * r.view(1, -1, 1) + D * D * r.view(-1, 1, 1)
    for block in range(5):
        w = _philox(site, block, seed)
        for pair in (0, 1):
            i = 4 * block + 2 * pair
            a, b = w[2 * pair], w[2 * pair + 1]
            radius = ((((a >> 9).double() + 0.5) / 2 ** 23).log() * -2).sqrt()
            angle = 2 * math.pi * ((b >> 30).double() / 4 + 1 / 8) + \
                ((((b >> 8) & 0x3FFFFF).double() + 0.5) / 2 ** 22 - 0.5) * (math.pi / 2)
            for q, z in ((i, angle.cos()), (i + 1, angle.sin())):
                if q < 19:
                    f[q][2:-2, 2:-2, 2:-2] += SIGMA * radius * z
    return f


def _moments(g):
    rho = sum(g[1:], g[0])
    u = []
    for axis in range(3):
        j = None
        for i in range(19):
            if E[i][axis]:
                t = g[i] if E[i][axis] > 0 else -g[i]
                j = t if j is None else j + t
        u.append(j / rho)
    return rho, u


def _lid_density(f):
    """The density of the lid's sites (x, y in [2, D - 3]) after the replacements of the populations leaving it."""
    D = f[0].shape[0]
    return sum(f[OPP[i] if E[i][2] < 0 else i][D - 2, 2:-2, 2:-2] for i in range(19))


def _iterate(f, lid, omega):
    D = f[0].shape[0]
    g = [r[2:-2, 2:-2, 2:-2] for r in f]
    rho, u = _moments(g)
    u2 = u[0] * u[0] + u[1] * u[1] + u[2] * u[2]
    rl, lm = _lid_density(f), lid[2:-2, 2:-2]
    out = []
    for i, (ex, ey, ez) in enumerate(E):
        p = f[OPP[i]][1:-1, 1:-1, 1:-1].clone()  # bounce-back; FLUID, lid and corner sites follow
        p[1:-1, 1:-1, 1:-1] = g[i] + omega * (_equilibrium(i, rho, u, u2) - g[i])
        p[-1, 1:-1, 1:-1] = rl * _lid_equilibrium(i, lm)
        for y in (0, -1):
            for x in (0, -1):
                p[0, y, x] = f[i][1:-1, 1:-1, 1:-1][0, y, x]
        r = torch.full_like(f[i], math.nan)
        r[1 + ez:D - 1 + ez, 1 + ey:D - 1 + ey, 1 + ex:D - 1 + ex] = p
        out.append(r)
    return _walls(out, lid)


def _fields(f, lid):
    D = f[0].shape[0]
    rho = torch.full((D, D, D), math.nan, dtype=torch.float64, device=lid.device)
    u = torch.full((3, D, D, D), math.nan, dtype=torch.float64, device=lid.device)
    r, v = _moments([t[2:-2, 2:-2, 2:-2] for t in f])
    rho[2:-2, 2:-2, 2:-2] = r
    rho[D - 2, 2:-2, 2:-2] = _lid_density(f)
    for axis in range(3):
        u[axis, 2:-2, 2:-2, 2:-2] = v[axis]
        u[axis, D - 2, 2:-2, 2:-2] = lid[2:-2, 2:-2] if axis == 0 else 0.0
    return rho.reshape(-1), u.reshape(-1)


def _exact_grad(case, seed, device):
    D = case["dim"]
    lid = torch.from_numpy(_lid(case, seed)).double().to(device).requires_grad_(True)
    tau = torch.tensor(float(np.float32(3 * NU + 0.5)), dtype=torch.float64, device=device, requires_grad=True)
    target = torch.from_numpy(_target(case, seed)).double().to(device)

    def step(lid, tau, *f):
        return tuple(_iterate(list(f), lid, 1 / tau))

    f = tuple(_rest(D, lid))
    for _ in range(case["steps"]):
        f = _recompute(step, lid, tau, *f, use_reentrant=False)
    y = D // 2
    _, u = _moments([r[2:-2, y, 2:-2] for r in f])
    loss = ((u[0] - target[2:-2, 2:-2]) ** 2).mean()
    loss.backward()
    out = {"loss": loss.detach().cpu(), "lid": lid.grad.cpu()}
    if case["tau"]:
        out["tau"] = tau.grad.cpu()
    return out


def exact(case, seed):
    D = case["dim"]
    device = "cuda" if torch.cuda.is_available() else "cpu"
    if case["kind"] == "grad":
        # every iteration's populations are kept
        if 19 * 8 * D ** 3 * case["steps"] > 100e9:
            return None
        return _exact_grad(case, seed, device)
    if case["steps"] * D ** 3 > 16e9:  # over about 20 seconds
        return None
    with torch.no_grad():
        lid = torch.from_numpy(_lid(case, seed)).double().to(device)
        omega = 1 / (3 * NU + 0.5)
        if case["kind"] == "checkpoint":
            f = list(_stored(case, seed, device).double().unbind(0))
            for r in f:
                r[0] = r[-1] = r[:, 0] = r[:, -1] = r[:, :, 0] = r[:, :, -1] = math.nan
            f = _walls(f, lid)
            for _ in range(case["steps"]):
                f = _iterate(f, lid, omega)
            return {"f": _csoa(torch.stack(f), _stride(case)).cpu()}
        f = _noise(_rest(D, lid), seed)
        for _ in range(case["steps"] - 1):
            f = _iterate(f, lid, omega)
        rho, u = _fields(f, lid)
        return {"rho": rho.cpu(), "u": u.cpu()}

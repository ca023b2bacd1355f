"""Performance cases of the micromagnetic library: what a user's program has it do.

Time stepping of single films and 3-D bodies, evaluations of the torque and of the field
terms, batches of relaxations, thermal ensembles, and the warm start's U-Net in inference
and training; each through the package's public entry points.  Sizes are written as the
user writes them, x, y, z.  exact() restates the physics in 64 bits with plain torch.
"""
import ctypes as C
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "2_b200"))

from mumax2 import Ensemble, Plan  # noqa: E402
from mumax2 import _native as nat  # noqa: E402
from mumax2 import unet as U  # noqa: E402
from mumax2 import workloads as W  # noqa: E402

MU0 = 4.0 * math.pi * 1e-7
KB, MUB, QE, HBAR = 1.380650424e-23, 9.2740091523e-24, 1.60217646e-19, 1.054571726e-34
GAMMA = 2.211e5
MAXERR = {"rk12": 1.0 / 2000, "rk23": 1e-5, "rk45": 1e-5, "heun": 1.0, "euler": 1.0}
EVALS = {"euler": 1, "heun": 2, "rk12": 2, "rk23": 3, "rk45": 6}


def listed():
    return [
        # the standard-problem film: the smallest run that anybody makes, launch latency counts
        dict(name="film_128x32_rk45", kind="step", nx=128, ny=32, nz=1, term="zeeman", solver="rk45", steps=12),
        # a spin-torque nano-oscillator: a masked disk under a current through the film
        dict(name="disk_128x128_rk45", kind="step", nx=128, ny=128, nz=1, term="slonczewski", solver="rk45", steps=8),
        # a domain wall in a strip driven by an in-plane current
        dict(name="strip_512x128_rk45", kind="step", nx=512, ny=128, nz=1, term="zhangli", solver="rk45", steps=8),
        # the headline film: a million cells with perpendicular anisotropy
        dict(name="body_256x256x16_rk23", kind="step", nx=256, ny=256, nz=16, term="anis", solver="rk23", steps=8),
        # a recommended size 2^n * 3 with the reference's own adaptive solver
        dict(name="body_192x192x8_rk12", kind="step", nx=192, ny=192, nz=8, term="anis", solver="rk12", steps=8),
        # ragged sizes with a geometry mask: a shape imported from elsewhere
        dict(name="body_150x75x3_rk23", kind="step", nx=150, ny=75, nz=3, term="masked", solver="rk23", steps=8),
        # one torque evaluation of a large film (the reference's convolution benchmark size)
        dict(name="film_1024x1024_torque", kind="torque", nx=1024, ny=1024, nz=1, term="zeeman"),
        # every field term of a cube, as a script that records them asks for
        dict(name="cube_64_fields", kind="fields", nx=64, ny=64, nz=64, term="anis"),
        # a relaxation pool: many masked films in one batch
        dict(name="relax_256_films", kind="relax", nsim=256, steps=6),
        # thermal realisations over five grid sizes, stepped together
        dict(name="ensemble_512_heun", kind="ensemble", nsim=512, steps=6),
        # warm starts predicted for a pool's problems
        dict(name="unet_predict_256", kind="unet_forward", batch=256),
        # one training step of the network
        dict(name="unet_train_64", kind="unet_train", batch=64),
    ]


def _size(rng, lo, hi):
    """A grid size in lo..hi, spread over its logarithm: recommended sizes 2^n * {1, 3, 5, 7}
    in half of the draws, else any whose transform the library takes (factors up to 31)."""
    while True:
        v = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
        if rng.random() < 0.5:
            v = min((k << n for k in (1, 3, 5, 7) for n in range(12) if lo <= k << n <= hi), key=lambda s: abs(s - v))
        r = v
        for f in (2, 3, 5, 7, 11, 13, 17, 19, 23, 29, 31):
            while r % f == 0:
                r //= f
        if r == 1 and lo <= v <= hi:
            return v


def draw(rng):
    kind = rng.choice(["film", "film", "body", "body", "torque", "fields", "relax", "ensemble", "unet"])
    if kind == "relax":
        return dict(kind="relax", nsim=_size(rng, 8, 256), steps=6)
    if kind == "ensemble":
        return dict(kind="ensemble", nsim=_size(rng, 16, 512), steps=rng.choice([3, 4, 6]))
    if kind == "unet":
        train = rng.random() < 0.5
        return dict(kind="unet_train" if train else "unet_forward", batch=_size(rng, 8, 64 if train else 256))
    if kind == "film":
        nx, ny = _size(rng, 32, 512), _size(rng, 16, 512)
        solver = rng.choice(["rk12", "heun", "rk23", "rk45"])
        term = rng.choice(["zeeman", "anis", "masked", "slonczewski", "zhangli"])
        return dict(kind="step", nx=nx, ny=ny, nz=1, term=term, solver=solver, steps=8)
    nx, ny, nz = _size(rng, 24, 256), _size(rng, 24, 256), _size(rng, 2, 16)
    if kind == "body":
        solver = rng.choice(["rk12", "heun", "rk23", "rk45"])
        return dict(kind="step", nx=nx, ny=ny, nz=nz, term=rng.choice(["zeeman", "anis", "masked"]), solver=solver,
                    steps=4)
    if rng.random() < 0.4:
        nx, ny, nz = _size(rng, 64, 1024), _size(rng, 64, 1024), 1
    return dict(kind=kind, nx=nx, ny=ny, nz=nz, term=rng.choice(["zeeman", "anis", "masked"]))


# ---------------------------------------------------------------- inputs
def _texture(n, seed):
    """A magnetisation as one meets it in a running simulation: a few long waves and some
    cell-to-cell noise, unit vectors, SoA (z, y, x) components on the GPU."""
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    z, y, x = (torch.arange(s, device="cuda", dtype=torch.float32).reshape(r) / s
               for s, r in zip(n, ((-1, 1, 1), (1, -1, 1), (1, 1, -1))))
    m = 0.1 * torch.randn((3,) + tuple(n), device="cuda", generator=g)
    m[2] += 0.5
    for _ in range(6):
        a = torch.randn(3, device="cuda", generator=g).reshape(3, 1, 1, 1)
        k = torch.randint(-3, 4, (3,), device="cuda", generator=g)
        p = torch.rand(1, device="cuda", generator=g)
        m += 0.5 * a * torch.cos(2 * math.pi * (k[0] * z + k[1] * y + k[2] * x + p))
    return m / m.norm(dim=0, keepdim=True)


def _problem(case, seed):
    """(problem, masks, m0) of a single simulation; arrays in internal (z, y, x) order."""
    rng = np.random.default_rng(seed)
    n = (case["nz"], case["ny"], case["nx"])
    N = n[0] * n[1] * n[2]
    term = case["term"]
    phi = rng.uniform(0, 2 * np.pi)
    b = rng.uniform(0.01, 0.03)
    pr = dict(n=n, cell=(3e-9, 4e-9, 4e-9), pbc=(0, 0, 0), demag=1, exchange=1, zeeman=1, demag_accuracy=6, msat=8e5,
              aex=1.3e-11, alpha=0.02, gamma=GAMMA, bext=(0.0, b * math.sin(phi), b * math.cos(phi)))
    masks = {}
    m0 = _texture(n, seed)
    if term == "anis":
        pr.update(cell=(2e-9, 4e-9, 4e-9), anis=1, ku=5e5, anisu=(1.0, 0.0, 0.0), alpha=0.1)
    elif term == "zhangli":
        pr.update(cell=(2e-9, 2e-9, 2e-9), zeeman=0, bext=(0.0, 0.0, 0.0), zhangli=1, zl_pol=0.5, xi=0.05,
                  j=(0.0, 0.0, float(rng.uniform(5e11, 1e12))))
    elif term in ("slonczewski", "masked"):
        z, y, x = np.mgrid[0:n[0], 0:n[1], 0:n[2]]
        geo = (((x + 0.5) / n[2] - 0.5) ** 2 + ((y + 0.5) / n[1] - 0.5) ** 2 <= 0.25).astype(np.float32)
        masks["msat"] = geo.ravel()
        if term == "slonczewski":
            pr.update(cell=(2e-9, 2e-9, 2e-9), zeeman=0, bext=(0.0, 0.0, 0.0), slonczewski=1, p=(1.0, 0.0, 0.0),
                      sl_pol=0.5, eps_prime=0.0, t_fl=2e-9, j=(float(rng.uniform(5e10, 1e11)), 0.0, 0.0),
                      **{"lambda": 1.0})
        else:  # a softer grain in one half of the body
            masks["msat"] = (geo * np.where(x < n[2] // 2, 1.0, 0.75)).astype(np.float32).ravel()
            masks["aex"] = np.where(x < n[2] // 2, 1.0, 0.8).astype(np.float32).ravel()
        m0 = m0 * torch.from_numpy((masks["msat"] != 0).astype(np.float32)).cuda().reshape(1, *n)
    return pr, masks, m0.reshape(-1).contiguous()


def _dt0(case):
    # the engine's initial step for the adaptive solvers: it grows by the controller's limit
    # for about the number of steps listed here, so the times reached do not hang on the
    # rounding of the error estimate
    return 1e-14 if case["solver"] in ("heun", "euler") else 1e-15


def _relax_inputs(case, seed):
    problem, sims, masks = W.relax_set(case["nsim"], seed=seed)
    masks = np.stack(masks).astype(np.float32)
    m = torch.stack([_texture(problem["n"], seed * 1009 + b).reshape(3, -1) for b in range(len(sims))])
    m = m * torch.from_numpy((masks != 0).astype(np.float32)).cuda()[:, None]
    return problem, sims, masks, m.reshape(-1).contiguous()


def _ensemble_inputs(case, seed):
    """The simulations of each of the ensemble's grid sizes, an equal share of every size, with
    the generator's distributions of the material, the field and the initial direction."""
    rng = np.random.default_rng(seed)
    out = []
    for q, grid in enumerate(W.ENSEMBLE_GRIDS_USER):
        count = (case["nsim"] + q) // len(W.ENSEMBLE_GRIDS_USER)
        n, cell = grid[::-1], W.ENSEMBLE_CELL_USER[::-1]
        unit = rng.normal(size=(2, count, 3))
        unit /= np.linalg.norm(unit, axis=2, keepdims=True)
        sims = [dict(msat=rng.uniform(4e5, 1.2e6), aex=rng.uniform(5e-12, 2e-11), alpha=rng.uniform(0.01, 0.1),
                     bext=tuple(rng.uniform(0.0, 0.05) * unit[0, i]), ku=0.0, anisu=(0.0, 0.0, 1.0),
                     temp=W.ENSEMBLE_TEMP, seed=int(seed) * 1_000_003 + 1000 * q + i) for i in range(count)]
        problem = dict(n=n, cell=cell, pbc=(0, 0, 0), demag=1, exchange=1, zeeman=1, anis=0, thermal=1, gamma=GAMMA,
                       demag_accuracy=6, **{k: sims[0][k] for k in ("msat", "aex", "alpha", "temp")})
        out.append((dict(n=n, problem=problem, sims=sims), torch.from_numpy(W.uniform_state(n, unit[1])).cuda()))
    return out


def _unet_inputs(case, seed):
    _, sims, masks = W.relax_set(case["batch"], seed=seed)
    masks = np.stack(masks).astype(np.float32)
    tgt = torch.stack([_texture((1, 64, 64), seed * 1009 + b).reshape(3, -1).t() for b in range(len(sims))])
    return sims, masks, tgt.contiguous()


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind in ("step", "torque", "fields"):
        pr, masks, s["m"] = _problem(case, seed)
        s["plan"] = Plan(pr, masks=masks)
        if kind == "step":
            s["plan"].solver(case["solver"], dt=_dt0(case), maxerr=MAXERR[case["solver"]])
            s["out"] = torch.empty_like(s["m"])
    elif kind == "relax":
        pr, sims, masks, s["m"] = _relax_inputs(case, seed)
        s["plan"] = Plan(pr, masks={"msat": masks.ravel()}, sims=sims, masks_per_sim=True)
        s["plan"].solver("rk23", dt=1e-15, maxerr=1e-6)
        s["out"] = torch.empty_like(s["m"])
    elif kind == "ensemble":
        s["m"], s["plans"] = [], []
        for c, m in _ensemble_inputs(case, seed):
            p = Plan(c["problem"], sims=c["sims"])
            p.solver("heun", dt=W.ENSEMBLE_DT)
            s["m"].append(m)
            s["plans"].append(p)
        s["ens"] = Ensemble(s["plans"], attempts=case["steps"])
        s["out"] = [torch.empty_like(m) for m in s["m"]]
    else:
        sims, masks, tgt = _unet_inputs(case, seed)
        s["net"] = U.UNet(case["batch"], seed=seed)
        s["masks"] = torch.from_numpy(masks).cuda()
        s["prm"] = torch.from_numpy(U.param_table(sims)).cuda()
        s["count"] = float(masks.sum())
        if kind == "unet_train":
            s["target"] = tgt
        else:
            s["out"] = torch.empty(case["batch"] * 3 * 64 * 64, device="cuda")
    torch.cuda.synchronize()
    return s


def _state(plan, out):
    nat.check(nat.lib().mm_get_state(plan.h, C.c_void_p(out.data_ptr()), 0, None))
    return out


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "step" or kind == "relax":
        p = s["plan"]
        p.set_time(0.0, _dt0(case) if kind == "step" else 1e-15)
        p.set_state(s["m"])
        p.steps(case["steps"])
        return _state(p, s["out"])
    if kind == "torque":
        return s["plan"].torque(s["m"])
    if kind == "fields":
        return s["plan"].fields(s["m"])
    if kind == "ensemble":
        for p, m in zip(s["plans"], s["m"]):
            p.set_state(m)
        s["ens"].steps(case["steps"])
        return [_state(p, o) for p, o in zip(s["plans"], s["out"])]
    net = s["net"]
    net.set_features(s["masks"].view(-1), s["prm"].view(-1))
    out = net.forward()
    if kind == "unet_forward":
        net.states(s["masks"].view(-1), s["out"])
        return {"out": out, "states": s["out"]}
    net.set_target(s["target"], s["masks"], mask_count=s["count"])
    loss = net.loss_and_grad()
    net.backward()
    net.adam(lr=1e-3)
    return {"loss": loss, "out": out, "gw": [net.p[c[0]]["gw"] for c in U.CONVS],
            "gb": [net.p[c[0]]["gb"] for c in U.CONVS], "w": [net.p[c[0]]["w"] for c in U.CONVS]}


# ---------------------------------------------------------------- what a pass cannot do without
def _eval_work(n):
    """One field evaluation: m read, the derivative written, one octant of the kernel read;
    the real transforms of three components there and back over the padded box."""
    N = n[0] * n[1] * n[2]
    L = [2 * s if s > 1 else 1 for s in n]
    octant = (L[0] // 2 + 1) * (L[1] // 2 + 1) * (L[2] // 2 + 1)
    pad = L[0] * L[1] * L[2]
    return 24 * N, (4 if n[0] == 1 else 6) * 4 * octant, 6 * 2.5 * pad * math.log2(pad) + 15 * pad + 150 * N


def work(case):
    kind = case["kind"]
    if kind.startswith("unet"):
        B = case["batch"]
        fl = B * U.conv_flops(64, 64)
        wt = sum(2 * 9 * c[2] * c[4] for c in U.CONVS)
        io = B * 4096 * (2 * U.FEAT + 2 * U.OUTC + 12 + 4)
        return {"bytes": io + wt, "flops": fl} if kind == "unet_forward" else {"bytes": io + 14 * wt, "flops": 3 * fl}
    if kind == "ensemble":
        by = fl = 0.0
        for q, grid in enumerate(W.ENSEMBLE_GRIDS_USER):
            b, k, f = _eval_work(grid[::-1])
            count = (case["nsim"] + q) // len(W.ENSEMBLE_GRIDS_USER)
            by += 2 * (b * count + k) * case["steps"]
            fl += 2 * f * count * case["steps"]
        return {"bytes": by, "flops": fl}
    n, sims, evals = (1, 64, 64), case.get("nsim", 1), 1
    if kind == "relax":
        evals = 3 * case["steps"] + 1
    else:
        n = (case["nz"], case["ny"], case["nx"])
        if kind == "step":
            evals = EVALS[case["solver"]] * case["steps"] + (case["solver"] in ("rk23", "rk45"))
    b, k, f = _eval_work(n)
    if kind == "fields":
        b = 84 * n[0] * n[1] * n[2]
    return {"bytes": evals * (b * sims + k), "flops": evals * f * sims}


def tolerance(case):
    kind = case["kind"]
    if kind in ("torque", "fields"):
        return {"rel": 2e-6}
    if kind.startswith("unet"):
        return {"rel": 4e-2}
    return {"rel": 2e-6}


# ---------------------------------------------------------------- the same in 64 bits
def _arne(n, cell, accuracy=6):
    """Transform of the demag tensor by face-charge integration: for each source axis s the
    field of the charges of a cell's two faces, averaged over the destination cell, with a
    number of points that falls with distance.  {(s, d): real [L0][L1][L2/2+1]}, s <= d."""
    dev = "cuda"
    L = [2 * v if v > 1 else 1 for v in n]
    cs = [float(c) for c in cell]
    ax = [torch.arange(v, device=dev, dtype=torch.float64) for v in n]
    far = [torch.clamp(a - 1, min=0) * c for a, c in zip(ax, cs)]
    d = torch.sqrt(far[0][:, None, None] ** 2 + far[1][None, :, None] ** 2 + far[2][None, None, :] ** 2).reshape(-1)
    d = torch.where(d == 0, torch.full_like(d, min(cs)), d)
    # tensor by tensor, which torch divides exactly: the quotients hit ties of the rounding
    size = d / torch.full_like(d, accuracy)
    num = torch.stack([(torch.clamp(torch.full_like(d, c) / size, min=1.0) + 0.5).floor().long() for c in cs])
    R = torch.stack(torch.meshgrid(*[a * c for a, c in zip(ax, cs)], indexing="ij")).reshape(3, -1)
    uniq, inv = torch.unique(num, dim=1, return_inverse=True)
    out = {}
    for s in range(3):
        v, w = (s + 1) % 3, (s + 2) % 3
        B = torch.zeros_like(R)
        for q in range(uniq.shape[1]):
            k = uniq[:, q].tolist()
            dest = [(-c / 2 + c / (2 * a) + c / a * torch.arange(a, device=dev, dtype=torch.float64)) for c, a in zip(cs, k)]
            off = list(dest)
            poles = 1
            for a in (v, w):
                m = 2 * k[a]
                pole = -cs[a] / 2 + cs[a] / (2 * m) + cs[a] / m * torch.arange(m, device=dev, dtype=torch.float64)
                off[a] = (dest[a][:, None] - pole[None, :]).reshape(-1)
                poles *= m
            P = torch.stack(torch.meshgrid(*off, indexing="ij")).reshape(3, -1)
            charge = cs[v] * cs[w] / (poles * k[0] * k[1] * k[2]) / (4 * math.pi)
            idx = torch.nonzero(inv == q).reshape(-1)
            for part in torch.split(idx, max(1, 4_000_000 // P.shape[1])):
                acc = torch.zeros((3, part.numel()), device=dev, dtype=torch.float64)
                for sign in (1.0, -1.0):
                    X = R[:, part, None] + P[:, None, :]
                    X[s] -= sign * cs[s] / 2
                    acc += sign * charge * (X / X.square().sum(0).pow(1.5)).sum(-1)
                B[:, part] = acc
        for t in range(s, 3):
            K = torch.zeros(L, device=dev, dtype=torch.float64)
            o = B[t].reshape(n)
            for axis in range(3):  # mirror to the negative offsets; the Nyquist plane stays zero
                if L[axis] == 1:
                    continue
                odd = s != t and axis in (s, t)
                rest = torch.flip(o.narrow(axis, 1, n[axis] - 1), [axis])
                o = torch.cat([o, torch.zeros_like(o.narrow(axis, 0, 1)), -rest if odd else rest], axis)
            if s != t and L[s] == 1 or s != t and L[t] == 1:
                o = torch.zeros_like(o)  # odd along an axis with one plane
            K += o
            out[(s, t)] = torch.fft.rfftn(K).real
    return out


def _normals(seed, N, step):
    """Box-Muller normals of Philox4x32-10 keyed by (seed, cell, step), as the thermal field
    defines them: float64 [3][N]."""
    M32 = 0xFFFFFFFF
    c = [torch.arange(N, dtype=torch.int64, device="cuda"), *(torch.full((N,), v, dtype=torch.int64, device="cuda")
                                                              for v in (step & M32, step >> 32, 0x7E57))]
    k0, k1 = seed & M32, (seed >> 32) & M32

    def mul(a, x):  # 32 x 32 -> (high, low) in 64-bit integers without overflow
        lo16, hi16 = (x & 0xFFFF) * a, (x >> 16) * a
        t = hi16 + (lo16 >> 16)
        return (t >> 16) & M32, ((t << 16) | (lo16 & 0xFFFF)) & M32

    for _ in range(10):
        h0, l0 = mul(0xD2511F53, c[0])
        h1, l1 = mul(0xCD9E8D57, c[2])
        c = [h1 ^ c[1] ^ k0, l1, h0 ^ c[3] ^ k1, l0]
        k0, k1 = (k0 + 0x9E3779B9) & M32, (k1 + 0xBB67AE85) & M32
    u = [((x >> 8).double() + 0.5) * 2.0 ** -24 for x in c]
    r0, r1 = torch.sqrt(-2 * torch.log(u[0])), torch.sqrt(-2 * torch.log(u[2]))
    return torch.stack([r0 * torch.cos(2 * math.pi * u[1]), r0 * torch.sin(2 * math.pi * u[1]),
                        r1 * torch.cos(2 * math.pi * u[3])])


def _cross(a, b):
    return torch.stack([a[:, 1] * b[:, 2] - a[:, 2] * b[:, 1], a[:, 2] * b[:, 0] - a[:, 0] * b[:, 2],
                        a[:, 0] * b[:, 1] - a[:, 1] * b[:, 0]], 1)


class _Ref:
    """The right-hand side and the solvers in 64 bits: states [B][3][n0][n1][n2]."""

    def __init__(self, pr, masks=None, sims=None):
        self.pr, self.n, self.sims = pr, tuple(pr["n"]), sims or [pr]
        self.B = len(self.sims)
        self.K = _arne(self.n, pr["cell"])
        self.mk = {k: torch.as_tensor(np.asarray(v), device="cuda").double().reshape(-1, 1, *self.n)
                   for k, v in (masks or {}).items()}
        self.noise = 0

    def sc(self, key, default=0.0):
        return torch.tensor([float(s.get(key, self.pr.get(key, default))) for s in self.sims], device="cuda",
                            dtype=torch.float64).reshape(-1, 1, 1, 1, 1)

    def vec(self, key):
        return torch.tensor([list(s.get(key, self.pr.get(key, (0.0, 0.0, 0.0)))) for s in self.sims], device="cuda",
                            dtype=torch.float64).reshape(-1, 3, 1, 1, 1)

    def unit(self, v):
        nrm = v.norm(dim=1, keepdim=True)
        out = torch.where(nrm > 0, v / torch.where(nrm > 0, nrm, torch.ones_like(nrm)), torch.zeros_like(v))
        return torch.where(self.mk["msat"] != 0, out, torch.zeros_like(out)) if "msat" in self.mk else out

    def demag(self, m):
        n = self.n
        L = [2 * v if v > 1 else 1 for v in n]
        src = m * self.mk["msat"] if "msat" in self.mk else m
        out = torch.empty_like(m)
        for b in range(self.B):  # one simulation at a time: bounded memory
            F = torch.fft.rfftn(src[b], s=L, dim=(1, 2, 3))
            H = torch.stack([sum(self.K[(min(s, t), max(s, t))] * F[s] for s in range(3)) for t in range(3)])
            out[b] = torch.fft.irfftn(H, s=L, dim=(1, 2, 3))[:, :n[0], :n[1], :n[2]]
        return out * self.sc("msat")

    def exchange(self, m):
        zero = torch.zeros_like(m)
        ratio = lambda a, b: torch.where(b != 0, a / torch.where(b != 0, b, torch.ones_like(b)), torch.zeros_like(a))  # noqa: E731
        one = torch.ones((1, 1) + self.n, device="cuda", dtype=torch.float64)
        lex = ratio(self.mk.get("aex", one), self.mk.get("msat", one) + zero[:, :1])
        H = torch.zeros_like(m)
        for a in range(3):
            if self.n[a] == 1:
                continue
            lo, hi = (lambda x: x.narrow(a + 2, 0, self.n[a] - 1)), (lambda x: x.narrow(a + 2, 1, self.n[a] - 1))
            wgt = ratio(2 * lo(lex) * hi(lex), lo(lex) + hi(lex)) * (hi(m) - lo(m)) / self.pr["cell"][a] ** 2
            H.narrow(a + 2, 0, self.n[a] - 1).add_(wgt)
            H.narrow(a + 2, 1, self.n[a] - 1).sub_(wgt)
        return H * 2 * self.sc("aex") / (MU0 * self.sc("msat"))

    def terms(self, m, dt=None):
        z = torch.zeros_like(m)
        pr = self.pr
        out = {"demag": self.demag(m), "ex": self.exchange(m), "anis": z, "zee": z, "therm": z}
        ms = self.mk.get("msat")
        if pr.get("zeeman"):
            out["zee"] = self.vec("bext") / MU0 + z
        if pr.get("anis"):
            u = self.vec("anisu")
            k2 = 2 * self.sc("ku") / (MU0 * self.sc("msat"))
            k2 = k2 / torch.where(ms == 0, torch.ones_like(ms), ms) if ms is not None else k2
            out["anis"] = k2 * (m * u).sum(1, keepdim=True) * u
        if pr.get("thermal"):
            vol = pr["cell"][0] * pr["cell"][1] * pr["cell"][2]
            s = torch.sqrt(2 * KB * self.sc("alpha") * self.sc("temp") / (MU0 * vol * pr["gamma"] * self.sc("msat") * dt))
            N = self.n[0] * self.n[1] * self.n[2]
            eta = torch.stack([_normals(int(q["seed"]), N, self.noise) for q in self.sims])
            out["therm"] = eta.reshape(m.shape) * s
        out["eff"] = sum(out[k] for k in ("demag", "ex", "anis", "zee", "therm"))
        return out

    def rhs(self, m, dt=None):
        pr = self.pr
        H = self.terms(m, dt)["eff"]
        al = self.sc("alpha")
        c = _cross(m, H)
        k = (c - al * _cross(m, c)) / (1 + al * al)
        ms = self.mk.get("msat")
        inv_ms = 1.0 if ms is None else torch.where(ms != 0, 1 / torch.where(ms != 0, ms, torch.ones_like(ms)), 0 * ms)
        if pr.get("zhangli"):
            j = np.array(pr["j"], dtype=np.float64)
            jn = float(np.linalg.norm(j))
            pre = jn * pr["zl_pol"] * MUB / (QE * pr["msat"]) / ((1 + pr["xi"] ** 2) * (1 + pr["alpha"] ** 2))
            dm = torch.zeros_like(m)
            for a in range(3):
                if j[a] == 0:
                    continue
                i = torch.arange(self.n[a], device="cuda")
                at = lambda o: m.index_select(a + 2, torch.where((i + o < 0) | (i + o >= self.n[a]), i, i + o))  # noqa: E731
                dm += j[a] / jn / (12 * pr["cell"][a]) * (at(-2) - 8 * at(-1) + 8 * at(1) - at(2))
            f = -_cross(dm, m)
            k = k + inv_ms / pr["gamma"] * pre * (-(1 + pr["xi"] * pr["alpha"]) * _cross(m, f)
                                                  + (pr["xi"] - pr["alpha"]) * f)
        if pr.get("slonczewski"):
            j = np.array(pr["j"], dtype=np.float64)
            nj = float(np.linalg.norm(j)) * float(np.sign(j.sum()))
            beta = HBAR * pr["gamma"] / (MU0 * QE * pr["msat"])
            p = torch.tensor(pr["p"], device="cuda", dtype=torch.float64).reshape(1, 3, 1, 1, 1)
            p = (p / p.norm()).expand_as(m)
            l2 = pr["lambda"] ** 2
            eps = l2 / ((l2 + 1) + (l2 - 1) * (p * m).sum(1, keepdim=True))
            fx = pr["sl_pol"] * beta * inv_ms * nj / pr["t_fl"] * eps
            fy = beta * pr["eps_prime"] * inv_ms * nj / pr["t_fl"]
            pxm = -_cross(p, m)
            a2 = 1 + pr["alpha"] ** 2
            k = k + ((fx - pr["alpha"] * fy) / a2 * -_cross(m, pxm) + (fy - pr["alpha"] * fx) / a2 * pxm) / pr["gamma"]
        return k

    TAB = {"rk23": ([[0.5], [0, 0.75], [2 / 9, 1 / 3, 4 / 9]], [5 / 72, -1 / 12, -1 / 9, 1 / 8], 2),
           "rk45": ([[1 / 5], [3 / 40, 9 / 40], [44 / 45, -56 / 15, 32 / 9],
                     [19372 / 6561, -25360 / 2187, 64448 / 6561, -212 / 729],
                     [9017 / 3168, -355 / 33, 46732 / 5247, 49 / 176, -5103 / 18656],
                     [35 / 384, 0, 500 / 1113, 125 / 192, -2187 / 6784, 11 / 84]],
                    [71 / 57600, 0, -71 / 16695, 71 / 1920, -17253 / 339200, 22 / 525, -1 / 40], 4)}

    def steps(self, m, solver, dt, maxerr, count):
        m = self.unit(m)
        dt = torch.full((self.B,), dt, device="cuda", dtype=torch.float64)
        left = torch.full((self.B,), count, device="cuda")
        fsal = solver in self.TAB
        k0 = self.rhs(m) if fsal else None
        while bool((left > 0).any()):
            h = (dt * self.pr["gamma"]).reshape(-1, 1, 1, 1, 1)
            d5 = dt.reshape(-1, 1, 1, 1, 1)
            if fsal:
                A, E, q = self.TAB[solver]
                ks, y = [k0], m
                for row in A:
                    y = self.unit(m + h * sum(a * k for a, k in zip(row, ks)))
                    ks.append(self.rhs(y, d5))
                e = sum(a * k for a, k in zip(E, ks))
            else:
                q = 1
                k0 = self.rhs(m, d5)
                y = self.unit(m + h * k0)
                if solver != "euler":
                    k1 = self.rhs(y, d5)
                    y = self.unit(y + 0.5 * h * (k1 - k0))
                    e = k1 - k0
            ok = left > 0
            if solver not in ("heun", "euler"):
                err = e.abs().reshape(self.B, -1).amax(1) * dt * self.pr["gamma"]
                bad = err > maxerr
                fac = 0.8 * torch.where(bad, (maxerr / err) ** (1.0 / (q + 2)), (maxerr / err) ** (1.0 / (q + 1)))
                dt = torch.where(ok, dt * torch.clamp(fac, 0.1, 1.5), dt)
                ok = ok & ~bad
            w = ok.reshape(-1, 1, 1, 1, 1)
            m = torch.where(w, y, m)
            if fsal:
                k0 = torch.where(w, ks[-1], k0)
            left = left - ok.long()
            self.noise += 1
        return m


def _unet_exact(case, seed):
    sims, masks, tgt = _unet_inputs(case, seed)
    B = case["batch"]
    params = U.init_params(seed)
    bf = lambda a: torch.tensor(a, device="cuda").to(torch.bfloat16).double()  # noqa: E731
    w = {k: bf(v[0]).requires_grad_(True) for k, v in params.items()}
    b = {k: torch.tensor(v[1], device="cuda").double().requires_grad_(True) for k, v in params.items()}
    convs = {c[0]: c for c in U.CONVS}
    x = torch.tensor(U.features(sims, masks, (1, 64, 64)), device="cuda").double().reshape(B, 64, 64, -1).permute(0, 3, 1, 2)
    parts = {("in", 0): x}

    def view(name, off, ch):
        got = sorted((o, v) for (nm, o), v in parts.items() if nm == name and off <= o < off + ch)
        return torch.cat([v for _, v in got], 1)

    for op in U.SCHEDULE:
        if op.startswith("pool"):
            (sv, so), (dv, do), ch, _ = U.POOLS[int(op[4:])]
            parts[(dv, do)] = torch.nn.functional.avg_pool2d(view(sv, so, ch), 2)
        elif op.startswith("up"):
            (sv, so), (dv, do), ch, _ = U.UPS[int(op[2:])]
            parts[(dv, do)] = view(sv, so, ch).repeat_interleave(2, 2).repeat_interleave(2, 3)
        else:
            name, (iv, io), cin, (ov, oo), cout, relu = convs[op]
            xi = torch.nn.functional.pad(view(iv, io, cin), (1, 1, 1, 1))
            H, Wd = xi.shape[2] - 2, xi.shape[3] - 2
            y = b[name].reshape(1, -1, 1, 1)
            for tap in range(9):  # one matrix product per tap
                dy, dx = tap // 3, tap % 3
                y = y + torch.einsum("bchw,oc->bohw", xi[:, :, dy:dy + H, dx:dx + Wd], w[name][:, tap])
            parts[(ov, oo)] = torch.relu(y) if relu else y
    out = parts[("out", 0)].permute(0, 2, 3, 1).reshape(B, 4096, U.OUTC)
    mk = torch.from_numpy(masks).cuda().double()
    if case["kind"] == "unet_forward":
        o3 = out[..., :3]
        st = o3 / o3.norm(dim=2, keepdim=True) * mk[..., None]
        return {"out": out.detach().reshape(-1),
                "states": torch.stack([st[..., 2], st[..., 1], st[..., 0]], 1).detach().reshape(-1)}
    loss = (mk[..., None] * (out[..., :3] - tgt.double()).square()).sum() / (3 * max(1.0, float(masks.sum())))
    names = [c[0] for c in U.CONVS]
    g = torch.autograd.grad(loss, [w[k] for k in names] + [b[k] for k in names])
    gw, gb = g[:len(names)], g[len(names):]
    upd = []
    for k, d in zip(names, gw):  # the first Adam step
        v = torch.tensor(params[k][0], device="cuda").double() - 1e-3 * d / (d.abs() + 1e-8)
        if k == "out":
            v[3:] = 0
        upd.append(v.reshape(-1))
    return {"loss": loss.detach().reshape(1), "out": out.detach().reshape(-1), "gw": [d.reshape(-1) for d in gw],
            "gb": [d.reshape(-1) for d in gb], "w": upd}


def exact(case, seed):
    kind = case["kind"]
    if kind.startswith("unet"):
        return _unet_exact(case, seed) if case["batch"] <= 64 else None
    if kind == "ensemble":
        outs = []
        for c, m in _ensemble_inputs(case, seed):
            r = _Ref(c["problem"], sims=c["sims"])
            m = m.double().reshape(len(c["sims"]), 3, *c["n"])
            outs.append(r.steps(m, "heun", W.ENSEMBLE_DT, 1.0, case["steps"]).reshape(-1))
        return outs
    if kind == "relax":
        pr, sims, masks, m = _relax_inputs(case, seed)
        r = _Ref(pr, masks={"msat": masks}, sims=sims)
        return r.steps(m.double().reshape(len(sims), 3, *pr["n"]), "rk23", 1e-15, 1e-6, case["steps"]).reshape(-1)
    pr, masks, m = _problem(case, seed)
    r = _Ref(pr, masks=masks)
    m = m.double().reshape(1, 3, *pr["n"])
    if kind == "fields":
        return {k: v.reshape(-1) for k, v in r.terms(m).items()}
    if kind == "torque":
        m = r.unit(m)
        return r.rhs(m).reshape(-1), m.reshape(-1)
    return r.steps(m, case["solver"], _dt0(case), MAXERR[case["solver"]], case["steps"]).reshape(-1)

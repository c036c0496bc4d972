"""The work that users of this library have it do, as cases to be timed.

A case is one call (or the few calls that belong together) through the public
Python entry points: the reference's default run, large SOR batches in both
precisions, the host-buffer call sequence of the reference's API, multigrid
with 5-point gravity, a mixed-ghost-size batch plan, and the learned starts
with their training steps.  Inputs are the seeded power-law patches of
gpg.inputs, made on the GPU.  The patch counts are those of bench.py, of the
reference's own runs and of learned.py's training, with odd ones among them.
"""
import math
import os
import sys

import numpy as np
import torch

PKG = os.path.join(os.getcwd(), "gpu_testbed_poisson-gravity_b200")
if PKG not in sys.path:
    sys.path.insert(0, PKG)

import learned  # noqa: E402
from gpg.abi import (GPG_INIT_GUESS, GPG_INIT_INTERP, GPG_INIT_ZERO, GPG_INT_CQUAD, GPG_INT_QUAD, GPG_MG,  # noqa: E402
                     GPG_SOR, default_params, fixed_residual_params, patch_sizes)
from gpg.lib import BatchPlan, Context, solve_batch_device, solve_device  # noqa: E402
from gpg.linear import LinearGuess  # noqa: E402
from gpg.net import LAYERS, Net  # noqa: E402

DEV = "cuda"
POI = 4.0 * math.pi * 1.0e-5
BOX, PATCH, R0 = 16, 8, 8.0
MIX = (0.3, 0.3, 0.2, 0.1, 0.1)          # ghost 1..5 shares of a mixed batch


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def _solve(name, scheme, bits, ghost, npatch, **kw):
    c = {"kind": "solve", "scheme": scheme, "bits": bits, "ghost": ghost, "npatch": npatch, "gra_ghost": 1,
         "quad": False, "gravity": False, "p5": False, "fixed": False}
    c.update(kw)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the reference's default run: a small call of a running simulation, latency bound
        _solve("sor_f32_g1_256", "sor", 32, 1, 256, gravity=True),
        # a batch of the headline workload in single precision
        _solve("sor_f32_g3_4096", "sor", 32, 3, 4096),
        # an odd number of patches, the other interpolation, gravity in the same call, double precision
        _solve("sor_f64_g2_1001_quad", "sor", 64, 2, 1001, quad=True, gravity=True),
        # the largest cubes in double precision: the longest batch of the headline workload
        _solve("sor_f64_g5_4096", "sor", 64, 5, 4096),
        # multigrid with 5-point gravity, single precision, a full level of a run
        _solve("mg_f32_g3_p5_16384", "mg", 32, 3, 16384, gra_ghost=2, gravity=True, p5=True),
        # multigrid in double precision, an ordinary number of patches
        _solve("mg_f64_g4_1000", "mg", 64, 4, 1000, gravity=True),
        # the reference-shaped call sequence: host buffers in, solver and gravity, host buffers out
        {"name": "host_f32_g2_4096", "kind": "host", "bits": 32, "ghost": 2, "npatch": 4096},
        # one batch plan over patches of all five ghost sizes, launched again each step
        {"name": "plan_f32_65536", "kind": "plan", "bits": 32, "npatch": 65536, "mode": 1},
        # the learned linear start and SOR to the fixed residual
        {"name": "lin_solve_65536", "kind": "lin_solve", "npatch": 65536, "gravity": False},
        # the learned network's start and SOR from it
        {"name": "net_solve_4096", "kind": "net_solve", "npatch": 4096},
        # one training step of the linear start (gradient, then Adam), learned.py's batch
        {"name": "lin_train_2048", "kind": "lin_train", "npatch": 2048},
        # a data-parallel rank's gradient of the network, learned.py's batch
        {"name": "net_train_1024", "kind": "net_train", "npatch": 1024},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["sor", "sor", "sor", "sor", "mg", "mg", "host", "plan", "lin_solve", "net_solve", "lin_train",
                       "net_train"])
    bits = rng.choice([32, 64])
    ghost = rng.randint(1, 5)
    gravity = rng.random() < 0.5
    p5 = gravity and ghost >= 2 and rng.random() < 0.3
    opt = {"gravity": gravity, "p5": p5, "gra_ghost": 2 if p5 else 1, "quad": rng.random() < 0.25}
    if kind == "sor":
        fixed = rng.random() < 0.25
        hi = (16384 if ghost <= 3 else 8192) if bits == 32 else 4096
        return _solve(None, "sor", bits, ghost, _log(rng, 64, hi // 3 if fixed else hi), fixed=fixed, **opt)
    if kind == "mg":
        hi = {32: 16384 if ghost <= 3 else 4096, 64: 2048 if ghost <= 3 else 1000}[bits]
        return _solve(None, "mg", bits, ghost, _log(rng, 64, hi), **opt)
    if kind == "host":
        hi = (512 if ghost <= 2 else 256) * 32 // bits
        return {"kind": "host", "bits": bits, "ghost": ghost, "npatch": 8 * _log(rng, 8, hi)}
    if kind == "plan":
        return {"kind": "plan", "bits": 32, "npatch": _log(rng, 500, 65536), "mode": rng.choice([0, 1, 1, 2])}
    if kind == "lin_solve":
        return {"kind": kind, "npatch": _log(rng, 100, 65536), "gravity": gravity}
    if kind == "net_solve":
        return {"kind": kind, "npatch": _log(rng, 64, 4096)}
    if kind == "lin_train":
        return {"kind": kind, "npatch": _log(rng, 64, 4096)}
    return {"kind": kind, "npatch": _log(rng, 32, 1024)}


# ---------------------------------------------------------------------------
# inputs (the profiles of gpg.inputs.make_patches, on the GPU)
# ---------------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _radius(n_patch, first, count, spacing):
    """[P][n][n][n] radius of the cell centres of a window that begins `first`
    fine cells below each patch's corner."""
    p = torch.arange(n_patch, device=DEV)
    idx = (torch.arange(count, device=DEV, dtype=torch.float64) + 0.5) * spacing - first - 0.5 * BOX * PATCH
    x, y, z = ((((p // BOX ** k) % BOX) * PATCH).double()[:, None] + idx[None, :] for k in range(3))
    return (x[:, None, None, :] ** 2 + y[:, None, :, None] ** 2 + z[:, :, None, None] ** 2).sqrt_()


def _patches(n, ghost, seed, dtype, fluid, rho0=None, index=None):
    g = _gen(seed)
    pn, m = 4 + 2 * ((ghost + 3) // 2), 6 + 2 * ghost
    bc = (slice(None), None, None, None)
    rho0 = torch.ones(n, device=DEV, dtype=torch.float64) if rho0 is None else rho0
    index = torch.full((n,), 2.0, device=DEV, dtype=torch.float64) if index is None else index
    rho = rho0[bc] * (_radius(n, ghost - 1, m, 1.0) / R0) ** (-index[bc])
    rho *= 1.0 + 0.05 * torch.randn(rho.shape, generator=g, device=DEV, dtype=torch.float64)
    ln_s = (_radius(n, 2 * ((ghost + 3) // 2), pn, 2.0) / R0).log_()
    two_n = (2.0 - index)[bc]
    small = two_n.abs() < 1e-9
    prof = torch.where(small, ln_s, torch.expm1(two_n * ln_s) / torch.where(small, torch.ones_like(two_n), two_n))
    pot = POI * R0 * R0 * rho0[bc] * prof / (3.0 - index)[bc]
    out = {"rho": rho.to(dtype), "pot_in": pot.to(dtype)}
    if fluid:
        lo = ghost - 1
        dens = rho[:, lo:lo + 8, lo:lo + 8, lo:lo + 8]
        flu = torch.empty((n, 5, 8, 8, 8), device=DEV, dtype=torch.float64)
        flu[:, 0] = dens
        flu[:, 1:4] = dens[:, None] * 0.1 * torch.randn((n, 3, 8, 8, 8), generator=g, device=DEV, dtype=torch.float64)
        flu[:, 4] = 1.0 + 0.1 * torch.rand((n, 8, 8, 8), generator=g, device=DEV, dtype=torch.float64)
        out["flu"] = flu.to(dtype)
    return out


def _spread(n, seed):
    """rho0 over four decades and the power index in [1.5, 2.5], the learned starts' patches."""
    g = _gen(seed + 1_000_003)
    rho0 = 10.0 ** (4.0 * torch.rand(n, generator=g, device=DEV, dtype=torch.float64))
    return rho0, 1.5 + torch.rand(n, generator=g, device=DEV, dtype=torch.float64)


def _dtype(c):
    return torch.float32 if c.get("bits", 32) == 32 else torch.float64


def _params(c):
    rs = c["bits"] // 8
    kw = dict(gra_ghost=c["gra_ghost"], gra_acc=int(c["gravity"]), p5_gradient=int(c["p5"]),
              int_scheme=GPG_INT_QUAD if c["quad"] else GPG_INT_CQUAD)
    if c["scheme"] == "mg":
        return default_params(rs, c["ghost"], GPG_MG, **kw)
    if c["fixed"]:
        return fixed_residual_params(rs, c["ghost"], init_mode=GPG_INIT_ZERO, **kw)
    return default_params(rs, c["ghost"], GPG_SOR, **kw)


def _mix(n):
    m = [int(f * n) for f in MIX]
    m[0] += n - sum(m)
    return m


def _outputs(n, gn, dtype):
    return {"pot_out": torch.empty((n, gn, gn, gn), device=DEV, dtype=dtype),
            "iters": torch.empty(n, device=DEV, dtype=torch.int32),
            "resid": torch.empty(n, device=DEV, dtype=torch.float64)}


def _inputs(c, seed):
    """What the case's arrays hold; also what exact() starts from."""
    kind, n = c["kind"], c["npatch"]
    if kind == "solve":
        return _patches(n, c["ghost"], seed, _dtype(c), c["gravity"])
    if kind == "host":
        return _patches(n, c["ghost"], seed, _dtype(c), True)
    if kind == "plan":
        rho0 = 10.0 ** (4.0 * torch.rand(n, generator=_gen(seed + 7), device=DEV, dtype=torch.float64))
        at, groups = 0, []
        for g, m in enumerate(_mix(n), 1):
            if m:
                groups.append(dict(_patches(m, g, seed + g, _dtype(c), False, rho0=rho0[at:at + m]), ghost=g))
            at += m
        return groups
    rho0, index = _spread(n, seed)
    d = _patches(n, 1, seed, torch.float32, c.get("gravity", False), rho0=rho0, index=index)
    if kind == "lin_train":
        return _lin_features(d)
    if kind == "net_train":
        d["target"] = _poisson(d["rho"].double(), d["pot_in"].double(), 1, False)[:, 1:-1, 1:-1, 1:-1].float()
        d["weights"] = _net_weights(seed)
    return d


def _lin_weights(seed):
    return (0.02 * torch.randn(4 * 64 * 64, generator=_gen(seed + 11), device=DEV)).cpu().numpy()


def _net_weights(seed):
    """He-normal weights of the four layers (channels 3..7 of the input and 1..15 of the output unused)."""
    g, flat = _gen(seed + 13), []
    for k, (cin, cout) in enumerate(LAYERS):
        ci, co = (3 if k == 0 else cin), (1 if k == 3 else cout)
        w = torch.zeros((27, cin, cout), device=DEV)
        w[:, :ci, :co] = math.sqrt(2.0 / (27 * ci)) * torch.randn((27, ci, co), generator=g, device=DEV)
        flat += [w.reshape(-1), torch.zeros(cout, device=DEV)]
    return torch.cat(flat).cpu().numpy()


# ---------------------------------------------------------------------------
# prepare and run
# ---------------------------------------------------------------------------
class _Held(dict):
    """The arrays of a host call, and the context that owns them."""


class _Context(Context):
    def __del__(self):
        try:
            self.close()
        except Exception:
            pass


def prepare(case, seed):
    kind, n = case["kind"], case["npatch"]
    d = _inputs(case, seed)
    if kind == "solve":
        p = _params(case)
        return {"kind": kind, "p": p, "in": d, "out": _outputs(n, patch_sizes(p)["gra_nxt"], _dtype(case))}
    if kind == "host":
        p = default_params(case["bits"] // 8, case["ghost"], GPG_SOR)
        ctx = _Context(torch.cuda.current_device(), 4)
        rho, pot_in, pot_out, flu = ctx.allocate(p, n // 8)
        for dst, k in ((rho, "rho"), (pot_in, "pot_in"), (flu, "flu")):
            torch.from_numpy(dst).copy_(d[k])
        out = _Held(pot_out=pot_out, flu=flu)
        out.owner = ctx
        return {"kind": kind, "p": p, "ctx": ctx, "groups": n // 8, "out": out}
    if kind == "plan":
        p = default_params(4, 1, GPG_SOR, gra_acc=0)
        for g in d:
            g.update(_outputs(g["rho"].shape[0], 10, _dtype(case)))
        st = {"kind": kind, "p": p, "groups": d, "out": [{k: g[k] for k in ("pot_out", "iters", "resid")} for g in d]}
        if case["mode"] < 2:
            st["plan"] = BatchPlan(p, d, torch.cuda.current_device(), mode=case["mode"])
        else:
            st["counter"] = torch.zeros(1, device=DEV, dtype=torch.int32)
        return st
    if kind == "lin_solve":
        lin = LinearGuess(max_batch=1, device_id=torch.cuda.current_device())
        learned.load_lin(lin)
        kw = dict(gra_acc=1, gra_ghost=1) if case["gravity"] else {}
        p = fixed_residual_params(4, 1, init_mode=GPG_INIT_INTERP, **kw)
        return {"kind": kind, "lin": lin, "p": p, "in": d, "out": _outputs(n, 8 + 2 * p.gra_ghost, torch.float32)}
    if kind == "net_solve":
        net = Net(max_batch=1, device_id=torch.cuda.current_device())
        learned.load(net, learned.DEFAULT_WEIGHTS)
        return {"kind": kind, "net": net, "p": fixed_residual_params(4, 1, init_mode=GPG_INIT_GUESS), "in": d,
                "guess": torch.empty((n, 8, 8, 8), device=DEV), "out": _outputs(n, 8, torch.float32)}
    if kind == "lin_train":
        lin = LinearGuess(max_batch=n, device_id=torch.cuda.current_device())
        lin.set_params(_lin_weights(seed))
        return {"kind": kind, "lin": lin, "in": d, "grad": torch.empty(lin.nparams, device=DEV),
                "loss": torch.empty(1, device=DEV)}
    net = Net(max_batch=n, device_id=torch.cuda.current_device())
    net.set_params(d["weights"])
    return {"kind": kind, "net": net, "in": d, "grad": torch.empty(net.nparams, device=DEV),
            "loss": torch.empty(1, device=DEV)}


def run(state):
    kind = state["kind"]
    if kind == "solve":
        d, o = state["in"], state["out"]
        solve_device(state["p"], d["rho"], d["pot_in"], pot_out=o["pot_out"], flu=d.get("flu"), iters=o["iters"],
                     resid=o["resid"])
        return dict(o, flu=d["flu"]) if "flu" in d else o
    if kind == "host":
        state["ctx"].asyn_solve(state["p"], state["groups"])
        state["ctx"].synchronize()
        return state["out"]
    if kind == "plan":
        if "plan" in state:
            state["plan"].launch()
        else:
            solve_batch_device(state["p"], state["groups"], state["counter"])
        return state["out"]
    if kind == "lin_solve":
        d, o = state["in"], state["out"]
        state["lin"].solve(state["p"], d["rho"], d["pot_in"], pot_out=o["pot_out"], flu=d.get("flu"),
                           iters=o["iters"], resid=o["resid"])
        return dict(o, flu=d["flu"]) if "flu" in d else o
    if kind == "net_solve":
        d, o = state["in"], state["out"]
        state["net"].predict(d["rho"], d["pot_in"], state["guess"], learned.CNST)
        solve_device(state["p"], d["rho"], d["pot_in"], pot_out=o["pot_out"], guess=state["guess"], iters=o["iters"],
                     resid=o["resid"])
        return dict(o, guess=state["guess"])
    if kind == "lin_train":
        u, t = state["in"]
        state["lin"].gradients(u, t, grad=state["grad"], loss=state["loss"])
        state["lin"].apply_gradient(state["grad"], 2e-3)
    else:
        d = state["in"]
        state["net"].gradients(d["rho"], d["pot_in"], d["target"], learned.CNST, grad=state["grad"],
                               loss=state["loss"])
    return {"grad": state["grad"], "loss": state["loss"]}


# ---------------------------------------------------------------------------
# what one pass cannot do without
# ---------------------------------------------------------------------------
def _solve_work(bits, ghost, n, gn, gravity, sweeps):
    m, pn = 6 + 2 * ghost, 4 + 2 * ((ghost + 3) // 2)
    values = m ** 3 + pn ** 3 + gn ** 3 + (2560 + 2048 if gravity else 0)
    return {"bytes": n * (values * bits // 8 + 12), "flops": n * m ** 3 * 10 * sweeps}


def work(case):
    kind, n = case["kind"], case["npatch"]
    if kind == "solve":
        # at least the reference's Min_Iter sweeps, or two V-cycles of six; about 26 sweeps from a zero start
        sweeps = 12 if case["scheme"] == "mg" else 26 if case["fixed"] else 10
        return _solve_work(case["bits"], case["ghost"], n, 8 + 2 * case["gra_ghost"], case["gravity"], sweeps)
    if kind == "host":
        return _solve_work(case["bits"], case["ghost"], n, 10, True, 10)
    if kind == "plan":
        parts = [_solve_work(32, g, m, 10, False, 10) for g, m in enumerate(_mix(n), 1)]
        return {k: sum(w[k] for w in parts) for k in ("bytes", "flops")}
    if kind == "lin_solve":
        w = _solve_work(32, 1, n, 10 if case["gravity"] else 8, case["gravity"], 1)
        return {"bytes": w["bytes"] + 4 * 16384, "flops": w["flops"] + n * learned.LIN_FLOP}
    if kind == "net_solve":
        w = _solve_work(32, 1, n, 8, False, 10)
        return {"bytes": w["bytes"] + n * 2048, "flops": w["flops"] + n * learned.NET_FLOP}
    if kind == "lin_train":
        return {"bytes": n * 4096 + 4 * 16384 * 8, "flops": 2 * n * learned.LIN_FLOP}
    return {"bytes": n * 3 * 2048 + 4 * 76144 * 2, "flops": 3 * n * learned.NET_FLOP}


# ---------------------------------------------------------------------------
# the same in 64 bits
# ---------------------------------------------------------------------------
def _matrix(ghost, quad):
    """[8+2G][POT_NXT] interpolation along one axis; both schemes are tensor products of it."""
    pn, n, u = 4 + 2 * ((ghost + 3) // 2), 8 + 2 * ghost, ghost % 2
    rows = ((5 / 32, 30 / 32, -3 / 32), (-3 / 32, 30 / 32, 5 / 32)) if quad else ((1 / 8, 1, -1 / 8), (-1 / 8, 1, 1 / 8))
    a = torch.zeros((n, pn), device=DEV, dtype=torch.float64)
    for x in range(n):
        i = 1 + (x + u) // 2
        for k in range(3):
            a[x, i - 1 + k] = rows[(x + u) % 2][k]
    return a


def _along(a, f):
    """The matrix `a` applied along the three axes of f."""
    return torch.einsum("za,yb,xc,pabc->pzyx", a, a, a, f)


def _laplacian(f):
    c = f[:, 1:-1, 1:-1, 1:-1]
    return (f[:, 2:, 1:-1, 1:-1] + f[:, :-2, 1:-1, 1:-1] + f[:, 1:-1, 2:, 1:-1] + f[:, 1:-1, :-2, 1:-1]
            + f[:, 1:-1, 1:-1, 2:] + f[:, 1:-1, 1:-1, :-2] - 6 * c)


def _poisson(rho, pot_in, ghost, quad):
    """The potential on the solver's cube [P][8+2G]^3: the exact solution of the discrete equation."""
    cube = _along(_matrix(ghost, quad), pot_in)
    m = 6 + 2 * ghost
    k = torch.arange(1, m + 1, device=DEV, dtype=torch.float64)
    s = math.sqrt(2.0 / (m + 1)) * torch.sin(math.pi * k[:, None] * k[None, :] / (m + 1))
    lam = 2.0 * torch.cos(math.pi * k / (m + 1)) - 2.0
    r = _along(s, POI * rho - _laplacian(cube))
    r /= lam[:, None, None] + lam[None, :, None] + lam[None, None, :]
    cube[:, 1:-1, 1:-1, 1:-1] += _along(s, r)
    return cube


def _gravity(flu, cube, ghost, p5, dt=1.0e-2):
    def at(dz, dy, dx):
        return cube[:, ghost + dz:ghost + dz + 8, ghost + dy:ghost + dy + 8, ghost + dx:ghost + dx + 8]
    out = flu.clone()
    half = 0.5 / flu[:, 0]
    inner = flu[:, 4] - half * (flu[:, 1:4] ** 2).sum(1)
    for k, (dz, dy, dx) in enumerate(((0, 0, 1), (0, 1, 0), (1, 0, 0))):
        if p5:
            a = dt / 12 * (at(-2 * dz, -2 * dy, -2 * dx) - at(2 * dz, 2 * dy, 2 * dx)
                           + 8 * at(dz, dy, dx) - 8 * at(-dz, -dy, -dx))
        else:
            a = dt / 2 * (at(dz, dy, dx) - at(-dz, -dy, -dx))
        out[:, 1 + k] -= flu[:, 0] * a
    out[:, 4] = inner + half * (out[:, 1:4] ** 2).sum(1)
    return out


def _window(cube, ghost, gra_ghost):
    lo = ghost - gra_ghost
    return cube[:, lo:lo + 8 + 2 * gra_ghost, lo:lo + 8 + 2 * gra_ghost, lo:lo + 8 + 2 * gra_ghost]


def _exact_solve(d, ghost, gra_ghost, quad=False, p5=False):
    """Sweep counts and residuals depend on the rounding and have no 64-bit value."""
    cube = _poisson(d["rho"].double(), d["pot_in"].double(), ghost, quad)
    out = {"pot_out": _window(cube, ghost, gra_ghost), "iters": None, "resid": None}
    if "flu" in d:
        out["flu"] = _gravity(d["flu"].double(), cube, ghost, p5)
    return out


def _fold(r):
    """[P][8]^3 -> [P][8 parities][64]: even and odd parts along z, y, x, each
    block's axes permuted into those of its class."""
    for ax in (1, 3, 5):
        a, b = r.narrow(ax, 0, 4), r.narrow(ax, 4, 4).flip(ax)
        r = torch.stack((a + b, a - b), dim=ax)
    r = r.permute(0, 1, 3, 5, 2, 4, 6).reshape(-1, 8, 4, 4, 4)     # [P][pz py px][k][j][i]
    swap = {2: (2, 3), 4: (1, 3), 6: (1, 3), 5: (1, 2)}
    return torch.stack([r[:, b].transpose(*swap[b]) if b in swap else r[:, b] for b in range(8)], 1).reshape(-1, 8, 64)


def _lin_features(d):
    """(u, t): folded residual of the interpolated start and folded correction, scaled per patch."""
    rho, pin = d["rho"].double(), d["pot_in"].double()
    cube = _along(_matrix(1, False), pin)
    u = _fold(_laplacian(cube) - POI * rho)
    t = _fold((_poisson(rho, pin, 1, False) - cube)[:, 1:-1, 1:-1, 1:-1]) / 8.0
    e = torch.frexp(cube[:, 1:-1, 1:-1, 1:-1].abs().amax((1, 2, 3)))[1]
    sc = torch.ldexp(torch.ones_like(e, dtype=torch.float64), 17 - e)[:, None, None]
    return (sc * u).float().contiguous(), (sc * t).float().contiguous()


def _exact_lin_train(u, t, flat):
    w = torch.from_numpy(flat).to(DEV).double().reshape(4, 64, 64)
    cls = torch.tensor([bin(b).count("1") for b in range(8)], device=DEV)
    u, t = u.double(), t.double()
    e = torch.einsum("brk,pbk->pbr", w[cls], u) - t
    g = torch.einsum("pbr,pbk->brk", e, u) * (2.0 / (512 * u.shape[0]))
    grad = torch.zeros_like(w).index_add_(0, cls, g)
    return {"grad": grad.reshape(-1), "loss": (e ** 2).mean().reshape(1)}


def _net_forward(d, flat):
    """(y4 [P][10]^3 of output channel 0, scale [P]) of the network in 64 bits."""
    n = d["rho"].shape[0]
    cube = _along(_matrix(1, False), d["pot_in"].double())
    inner = torch.zeros((10, 10, 10), device=DEV, dtype=torch.float64)
    inner[1:-1, 1:-1, 1:-1] = 1.0
    s = (cube * (1 - inner)).abs().amax((1, 2, 3))[:, None, None, None]
    a = torch.zeros((n, 10, 10, 10, 8), device=DEV, dtype=torch.float64)
    a[:, 1:-1, 1:-1, 1:-1, 0] = learned.CNST * d["rho"].double() / s
    a[..., 1] = cube * (1 - inner) / s
    a[..., 2] = inner
    at = 0
    for k, (cin, cout) in enumerate(LAYERS):
        w = flat[at:at + 27 * cin * cout].reshape(27, cin, cout)
        b = flat[at + 27 * cin * cout:at + 27 * cin * cout + cout]
        at += 27 * cin * cout + cout
        pad = torch.nn.functional.pad(a, (0, 0, 1, 1, 1, 1, 1, 1))
        y = b
        for q in range(27):
            z, yy, x = q // 9, (q // 3) % 3, q % 3
            y = y + pad[:, z:z + 10, yy:yy + 10, x:x + 10] @ w[q]
        a = torch.relu(y) if k < 3 else y
    return a[..., 0], s


def exact(case, seed):
    kind = case["kind"]
    d = _inputs(case, seed)
    if kind == "solve":
        return _exact_solve(d, case["ghost"], case["gra_ghost"], case["quad"], case["p5"])
    if kind == "host":
        out = _exact_solve(d, case["ghost"], 1)
        return {"pot_out": out["pot_out"], "flu": out["flu"]}
    if kind == "plan":
        return [_exact_solve(g, g["ghost"], 1) for g in d]
    if kind == "lin_solve":
        return _exact_solve(d, 1, 1 if case["gravity"] else 0)
    if kind == "net_solve":
        flat = torch.from_numpy(np.fromfile(learned.DEFAULT_WEIGHTS + ".bin", dtype=np.float32)).to(DEV).double()
        with torch.no_grad():
            y, s = _net_forward(d, flat)
        return dict(_exact_solve(d, 1, 0), guess=(y * s)[:, 1:-1, 1:-1, 1:-1])
    if kind == "lin_train":
        return _exact_lin_train(*d, _lin_weights(seed))
    flat = torch.from_numpy(d["weights"]).to(DEV).double().requires_grad_()
    y, s = _net_forward(d, flat)
    diff = y[:, 1:-1, 1:-1, 1:-1] - d["target"].double() / s
    loss = (diff ** 2).mean()
    loss.backward()
    return {"grad": flat.grad, "loss": loss.detach().reshape(1)}

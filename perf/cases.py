"""The calls that users of this framework make, as cases to be timed and compared.

Kinds of case (`kind`), each one pass through public entry points of nbody_b200:

  step      Engine: `steps` captured Hermite steps, then the state read back
            (a run with snapshots).  FP64 or mixed precision.
  dropin    force_calculation: host arrays in, acc and jerk out (the
            reference's force_calculation contract).
  device    Engine.acc_jerk_device inside a user's own torch Hermite step:
            state on the GPU, positions and velocities out.
  ensemble  Ensemble: `steps` steps of many clusters, then the state read back.
  adjoint   hermite_rollout forward and backward: final state and the
            gradients with respect to the initial state and the masses.
  energy    Engine.energy: the kinetic and potential energy of a state.

Bodies are Plummer spheres in Henon units (G = M = 1, E = -1/4), sampled here
with torch; softenings and steps are those of the repository's benchmark, with
steps small enough to resolve the softening.
"""
import math
import os
import sys

import numpy as np
import torch
import torch.utils.checkpoint

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "n-body-code_b200"))

import nbody_b200 as nb  # noqa: E402

DEV = "cuda:0"
STATE_KEYS = ("x", "y", "z", "vx", "vy", "vz")


def listed():
    return [
        # the reference's default run: 1024 bodies, 10 cycles
        dict(name="step_fp64_n1024", kind="step", precision="fp64", n=1024, steps=10, eps=1e-2, dt=1 / 1024),
        # a mid-sized system in full double precision
        dict(name="step_fp64_n16384", kind="step", precision="fp64", n=16384, steps=4, eps=1e-2, dt=1 / 1024),
        # the benchmark's FP64 arm
        dict(name="step_fp64_n65536", kind="step", precision="fp64", n=65536, steps=2, eps=1e-2, dt=1 / 1024),
        # a small ragged system in mixed precision (packed hi/lo kernel)
        dict(name="step_mixed_n5003", kind="step", precision="mixed", n=5003, steps=8, eps=1e-2, dt=1 / 4096),
        # the benchmark's headline system in mixed precision (near/far kernel)
        dict(name="step_mixed_n65536", kind="step", precision="mixed", n=65536, steps=8, eps=1e-2, dt=1 / 4096),
        # the benchmark's large system
        dict(name="step_mixed_n262144", kind="step", precision="mixed", n=262144, steps=2, eps=4e-3, dt=1 / 4096),
        # the reference's back end replaced at its default size: one call per
        # step from host arrays, where latency counts
        dict(name="dropin_fp64_n1024", kind="dropin", precision="fp64", n=1024, eps=1e-2),
        # the same at a ragged larger size
        dict(name="dropin_fp64_n30011", kind="dropin", precision="fp64", n=30011, eps=1e-2),
        # a torch program with its own integrator (ragged size, mixed precision)
        dict(name="device_mixed_n40009", kind="device", precision="mixed", n=40009, eps=1e-2, dt=1 / 1024),
        # the benchmark's ensemble at half its cluster count: uneven clusters,
        # softening 4/N, a step that resolves the smallest softening
        dict(name="ensemble_mixed_c256", kind="ensemble", precision="mixed", clusters=256, nmin=256, nmax=8192,
             steps=8, dt=1 / 8192),
        # the benchmark's gradient size (16 of its steps, one checkpoint segment)
        dict(name="adjoint_fp64_n4096", kind="adjoint", precision="fp64", n=4096, steps=16, checkpoint=16,
             eps=1e-2, dt=1 / 256),
        # the energy diagnostic that brackets every run
        dict(name="energy_n32768", kind="energy", precision="fp64", n=32768, eps=1e-2),
    ]


def _log_int(rng, lo, hi):
    n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    return max(lo, min(hi, n | 1 if rng.random() < 0.7 else n))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "dropin", "device", "ensemble", "adjoint", "energy"])
    eps = rng.choice([4e-3, 1e-2, 2e-2])
    if kind == "step":
        precision = rng.choice(["fp64", "mixed"])
        n = _log_int(rng, 256, 131072 if precision == "fp64" else 262144)
        steps = rng.choice([1, 2, 4, 8])
        while steps > 1 and float(n) * n * steps > (1 if precision == "fp64" else 2) * 262144.0 ** 2:
            steps //= 2
        return dict(kind=kind, precision=precision, n=n, steps=steps, eps=eps, dt=1 / 4096)
    if kind == "dropin":
        return dict(kind=kind, precision="fp64", n=_log_int(rng, 256, 65536), eps=eps)
    if kind == "device":
        return dict(kind=kind, precision=rng.choice(["fp64", "mixed"]), n=_log_int(rng, 256, 100000), eps=eps,
                    dt=1 / 1024)
    if kind == "ensemble":
        return dict(kind=kind, precision=rng.choice(["mixed", "mixed", "fp64"]), clusters=_log_int(rng, 8, 256),
                    nmin=256, nmax=rng.choice([1024, 2048, 4096, 8192]), steps=rng.choice([2, 4, 8]), dt=1 / 8192)
    if kind == "adjoint":
        steps = rng.choice([8, 16, 32])
        return dict(kind=kind, precision="fp64", n=_log_int(rng, 256, 8192), steps=steps,
                    checkpoint=rng.choice([8, 16]), eps=1e-2, dt=1 / 256)
    return dict(kind="energy", precision="fp64", n=_log_int(rng, 1024, 131072), eps=eps)


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _plummer(n, gen):
    """(3, n) positions and velocities and (n,) masses on the GPU, float64."""
    def u(*shape):
        return torch.rand(*shape, generator=gen, device=DEV, dtype=torch.float64)

    def direction():
        z = 2.0 * u(n) - 1.0
        phi = 2.0 * math.pi * u(n)
        s = torch.sqrt(1.0 - z * z)
        return torch.stack([s * torch.cos(phi), s * torch.sin(phi), z])

    mass = 0.98 * u(n) + 1e-4  # enclosed mass fraction; the outermost 2 % are cut
    r = 1.0 / torch.sqrt(mass ** (-2.0 / 3.0) - 1.0)
    # speed: q in [0, 1] with density q^2 (1 - q^2)^(7/2), by its tabulated inverse
    q = torch.linspace(0.0, 1.0, 4097, device=DEV, dtype=torch.float64)
    cdf = torch.cumsum(q * q * (1.0 - q * q) ** 3.5, 0)
    cdf = cdf / cdf[-1]
    t = u(n)
    k = torch.searchsorted(cdf, t).clamp(1, 4096)
    w = (t - cdf[k - 1]) / (cdf[k] - cdf[k - 1]).clamp_min(1e-300)
    speed = (q[k - 1] + w * (q[k] - q[k - 1])) * math.sqrt(2.0) * (1.0 + r * r) ** -0.25
    x = r * direction() * (3.0 * math.pi / 16.0)
    v = speed * direction() * math.sqrt(16.0 / (3.0 * math.pi))
    x = x - x.mean(1, keepdim=True)
    v = v - v.mean(1, keepdim=True)
    return x.contiguous(), v.contiguous(), torch.full((n,), 1.0 / n, device=DEV, dtype=torch.float64)


def _sizes(case):
    """Cluster sizes of an ensemble: log-uniform over [nmin, nmax], in a fixed mixed order."""
    c = case["clusters"]
    ratio = case["nmax"] / case["nmin"]
    s = [int(round(case["nmin"] * ratio ** ((k + 0.5) / c))) for k in range(c)]
    return [s[(k * 97) % c] for k in range(c)] if c % 97 else s


def _generator(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed) * 7919 + 12345)
    return g


def _host(x, v, m):
    a = torch.cat([x, m[None], v]).cpu().numpy()
    return {k: np.ascontiguousarray(a[i]) for i, k in enumerate(("x", "y", "z", "m", "vx", "vy", "vz"))}


def _target(case, gen, x):
    sel = torch.randperm(case["n"], generator=gen, device=DEV)[:min(64, case["n"])]
    return sel, x[:, sel] + 0.1 * torch.randn(3, sel.numel(), generator=gen, device=DEV, dtype=torch.float64)


def prepare(case, seed):
    gen = _generator(seed)
    kind = case["kind"]
    st = dict(case=case)
    if kind == "ensemble":
        sizes = _sizes(case)
        parts = [_plummer(n, gen) for n in sizes]
        cat = _host(*(torch.cat([p[k] for p in parts], dim=-1) for k in range(3)))
        eps2 = (4.0 / np.array(sizes, dtype=np.float64)) ** 2
        st["ens"] = nb.Ensemble(sizes, eps2, case["dt"], precision=case["precision"])
        st["ens"].set_state(cat)
        return st
    x, v, m = _plummer(case["n"], gen)
    eps2 = case["eps"] ** 2
    if kind == "dropin":
        st["bodies"] = _host(x, v, m)
    elif kind == "adjoint":
        st.update(x=x.requires_grad_(), v=v.requires_grad_(), m=m.requires_grad_())
        st["sel"], st["target"] = _target(case, gen, x.detach())
        st["adjoint"] = nb.Adjoint(case["n"], eps2, case["dt"], case["steps"], case["checkpoint"], case["precision"])
    elif kind == "device":
        st["engine"] = nb.Engine(case["n"], eps2=eps2, precision=case["precision"], dt=case["dt"])
        st["stream"] = torch.cuda.Stream()
        f = torch.empty(6, case["n"], device=DEV, dtype=torch.float64)
        torch.cuda.synchronize()
        st["engine"].acc_jerk_device(x[0], x[1], x[2], m, v[0], v[1], v[2], list(f), st["stream"].cuda_stream)
        torch.cuda.synchronize()
        st.update(x=x, v=v, m=m, a=f[:3], j=f[3:])
    else:
        st["engine"] = nb.Engine(case["n"], eps2=eps2, precision=case["precision"], dt=case.get("dt", 1 / 1024))
        st["engine"].set_state(_host(x, v, m))
    return st


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def _predict(x, v, a, j, h):
    xp = torch.add(x, v, alpha=h).add_(a, alpha=h * h / 2).add_(j, alpha=h ** 3 / 6)
    return xp, torch.add(v, a, alpha=h).add_(j, alpha=h * h / 2)


def _correct(xp, vp, a, j, a1, j1, h):
    """The Hermite corrector (snap and crackle expanded)."""
    da = a - a1
    x = torch.add(xp, da, alpha=-0.15 * h * h).add_(j, alpha=-7 * h ** 3 / 60).add_(j1, alpha=-h ** 3 / 30)
    return x, torch.add(vp, da, alpha=-0.5 * h).add_(j, alpha=-5 * h * h / 12).add_(j1, alpha=-h * h / 12)


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "step":
        st["engine"].timestepping(case["steps"])
        return st["engine"].get_state()
    if kind == "dropin":
        return nb.force_calculation(st["bodies"], eps2=case["eps"] ** 2, precision=case["precision"])
    if kind == "device":
        h = case["dt"]
        with torch.cuda.stream(st["stream"]):
            xp, vp = _predict(st["x"], st["v"], st["a"], st["j"], h)
            f = torch.empty(6, case["n"], device=DEV, dtype=torch.float64)
            st["engine"].acc_jerk_device(xp[0], xp[1], xp[2], st["m"], vp[0], vp[1], vp[2], list(f),
                                         st["stream"].cuda_stream)
            st["x"], st["v"] = _correct(xp, vp, st["a"], st["j"], f[:3], f[3:], h)
            st["a"], st["j"] = f[:3], f[3:]
        return [st["x"], st["v"]]
    if kind == "ensemble":
        st["ens"].timestepping(case["steps"])
        return st["ens"].get_state()
    if kind == "adjoint":
        x1, v1 = nb.hermite_rollout(st["x"], st["v"], st["m"], eps2=case["eps"] ** 2, dt=case["dt"],
                                    nsteps=case["steps"], checkpoint_every=case["checkpoint"],
                                    precision=case["precision"], adjoint=st["adjoint"])
        loss = ((x1[:, st["sel"]] - st["target"]) ** 2).sum()
        gx, gv, gm = torch.autograd.grad(loss, (st["x"], st["v"], st["m"]))
        return dict(x=x1.detach(), v=v1.detach(), gx=gx, gv=gv, gm=gm)
    return list(st["engine"].energy())


# ---------------------------------------------------------------------------
# work and exact results
# ---------------------------------------------------------------------------
# Arithmetic of one unordered pair (each FMA two operations): separation 6,
# r^2 6, r.v 5, 1/sqrt 1, s^-3/2 and 1/s 2, masses 2, tidal factor 2, jerk
# vector 6, and 24 for the sums of both bodies' acc and jerk.
PAIR_FLOPS = 54
# the pair's contribution to the gradients with respect to both bodies
PAIR_VJP_FLOPS = 130
# separation 3, r^2 6, 1/sqrt 1, the two bodies' sums 4
PAIR_ENERGY_FLOPS = 14


def work(case):
    kind = case["kind"]
    if kind == "ensemble":
        s = _sizes(case)
        return {"bytes": 8.0 * 13 * sum(s),
                "flops": PAIR_FLOPS * case["steps"] * sum(n * (n - 1) / 2 for n in s)}
    n = case["n"]
    pairs = n * (n - 1) / 2
    if kind == "adjoint":
        return {"bytes": 8.0 * 20 * n,
                "flops": (PAIR_FLOPS + PAIR_VJP_FLOPS) * (case["steps"] + 1) * pairs}
    if kind == "energy":
        return {"bytes": 8.0 * 7 * n, "flops": PAIR_ENERGY_FLOPS * pairs}
    evals = case["steps"] if kind == "step" else 1
    return {"bytes": 8.0 * 13 * n, "flops": PAIR_FLOPS * evals * pairs}


def _acc_jerk(x, v, m, eps2):
    """Direct sums in 64 bits, in row chunks."""
    n = x.shape[1]
    rows = max(1, min(n, (1 << 21) // n))
    acc, jerk = [], []
    for i in range(0, n, rows):
        d = [x[k][None, :] - x[k][i:i + rows, None] for k in range(3)]
        u = [v[k][None, :] - v[k][i:i + rows, None] for k in range(3)]
        s = d[0] * d[0] + d[1] * d[1] + d[2] * d[2] + eps2
        c = (d[0] * u[0] + d[1] * u[1] + d[2] * u[2]) / s * -3.0
        q = m[None, :] / (s * torch.sqrt(s))
        acc.append(torch.stack([(q * d[k]).sum(1) for k in range(3)]))
        jerk.append(torch.stack([(q * (u[k] + c * d[k])).sum(1) for k in range(3)]))
    return torch.cat(acc, 1), torch.cat(jerk, 1)


def _hermite(x, v, m, eps2, h, steps, force=_acc_jerk):
    a, j = force(x, v, m, eps2)
    for _ in range(steps):
        xp = x + h * v + h * h / 2 * a + h ** 3 / 6 * j
        vp = v + h * a + h * h / 2 * j
        a1, j1 = force(xp, vp, m, eps2)
        x = xp - 0.15 * h * h * (a - a1) - h ** 3 * (7 / 60 * j + 1 / 30 * j1)
        v = vp - 0.5 * h * (a - a1) - h * h * (5 / 12 * j + 1 / 12 * j1)
        a, j = a1, j1
    return x, v


def exact(case, seed):
    gen = _generator(seed)
    kind = case["kind"]
    if kind == "ensemble":
        out = []
        parts = [_plummer(n, gen) for n in _sizes(case)]
        for x, v, m in parts:
            out.append(torch.cat(_hermite(x, v, m, (4.0 / m.numel()) ** 2, case["dt"], case["steps"])))
        return dict(zip(STATE_KEYS, torch.cat(out, dim=1).cpu().numpy()))
    x, v, m = _plummer(case["n"], gen)
    eps2 = case["eps"] ** 2
    n = case["n"]
    if kind == "dropin":
        return torch.cat(_acc_jerk(x, v, m, eps2)).cpu().numpy()
    if kind == "energy":
        rows = max(1, min(n, (1 << 22) // n))
        u = torch.zeros((), device=DEV, dtype=torch.float64)
        for i in range(0, n, rows):
            s = sum((x[k][None, :] - x[k][i:i + rows, None]) ** 2 for k in range(3)) + eps2
            phi = (m / torch.sqrt(s)).sum(1) - m[i:i + rows] / math.sqrt(eps2)  # without the self term
            u -= 0.5 * (m[i:i + rows] * phi).sum()
        return [float((0.5 * m * (v * v).sum(0)).sum()), float(u)]
    if kind == "adjoint":
        sel, target = _target(case, gen, x)
        for t in (x, v, m):
            t.requires_grad_()
        if float(n) * n * case["steps"] > 16.0 * 4096 ** 2:
            return None  # the recomputed graph takes too long

        def force(x, v, m, eps2):
            return torch.utils.checkpoint.checkpoint(_acc_jerk_whole, x, v, m, eps2, use_reentrant=False)
        x1, v1 = _hermite(x, v, m, eps2, case["dt"], case["steps"], force)
        gx, gv, gm = torch.autograd.grad(((x1[:, sel] - target) ** 2).sum(), (x, v, m))
        return dict(x=x1.detach(), v=v1.detach(), gx=gx, gv=gv, gm=gm)
    evals = (case["steps"] if kind == "step" else 1) + 1
    if float(n) * n * evals > 9.5 * 65536.0 ** 2:
        return None  # over twenty seconds of direct sums
    x, v = _hermite(x, v, m, eps2, case["dt"], case.get("steps", 1))
    if kind == "device":
        return [x, v]
    return dict(zip(STATE_KEYS, torch.cat([x, v]).cpu().numpy()))


def _acc_jerk_whole(x, v, m, eps2):
    """_acc_jerk in one block (differentiable)."""
    d = [x[k][None, :] - x[k][:, None] for k in range(3)]
    u = [v[k][None, :] - v[k][:, None] for k in range(3)]
    s = d[0] * d[0] + d[1] * d[1] + d[2] * d[2] + eps2
    c = (d[0] * u[0] + d[1] * u[1] + d[2] * u[2]) / s * -3.0
    q = m[None, :] / (s * torch.sqrt(s))
    return (torch.stack([(q * d[k]).sum(1) for k in range(3)]),
            torch.stack([(q * (u[k] + c * d[k])).sum(1) for k in range(3)]))

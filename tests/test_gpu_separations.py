"""Mixed precision where no caller chose the ordered near/far form: bodies in
the caller's order keep the separations of the hi/lo kernels whatever that
order is and whatever bodies lie far out.

Bound per component: a pair's term in float from a separation of two rounded
adds (2 x 2^-24 each of three factors of it), 1/sqrt and 1/s of a few ulp, and
float sums of at most 128 terms: (128 + 32) 2^-24 = 1e-5 of the sum of the
terms' magnitudes."""
import numpy as np
import pytest

import nbody_b200 as nb
import oracle as O

pytestmark = pytest.mark.gpu

EPS2 = {"binaries": 1e-10}  # else 1e-4
BOUND = 160 * 2.0 ** -24


def bodies(n, kind):
    s = nb.plummer(n, seed=11)
    if kind == "two clusters":  # one after the other
        s["x"] = s["x"] + np.where(np.arange(n) < n // 2, 8.0, -8.0)
    elif kind == "radius":
        r = s["x"] ** 2 + s["y"] ** 2 + s["z"] ** 2
        s = {k: np.ascontiguousarray(v[np.argsort(r)]) for k, v in s.items()}
    elif kind == "lattice":
        side = int(np.ceil(n ** (1 / 3)))
        k = np.arange(n)
        s["x"], s["y"], s["z"] = (0.1 * v for v in (k % side, k // side % side, k // side ** 2))
        s = {k: np.ascontiguousarray(v, dtype=np.float64) for k, v in s.items()}
    else:  # one escaper in every 64 bodies
        if kind == "binaries":  # 1e-4 apart, co-moving, and escapers among them
            for k in ("x", "y", "z", "vx", "vy", "vz"):
                s[k][1::2] = s[k][:n // 2 * 2:2]
            s["x"][1::2] += 1e-4
        for k in "xyz":
            s[k][5::64] *= 1e13 if kind == "far escapers" else 1e10
    return s


def softening2(kind):
    return EPS2.get(kind, 1e-4)


def rows_of(n, step, kind):
    """Every step-th body; beyond 1e12 a term is below the smallest float, so
    the far escapers' own sums are not looked at."""
    rows = np.arange(0, n, step)
    return rows[rows % 64 != 5] if kind == "far escapers" else rows


def scale(s, rows, eps2):
    """Sums of the magnitudes of the acc and jerk terms of the given rows."""
    x, v = (np.stack([s[k] for k in q]) for q in (("x", "y", "z"), ("vx", "vy", "vz")))
    acc, jerk = [], []
    for i in rows:
        d, u = x - x[:, i:i + 1], v - v[:, i:i + 1]
        r2 = (d * d).sum(0) + eps2
        q = s["m"] * r2 ** -1.5
        r, w = np.sqrt((d * d).sum(0)), np.sqrt((u * u).sum(0))
        acc.append((q * r).sum())
        jerk.append((q * (w + 3 * r * r * w / r2)).sum())
    return np.array(acc), np.array(jerk)


def check(d, s, rows, eps2):
    ref = O.force_rows(s, eps2, rows)
    sa, sj = scale(s, rows, eps2)
    ea = np.abs(d[:3, rows] - ref[:3]).max(axis=0) / sa
    ej = np.abs(d[3:, rows] - ref[3:]).max(axis=0) / sj
    assert ea.max() <= BOUND and ej.max() <= BOUND, (ea.max(), ej.max())
    return ea, ej


KINDS = ["two clusters", "radius", "lattice", "escapers", "far escapers", "binaries"]


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("n", [1025, 3001, 12000])
def test_engine_below_the_order_limit(n, kind):
    s = bodies(n, kind)
    rows = rows_of(n, max(1, n // 300), kind)
    err = {}
    for variant in (0, 3):
        with nb.Engine(n, eps2=softening2(kind), precision="mixed", dt=1.0, pair_variant=variant) as e:
            e.set_state(s)
            e.force_calculation()
            err[variant] = check(e.get_derivs(), s, rows, softening2(kind))
            if variant == 0:
                assert e.timers()["near_tile_fraction"] == 1.0
    # the same separations, other orders of the float sums
    for a, b in zip(err[0], err[3]):
        assert np.quantile(a, 0.99) <= 2 * np.quantile(b, 0.99)


@pytest.mark.parametrize("kind", KINDS)
def test_calls_on_the_callers_arrays_below_their_order_limit(kind):
    import torch
    n, eps2 = 17000, softening2(kind)
    s = bodies(n, kind)
    rows = rows_of(n, 61, kind)
    check(nb.force_calculation(s, eps2=eps2, precision="mixed"), s, rows, eps2)
    t = [torch.tensor(s[k], device="cuda") for k in nb.FIELDS]
    out = torch.empty(6, n, dtype=torch.float64, device="cuda")
    with nb.Engine(n, eps2=eps2, precision="mixed", dt=1.0) as e:
        e.acc_jerk_device(*t, list(out), stream=torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
    check(out.cpu().numpy(), s, rows, eps2)


@pytest.mark.parametrize("n", [1025, 3001])
def test_steps_from_records_of_the_predictor(n):
    """Ten steps of 1e-9 in one call (records written by the predictor and by
    the joined corrector).  They move a body by 1e-8, and a binary's two by
    1e-12 against each other: the derivatives stay those of the start to 3e-6 of
    the terms, and the pairs of other bodies, at 1e-3 and beyond, add less."""
    kind = "binaries"
    s = bodies(n, kind)
    with nb.Engine(n, eps2=softening2(kind), precision="mixed", dt=1e-9) as e:
        e.set_state(s)
        e.timestepping(10)
        d = e.get_derivs()
    rows = np.arange(0, n, 7)
    ref = O.force_rows(s, softening2(kind), rows)
    sa, _ = scale(s, rows, softening2(kind))
    assert (np.abs(d[:3, rows] - ref[:3]).max(axis=0) / sa).max() <= BOUND + 3e-6


@pytest.mark.parametrize("n", [1000, 5003])
def test_adjoint_forward(n):
    """One step of h = 1e-9 of the mixed forward against the FP64 one: the
    velocity changes by h (a0 + a1) / 2 and terms of higher order, so the
    derivatives' errors show as at most h times the bound on acc and h^2 / 6
    times that on jerk; twice that, and the rounding of v."""
    import torch
    kind, h = "binaries", 1e-9
    s, eps2 = bodies(n, kind), softening2(kind)
    x = torch.tensor(np.stack([s[k] for k in "xyz"]), device="cuda")
    v = torch.tensor(np.stack([s[k] for k in ("vx", "vy", "vz")]), device="cuda")
    m = torch.tensor(s["m"], device="cuda")
    out = {}
    for precision in ("fp64", "mixed"):
        adj = nb.Adjoint(n, eps2, h, 1, 1, precision)
        x1, v1 = torch.empty_like(x), torch.empty_like(v)
        adj.forward(x, v, m, x1, v1, torch.cuda.current_stream().cuda_stream)
        out[precision] = v1.cpu().numpy()
        adj.close()
    rows = np.arange(0, n, 7)
    sa, sj = scale(s, rows, eps2)
    err = np.abs(out["mixed"] - out["fp64"])[:, rows].max(axis=0)
    assert (err <= 2 * BOUND * (h * sa + h * h / 6 * sj) + 2e-15).all(), (err / (h * sa)).max()

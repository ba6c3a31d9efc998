"""The symmetric kernels on whole systems with one body that outweighs all
others: a pair with it that is left out, met twice or given to another row is
most of that row's sum, in mixed precision too."""
import numpy as np
import pytest

import nbody_b200 as nb
import oracle as O
from _util import derivs_rel, vec_rel

pytestmark = pytest.mark.gpu

EPS2 = 1e-4
# float pair terms and sums of at most 128 of them: (128 + 32) 2^-24 of the sum of
# the terms' magnitudes; FP64: sums of n <= 2^17 terms of relative error ~2^-52
BOUND = {"mixed": 160 * 2.0 ** -24, "fp64": 1e-12}


def system(n):
    """Bodies spread through a unit cube, so that no pair's term is small."""
    rng = np.random.default_rng(n)
    s = {k: rng.uniform(-0.5, 0.5, n) for k in ("x", "y", "z", "vx", "vy", "vz")}
    s["m"] = np.full(n, 1.0 / n)
    return s


def exact(s):
    """(acc and jerk, magnitudes of their terms) of all rows, torch FP64."""
    import torch
    t = {k: torch.tensor(v, device="cuda") for k, v in s.items()}
    x, v = (torch.stack([t[k] for k in q]) for q in (("x", "y", "z"), ("vx", "vy", "vz")))
    n = x.shape[1]
    d, size = torch.empty(6, n, dtype=torch.float64, device="cuda"), torch.empty(2, n, dtype=torch.float64, device="cuda")
    for i in range(0, n, 512):
        w = slice(i, min(n, i + 512))
        terms = pair_terms(x, v, t["m"], w)
        d[:, w], size[:, w] = terms[0].sum(-1), terms[1].sum(-1)
    return d.cpu().numpy(), size.cpu().numpy()


def pair_terms(x, v, m, rows):
    import torch
    r, u = x[:, None, :] - x[:, rows, None], v[:, None, :] - v[:, rows, None]
    r2 = (r * r).sum(0)
    s = r2 + EPS2
    q = m / (s * torch.sqrt(s))
    c = -3.0 * (r * u).sum(0) / s
    un = torch.sqrt((u * u).sum(0))
    return torch.cat([q * r, q * (u + c * r)]), torch.stack([q * torch.sqrt(r2), q * un * (1 + 3 * r2 / s)])


def heavy_term(s, h):
    """The terms of body h at unit mass in all rows, and their magnitudes."""
    x, v = (np.stack([s[k] for k in q]) for q in (("x", "y", "z"), ("vx", "vy", "vz")))
    r, u = x[:, h:h + 1] - x, v[:, h:h + 1] - v
    r2 = (r * r).sum(0)
    w = r2 + EPS2
    q = w ** -1.5
    un = np.sqrt((u * u).sum(0))
    return (np.concatenate([q * r, q * (u - 3 * (r * u).sum(0) / w * r)]),
            np.stack([q * np.sqrt(r2), q * un * (1 + 3 * r2 / w)]))


# blocks of 256 and 512 rows, short last ones; from 65537 two sub-blocks each
@pytest.mark.parametrize("precision,n", [("fp64", 5003), ("fp64", 16897), ("fp64", 70017),
                                         ("mixed", 5003), ("mixed", 20000), ("mixed", 65537), ("mixed", 70017)])
def test_every_row_feels_one_heavy_body(precision, n):
    s = system(n)
    base, size = exact(s)
    for h in (0, 31, 511, 512, n // 2, n - 33, n - 1):
        m = s["m"].copy()
        m[h] = 1.0
        with nb.Engine(n, eps2=EPS2, precision=precision, dt=1.0) as e:
            e.set_state({**s, "m": m})
            e.force_calculation()
            d = e.get_derivs()
        term, mag = heavy_term(s, h)
        want = base + (1.0 - 1.0 / n) * term
        limit = BOUND[precision] * (size + (1.0 - 1.0 / n) * mag)
        for k in range(2):
            err = np.abs(d[3 * k:3 * k + 3] - want[3 * k:3 * k + 3]).max(axis=0)
            assert (err <= limit[k]).all(), (h, k, int(np.argmax(err / limit[k])), (err / limit[k]).max())


@pytest.mark.parametrize("n", [65537, 70001])
def test_energy_of_blocks_with_two_sub_blocks(n):
    """Both potentials against all pairs in torch FP64: sums of positive terms of
    relative error a few 2^-52, 1e-12."""
    import torch
    s = system(n)
    s["m"] *= np.random.default_rng(1).uniform(0.0, 2.0, n)
    with nb.Engine(n, eps2=EPS2, dt=1.0) as e:
        e.set_state(s)
        _, U = e.energy()
        _, Uc = e.energy(ref_compat=True)
    x = torch.tensor(np.stack([s[k] for k in "xyz"]), device="cuda")
    m = torch.tensor(s["m"], device="cuda")
    j = torch.arange(n, device="cuda")
    want, compat = 0.0, 0.0
    for i in range(0, n, 1024):
        r = x[:, None, :] - x[:, i:i + 1024, None]
        y = torch.rsqrt((r * r).sum(0) + EPS2) * (j[None, :] > j[i:i + 1024, None])
        want -= float((y * m[None, :] * m[i:i + 1024, None]).sum())
        compat -= float((y * (m * m)[None, :]).sum())
    assert abs(U - want) <= 1e-12 * abs(want), (U, want)
    assert abs(Uc - compat) <= 1e-12 * abs(compat), (Uc, compat)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_systems_of_fewer_than_128_slots(precision):
    """From 1.4e6 bodies memory bounds the blocks: several sub-blocks of each."""
    n = 1500001
    s = nb.plummer(n, seed=4)
    rows = np.unique(np.concatenate([np.arange(0, n, 60013), [1, 511, 512, n - 2, n - 1]]))
    with nb.Engine(n, eps2=EPS2, precision=precision, dt=1.0) as e:
        e.set_state(s)
        e.force_calculation()
        d = e.get_derivs()[:, rows]
    ref = O.force_rows(s, EPS2, rows)
    if precision == "fp64":
        ea, ej = derivs_rel(d, ref)
        assert ea <= 1e-12 and ej <= 1e-11, (ea, ej)
    else:
        ea = vec_rel(d[:3], ref[:3])
        assert np.median(ea) <= 2e-6 and ea.max() <= 2e-4, (np.median(ea), ea.max())


@pytest.mark.parametrize("precision,kw", [("fp64", {}), ("mixed", {}), ("mixed", dict(pair_variant=4, sort_every=3))])
def test_adaptive_steps_of_one_call_equal_single_steps(precision, kw):
    """The eight-step graphs of an engine whose every step sets the next one's
    length."""
    s = nb.plummer(1300, seed=6)
    with nb.Engine(1300, eps2=EPS2, precision=precision, **kw) as a, \
            nb.Engine(1300, eps2=EPS2, precision=precision, **kw) as b:
        for e in (a, b):
            e.set_state(s)
            e.force_calculation()
        for k in (1, 9, 25):
            a.timestepping(k)
            for _ in range(k):
                b.timestepping(1)
        sa, sb, ta, tb = a.get_state(), b.get_state(), a.timers(), b.timers()
    assert all(np.array_equal(sa[k], sb[k]) for k in sa)
    assert ta["steps"] == tb["steps"] == 35 and ta["reorders"] == tb["reorders"]
    assert ta["t"] == tb["t"] and ta["dt"] == tb["dt"] and ta["dt"] > 0

"""The symmetric pair kernels (each unordered pair evaluated once) at the edges
of their tiles, blocks and schedules, against the oracle's direct sums.

Masses are unequal and some are zero, so a pair that is missed, met twice or
given the wrong body's mass shows at once.  FP64 bound 1e-12: the parity bound
of the FP64 engine (sums of n terms of relative error ~2^-52, n <= 2^17)."""
import numpy as np
import pytest

import nbody_b200 as nb
import oracle as O
from _util import derivs_rel, vec_rel

pytestmark = pytest.mark.gpu

EPS2 = 1e-4


def bodies(n, seed=3):
    s = nb.plummer(max(n, 2), seed=seed)
    s = {k: v[:n].copy() for k, v in s.items()}
    s["m"] = s["m"] * np.random.default_rng(seed).uniform(0.0, 2.0, n)
    s["m"][::7] = 0.0
    return s


def derivs(s, precision, **kw):
    with nb.Engine(s["x"].size, eps2=EPS2, precision=precision, dt=1.0, **kw) as e:
        e.set_state(s)
        e.force_calculation()
        return e.get_derivs(), e.timers()


# one block; tiles of 32; blocks of 256 rows, odd and even counts, short last
# blocks
@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 256, 257, 511, 513, 768, 769, 1025, 2047, 4097])
def test_fp64_small_edges(n):
    s = bodies(n)
    d, _ = derivs(s, "fp64")
    if n == 1:
        assert np.all(d == 0.0)
        return
    ref = O.force(s, EPS2)
    ok = np.abs(ref[:3]).max(axis=0) > 0  # a body whose partners are all massless feels nothing
    assert np.all(d[:, ~ok] == 0.0)
    ea, ej = derivs_rel(d[:, ok], ref[:, ok])
    assert ea <= 1e-12 and ej <= 1e-12, (n, ea, ej)


# the last n of one block size and the first of the next; blocks of two
# sub-blocks (from 65537), odd and even block counts
# (the four-row kernel serves 8192 and up, smaller ones where it fills the GPU better)
@pytest.mark.parametrize("n", [3001, 5003, 8192, 8193, 16383, 16384, 16897, 65536, 65537, 70001])
def test_fp64_block_edges_sampled_rows(n):
    s = bodies(n)
    d, t = derivs(s, "fp64")
    if n in (8192, 65536):  # the choice by predicted time reaches both kernels
        assert t["i_per_thread"] == 4
    if n == 3001:
        assert t["i_per_thread"] == 2
    rows = np.unique(np.concatenate([np.arange(0, n, n // 60), [n - 1, n - 2, n // 2, n // 2 - 1]]))
    ref = O.force_rows(s, EPS2, rows)
    ea, ej = derivs_rel(d[:, rows], ref)
    assert ea <= 1e-12 and ej <= 1e-12, (n, ea, ej)
    # the same sums from the one-sided kernel, every row
    one, _ = derivs(s, "fp64", threads=128, i_per_thread=2, j_tile=128)
    assert vec_rel(d[:3], one[:3]).max() <= 1e-12 and vec_rel(d[3:], one[3:]).max() <= 1e-11


def test_fewer_bodies_than_the_engine_and_row_ranges():
    """A device-array call on fewer bodies than the engine holds between its
    own steps, and a drop-in row range after the autotuner cached a symmetric
    tiling for another size with the same padding and row count."""
    import torch
    n, m = 3000, 2500
    s = bodies(n)
    sub = {k: v[:m] for k, v in s.items()}
    t = [torch.tensor(sub[k], dtype=torch.float64, device="cuda") for k in nb.FIELDS]
    out = torch.empty(6, m, dtype=torch.float64, device="cuda")
    with nb.Engine(n, eps2=EPS2, dt=1 / 1024) as e, nb.Engine(n, eps2=EPS2, dt=1 / 1024) as f:
        for g in (e, f):
            g.set_state(s)
            g.timestepping(2)
        e.acc_jerk_device(*t, list(out), stream=torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
        for g in (e, f):
            g.timestepping(2)
        a, b = e.get_state(), f.get_state()
    assert all(np.array_equal(a[k], b[k]) for k in a)
    ea, ej = derivs_rel(out.cpu().numpy(), O.force(sub, EPS2))
    assert ea <= 1e-12 and ej <= 1e-12, (ea, ej)
    big = bodies(5100)
    nb.release_force_cache()
    try:
        nb.force_calculation_tune({k: v[:5000] for k, v in big.items()}, eps2=EPS2)
        part = nb.force_calculation(big, eps2=EPS2, i_begin=0, i_end=5000)
    finally:
        nb.release_force_cache()
    assert np.all(part[:, 5000:] == 0.0)
    ea, ej = derivs_rel(part[:, :5000], O.force_rows(big, EPS2, np.arange(5000)))
    assert ea <= 1e-12 and ej <= 1e-12, (ea, ej)


# subtiles of 64, tiles of 64 (two rows per lane) and 128 bodies (four rows),
# a last tile whose second subtile is empty, odd and even block counts; bodies
# in the caller's order (automatic, below 16384) and in Hilbert order
# (pair_variant 4, or from 16384).  Bounds: those of the mixed kernels against
# FP64 (median 2e-6, worst 2e-4 acc; median 1e-5 jerk).
@pytest.mark.parametrize("variant", [0, 4])
@pytest.mark.parametrize("n", [1, 2, 63, 64, 65, 255, 257, 513, 1025, 4097, 5003])
def test_mixed_small_edges(n, variant):
    s = bodies(n)
    d, _ = derivs(s, "mixed", pair_variant=variant)
    if n == 1:
        assert np.all(d == 0.0)
        return
    ref = O.force(s, EPS2)
    ok = np.abs(ref[:3]).max(axis=0) > 0
    assert np.all(d[:, ~ok] == 0.0)
    ea, ej = vec_rel(d[:3, ok], ref[:3, ok]), vec_rel(d[3:, ok], ref[3:, ok])
    assert np.median(ea) <= 2e-6 and ea.max() <= 2e-4, (n, np.median(ea), ea.max())
    assert np.median(ej) <= 1e-5, (n, np.median(ej))


@pytest.mark.parametrize("n", [16384, 20000, 65537, 70017])
def test_mixed_block_edges_against_the_one_sided_kernel(n):
    """Every row against the packed hi/lo kernel of the same float arithmetic
    class: a pair missed or met twice would be off by its whole term.  Bounds:
    the mixed kernels' against FP64, twice."""
    s = bodies(n)
    d, t = derivs(s, "mixed")
    assert t["record_format"] == 3
    one, _ = derivs(s, "mixed", pair_variant=3)
    ea, ej = vec_rel(d[:3], one[:3]), vec_rel(d[3:], one[3:])
    assert np.median(ea) <= 4e-6 and ea.max() <= 4e-4, (n, np.median(ea), ea.max())
    assert np.median(ej) <= 2e-5, (n, np.median(ej))
    again, _ = derivs(s, "mixed")
    assert np.array_equal(d, again)


@pytest.mark.parametrize("n", [3001, 33000])
def test_mixed_calls_on_the_callers_arrays(n):
    """Host and device calls in the caller's order (below 32768 bodies) and
    through the Hilbert order (from there) give the engine's accuracy, and
    leave a stepping engine's own bodies alone."""
    import torch
    s = bodies(n)
    rows = np.arange(0, n, max(1, n // 200))
    ref = O.force_rows(s, EPS2, rows)
    ok = np.abs(ref[:3]).max(axis=0) > 0
    t = [torch.tensor(s[k], dtype=torch.float64, device="cuda") for k in nb.FIELDS]
    out = torch.empty(6, n, dtype=torch.float64, device="cuda")
    with nb.Engine(n, eps2=EPS2, dt=1 / 1024, precision="mixed") as e, \
            nb.Engine(n, eps2=EPS2, dt=1 / 1024, precision="mixed") as f:
        for g in (e, f):
            g.set_state(s)
            g.timestepping(2)
        e.acc_jerk_device(*t, list(out), stream=torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
        for g in (e, f):
            g.timestepping(2)
        a, b = e.get_state(), f.get_state()
    assert all(np.array_equal(a[k], b[k]) for k in a)
    for d in (out.cpu().numpy(), nb.force_calculation(s, eps2=EPS2, precision="mixed")):
        ea = vec_rel(d[:3, rows][:, ok], ref[:3, ok])
        assert np.median(ea) <= 2e-6 and ea.max() <= 2e-4, (n, np.median(ea), ea.max())


def _vjp_rows(s, ab, jb, rows):
    """d/d(x_k, v_k, m_k) of sum_i ab_i . acc_i + jb_i . jerk_i for the given
    rows k, by autograd of the terms that contain body k (plain torch, FP64)."""
    import torch
    dev = "cuda"
    X = torch.tensor(np.stack([s["x"], s["y"], s["z"]]), device=dev)
    V = torch.tensor(np.stack([s["vx"], s["vy"], s["vz"]]), device=dev)
    M = torch.tensor(s["m"], device=dev)
    A, J = torch.tensor(ab, device=dev), torch.tensor(jb, device=dev)
    k = torch.tensor(rows, device=dev)
    x, v, m = (t[..., k].clone().requires_grad_() for t in (X, V, M))
    d = X[:, None, :] - x[:, :, None]
    u = V[:, None, :] - v[:, :, None]
    s2 = (d * d).sum(0) + EPS2
    q = s2 ** -1.5
    q = torch.where(torch.arange(M.numel(), device=dev)[None, :] == k[:, None], torch.zeros_like(q), q)
    c = -3.0 * (d * u).sum(0) / s2
    own = ((A[:, k, None] * d).sum(0) + (J[:, k, None] * (u + c * d)).sum(0)) * q * M[None, :]
    partner = -((A[:, None, :] * d).sum(0) + (J[:, None, :] * (u + c * d)).sum(0)) * q * m[:, None]
    gx, gv, gm = torch.autograd.grad((own + partner).sum(), (x, v, m))
    return gx.cpu().numpy(), gv.cpu().numpy(), gm.cpu().numpy()


# blocks of 256 rows, odd and even counts, tiles of 32; blocks of two
# sub-blocks from 32769.  Sums of n terms of relative error a few 2^-52: 1e-11
# of each kind's largest value.
@pytest.mark.parametrize("n", [1, 2, 31, 33, 255, 257, 513, 1000, 4097, 33001])
def test_pair_vjp_edges(n):
    import torch
    s = bodies(n)
    rng = np.random.default_rng(n)
    ab, jb = rng.normal(size=(3, n)), rng.normal(size=(3, n))
    t = {k: torch.tensor(v, device="cuda") for k, v in
         dict(x=np.stack([s["x"], s["y"], s["z"]]), v=np.stack([s["vx"], s["vy"], s["vz"]]),
              m=s["m"], a=ab, j=jb).items()}
    gx, gv = torch.empty(3, n, dtype=torch.float64, device="cuda"), torch.empty(3, n, dtype=torch.float64, device="cuda")
    gm = torch.empty(n, dtype=torch.float64, device="cuda")
    adj = nb.Adjoint(n, EPS2, 1 / 256, 1, 1)
    adj.vjp_acc_jerk(t["x"], t["v"], t["m"], t["a"], t["j"], gx, gv, gm,
                     torch.cuda.current_stream().cuda_stream)
    rows = np.arange(n) if n <= 1000 else np.unique(np.concatenate([np.arange(0, n, n // 100), [n - 2, n - 1]]))
    for got, want in zip((gx, gv, gm), _vjp_rows(s, ab, jb, rows)):
        got = got.cpu().numpy()
        err = np.abs(got[..., rows] - want).max()
        assert err <= 1e-11 * max(np.abs(want).max(), np.abs(got).max()) + (0.0 if n > 1 else 1e-300), (n, err)
    adj.close()


@pytest.mark.parametrize("precision,kw", [("fp64", {}), ("mixed", {}), ("mixed", dict(pair_variant=4, sort_every=3)),
                                          ("mixed", dict(pair_variant=4, sort_every=10))])
def test_steps_of_one_call_equal_single_steps(precision, kw):
    """A call's steps run from graphs of one and of eight steps, re-ordered
    when due; the result, the step count and the number of re-orderings are
    those of one call per step."""
    s = bodies(1300)
    args = dict(eps2=EPS2, dt=1 / 1024, precision=precision, **kw)
    with nb.Engine(1300, **args) as a, nb.Engine(1300, **args) as b:
        for e in (a, b):
            e.set_state(s)
            e.force_calculation()
        for k in (1, 2, 9, 10, 25):
            a.timestepping(k)
            for _ in range(k):
                b.timestepping(1)
        sa, sb, ta, tb = a.get_state(), b.get_state(), a.timers(), b.timers()
    assert all(np.array_equal(sa[k], sb[k]) for k in sa)
    assert ta["steps"] == tb["steps"] == 47 and ta["t"] == tb["t"] and ta["reorders"] == tb["reorders"]
    assert ta["pred_ms"] > 0 and ta["eval_ms"] > 0 and ta["corr_ms"] > 0


# blocks of 256 rows with tiles of 64, of 512 rows with tiles of 128 (from
# 16384), odd and even counts.  A sum of positive terms of relative error a few
# 2^-52: 1e-12.
@pytest.mark.parametrize("n", [1, 2, 63, 64, 65, 255, 257, 513, 1024, 4097, 16383, 16384, 20001])
def test_energy_edges(n):
    s = bodies(n)
    with nb.Engine(n, eps2=EPS2, dt=1.0) as e:
        e.set_state(s)
        T, U = e.energy()
        _, Uc = e.energy(ref_compat=True)
    kin = 0.5 * (s["m"] * (s["vx"] ** 2 + s["vy"] ** 2 + s["vz"] ** 2)).sum()
    assert abs(T - kin) <= 1e-12 * kin
    for got, compat in ((U, False), (Uc, True)):
        want = O.potential(s, EPS2, compat=compat) if n > 1 else 0.0
        assert abs(got - want) <= 1e-12 * abs(want), (n, compat, got, want)


# clusters around the edges of tiles (32, 64) and blocks (256), odd and even
# block counts, one of more than 128 blocks (two 256-row sub-blocks per block);
# items of one tile and of more than a run.  Bounds of the FP64 and mixed
# kernels against the oracle.
@pytest.mark.parametrize("precision,variant", [("fp64", 0), ("mixed", 0), ("mixed", 4)])
@pytest.mark.parametrize("tpi", [0, 1, 1000])
def test_ensemble_edges(precision, variant, tpi):
    sizes = [1, 31, 33, 64, 255, 256, 257, 513, 1000, 1281, 2] + ([33000] if tpi != 1 else [])
    parts = [bodies(n, seed=5 + c) for c, n in enumerate(sizes)]
    cat = {k: np.concatenate([p[k] for p in parts]) for k in nb.FIELDS}
    with nb.Ensemble(sizes, EPS2, 1 / 512, precision=precision, pair_variant=variant, tiles_per_item=tpi) as e:
        e.set_state(cat)
        e.force_calculation()
        d, off = e.get_derivs(), e.offsets
        st = e.get_state()
    for k in st:
        assert np.array_equal(st[k], cat[k]), k
    for c, n in enumerate(sizes):
        if n == 1:
            assert np.all(d[:, off[c]] == 0.0)
            continue
        rows = np.arange(n) if n <= 2000 else np.arange(0, n, 331)
        ref = O.force_rows(parts[c], EPS2, rows)
        ok = np.abs(ref[:3]).max(axis=0) > 0
        got = d[:, off[c]:off[c + 1]][:, rows]
        assert np.all(got[:, ~ok] == 0.0)
        ea, ej = vec_rel(got[:3, ok], ref[:3, ok]), vec_rel(got[3:, ok], ref[3:, ok])
        if precision == "fp64":
            assert ea.max() <= 1e-12 and ej.max() <= 1e-12, (c, n, ea.max(), ej.max())
        else:
            assert np.median(ea) <= 2e-6 and ea.max() <= 2e-4 and np.median(ej) <= 1e-5, (c, n)


# steps of one call share a kernel between the corrector and the next step's
# predictor; steps of their own calls do not: the same arithmetic, bit for bit
# (short last subtile and CTA, one body more than a CTA's rows, no full subtile)
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("n", [33, 300, 1025, 4095, 16385])
def test_chained_steps_equal_single_steps(n, precision):
    s = bodies(n)
    out = []
    for calls in ([11], [1] * 11):
        with nb.Engine(n, eps2=EPS2, precision=precision, dt=1 / 1024) as e:
            e.set_state(s)
            e.force_calculation()
            for k in calls:
                e.timestepping(k)
            out.append((e.get_state(), e.get_derivs()))
    (a, da), (b, db) = out
    for k in a:
        assert np.array_equal(a[k], b[k]), k
    assert np.array_equal(da, db)

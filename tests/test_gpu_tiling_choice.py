"""Which kernel, order and work list a call gets."""
import numpy as np
import pytest

import nbody_b200 as nb
import oracle as O
from _util import vec_rel

pytestmark = pytest.mark.gpu

EPS2 = 1e-4


def device_arrays(s):
    import torch
    n = s["x"].size
    return [torch.tensor(s[k], device="cuda") for k in nb.FIELDS], \
        torch.empty(6, n, dtype=torch.float64, device="cuda")


def stream():
    import torch
    return torch.cuda.current_stream().cuda_stream


def test_one_sided_near_far_calls_get_their_bodies_in_order():
    """An explicit shape of the near/far kernel between 16384 and 32768 bodies:
    device-array calls order the caller's bodies (in no order, every tile of
    128 of them is near)."""
    import torch
    n = 20000
    s = nb.plummer(n, seed=5)
    t, out = device_arrays(s)
    with nb.Engine(n, eps2=EPS2, precision="mixed", dt=1.0, threads=128, i_per_thread=4, j_tile=128) as e:
        e.set_state(s)
        e.force_calculation()
        own = e.timers()["near_tile_fraction"]
        e.acc_jerk_device(*t, list(out), stream=stream())
        torch.cuda.synchronize()
        called = e.timers()["near_tile_fraction"]
    assert own < 0.9 and called < 0.9, (own, called)
    rows = np.arange(0, n, 97)
    ref = O.force_rows(s, EPS2, rows)
    ea = vec_rel(out.cpu().numpy()[:3, rows], ref[:3])
    assert np.median(ea) <= 2e-6 and ea.max() <= 2e-4


def test_tuned_tilings_of_ordered_and_unordered_passes_are_apart():
    """Between 16384 and 32768 bodies an engine's passes run on bodies in
    Hilbert order and a drop-in call's do not: neither takes the tiling that
    was timed for the other."""
    n = 20011
    s = nb.plummer(n, seed=5)
    nb.release_force_cache()
    try:
        nb.force_calculation_tune(s, eps2=EPS2, precision="mixed")
        source = []
        for _ in range(2):
            with nb.Engine(n, eps2=EPS2, precision="mixed", dt=1.0, tune=True) as e:
                e.set_state(s)
                e.force_calculation()
                source.append(e.timers()["tiling_source"])
    finally:
        nb.release_force_cache()
    assert source == [2, 3]  # timed for this engine, then taken from the cache


def test_device_calls_of_alternating_sizes():
    """The kept tiling of a device-array call is that of its size."""
    import torch
    s = nb.plummer(3000, seed=5)
    t, out = device_arrays(s)
    with nb.Engine(3000, eps2=EPS2, dt=1.0) as e:
        for n in (3000, 100, 2500, 2500, 3000):
            sub = [a[:n] for a in t]
            got = torch.empty(6, n, dtype=torch.float64, device="cuda")
            e.acc_jerk_device(*sub, list(got), stream=stream())
            with nb.Engine(3000, eps2=EPS2, dt=1.0) as f:
                want = torch.empty_like(got)
                f.acc_jerk_device(*sub, list(want), stream=stream())
                torch.cuda.synchronize()
            assert torch.equal(got, want), n


@pytest.mark.parametrize("tpi", [1, 8, 100])
def test_fp64_ensemble_items_are_given_in_tiles_of_128_bodies(tpi):
    """tiles_per_item = 8: 1024 bodies per item, as the packed hi/lo ensembles'."""
    sizes = [5000, 700, 100]
    s = [nb.plummer(n, seed=n) for n in sizes]
    with nb.Ensemble(sizes, EPS2, 1 / 512, precision="fp64", tiles_per_item=tpi) as e:
        e.set_state({k: np.concatenate([p[k] for p in s]) for k in nb.FIELDS})
        e.force_calculation()
        info, d, off = e.info(), e.get_derivs(), e.offsets
    assert info["tiles_per_item"] == tpi and info["j_tile"] == 128
    items = 0
    for n in sizes:
        blocks, tiles = -(-n // 256), -(-n // 32)  # tiles of the kernel
        first = min((blocks // 2 + 1) * 8, tiles)  # the first block's run
        items += blocks * -(-first // (4 * tpi))
    assert info["items"] == items
    for c, p in enumerate(s):
        rows = np.arange(0, sizes[c], 7)
        got, ref = d[:, off[c]:off[c + 1]][:, rows], O.force_rows(p, EPS2, rows)
        assert vec_rel(got[:3], ref[:3]).max() <= 1e-12


@pytest.mark.parametrize("precision,variant", [("fp64", 0), ("mixed", 0), ("mixed", 4)])
def test_ensemble_tuning_tries_the_default_item_size(precision, variant, capfd, monkeypatch):
    """A small ensemble's default items are shorter than 256 bodies."""
    rng = np.random.default_rng(1)
    sizes = rng.integers(256, 2048, 16)
    parts = [nb.plummer(int(n), seed=int(n)) for n in sizes]
    state = {k: np.concatenate([p[k] for p in parts]) for k in nb.FIELDS}
    kw = dict(precision=precision, pair_variant=variant)
    with nb.Ensemble(sizes, EPS2, 1 / 512, **kw) as e:
        default = e.info()
    bodies = default["tiles_per_item"] * default["j_tile"]
    assert bodies <= 128
    monkeypatch.setenv("NBODY_TUNE_VERBOSE", "1")
    with nb.Ensemble(sizes, EPS2, 1 / 512, tune=True, **kw) as e:
        e.set_state(state)
        e.force_calculation()
    tried = []
    for line in capfd.readouterr().err.splitlines():
        if "[nbody ens tune]" in line:
            f = dict(w.split("=") for w in line.split() if "=" in w)
            tried.append(int(f["tile"]) * int(f["tiles_per_item"]))
    assert tried and any(t <= bodies for t in tried), (bodies, sorted(set(tried)))

"""Partial-sum slots on a device with little memory left."""
import numpy as np
import pytest

import nbody_b200 as nb
import oracle as O
from _util import derivs_rel, vec_rel

pytestmark = pytest.mark.gpu

EPS2 = 1e-4


@pytest.fixture
def crowded():
    """Leaves `keep` bytes of device memory free."""
    import torch
    held = []

    def hold(keep):
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        free, _ = torch.cuda.mem_get_info()
        assert free > keep
        held.append(torch.empty(int(free - keep), dtype=torch.uint8, device="cuda"))
    yield hold
    held.clear()
    torch.cuda.empty_cache()


def test_the_largest_engine_is_created():
    """2^28 bodies, the largest n: 62 GB of state and records; the slots of a
    symmetric pass (up to 412 GB) wait for a pass."""
    with nb.Engine(1 << 28, eps2=EPS2, dt=1.0) as e:
        assert e.timers()["tiling_source"] == 0


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_passes_without_room_for_the_symmetric_slots(precision, crowded):
    """600001 bodies want 2.5 GB and more of slots: with 1.2 GB left the pass is
    one-sided; device-array calls likewise."""
    import torch
    n = 600001
    s = nb.plummer(n, seed=2)
    rows = np.arange(0, n, 9973)
    ref = O.force_rows(s, EPS2, rows)
    t = [torch.tensor(s[k], device="cuda") for k in nb.FIELDS]
    out = torch.empty(6, n, dtype=torch.float64, device="cuda")
    crowded(1.2e9)
    got = []
    with nb.Engine(n, eps2=EPS2, precision=precision, dt=1.0) as e:
        e.set_state(s)
        e.force_calculation()
        got.append(e.get_derivs()[:, rows])
        assert e.timers()["split_j"] * 48 * n < 1.2e9
    with nb.Engine(n, eps2=EPS2, precision=precision, dt=1.0) as e:
        e.acc_jerk_device(*t, list(out), stream=torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
        got.append(out.cpu().numpy()[:, rows])
    for d in got:
        if precision == "fp64":
            ea, ej = derivs_rel(d, ref)
            assert ea <= 1e-12 and ej <= 1e-12, (ea, ej)
        else:
            ea = vec_rel(d[:3], ref[:3])
            assert np.median(ea) <= 2e-6 and ea.max() <= 2e-4, (np.median(ea), ea.max())


def test_adjoint_without_room_for_all_slots(crowded):
    """200003 bodies want 1.3 GB of slots; with less left the schedules get fewer
    blocks and splits.  Same sums in another order: 1e-11 of each kind's
    largest value."""
    import torch
    n = 200003
    s = nb.plummer(n, seed=2)
    rng = np.random.default_rng(3)
    x, v, a, j = (torch.tensor(w, device="cuda") for w in
                  (np.stack([s[k] for k in "xyz"]), np.stack([s[k] for k in ("vx", "vy", "vz")]),
                   rng.normal(size=(3, n)), rng.normal(size=(3, n))))
    m = torch.tensor(s["m"], device="cuda")
    out = []
    for crowd in (False, True):
        g = [torch.empty_like(x), torch.empty_like(x), torch.empty_like(m), torch.empty_like(x), torch.empty_like(x)]
        if crowd:
            crowded(0.7e9)
        adj = nb.Adjoint(n, EPS2, 1 / 256, 1, 1)
        adj.vjp_acc_jerk(x, v, m, a, j, g[0], g[1], g[2], torch.cuda.current_stream().cuda_stream)
        adj.forward(x, v, m, g[3], g[4], torch.cuda.current_stream().cuda_stream)
        adj.close()
        out.append([w.cpu().numpy() for w in g])
    for p, q in zip(*out):
        assert np.abs(p - q).max() <= 1e-11 * np.abs(p).max()


def test_a_create_without_memory_leaves_nothing_behind(crowded):
    """Each kind of object that finds no memory says so; the calls after it work."""
    s = nb.plummer(1000, seed=1)
    ref = O.force(s, EPS2)
    crowded(2e9)
    for refused in (lambda: nb.Engine(1 << 28, eps2=EPS2, dt=1.0),
                    lambda: nb.Ensemble([1 << 20] * 40, EPS2, 1 / 512),
                    lambda: nb.Adjoint(1 << 22, EPS2, 1 / 256, 160, 16)):
        with pytest.raises(nb.NBodyError) as err:
            refused()
        assert "OOM" in str(err.value)
        with nb.Engine(1000, eps2=EPS2, dt=1.0) as e:
            e.set_state(s)
            e.force_calculation()
            ea, ej = derivs_rel(e.get_derivs(), ref)
        assert ea <= 1e-12 and ej <= 1e-12

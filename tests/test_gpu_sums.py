"""The particle kernels' sums and grouping at the sizes where they can go
wrong: particle counts around warps, chunks and windows, all in one cell, in
two, or anywhere; grids that are no multiple of a tile.

  * the deposits of the fused FP64 push and of the mixed tiles (particles at
    rest in no field stay where they are) against the one-particle-at-a-time
    deposits of the loaders: the FP64 weights summed in another order, 1e-13
    of the largest node; the mixed ones are the same integers, scaled once
    per window instead of once per particle, 1e-13 as well;
  * the mixed sort: tile order, offsets, and the same particles per cell;
  * the losses of one push, counted by label and summed over copies, against
    the particles that left."""
import numpy as np
import pytest

from tests.conftest import have_gpu

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not have_gpu(), reason="needs a CUDA GPU")]


def _setup(n):
    from essaitemporaire_lepic_module_b200 import config
    box = [0.0, 0.0, 0.0] + [v * 1e-2 for v in n]
    return config.build(config.Workload("sums", n, 1e-4, [box + [1]], [0.0, 0.0],
                                        [("[Ar+]", 39.95, 1.0, 0.026, 1.0)], Te=2.0, n0=1e15, ppc=4, dt=2e-11,
                                        steps=1, ng=1))


def _place(st, count, how, seed=1):
    rng = np.random.default_rng(seed)
    n, h = np.asarray(st.n), np.asarray(st.h)
    cell = rng.integers(0, n, size=(count, 3))
    if how == "one":
        cell[:] = n // 2
    elif how == "two":
        cell[:] = n // 2
        cell[::2, 0] += 1
    elif how == "sorted":
        cell = cell[np.lexsort(cell.T)]
    v = np.zeros((st.ntype, count, 6))
    for p in range(st.ntype):
        v[p, :, :3] = (cell + rng.random((count, 3)) * 0.999) * h
    return v


@pytest.mark.parametrize("n", [(16, 16, 16), (12, 20, 9)])
@pytest.mark.parametrize("how", ["one", "two", "any", "sorted"])
@pytest.mark.parametrize("count", [1, 31, 33, 1025, 2047, 2049, 20000])
@pytest.mark.parametrize("precision", ["f64", "mixed"])
def test_deposit_of_resting_particles(precision, count, how, n):
    import ctypes as C

    from essaitemporaire_lepic_module_b200._lib import lib
    from essaitemporaire_lepic_module_b200.sim import Simulation
    st = _setup(n)
    sim = Simulation(st, cap=count + 37, precision=precision)
    sim.load_from_host(_place(st, count, how), [count] * st.ntype)
    if precision == "mixed":                     # loaded with FP64 weights: here with the integer ones
        sim.np.zero_()
        for p, s in enumerate(sim.sp):
            assert lib().lepic_dev_deposit_mixed(C.byref(sim.grid), C.byref(s.s), p + 1, C.byref(sim.P),
                                                 C.c_void_p(sim.np[p].data_ptr()), count, sim._s()) == 0
    want = sim.np.clone()
    sim.sort()
    sim.move_deposit()
    sim.check_device()
    assert [s.n() for s in sim.sp] == [count] * st.ntype
    assert float((sim.np - want).abs().max()) <= 1e-13 * float(want.abs().max())


@pytest.mark.parametrize("n", [(16, 16, 16), (12, 20, 9)])
@pytest.mark.parametrize("how", ["one", "any", "sorted"])
@pytest.mark.parametrize("count", [1, 33, 1023, 1025, 4096, 20000])
def test_mixed_sort(count, how, n):
    from essaitemporaire_lepic_module_b200.sim import Simulation
    st = _setup(n)
    sim = Simulation(st, cap=count + 37, precision="mixed")
    v = _place(st, count, how)
    v[:, :, 3:] = np.random.default_rng(2).normal(size=v[:, :, 3:].shape)
    sim.load_from_host(v, [count] * st.ntype)
    s = sim.sp[0]

    def state():
        c = s.cell[:count].cpu().numpy()
        p = s.p[:, :count].cpu().numpy()
        xyz = np.stack([c & 1023, (c >> 10) & 1023, c >> 20])
        nt = [(k + 7) // 8 for k in n]
        t = xyz // 8
        tile = t[0] + nt[0] * (t[1] + nt[1] * t[2])
        key = tile * 512 + (xyz[0] % 8) + 8 * ((xyz[1] % 8) + 8 * (xyz[2] % 8))
        rows = np.concatenate([key[None], p], 0)
        return key, tile, rows[:, np.lexsort(rows[::-1])]

    _, _, before = state()
    sim.sort([0])
    key, tile, after = state()
    assert np.all(np.diff(key) >= 0)
    ntiles = s.tile_off.numel() - 1
    off = np.concatenate([[0], np.cumsum(np.bincount(tile, minlength=ntiles))])
    assert np.array_equal(s.tile_off.cpu().numpy(), off)
    assert np.array_equal(before, after)


@pytest.mark.parametrize("precision", ["f64", "mixed"])
def test_losses_are_all_counted(precision):
    from essaitemporaire_lepic_module_b200.sim import Simulation
    st = _setup((16, 16, 16))
    count = 30000
    v = _place(st, count, "any")
    v[:, :, 3] = 6e6 * np.where(np.arange(count) % 2, 1.0, -1.0)     # 1.2 cells a step along x
    sim = Simulation(st, cap=count + 37, precision=precision)
    sim.load_from_host(v, [count] * st.ntype)
    sim.sort()
    for _ in range(2):
        sim.move_deposit()
        sim.check_device()
    pm, pl = sim.loss_stats()
    for p in range(st.ntype):
        lost = count - sim.sp[p].n()
        ek = 0.5 * st.Nm[p] * abs(st.mass[p]) * 6e6 ** 2
        assert lost > 1000
        assert pm[1, 0, p] == lost
        assert abs(pl[p, 0] - lost * ek) <= 1e-5 * lost * ek         # FP32 velocities in the mixed form
        assert abs(pm[1, 1, p] - pl[p, 0]) <= 1e-12 * pl[p, 0]


@pytest.mark.parametrize("precision", ["f64", "mixed"])
def test_losses_of_pushes_on_two_streams_share_an_array(precision):
    """Two species pushed on two streams at once, their losses added to one
    array: every lost particle of both is counted in it."""
    import ctypes as C

    import torch
    from essaitemporaire_lepic_module_b200._lib import lib
    from essaitemporaire_lepic_module_b200.sim import Simulation
    st = _setup((16, 16, 16))
    count = 4000
    v = _place(st, count, "any")
    v[:, :, 3] = 6e6 * np.where(np.arange(count) % 2, 1.0, -1.0)
    sim = Simulation(st, cap=count + 37, precision=precision)
    sim.load_from_host(v, [count] * st.ntype)
    sim.sort()
    sim.move_deposit()                           # the first call allocates
    acc = torch.zeros(2 + 2 * (st.geom.ngrid + 1), dtype=torch.float64, device="cuda")
    push = lib().lepic_dev_push_deposit_mixed if precision == "mixed" else lib().lepic_dev_push_deposit
    E = sim.E32 if precision == "mixed" else sim.Ei
    streams = [torch.cuda.Stream() for _ in sim.sp]
    lost = 0
    for _ in range(40):
        sim.load_from_host(v, [count] * st.ntype)
        sim.sort()
        torch.cuda.synchronize()
        for p, s in enumerate(sim.sp):
            assert push(C.byref(sim.grid), C.c_void_p(E.data_ptr()), C.byref(s.s), p + 1, st.geom.ngrid,
                        C.byref(sim.P), C.c_void_p(sim.np[p].data_ptr()), C.c_void_p(acc.data_ptr()), -1,
                        C.c_void_p(streams[p].cuda_stream)) == 0
        torch.cuda.synchronize()
        lost += sum(count - s.n() for s in sim.sp)
    sim.check_device()
    assert lost > 1000
    assert float(acc[2::2].sum()) == lost

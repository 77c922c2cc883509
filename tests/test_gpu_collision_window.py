"""The differentiable window of the collisional step (adjoint.CollisionWindow):
electrons and Ar+ of a Penning-like box (16x16x32 cells, end plates at
200 V, B_z = 0.1 T) with the Ar null-collision MCC (elastic, excitation,
ionization, charge exchange) every 4 steps of a 12-step window, the
collisions recorded by the first forward pass and replayed by every later
one.

Bars:
  * the backward pass undoes the window: after it the particles are back at
    their initial state (cells equal, offsets within 1e-5, velocities within
    1e-4 of the species' largest speed; FP32 rounding of the reversed pushes);
  * the FP64 adjoint (the same events, FP64 particles and multigrid) against
    central finite differences of the FP64 window (events replayed):
    dJ/dV per wall label and dJ/dB_z within 1e-4, a directional derivative in
    the initial velocities within 1e-3 (steps of 1e-5 V, 1e-9 T, 1e-2 m/s),
    for the mean electron energy and the probe potential at the box centre;
  * the mixed-precision adjoint (FP32 particles and pushes, FP32 V-cycles in
    FP64 refinement) against the FP64 adjoint for all three observables
    (energy, probe potential, wall energy flux): J, dJ/dV and dJ/dB_z within
    1e-4 (dJ/dB_z of the wall flux within 1e-3), the gradient in the initial
    velocities within 8e-6 in the 2-norm, but for at most 1e-4 of the
    particles (whose wall crossing differs between the two windows, or whose
    replayed ionization is just above its threshold);
  * the torch.autograd.Function returns the window's own gradients.
"""
import dataclasses

import numpy as np
import pytest

from tests.conftest import have_gpu

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not have_gpu(), reason="needs a CUDA GPU")]


@pytest.fixture(scope="module")
def windows():
    import torch
    from essaitemporaire_lepic_module_b200 import config
    from essaitemporaire_lepic_module_b200.adjoint import CollisionWindow
    from essaitemporaire_lepic_module_b200.sim import Simulation
    wl = dataclasses.replace(config.workload("penning_small"), name="mccpen16",
                             ions=[("[Ar+]", 39.95, 1.0, 0.026, 1.0)], gas_pressure=20.0)
    st = config.build(wl)
    sim = Simulation(st, precision="mixed", seed=7)
    sim.load_uniform()
    for _ in range(3):
        sim.step()
    torch.cuda.synchronize()
    # sorted by cell first: the FP32 window scatters tile by tile (slots past
    # the tiles, the collision products, untiled)
    w64 = CollisionWindow(sim, K=12, ns_coll=4, fp64=True, keep_initial=True, sort=True)
    w32 = CollisionWindow(sim, K=12, ns_coll=4, keep_initial=True)
    V = [float(st.wl.V[lab]) for lab in range(1, st.geom.ngrid + 1)]
    Bz = float(st.Bconst[2])
    w32.forward(V, Bz)                  # records the collisions
    w64.use_log_of(w32)
    return st, w32, w64, V, Bz


def _close(a, b, rel):
    a, b = np.atleast_1d(a), np.atleast_1d(b)
    scale = max(np.abs(b).max(), 1e-300)
    return np.abs(a - b).max() <= rel * scale


def test_events_recorded(windows):
    st, w32, _, _, _ = windows
    assert len(w32.ev_range) == 3                         # steps 1, 5, 9
    assert all(b - a > 1000 for a, b in w32.ev_range.values())
    T = st.tables
    types = {int(T.col_info[c, 2 + T.col_info[c, 0] + T.col_info[c, 1]]) for c in range(T.sig.shape[0])
             if w32.counts[c] > 0}
    assert types == {1, 3, 2, 4}, types                   # elastic, excitation, ionization, charge exchange


def test_backward_returns_to_the_initial_state(windows):
    _, w32, _, V, Bz = windows
    w32.forward(V, Bz, observable="energy")
    w32.backward()
    for p, (c0, p0, _) in enumerate(w32.initial):
        n = w32.count0[p]
        d = w32.stores[p]
        x = (d["cell"][:n] & 1023).double() + d["p"][0, :n].double()
        x0 = (c0[:n] & 1023).double() + p0[0, :n].double()
        assert float((x - x0).abs().max()) <= 1e-5
        vmax = float(p0[3:6, :n].abs().max())
        assert float((d["p"][3:6, :n] - p0[3:6, :n]).abs().max()) <= 1e-4 * vmax


@pytest.mark.parametrize("observable", ["energy", "probe"])
def test_fp64_adjoint_vs_central_differences(windows, observable):
    import torch
    _, _, w64, V, Bz = windows
    w64.forward(V, Bz, observable=observable)
    gV, gB, gv = w64.backward()
    # small steps: the replayed events are fixed, but an ionization just
    # above its threshold gives its products a speed growing as the square
    # root of the energy above it, which curves J within a larger step (the
    # events a run records depend on the FP32 window's rounding)
    hV = 1e-5
    fd = []
    for lab in range(len(V)):
        Vp, Vm = list(V), list(V)
        Vp[lab] += hV
        Vm[lab] -= hV
        fd.append((w64.forward(Vp, Bz, observable=observable) - w64.forward(Vm, Bz, observable=observable)) / (2 * hV))
    assert _close(gV, np.array(fd), 1e-4), (gV, fd)
    hB = 1e-9
    fB = (w64.forward(V, Bz + hB, observable=observable) - w64.forward(V, Bz - hB, observable=observable)) / (2 * hB)
    assert _close(gB, fB, 1e-4), (gB, fB)
    torch.manual_seed(0)
    n0 = w64.count0[0]
    dv = torch.randn((3, n0), dtype=torch.float64, device="cuda")
    v0 = w64.initial[0][1][3:6, :n0].clone()
    hv = 1e-2
    fv = (w64.forward(V, Bz, v0=v0 + hv * dv, observable=observable)
          - w64.forward(V, Bz, v0=v0 - hv * dv, observable=observable)) / (2 * hv)
    assert _close(float((gv * dv).sum()), fv, 1e-3), (float((gv * dv).sum()), fv)


@pytest.mark.parametrize("observable", ["energy", "probe", "flux"])
def test_mixed_adjoint_vs_fp64_adjoint(windows, observable):
    _, w32, w64, V, Bz = windows
    J32 = w32.forward(V, Bz, observable=observable)
    g32 = w32.backward()
    J64 = w64.forward(V, Bz, observable=observable)
    g64 = w64.backward()
    assert abs(J32 - J64) <= 1e-4 * abs(J64)
    assert _close(g32[0], g64[0], 1e-4), (g32[0], g64[0])
    # the wall flux counts particles reaching a wall: a particle that
    # reaches it in one window and not in the other (their rounding differs)
    # moves dJ/dBz by up to a few 1e-4 of its value (seen once in many runs;
    # typically 1e-6), so that derivative is held to 1e-3
    rel_bz = 1e-3 if observable == "flux" else 1e-4
    assert _close(g32[1], g64[1], rel_bz), (g32[1], g64[1])
    # the gradient in the initial velocities, particle by particle: FP32
    # rounding through the window leaves the 2-norm of the difference at 2e-7
    # to 6e-7 of the gradient's.  A few of the 247,000 particles are further
    # off: one that reaches a wall in one window and not in the other (one run
    # of twelve; by 0.6 of the rms, which is as much as 2 % of the derivative
    # along a random direction, whose terms cancel), or one whose replayed
    # ionization is just above its threshold.  Those off by more than 1e-3 of
    # the rms are counted instead (at most 1e-4 of all); the rest holds 6e-7
    # and twelve just below that line, 1e-3 sqrt(12 / 247,000) = 7e-6.
    n = g64[2].shape[1]
    off = (g32[2] - g64[2]).norm(dim=0) > 1e-3 * g64[2].norm() / n ** 0.5
    assert int(off.sum()) <= 1e-4 * n, int(off.sum())
    assert float((g32[2] - g64[2])[:, ~off].norm()) <= 8e-6 * float(g64[2].norm())
    # backward no dearer than 3 forward passes of the window
    assert w32.timing["backward_ms"] <= 3.0 * w32.timing["forward_ms"] + 5.0


def test_autograd_function(windows):
    import torch
    from essaitemporaire_lepic_module_b200.adjoint import collision_window_objective
    _, w32, _, V, Bz = windows
    Vt = torch.tensor(V, dtype=torch.float64, requires_grad=True)
    Bt = torch.tensor(Bz, dtype=torch.float64, requires_grad=True)
    v0 = w32.initial[0][1][3:6, :w32.count0[0]].to(torch.float64).clone().requires_grad_(True)
    J = collision_window_objective(w32, Vt, Bt, v0, observable="probe")
    J.backward()
    assert float(J.detach()) == pytest.approx(w32.forward(V, Bz, v0=v0.detach(), observable="probe"), rel=1e-9)
    gV, gB, gv = w32.backward()
    np.testing.assert_allclose(Vt.grad.numpy(), gV, rtol=1e-6, atol=0)
    assert float(Bt.grad) == pytest.approx(gB, rel=1e-6)
    scale = float(gv.abs().max())
    assert float((v0.grad - gv.to(torch.float64)).abs().max()) <= 1e-5 * scale


def test_tiled_and_untiled_scatters_agree(windows):
    """The FP32 window's deposit and push adjoint tile by tile (shared-memory
    node boxes, FP32 partial sums) against the untiled kernels (warp run sums,
    FP64 atomics) on the same events: J and the gradients within 1e-4."""
    import torch
    _, w32, _, V, Bz = windows
    assert any(int(w.tile_end) > 0 for w in w32.ws)
    J1 = w32.forward(V, Bz, observable="probe")
    g1 = w32.backward()
    g1 = (g1[0].copy(), g1[1], g1[2].clone())
    saved = [(w.tile_off, w.tile_end) for w in w32.ws]
    try:
        for w in w32.ws:
            w.tile_off, w.tile_end = None, 0
        J2 = w32.forward(V, Bz, observable="probe")
        g2 = w32.backward()
    finally:
        for w, (a, b) in zip(w32.ws, saved):
            w.tile_off, w.tile_end = a, b
    assert abs(J1 - J2) <= 1e-4 * abs(J2)
    assert _close(g1[0], g2[0], 1e-4), (g1[0], g2[0])
    assert _close(g1[1], g2[1], 1e-4), (g1[1], g2[1])
    torch.manual_seed(2)
    dv = torch.randn(g2[2].shape, dtype=torch.float64, device="cuda")
    assert _close(float((g1[2].double() * dv).sum()), float((g2[2].double() * dv).sum()), 1e-4)

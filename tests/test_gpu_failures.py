"""Failure detection without faulting the GPU: bad inputs are made on the
host, the kernels record a status in the device error word instead of
trapping, the host turns it into LepicError with the status code, and the
context stays usable afterwards.

  * a particle in a cell outside the grid         -> LEPIC_ERR_CELL (22)
  * ionization products beyond the capacity       -> LEPIC_ERR_CAPACITY (1)
  * a refinement cap too small for the tolerance  -> LEPIC_ERR_NOT_CONVERGED (23)
  * a NaN in the right-hand side                  -> a non-zero status, then a
                                                     clean solve succeeds
  * a solve whose barrier is given up             -> LEPIC_ERR_TIMEOUT (25),
                                                     then solves are right
  * a bounded device wait that nothing completes  -> LEPIC_ERR_TIMEOUT (25)
                                                     after its limit, then the
                                                     context runs a step
"""
import numpy as np
import pytest

from essaitemporaire_lepic_module_b200 import config
from tests.conftest import have_gpu

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not have_gpu(), reason="needs a CUDA GPU")]


def test_cell_outside_grid_raises_then_recovers():
    from essaitemporaire_lepic_module_b200._lib import LepicError
    from essaitemporaire_lepic_module_b200.sim import Simulation
    st = config.build("box16")
    sim = Simulation(st, precision="mixed")
    sim.load_uniform()
    sim.step()
    n1 = st.n[0]
    sim.sp[0].cell[7] = (n1 + 4) | (2 << 10) | (2 << 20)   # ix beyond the grid
    with pytest.raises(LepicError) as e:
        sim.step()
    assert e.value.code == 22
    sim.step()                                             # the bad particle became a hole


def test_capacity_overflow_in_collisions():
    import torch
    from essaitemporaire_lepic_module_b200._lib import LepicError
    from essaitemporaire_lepic_module_b200.sim import Simulation
    st = config.build("mcc32")
    n = st.n_particles()
    sim = Simulation(st, cap=n)
    sim.load_uniform()
    s = sim.sp[0]
    s.p[3:6, :n] *= 4.0             # 32 eV electrons: every call ionizes many
    torch.cuda.synchronize()
    sim.it = 11
    with pytest.raises(LepicError) as e:
        sim.collisions()
    assert e.value.code == 1
    sim.check_device()              # the error word was cleared by the raise


def _poisson_sim():
    import torch
    from essaitemporaire_lepic_module_b200.sim import Simulation
    st = config.build("poisson32")
    sim = Simulation(st, cap=1024, precision="mixed")
    sim.rhs.copy_(torch.as_tensor(st.rhs_blobs, device="cuda"))
    sim.phi.copy_(torch.as_tensor(st.geom.phi, device="cuda"))
    return st, sim


def test_refinement_cap_reports_not_converged():
    from essaitemporaire_lepic_module_b200._lib import LepicError
    st, sim = _poisson_sim()
    with pytest.raises(LepicError) as e:
        sim.pdesolver_mixed(eps=1e-15, max_refine=1)
    assert e.value.code == 23
    it, _, res = sim.pdesolver_mixed()
    assert res < st.wl.eps


def test_nan_in_rhs_is_reported_and_the_next_solve_works():
    import torch
    from essaitemporaire_lepic_module_b200._lib import LepicError
    st, sim = _poisson_sim()
    good = sim.rhs.clone()
    sim.rhs.view(-1)[12345] = float("nan")
    with pytest.raises(LepicError):
        sim.pdesolver_mixed(max_refine=5)
    sim.rhs.copy_(good)
    sim.phi.copy_(torch.as_tensor(st.geom.phi, device="cuda"))
    it, _, res = sim.pdesolver_mixed()
    assert res < st.wl.eps and bool(torch.isfinite(sim.phi).all())


def test_bounded_wait_times_out_and_context_stays_usable():
    """A barrier that one of two blocks never reaches: the wait gives up after
    its limit (50 ms here; the solves' allow about a second in which nothing
    moves) and LEPIC_ERR_TIMEOUT is recorded instead of a hang; the
    status is read once and cleared, and a step runs afterwards."""
    import ctypes as C
    import time
    import torch
    from essaitemporaire_lepic_module_b200._lib import lib
    from essaitemporaire_lepic_module_b200.sim import Simulation
    torch.cuda.synchronize()
    L = lib()
    t0 = time.perf_counter()
    assert L.lepic_dev_wait_selftest(50_000_000, None) == 0
    detail = C.c_int(-1)
    assert L.lepic_dev_check(None, C.byref(detail)) == 25
    elapsed = time.perf_counter() - t0
    assert 0.045 <= elapsed < 5.0, elapsed
    assert L.lepic_dev_check(None, C.byref(detail)) == 0          # read once, then cleared
    assert L.lepic_dev_wait_selftest(0, None) == 21                # limit out of range: LEPIC_ERR_ARG
    st = config.build("box16")
    sim = Simulation(st, precision="mixed")
    sim.load_uniform()
    sim.step()
    torch.cuda.synchronize()
    assert L.lepic_dev_check(None, C.byref(detail)) == 0


@pytest.mark.parametrize("how", ["f64", "mixed", "mixed_nonblocking"])
def test_a_solve_whose_barrier_is_given_up_says_so(how):
    """Blocks that wait a few milliseconds only, while block 0 smooths the
    coarsest level for longer: the solve ends with LEPIC_ERR_TIMEOUT (without
    a wait, in the error word, read here without clearing anything else), and
    the next 70 solves, which come round to the same barrier, are those of
    before."""
    import ctypes as C

    import torch
    from essaitemporaire_lepic_module_b200._lib import LepicGrid, lib, phys_struct
    L = lib()
    st = config.build("box16")
    mixed = how != "f64"
    n, ng = (64, 64, 64), 3 if mixed else 4
    shape = tuple(v + 3 for v in n)
    bc = np.ones(shape, dtype=np.int32)
    bc[2:-2, 2:-2, 2:-2] = -1
    bct = torch.as_tensor(bc, device="cuda")
    rt = torch.as_tensor(np.random.default_rng(3).normal(size=tuple(v - 1 for v in shape)) * 1e-5, device="cuda")
    grid = LepicGrid()
    for a in range(3):
        grid.n[a], grid.h[a] = n[a], 1.0e-4
    grid.bcnd = bct.data_ptr()
    P = phys_struct(st)
    s = C.c_void_p(torch.cuda.current_stream().cuda_stream)

    def solve(entry):
        u = torch.zeros(shape, dtype=torch.float64, device="cuda")
        k, kt, res = C.c_int(0), C.c_double(0), C.c_double(0)
        if entry == "f64":
            rc = L.lepic_dev_pdesolver(C.byref(grid), C.c_void_p(u.data_ptr()), C.c_void_p(rt.data_ptr()), 1, 1e-9,
                                       1.4, 4, C.byref(P), C.byref(k), C.byref(kt), C.byref(res), s)
        else:
            rc = L.lepic_dev_pdesolver_mixed(C.byref(grid), C.c_void_p(u.data_ptr()), C.c_void_p(rt.data_ptr()), 1e-9,
                                             1.3, 4, C.byref(P), 40, 1, 3, 2, 2, 4, C.byref(k), C.byref(res), s)
        assert rc == 0, (entry, rc)
        return u

    before = {e: solve(e) for e in ("f64", "mixed")}
    u = torch.zeros(shape, dtype=torch.float64, device="cuda")
    rc = L.lepic_dev_solve_selftest(C.byref(grid), C.c_void_p(u.data_ptr()), C.c_void_p(rt.data_ptr()), ng,
                                    C.byref(P), int(mixed), int(how == "mixed"), s)
    word = torch.zeros(2, dtype=torch.int32).pin_memory()
    if how == "mixed_nonblocking":
        assert rc == 0
        assert L.lepic_dev_check_async(s, C.c_void_p(word.data_ptr())) == 0
        torch.cuda.synchronize()
        assert int(word[0]) == 25
    else:
        assert rc == 25
        assert L.lepic_dev_check(s, None) == 0
    for i in range(70):
        e = ("f64", "mixed")[i % 2]
        assert bool((solve(e) == before[e]).all())


def test_nonblocking_loop_reports_failures_later():
    """Nonblocking mode (no wait in the step loop): a particle moved outside
    the grid is reported by a later step's check or at flush_checks, with
    the same status code, and the loop goes on afterwards."""
    from essaitemporaire_lepic_module_b200._lib import LepicError
    from essaitemporaire_lepic_module_b200.sim import Simulation
    st = config.build("box16")
    sim = Simulation(st, precision="mixed", nonblocking=True)
    sim.load_uniform()
    sim.step()
    sim.flush_checks()
    n1 = st.n[0]
    sim.sp[0].cell[7] = (n1 + 4) | (2 << 10) | (2 << 20)
    with pytest.raises(LepicError) as e:
        for _ in range(4):
            sim.step()
        sim.flush_checks()
    assert e.value.code == 22
    sim.flush_checks()
    sim.step()
    sim.flush_checks()

"""The FP64 Poisson solve on colour-split levels (Dirichlet walls) against
the general kernel (lepic_dev_pdesolver_noalloc runs it): the same node
arithmetic in the same order, so phi, cycles and sweeps are compared bit for
bit.  Grids at the edges of the split layout: odd and even row lengths, one
level, levels on the grid and on chip; walls anywhere, free ghost nodes and
labels 0 and -2 among them."""
import ctypes as C

import numpy as np
import pytest

from tests.conftest import have_gpu

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not have_gpu(), reason="needs a CUDA GPU")]


@pytest.mark.parametrize("n,ng", [((5, 9, 7), 1), ((6, 10, 14), 2), ((30, 22, 26), 2), ((16, 16, 16), 5),
                                  ((32, 16, 24), 4), ((40, 24, 32), 4), ((66, 34, 18), 2), ((64, 64, 64), 7)])
@pytest.mark.parametrize("walls", ["box", "any"])
def test_split_equals_general_kernel(n, ng, walls):
    import torch
    from essaitemporaire_lepic_module_b200 import config
    from essaitemporaire_lepic_module_b200._lib import LepicGrid, lib, phys_struct

    st = config.build("box16")
    rng = np.random.default_rng(n[0] * 100 + n[2])
    shape = (n[2] + 3, n[1] + 3, n[0] + 3)
    bc = np.ones(shape, dtype=np.int32)
    bc[2:-2, 2:-2, 2:-2] = -1
    if walls == "any":
        bc[rng.random(shape) < 0.15] = 2
        bc[rng.random(shape) < 0.03] = -1
        bc[rng.random(shape) < 0.01] = 0
        bc[rng.random(shape) < 0.01] = -2
    phi0 = np.where(bc > 0, rng.normal(size=shape), 0.0)
    rhs = rng.normal(size=tuple(v - 1 for v in shape)) * 1e-5
    dev = torch.device("cuda")
    bct = torch.as_tensor(bc, device=dev)
    grid = LepicGrid()
    for a in range(3):
        grid.n[a] = n[a]
        grid.h[a] = (1.0e-4, 1.1e-4, 0.9e-4)[a]
    grid.bcnd = bct.data_ptr()
    P = phys_struct(st)
    rt = torch.as_tensor(rhs, device=dev)
    got = []
    for entry in (lib().lepic_dev_pdesolver, lib().lepic_dev_pdesolver_noalloc):
        phi = torch.as_tensor(phi0, device=dev).clone()
        for ncycl in (1, 6):   # a cold solve, then a warm one
            k, kt, res = C.c_int(0), C.c_double(0), C.c_double(0)
            # masks drawn at random need not converge: the iterates are compared
            rc = entry(C.byref(grid), C.c_void_p(phi.data_ptr()), C.c_void_p(rt.data_ptr()), ncycl, 1e-9, 1.4, ng,
                       C.byref(P), C.byref(k), C.byref(kt), C.byref(res),
                       C.c_void_p(torch.cuda.current_stream().cuda_stream))
            got.append((rc, k.value, kt.value, res.value, phi.cpu().numpy()))
    half = len(got) // 2
    for a, b in zip(got[:half], got[half:]):
        assert a[:3] == b[:3]
        assert abs(a[3] - b[3]) <= 1e-11 * abs(b[3])     # the norm is summed in another order
        assert np.array_equal(a[4], b[4])

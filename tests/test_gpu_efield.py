"""The E-field pass at the sizes where its blocks and rows end (rows of 8 to
301 nodes) and on the walls it extrapolates from: boxes, slabs and
posts inside, Neumann and periodic planes.  The values are the oracle's, bit
for bit, for a potential whose ghost nodes continue those planes."""
import numpy as np
import pytest

from essaitemporaire_lepic_module_b200 import config
from tests.conftest import have_gpu

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not have_gpu(), reason="needs a CUDA GPU")]


@pytest.mark.parametrize("walls", ["box", "slabs", "posts", "neumann", "periodic"])
@pytest.mark.parametrize("n", [(30, 8, 9), (31, 12, 10), (32, 9, 8), (65, 7, 12), (7, 33, 18), (300, 8, 7)])
def test_efield_rows_and_walls(n, walls, oracle_lib):
    from essaitemporaire_lepic_module_b200 import dropin
    top = [v * 1e-2 for v in n]
    seg = [[0.0, 0.0, 0.0] + top + [1]]
    if walls in ("neumann", "periodic"):         # periodic planes in y and z
        seg.append([0.0, 0.0, 0.0] + top + [0])
    if walls == "slabs":
        seg.append([0.0, 0.0, 3e-2, top[0], top[1], 4e-2, -1])
    if walls == "posts":
        seg.append([3.5e-2, 3.5e-2, 0.0, 4.5e-2, 4.5e-2, top[2], -1])
    st = config.build(config.Workload("rows", n, 1e-4, seg, [0.0, 100.0], [("[Ar+]", 39.95, 1.0, 0.026, 1.0)], Te=2.0,
                                      n0=1e15, ppc=1, dt=2e-11, steps=1, ng=1, neumann_x=walls == "neumann"))
    dropin.set_commons(st)
    n1, n2, n3 = n
    phi = np.random.default_rng(sum(n)).standard_normal((n3 + 3, n2 + 3, n1 + 3))
    if walls == "neumann":
        phi[:, :, 0] = phi[:, :, 2]
    if walls in ("neumann", "periodic"):
        phi[n3 + 1], phi[n3 + 2], phi[0] = phi[1], phi[2], phi[n3]
        phi[:, n2 + 1], phi[:, n2 + 2], phi[:, 0] = phi[:, 1], phi[:, 2], phi[:, n2]
    g, o = dropin.calc_efield(st, phi), oracle_lib.calc_efield(st, phi)
    inner = (slice(1, n3 + 2), slice(1, n2 + 2), slice(1, n1 + 2))
    np.testing.assert_array_equal(g[inner], o[inner])

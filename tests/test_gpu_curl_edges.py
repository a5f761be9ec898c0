"""The curl and the confinement push where their planes and spans end (axes of one and two cells, planes and rows beyond a
block's last), at spacings with and without a division: the oracle's floats."""

import pytest

from oracle import oracle as O
from plume_b200.sim.vorticity import VorticityConfinement
from support import ALL_CLOSED, assert_same, host
from test_gpu_fused_advection import pair

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cell_m", [1.0 / 64.0, 0.05, 4.0])
@pytest.mark.parametrize("cells", [(1, 1, 1), (2, 1, 3), (1, 2, 33), (5, 9, 33), (9, 8, 70), (3, 2, 32)],
                         ids=lambda c: "x".join(map(str, c)))
def test_curl_and_push(cuda_device, cells, cell_m):
    o, c = pair(cells, ALL_CLOSED, cell_m=cell_m)
    oc, cc = O.VorticityConfinement(o), VorticityConfinement(c)
    assert_same(host(cc.measure_curl(c)), oc.measure_curl(o), "curl")
    oc.apply(o, 0.3, 0.02)
    cc.apply(c, 0.3, 0.02)
    assert_same(host(cc.push), oc.push, "push")
    for name in ("u", "v", "w"):
        assert_same(host(getattr(c, name).data), getattr(o, name).data, name)

"""What a context needs of the device beyond its creation: the field getters
nothing."""
import pytest

from swe_fvm_gb300 import Fluxes, SpaceDisc, scenarios

pytestmark = pytest.mark.gpu


def test_getters_take_no_device_memory(gpu):
    import torch

    m, prim = scenarios.sloped_bump_case(240, 3)
    for reorder in ("keep", "morton"):
        sd = SpaceDisc(Fluxes.HLLC(), m, prim, reorder=reorder)
        sd.run(1, 1e-5, 1)
        sd.synchronize()
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        sd.GetEdgField(), sd.GetSrcField(), sd.GetFluxes(), sd.GetNodeMax()
        assert torch.cuda.mem_get_info()[0] == before

"""Device memory of a mixed handle: the FP64 plans' slices count there for the EM sums alone, whose rows are K and 2 K long, so
they take no more than the Float32 plans' slices of gradients and Hessians (458.6 MB and 27.8 MB for these cohorts; with FP64
slices of full rows 462.9 and 30.3)."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("I,J,K,limit", [(20000, 50000, 6, 460e6), (2000, 8000, 5, 29e6)])
def test_mixed_handle_bytes(oa, I, J, K, limit):
    import torch
    g = oa.DeviceGenotypes(torch.full((J, (I + 3) // 4), 0x55, dtype=torch.uint8, device="cuda"), I, J)
    with oa.CuAdmixData(oa.AdmixData(I, J, K, 3), g, flags=oa.ADMIX_FLAG_MIXED) as h:
        assert h.device_bytes() <= limit

"""A CUDA error that an entry point has reported is not found again by the next call of another model or of torch:
here a shell whose fields (514 GB each) no GPU holds, refused by the allocator."""
import pytest

from atjup_b200.params import BC_ALL, resolve_params
from helpers import DRY_ENV, gpu_from, synthetic_case

pytestmark = pytest.mark.gpu


def test_reported_error_is_not_left_behind():
    import torch
    from atjup_b200.gpu import AtjupError, GpuModel
    x = torch.ones(8, device="cuda")
    p, g, f = synthetic_case()
    m = gpu_from(p, g, f)
    try:
        with pytest.raises(AtjupError, match="out of memory"):
            GpuModel(resolve_params(DRY_ENV, im=4000, jm=4000, km=4001), g)
        m.bc(BC_ALL)
        with pytest.raises(AtjupError, match="out of memory"):
            GpuModel(resolve_params(DRY_ENV, im=4000, jm=4000, km=4001), g)
        assert float((x + 1).sum()) == 16.0
    finally:
        m.close()

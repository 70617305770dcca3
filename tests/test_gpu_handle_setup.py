"""A handle is one allocation on the device and one of pinned host memory."""
import pytest
import torch
from torch.profiler import ProfilerActivity, profile

from nntc_b200 import materials
from nntc_b200.session import Session

pytestmark = pytest.mark.gpu


def test_one_allocation_of_each_kind():
    mat = materials.small(1, 40, 24, textures=2)
    torch.zeros(1, device="cuda")
    with Session(mat) as s:
        s.objective()
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        with Session(mat) as s:
            s.objective()
        torch.cuda.synchronize()
    calls = [e.name for e in prof.events() if e.name.startswith("cuda")]
    assert calls.count("cudaMalloc") == 1, calls
    assert sum(c in ("cudaMallocHost", "cudaHostAlloc") for c in calls) == 1, calls
    assert calls.count("cudaFreeHost") == 1, calls

"""GPU test of tensor-core batches whose products differ in inner dimension
(one bucket holds them all): k of one to a few chunks, tile edges and single
rows and columns beside long ones.  Every bit equals the single product's."""
import numpy as np
import pytest
import torch

from vcp_gb300 import batch, pidcuda
from vcp_gb300 import workloads as W

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1, 1), (129, 257, 63), (128, 256, 64), (5, 300, 65), (200, 3, 700), (130, 66, 1024),
          (64, 64, 1025), (257, 40, 2100), (33, 513, 130), (1, 1, 4096), (300, 300, 300)]


@pytest.mark.parametrize("slices", [0, 0x108])
@pytest.mark.parametrize("order", [1, -1])
def test_mixed_inner_dimensions(cuda_lib, slices, order):
    rng = np.random.default_rng(9)
    probs, want = [], []
    for m, n, k in SHAPES[::order]:
        A = torch.from_numpy(W.interval_ephi(rng, m, k, 4, 2.0 ** -40)).cuda()
        B = torch.from_numpy(W.interval_ephi(rng, k, n, 4, 2.0 ** -40)).cuda()
        C = torch.zeros(2 * m * n, dtype=torch.float64, device="cuda")
        R = torch.zeros_like(C)
        pidcuda.mulmm_dev(m, n, k, A, m, B, k, R, m, pidcuda.FORM_OZAKI, slices)
        probs.append((m, n, k, A, m, B, k, C, m))
        want.append(R)
    batch.run(probs, pidcuda.FORM_OZAKI, slices)
    torch.cuda.synchronize()
    for p, R in zip(probs, want):
        assert torch.equal(p[7].view(torch.int64), R.view(torch.int64)), p[:3]

"""The tensor-core batched sum's error against 64 bits.

Bounds: the relative L2 error that the FP32-pipe kernel had at these sizes on
complex Gaussian inputs (mean of 40 solves, to three digits).  Over the 4 x N^3
complex values of a batch the figure moves by about 0.5% with the input.
"""
import numpy as np
import pytest

from oracle.oracle import INDEX_ALIASED

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,bound", [(13, 1.63e-7), (14, 1.70e-7), (15, 1.76e-7), (17, 1.87e-7),
                                     (21, 2.06e-7), (25, 2.22e-7), (31, 2.46e-7)])
def test_no_larger_than_the_fp32_kernels(N, bound):
    import torch
    import entropydecreaseboltzmann_gb300 as edb

    S = 4
    rng = np.random.default_rng(N)
    fin = rng.standard_normal((S, N ** 3)) + 1j * rng.standard_normal((S, N ** 3))
    fin = torch.from_numpy(fin.astype(np.complex64)).cuda()
    q = edb.QCalculator(N, 0, gamma=0.0, L=6.0, filter=False, index_mode=INDEX_ALIASED)
    q.genB()
    q.set_fp64_kernel(1)  # native FP64
    got = torch.empty_like(fin)
    q.calQ_batch_f32(S, fin, got)
    want = torch.empty(S, N ** 3, dtype=torch.complex128, device="cuda")
    for s in range(S):
        q.calQ_device(fin[s].to(torch.complex128), want[s])
    torch.cuda.synchronize()
    err = (got.to(torch.complex128) - want).norm(dim=1) / want.norm(dim=1)
    assert float(err.mean()) <= bound

"""The double-float pair sum's error against the FP64 kernel on small odd grids.

Bounds: the mean relative L2 error of the (re, im) form of the sum, which kept
the products with the two parts of f_l in accumulators of their own, on the
same kind of inputs (400 complex Gaussian solves, to three digits).  The mean
over 200 solves moves by less than 1% with the inputs.
"""
import numpy as np
import pytest

from oracle.oracle import INDEX_ALIASED

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,bound", [(5, 4.45e-15), (6, 4.85e-15), (7, 4.93e-15), (9, 5.46e-15),
                                     (10, 5.88e-15), (11, 5.84e-15), (13, 6.38e-15)])
def test_no_larger_than_with_separate_accumulators(N, bound):
    import torch
    import entropydecreaseboltzmann_gb300 as edb

    S = 200
    rng = np.random.default_rng(N)
    f = torch.from_numpy(rng.standard_normal((S, N ** 3)) + 1j * rng.standard_normal((S, N ** 3)))
    f = f.cuda()
    q = edb.QCalculator(N, 0, gamma=0.0, L=6.0, filter=False, index_mode=INDEX_ALIASED)
    q.genB()
    q.fp64_shape(0)
    got, want = torch.empty_like(f), torch.empty_like(f)
    for kind, out in ((0, got), (1, want)):  # double-float, native FP64
        q.set_fp64_kernel(kind)
        for s in range(S):
            q.calQ_device(f[s], out[s])
    torch.cuda.synchronize()
    assert float(((got - want).norm(dim=1) / want.norm(dim=1)).mean()) <= bound

"""The tensor-core batched sum at the upper end of FP32's range.

It forms products before it weights them: a product of two modes may leave the
range where its weighted value, and the sum, do not.

Tolerance: the batched path's FP32 bound against FP64, relative L2 <= 5e-6.
"""
import numpy as np
import pytest

from oracle.oracle import INDEX_ALIASED

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [13, 18, 31])
@pytest.mark.parametrize("chunks", [1, 3])
def test_products_out_of_range_with_sums_in_range(N, chunks):
    import torch
    import entropydecreaseboltzmann_gb300 as edb

    S = 5
    rng = np.random.default_rng(N)
    f = rng.standard_normal((S, N ** 3)) + 1j * rng.standard_normal((S, N ** 3))
    f[1] *= 1e19
    f[2, 5] = 2.0 ** 127  # one mode; the others meet it with weights well below 1
    f[4, 0] = np.inf
    fin = torch.from_numpy(f.astype(np.complex64)).cuda()
    q = edb.QCalculator(N, 0, gamma=0.0, L=6.0, filter=False, index_mode=INDEX_ALIASED)
    q.genB()
    q.set_fp64_kernel(1)  # native FP64: the double-float one has the range of floats
    part = torch.empty(chunks * S * N ** 3 * 4, dtype=torch.float32, device="cuda")
    out, one = torch.empty_like(fin), torch.empty_like(fin[:1])
    q.calQ_batch_f32_ex(S, 0, chunks, part, fin, out)
    for s in range(4):
        want = torch.empty(N ** 3, dtype=torch.complex128, device="cuda")
        q.calQ_device(fin[s].to(torch.complex128), want)
        assert float((out[s].to(torch.complex128) - want).norm() / want.norm()) <= 5e-6, s
        q.calQ_batch_f32_ex(1, 0, chunks, part, fin[s:s + 1], one)
        assert torch.equal(one[0], out[s]), s
    assert not torch.isfinite(torch.view_as_real(out[4])).any()
    assert edb.device_status() == 0

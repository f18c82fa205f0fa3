"""The FP64 transforms' error against numpy's in extended precision.

Bounds: the relative error of the passes that evaluated their twiddles on the
device (complex Gaussian cubes, to three digits).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,bound", [(10, 3.37e-16), (17, 7.90e-16), (20, 3.98e-16),
                                     (32, 3.58e-16), (64, 4.04e-16)])
def test_no_larger_than_with_device_twiddles(N, bound):
    import torch
    import entropydecreaseboltzmann_gb300 as edb

    if np.finfo(np.longdouble).nmant < 60:
        pytest.skip("no extended precision here")
    B = max(2, 20000 // N ** 3)
    rng = np.random.default_rng(N)
    x = rng.standard_normal((B, N, N, N)) + 1j * rng.standard_normal((B, N, N, N))
    want = np.fft.fftn(x.astype(np.clongdouble), axes=(1, 2, 3))
    assert want.dtype == np.clongdouble
    d = torch.from_numpy(x).cuda()
    got = torch.empty_like(d)
    edb.fft3d.device(N, B, d, got, False, 0)
    e = got.cpu().numpy() - want
    assert np.sqrt((np.abs(e) ** 2).sum() / (np.abs(want) ** 2).sum()) <= bound

"""The table copies of the double-float sum over pairs.

Sizes: CTAs of under one warp (N = 3, 4, 6, 8), with a last warp that is partly
empty (N = 12, 20, 24, 28) and of full warps (N = 16); rows padded by one, two and
three entries (N = 3, 7 | 6, 18, 30 | 9, 17, 25); every launch shape, so every
number of rows a copy, and both rules for the l-line chunks.

Tolerance: the drop-in path's bound, relative L2 <= 1e-12.
"""
import numpy as np
import pytest

from oracle.oracle import INDEX_ALIASED

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def edb():
    import entropydecreaseboltzmann_gb300 as e

    return e


@pytest.mark.parametrize("N", [3, 4, 6, 7, 8, 9, 12, 16, 17, 18, 20, 24, 25, 28, 30])
def test_every_launch_shape_against_the_direct_sum(edb, oracle, N):
    L = 6.0
    rng = np.random.default_rng(N)
    fin = rng.standard_normal(N ** 3) + 1j * rng.standard_normal(N ** 3)
    modes = rng.choice(N ** 3, min(N ** 3, 96), replace=False)
    modes[:2] = 0, N ** 3 - 1
    want = oracle.direct_modes(N, fin, modes, gamma=0.0, R=L, filter=False)
    q = edb.QCalculator(N, 0, L=L, filter=False, index_mode=INDEX_ALIASED)
    q.genB()
    for shape in range(edb.lib.edb_qcalc_fp64_shapes()):
        q.fp64_shape(shape)
        got = q.calQ(None, fin)[modes]
        assert np.linalg.norm(got - want) <= 1e-12 * np.linalg.norm(want), shape
    # a wait that runs out is reported, and the next call is whole again
    edb.set_wait_limit_ns(0)
    try:
        with pytest.raises(edb.EdbError) as e:
            q.calQ(None, fin)
        assert e.value.status == 4
    finally:
        edb.set_wait_limit_ns(-1)
    assert np.array_equal(q.calQ(None, fin)[modes], got)


@pytest.mark.parametrize("N", [8, 16, 17])
def test_captured_and_back_to_back_sums_have_the_same_bits(edb, N):
    """The three launches of a sum overlap; a graph of two sums in a chain, replayed
    without waiting, and the same sums called one after another agree."""
    import torch

    rng = np.random.default_rng(N)
    f = torch.from_numpy(rng.standard_normal(N ** 3) + 1j * rng.standard_normal(N ** 3)).cuda()
    q = edb.QCalculator(N, 0, L=6.0, filter=False, index_mode=INDEX_ALIASED)
    q.genB()
    one, two = torch.empty_like(f), torch.empty_like(f)
    q.calQ_device(f, one)
    torch.cuda.synchronize()
    q.calQ_device(one, two)
    torch.cuda.synchronize()
    a, b = torch.zeros_like(f), torch.zeros_like(f)
    for _ in range(20):
        q.calQ_device(f, a)
        q.calQ_device(a, b)
    torch.cuda.synchronize()
    assert torch.equal(a, one) and torch.equal(b, two)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        st = torch.cuda.current_stream()
        q.calQ_device(f, a, stream=st)
        q.calQ_device(a, b, stream=st)
    a.zero_()
    b.zero_()
    for _ in range(20):
        g.replay()
    torch.cuda.synchronize()
    assert torch.equal(a, one) and torch.equal(b, two)

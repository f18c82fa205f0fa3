"""The one-solve-a-thread variants of the batched Q-hat (10 to 13), and the
remainder of a batch that is launched as one of them.

A solve's result has the same bits from every variant, so variant 0 is the
reference.  S leaves solve groups of four and of two partly empty or just full;
chunks split the lines; an input that starts 8 bytes past a 16-byte boundary
takes the fallback; the grids run from under one tile to several.  Batches of
whole groups of 16 and 1, 4, 5, 8 or 9 solves more, whose last group starts a new
wave of CTAs or does not, give each solve the bits it has alone.
"""
import numpy as np
import pytest

from oracle.oracle import INDEX_ALIASED

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [4, 8, 12, 20, 28, 32])
def test_same_bits_as_variant_0(N):
    import entropydecreaseboltzmann_gb300 as edb
    import torch

    rng = np.random.default_rng(N)
    f = rng.standard_normal((9, N ** 3)) + 1j * rng.standard_normal((9, N ** 3))
    fin = torch.from_numpy(f.astype(np.complex64)).cuda()
    q = edb.QCalculator(N, 0, L=6.0, filter=False, index_mode=INDEX_ALIASED)
    q.genB()
    for S in (1, 2, 3, 4, 5, 9):
        buf = torch.empty(S * N ** 3 + 1, dtype=torch.complex64, device="cuda")
        off = buf[1:].view(S, N ** 3)
        off.copy_(fin[:S])
        for chunks in (1, min(4, N)):
            part = torch.empty(chunks * S * N ** 3 * 4, dtype=torch.float32, device="cuda")
            want = torch.empty_like(fin[:S])
            q.calQ_batch_f32_ex(S, 0, chunks, part, fin[:S], want)
            for variant in (10, 11, 12, 13):
                for src in (fin[:S], off):
                    out = torch.full_like(want, float("nan"))
                    q.calQ_batch_f32_ex(S, variant, chunks, part, src, out)
                    torch.cuda.synchronize()
                    assert torch.equal(out, want), (S, chunks, variant)
    assert edb.device_status() == 0


@pytest.mark.parametrize("N,sizes", [(16, (65, 68, 72, 73)), (24, (33, 36, 37, 66, 72)),
                                     (32, (17, 20, 66, 69))])
def test_a_remainder_of_the_batch_has_its_own_bits(N, sizes):
    import entropydecreaseboltzmann_gb300 as edb
    import torch

    rng = np.random.default_rng(N)
    S = max(sizes)
    f = rng.standard_normal((S, N ** 3)) + 1j * rng.standard_normal((S, N ** 3))
    fin = torch.from_numpy(f.astype(np.complex64)).cuda()
    q = edb.QCalculator(N, 0, L=6.0, filter=False, index_mode=INDEX_ALIASED)
    q.genB()
    alone = torch.empty_like(fin)
    for s in range(S):
        q.calQ_batch_f32(1, fin[s:s + 1], alone[s:s + 1])
    for S in sizes:
        for variant in (0, 4):
            out = torch.full_like(fin[:S], float("nan"))
            q.calQ_batch_f32_ex(S, variant, 1, out, fin[:S], out)
            torch.cuda.synchronize()
            assert torch.equal(out, alone[:S]), (S, variant)
    assert edb.device_status() == 0

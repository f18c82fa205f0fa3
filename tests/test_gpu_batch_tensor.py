"""The tensor-core form of the batched Q-hat (N % 4 != 0, N = 13..31).

Sizes sit at the edges of its tiles: the smallest and the largest, 16, 24 and 32
weight columns (N = 15 | 17, 23 | 25), lines whose last step is not full.  S = 1, 2 and 5 leave groups of solves partly
empty; chunk counts leave chunks empty.

Tolerance: the batched path's FP32 bound against FP64, relative L2 <= 5e-6.
"""
import numpy as np
import pytest

from oracle.oracle import INDEX_ALIASED

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def edb():
    import entropydecreaseboltzmann_gb300 as e

    return e


def rel_l2(a, b):
    return float(np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300))


def _inputs(N, S, seed):
    import torch

    rng = np.random.default_rng(seed)
    fh = rng.standard_normal((S, N ** 3)) + 1j * rng.standard_normal((S, N ** 3))
    fh = fh.astype(np.complex64)
    return fh, torch.from_numpy(fh).cuda()


@pytest.mark.parametrize("N,gamma,filt", [
    (13, 0.5, True), (14, 1.0, False), (15, 0.0, True), (17, 1.0, False), (18, 0.0, False),
    (22, 0.0, True), (23, 1.0, False), (25, 0.0, False), (30, 0.0, False), (31, 1.0, True)])
def test_against_the_oracle(edb, oracle, N, gamma, filt):
    import torch

    L, S = 6.0, 5
    fh, fin = _inputs(N, S, seed=N)
    q = edb.QCalculator(N, int(gamma), gamma=gamma, L=L, filter=filt, index_mode=INDEX_ALIASED)
    q.genB()
    out = torch.full_like(fin, float("nan"))
    q.calQ_batch_f32(S, fin, out)
    chunks = 4
    part = torch.empty(chunks * S * N ** 3 * 4, dtype=torch.float32, device="cuda")
    cut = torch.full_like(fin, float("nan"))
    q.calQ_batch_f32_ex(S, 0, chunks, part, fin, cut)
    # a caller's view that starts 8 bytes past a 16-byte boundary
    shift = torch.empty(S * N ** 3 + 1, dtype=torch.complex64, device="cuda")
    shift[1:] = fin.reshape(-1)
    off = torch.full_like(fin, float("nan"))
    q.calQ_batch_f32(S, shift[1:], off)
    one, two = torch.empty_like(fin[:1]), torch.empty_like(fin[:2])
    q.calQ_batch_f32(1, fin[4:5].contiguous(), one)
    q.calQ_batch_f32(2, fin[3:5].contiguous(), two)
    torch.cuda.synchronize()
    assert edb.device_status() == 0
    assert torch.equal(off, out)
    assert torch.equal(one[0], out[4]) and torch.equal(two, out[3:5])
    got, got_cut = out.cpu().numpy(), cut.cpu().numpy()
    for s in (0, 4):
        f = fh[s].astype(np.complex128)
        if N <= 13:
            B = oracle.genB(N, gamma, L, filt, INDEX_ALIASED)
            want = oracle.calQ(N, B, f, INDEX_ALIASED)
        else:
            # the oracle's table would be gigabytes: the FP64 drop-in, itself
            # within 1e-12 of the oracle over these sizes, gives every mode
            want = q.calQ(None, f)
            k = np.argsort(np.abs(want))[-16:]
            top = oracle.direct_modes(N, f, k, gamma=gamma, R=L, filter=filt)
            assert rel_l2(want[k], top) <= 1e-12
        assert rel_l2(got[s], want) <= 5e-6
        assert rel_l2(got_cut[s], want) <= 5e-6


def test_wait_timeout_is_reported_and_recovers(edb):
    import torch

    N, L, S = 13, 6.0, 9
    _, fin = _inputs(N, S, seed=1)
    q = edb.QCalculator(N, 0, L=L, filter=False, index_mode=INDEX_ALIASED)
    q.genB()
    good, again = torch.empty_like(fin), torch.empty_like(fin)
    q.calQ_batch_f32(S, fin, good)
    torch.cuda.synchronize()
    assert edb.device_status(clear=True) == 0
    edb.set_wait_limit_ns(0)
    try:
        q.calQ_batch_f32(S, fin, again)
        torch.cuda.synchronize()
        assert edb.device_status(clear=True) & 1
    finally:
        edb.set_wait_limit_ns(-1)
    q.calQ_batch_f32(S, fin, again)
    torch.cuda.synchronize()
    assert edb.device_status(clear=True) == 0
    assert torch.equal(again, good)


@pytest.mark.parametrize("N,S", [(13, 50), (21, 37), (25, 31), (31, 17)])
def test_a_batch_in_two_launches_has_each_solves_own_bits(N, S):
    """Sizes whose solves go part in CTAs of four and part in CTAs of two; chunks
    keep their place in the caller's partial sums."""
    import torch
    import entropydecreaseboltzmann_gb300 as edb

    _, fin = _inputs(N, S, seed=N)
    q = edb.QCalculator(N, 0, gamma=0.0, L=6.0, filter=False, index_mode=INDEX_ALIASED)
    q.genB()
    for chunks in (1, 3):
        part = torch.empty(chunks * S * N ** 3 * 4, dtype=torch.float32, device="cuda")
        out = torch.full_like(fin, float("nan"))
        q.calQ_batch_f32_ex(S, 0, chunks, part, fin, out)
        for s in range(S):
            one = torch.empty_like(fin[:1])
            q.calQ_batch_f32_ex(1, 0, chunks, part, fin[s:s + 1], one)
            assert torch.equal(one, out[s:s + 1]), (chunks, s)
    assert edb.device_status() == 0

"""The tensor-core batched sum where it is used: batches, the server, mixed with bad solves.

Up to four solves share a CTA's operand buffers, tensor-memory tiles and staged
planes; a step is a captured graph.
"""
import numpy as np
import pytest

from oracle.oracle import INDEX_ALIASED

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def edb():
    import entropydecreaseboltzmann_gb300 as e

    return e


@pytest.mark.parametrize("N,S", [(13, 5), (21, 7), (30, 4)])
@pytest.mark.parametrize("bad", [complex(np.nan, 0.0), complex(0.0, np.inf), complex(1e30, 1e30)])
def test_a_bad_solve_leaves_its_neighbours_bits_alone(edb, N, S, bad):
    import torch

    rng = np.random.default_rng(N)
    fin = rng.standard_normal((S, N ** 3)) + 1j * rng.standard_normal((S, N ** 3))
    fin = torch.from_numpy(fin.astype(np.complex64)).cuda()
    q = edb.QCalculator(N, 0, gamma=0.0, L=6.0, filter=False, index_mode=INDEX_ALIASED)
    q.genB()
    good, out = torch.empty_like(fin), torch.empty_like(fin)
    q.calQ_batch_f32(S, fin, good)
    for at in (0, 2, S - 1):
        f = fin.clone()
        f[at, N + 1] = bad
        q.calQ_batch_f32(S, f, out)
        others = [s for s in range(S) if s != at]
        assert torch.equal(out[others], good[others]), at
        if not np.isfinite(bad):
            assert not torch.isfinite(torch.view_as_real(out[at])).all()
    assert edb.device_status() == 0


@pytest.mark.parametrize("N,S,scheme", [(17, 9, "SCHEME_RK4"), (21, 37, "SCHEME_SSP3")])
def test_a_batch_steps_each_solve_as_alone(edb, N, S, scheme):
    from entropydecreaseboltzmann_gb300 import data

    f0 = data.maxwellian_mixture_batch(S, N, 6.0, seed=N)
    q = edb.QCalculator(N, 1, gamma=1.0, L=6.0, filter=False, index_mode=INDEX_ALIASED)
    q.genB()

    def run(f):
        b = edb.BatchSolver(q, len(f), 6.0, getattr(edb, scheme), 0.01, fix_entropy=True)
        b.load(f)
        b.step(3)
        return b.read(real=True)

    together = run(f0)
    for s in (0, S // 2, S - 1):
        assert np.array_equal(run(f0[s:s + 1])[0], together[s]), s


def test_a_served_solve_has_the_bits_it_has_alone(edb):
    from entropydecreaseboltzmann_gb300 import data

    N, steps = 17, 6
    f0 = data.maxwellian_mixture_batch(7, N, 6.0, seed=3)

    def serve(which):
        srv = edb.Server(hbm_budget_bytes=4e9, scheme=edb.SCHEME_RK4, dt=0.01)
        ids = [srv.submit(N, 0.0, 6.0, steps + i, f0[i], want_result=True) for i in which]
        srv.run()
        res = [srv.result(r) for r in ids]
        srv.close()
        return res

    mix = serve(range(7))
    for i in (0, 6):
        (F, Fh), = serve([i])
        assert np.array_equal(F, mix[i][0]) and np.array_equal(Fh, mix[i][1]), i

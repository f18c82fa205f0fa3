"""The FP32 table of the tensor-core batched sum takes no columns beyond its own.

A server's budget that just holds a table (and the buffers of its transfers)
admits it.  Sizes whose columns, in fours, are fewer than the kernel's 24 or 32.
"""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,steps", [(17, 3), (19, 4), (25, 5), (26, 7)])
def test_a_budget_of_the_columns_in_use_holds_a_table(N, steps):
    import entropydecreaseboltzmann_gb300 as edb

    lines = N * (N // 2 + 1) * N  # of an output plane's visited l1 planes
    table = lines * steps * 128 * ((N + 3) // 4 * 4) * 4 + 256
    transfers = 64 * N ** 3 * 40 + 4096
    s = edb.Server(hbm_budget_bytes=table + transfers)
    s.prepare(N, 0.0, 6.0)

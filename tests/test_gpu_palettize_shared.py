"""Matrices whose rows several threads carry to the GPU and back: the bytes are those of the same rows in calls of their own, which
one thread serves (and which the other quantiser tests hold against the oracle).  Sizes: shares that end inside a row of a slot, fewer
rows than threads, rows of the thread-per-row kernel, and the first size that is shared."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n", [(1021, 2100), (2, 1 << 20), (3, 900000), (100003, 64), (4096, 512)])
def test_shares(backend, m, n):
    w = (np.random.default_rng(m).standard_normal((m, n)) * 0.02).astype(np.float32)
    assert w.nbytes >= 8 << 20
    got = backend.palettize(w)
    assert np.array_equal(got, backend.palettize(w))
    pal, idx = got[:m * 32].reshape(m, 32), got[m * 32:].reshape(m, n // 2)
    step = max(1, (2 << 20) // (4 * n))
    for a in list(range(0, m, max(step, m // 6 // step * step))) + [m - 1]:
        rows = w[a:a + step]
        if rows.nbytes >= 8 << 20:
            continue
        own = backend.palettize(rows)
        assert np.array_equal(own[:len(rows) * 32], pal[a:a + step].reshape(-1)) and np.array_equal(own[len(rows) * 32:], idx[a:a + step].reshape(-1)), a

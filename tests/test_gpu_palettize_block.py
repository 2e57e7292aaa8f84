"""The quantiser's one-block-per-row kernel against the CPU restatement, byte for byte, where it can go wrong: rows that
are no multiple of the 32 elements of a running sum or of the 128 threads, fewer elements than entries, more shared memory
than the default limit, the last row length that fits and the first that does not (one thread per row), distances that
overflow, infinities and NaN among the weights."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
FITS = (220 * 1024) // 132 * 32  # elements whose distances and running sums fit


@pytest.mark.parametrize("m,k", [(3, 2), (2, 14), (3, 30), (3, 32), (3, 34), (2, 126), (2, 130), (2, 4098), (2, 12290), (1, FITS), (1, FITS + 2)])
def test_row_lengths(backend, oracle, m, k):
    w = (np.random.default_rng(k).standard_normal((m, k)) * 0.5).astype(np.float32)
    assert np.array_equal(backend.palettize(w), oracle.palettize_to_payload(w, m, k, 16, 50))


@pytest.mark.parametrize("m,k", [(720 * 2, 2), (720 * 16 - 1, 16), (720 * 16, 16), (720 * 34 + 5, 34)])
def test_many_short_rows(backend, oracle, m, k):
    """Both sides of the line from which short rows take a thread each."""
    w = (np.random.default_rng(k).standard_normal((m, k)) * 0.5).astype(np.float32)
    assert np.array_equal(backend.palettize(w), oracle.palettize_to_payload(w, m, k, 16, 50))


@pytest.mark.parametrize("kind", ["huge", "inf", "nan", "zeros", "ties"])
def test_values(backend, oracle, kind):
    m, k = 4, 200
    rng = np.random.default_rng(5)
    w = rng.standard_normal((m, k)).astype(np.float32)
    if kind == "huge":
        w *= np.float32(3e19)  # squares near the largest float, their sum beyond it
    elif kind == "inf":
        w[0, 3], w[1, 100], w[2, 77] = np.inf, -np.inf, np.inf
    elif kind == "nan":
        w[0, 3] = w[1, 150] = np.nan
        w[2, k // 2] = np.nan  # the first centroid
    elif kind == "zeros":
        w[:] = 0.0
        w[1, 7] = 1.0
        w[2] = -0.0
    else:
        w = rng.integers(-9, 10, size=(m, k)).astype(np.float32) / 4  # equal distances to two entries
    got, want = backend.palettize(w), oracle.palettize_to_payload(w, m, k, 16, 50)
    # a NaN's payload is the machine's own
    assert np.array_equal(got[: m * 32].view(np.float16), want[: m * 32].view(np.float16), equal_nan=True)
    assert np.array_equal(got[m * 32:], want[m * 32:])

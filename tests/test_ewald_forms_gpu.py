"""The Ewald sum's forms away from the reference's k-vector order: vectors summed as given (not a mirrored integer cube) at the
edges of a tile and a block and above the tiled range, and mirrored sets in no order over several blocks of vectors. Bounds
as in test_ewald_sum, which holds the comparison."""
import numpy as np
import pytest

import tests.test_fp64_kernels_gpu as fp64

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 32, 257, 900, 49152, 49153])
@pytest.mark.parametrize("kind", ["free", "wide", "half"])
def test_vectors_as_given(n, kind):
    fp64.test_ewald_sum(n, kind)


@pytest.mark.parametrize("n", [1, 33, 900])
@pytest.mark.parametrize("kmax", [7, 10])
def test_mirrored_vectors_in_no_order(n, kmax, monkeypatch):
    """1418 and 4168 vectors: more runs of equal (x, y) in a block than its table of products holds."""
    m = np.arange(-kmax, kmax + 1)
    N = np.stack(np.meshgrid(m, m, m, indexing="ij"), -1).reshape(-1, 3)
    N = N[(np.sum(N ** 2, 1) <= kmax ** 2) & np.any(N != 0, 1)]
    rng = np.random.default_rng(kmax)
    N = N[rng.permutation(len(N))]

    def vectors(kind, box, alpha):
        kv = 2 * np.pi * N / box
        k2 = np.sum(kv ** 2, 1)
        return np.ascontiguousarray(kv), np.exp(-k2 / (4 * alpha ** 2)) / k2 * rng.uniform(0.5, 2, len(N))

    monkeypatch.setattr(fp64, "_ewald_vectors", vectors)
    fp64.test_ewald_sum(n, "order")

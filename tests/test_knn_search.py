"""The host's kNN search against all pairs: the k smallest (distance, id) of every point, in
the reference's float arithmetic (coord3::getDist, src/NeuCor.h:16-18)."""
import numpy as np
import pytest


@pytest.mark.parametrize("n,k,density,seed", [(2, 1, 8.0, 1), (33, 32, 8.0, 2), (130, 7, 0.01, 3), (257, 60, 8.0, 4),
                                              (700, 150, 1e6, 5), (1024, 1, 8.0, 6), (300, 299, 50.0, 7)])
def test_search_finds_the_nearest(nc, n, k, density, seed):
    xyz, pre, post, w = nc.build_knn(n, k, density, seed=seed)
    d = xyz.reshape(n, 1, 3) - xyz.reshape(1, n, 3)
    sq = d * d
    dist = np.sqrt((sq[..., 0] + sq[..., 1]) + sq[..., 2])
    assert dist.dtype == np.float32
    key = dist.view(np.uint32).astype(np.uint64) << np.uint64(32) | np.arange(n, dtype=np.uint64)
    np.fill_diagonal(key, np.iinfo(np.uint64).max)
    nearest = np.argsort(key, axis=1)[:, :k]
    assert np.array_equal(np.asarray(post).reshape(n, k), nearest)
    assert np.array_equal(np.asarray(pre), np.repeat(np.arange(n), k))
    assert np.asarray(w).min() >= 0.0 and np.asarray(w).max() < 1.0

"""Read-backs written straight into the caller's memory against those that pass through a copy
(buffers that are not on 16 bytes, and large ones), at the sizes where the way changes."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def at_offset(count, offset):
    """`count` floats, `offset` bytes past a 64-byte boundary, in memory nobody has touched."""
    raw = np.empty(4 * count + 192, np.uint8)
    start = (-raw.ctypes.data) % 64 + offset
    return raw[start:start + 4 * count].view(np.float32)


@pytest.mark.parametrize("n,k", [(2, 1), (40, 25), (1024, 64), (1025, 64), (4096, 17), (33000, 20)])
def test_same_values_either_way(nc, n, k):
    net = nc.NeuCor.knn(n, k, 8.0, seed=n, params=nc.default_params(seed=5))
    net.run(20)
    lib = nc.load_library()
    for call, count in ((lib.nc_read_weights, n * k), (lib.nc_read_potentials, n), (lib.nc_read_potact, 2 * n)):
        outs = []
        for offset in (0, 16, 4, 12):
            out = at_offset(count, offset)
            assert call(net._handle(), ctypes.c_void_p(out.ctypes.data)) == 0
            outs.append(out.copy())
        for o in outs[1:]:
            assert np.array_equal(o.view(np.uint32), outs[0].view(np.uint32)), (call, count)
    net.close()

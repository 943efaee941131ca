"""cac_cc_noalloc, one pass of union walks, on graphs with long chains, hubs and many components; labels against the oracle."""
import ctypes

import numpy as np
import pytest

import pyoracle as O
from test_cc_small_shapes_gpu import _shapes

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("offset", [0, 1])  # 1: edge arrays off the 16-byte boundary
@pytest.mark.parametrize("n", [33, 1025, 20001, 300007])
def test_labels(libcac, n, offset):
    out = torch.empty(n, dtype=torch.int32, device="cuda")
    count = torch.empty(1, dtype=torch.int32, device="cuda")
    for name, (u, v) in _shapes(n).items():
        want_count, want = O.cc_labels(n, u.astype(np.uint32), v.astype(np.uint32))
        a, b = (torch.empty(len(u) + 4, dtype=torch.int32, device="cuda") for _ in range(2))
        for t, x in ((a, u), (b, v)):
            t[offset:offset + len(x)] = torch.from_numpy(x.astype(np.int32)).cuda()
        torch.cuda.synchronize()
        ptr = [ctypes.c_void_p(t.data_ptr() + 4 * offset) for t in (a, b)]
        for labels in (out, None):
            st = libcac.lib().cac_cc_noalloc(n, len(u), *ptr, None if labels is None else ctypes.c_void_p(labels.data_ptr()),
                                             ctypes.c_void_p(count.data_ptr()),
                                             ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
            assert st == 0
            torch.cuda.synchronize()
            assert int(count.item()) == want_count, name
        assert np.array_equal(out.cpu().numpy().view(np.uint32), want), name

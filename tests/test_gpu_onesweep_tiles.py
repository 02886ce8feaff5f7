"""The onesweep sort at the edges of its look-back steps (eight tiles of 4096 keys at a time) and with digits that
many lanes share: exact against a stable argsort."""
import ctypes

import numpy as np
import pytest

from splatter_gb300 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [8 * 4096, 8 * 4096 + 1, 9 * 4096, 9 * 4096 + 1, 17 * 4096 + 33, 262_144])
@pytest.mark.parametrize("distinct", [1, 3, 40, 1 << 32])
def test_onesweep_is_stable_over_many_tiles(cuda, n, distinct):
    import torch
    lib = _lib.load()
    stream = torch.cuda.current_stream().cuda_stream
    rng = np.random.default_rng(n + distinct % 1000)
    keys = (rng.integers(0, distinct, n, dtype=np.int64) * 2654435761 % (1 << 32)).astype(np.uint32)
    vals = rng.permutation(n).astype(np.uint32)
    kd, vd = (torch.from_numpy(a.view(np.int32)).cuda() for a in (keys, vals))
    ko, vo = torch.empty_like(kd), torch.empty_like(vd)
    _lib.check(lib.spl_sort_pairs_no_alloc(*(ctypes.c_void_p(t.data_ptr()) for t in (kd, vd, ko, vo)), n, 32,
                                           ctypes.c_void_p(stream)))
    torch.cuda.synchronize()
    order = np.argsort(keys, kind="stable")
    assert np.array_equal(ko.cpu().numpy().view(np.uint32), keys[order])
    assert np.array_equal(vo.cpu().numpy().view(np.uint32), vals[order])
    err = ctypes.c_uint32(99)
    assert lib.spl_sort_pairs_no_alloc_status(ctypes.c_void_p(stream), ctypes.byref(err)) == 0 and err.value == 0

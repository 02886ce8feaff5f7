"""The sort's input and output arrays in every arrangement that it takes: apart, in place, exchanged, both
outputs one array (the values stay), and arrays that start between 16-byte boundaries, whether the kernel reads
and writes them itself or copies of them."""
import ctypes

import pytest

from splatter_gb300 import Configuration, Renderer, _lib

pytestmark = pytest.mark.gpu

SHAPES = ["apart", "in place", "exchanged", "one output", "keys into values", "input + 1", "output + 1", "shifted by 1"]


@pytest.mark.parametrize("n", [1, 700, 4097, 200_003])
@pytest.mark.parametrize("bits", [8, 16, 32])
@pytest.mark.parametrize("shape", SHAPES)
def test_arrangements(cuda, shape, bits, n):
    import torch
    gen = torch.Generator(device="cuda").manual_seed(n)
    big = torch.randint(0, 1 << 32, (n,), generator=gen, device="cuda")
    order = torch.sort(big & ((1 << bits) - 1), stable=True).indices
    keys = torch.where(big >= 1 << 31, big - (1 << 32), big).to(torch.int32)
    values = torch.randperm(n, generator=gen, device="cuda").to(torch.int32)
    want_k, want_v = keys[order], values[order]
    a, b, c, d = (torch.zeros(n + 8, dtype=torch.int32, device="cuda") for _ in range(4))
    at = {"input + 1": (1, 1, 0, 0), "output + 1": (0, 0, 1, 1)}.get(shape, (0, 0, 0, 0))
    ki, vi, ko, vo = a, b, c, d
    if shape == "in place":
        ko, vo = ki, vi
    elif shape == "exchanged":
        ko, vo = vi, ki
    elif shape == "one output":
        vo = ko
    elif shape == "keys into values":
        ko = vi
    elif shape == "shifted by 1":
        ko, vo, at = ki, vi, (0, 0, 1, 1)
    ki, vi, ko, vo = (t[o:o + n] for t, o in zip((ki, vi, ko, vo), at))
    ki.copy_(keys)
    vi.copy_(values)
    r = Renderer(Configuration(max_splat_count=n, max_pair_count=1024))
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    pointers = [ctypes.c_void_p(t.data_ptr()) for t in (ki, vi, ko, vo)]
    _lib.check(_lib.load().spl_sort_pairs(r.handle, *pointers, n, bits, stream))
    assert torch.equal(vo, want_v)
    if shape != "one output":
        assert torch.equal(ko, want_k)
    r.close()

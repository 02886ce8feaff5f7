"""The one-launch sort against torch's stable sort, whole results, at the sizes where its work is split
differently: one CTA, CTAs that exchange their counts directly or by groups, segments of up to half a
sub-tile, a sub-tile and several, last segments of a few keys; and keys that put every lane, or most of them,
on one digit."""
import pytest

from splatter_gb300 import Configuration, Renderer

pytestmark = pytest.mark.gpu

SUB_TILE, SHORTEST = 4096, 2048


def grid():
    import torch
    return 2 * torch.cuda.get_device_properties(0).multi_processor_count


def sizes():
    edges = [1, 31, SUB_TILE, 16 * SHORTEST, 32 * SHORTEST, 33 * SHORTEST, "short", "tile", "tile+tail", "long", "long+tail"]
    return [(e, d) for e in edges for d in (-1, 0, 1)][1:]


def count_of(edge):
    g = grid()
    return {"short": g * SHORTEST, "tile": g * SUB_TILE, "tile+tail": g * (SUB_TILE + 256) - 4000, "long": 3 * g * SUB_TILE,
            "long+tail": g * (3 * SUB_TILE + 256) - 12000}.get(edge, edge)


def keys_of(kind, n, gen):
    import torch
    big = torch.randint(0, 1 << 32, (n,), generator=gen, device="cuda")
    return {"random": big, "few": big % 3 * 0x01010101, "one": torch.full_like(big, 0x12FF0034),
            "rising": torch.arange(n, device="cuda") * 771 % (1 << 32), "high": (big >> 27) << 27 | 5}[kind]


@pytest.mark.parametrize("kind", ["random", "few", "one", "rising", "high"])
@pytest.mark.parametrize("edge,delta", sizes())
def test_sort_equals_stable_sort(cuda, edge, delta, kind):
    import torch
    n = count_of(edge) + delta
    if kind != "random" and (delta != 1 or n < SUB_TILE):
        pytest.skip("key kinds once per size")
    gen = torch.Generator(device="cuda").manual_seed(n)
    keys = keys_of(kind, n, gen)
    values = torch.randperm(n, generator=gen, device="cuda").to(torch.int32)
    r = Renderer(Configuration(max_splat_count=n, max_pair_count=1024))
    as_int = torch.where(keys >= 1 << 31, keys - (1 << 32), keys).to(torch.int32)
    for bits in (32, 8, 24) if delta == 1 else (32,):
        order = torch.sort(keys & ((1 << bits) - 1), stable=True).indices
        got_k, got_v = r.sort_pairs(as_int, values, key_bits=bits)
        assert torch.equal(got_k, as_int[order]) and torch.equal(got_v, values[order]), bits
    # again, with fewer keys than the table of counts last held
    m = max(1, n // 3)
    order = torch.sort(keys[:m], stable=True).indices
    got_k, got_v = r.sort_pairs(as_int[:m].contiguous(), values[:m].contiguous())
    assert torch.equal(got_k, as_int[:m][order]) and torch.equal(got_v, values[:m][order])
    r.close()

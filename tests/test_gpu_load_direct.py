"""Records copied straight from the caller's memory against the same records loaded from the device: counts around the
line (2^18 bytes) and around a staging piece, host addresses off the 16-byte boundary, the caller's memory overwritten
as soon as the call returns, and a frame's work still running on the stream."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LINE = (1 << 18) // 248  # records of the last staged chunk


def _records(n, seed):
    rng = np.random.default_rng(seed)
    rec = rng.standard_normal((n, 62)).astype(np.float32)
    rec[:, 55:58] = rec[:, 55:58] * 0.5 - 4.0
    return rec


def _splats(scene, n):
    import torch
    torch.cuda.synchronize()
    return scene.read_splats(0, n).tobytes()


@pytest.mark.parametrize("count,offset", [(LINE, 0), (LINE + 1, 0), (LINE + 1, 4), (5000, 12), (65536, 4), (65537, 0),
                                          (140000, 20)])
def test_direct_chunks_equal_device_loads(count, offset):
    import torch
    from splatter_gb300 import Configuration, Renderer, Scene
    n = count + 9
    renderer = Renderer(Configuration(max_splat_count=n, spherical_harmonics_order=3))
    rec = _records(n, count)
    scenes = [Scene(renderer, n), Scene(renderer, n)]
    for s in scenes:
        s.load_chunk_device(torch.from_numpy(_records(n, 1)).cuda())
    scenes[0].load_chunk_device(torch.from_numpy(rec[:count]).cuda(), 7)
    camera = np.eye(4, dtype=np.float32).reshape(16)
    renderer.render_frame(scenes[1], camera, 640, 400)
    store = bytearray(count * 248 + offset)
    host = np.frombuffer(store, np.float32, count * 62, offset).reshape(count, 62)
    host[:] = rec[:count]
    scenes[1].load_chunk(host, 7)
    host[:] = np.nan
    assert _splats(scenes[0], n) == _splats(scenes[1], n)

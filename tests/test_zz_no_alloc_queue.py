"""rast_render_noalloc at its scratch limit: frames of so many bins that the raster queue's six arrays
do not fit the 32 MiB beside the rest take one array (only empty bins are kept apart), from the first
attempt, after a regrowth of the bins, and with more triangles than a small frame. The image equals the
ordinary entry point's."""
import numpy as np
import pytest

from rusterizer_gb300 import _lib, renderer
from test_zz_no_alloc import _ndc_scene, _noalloc

pytestmark = pytest.mark.gpu

LIMIT = 32 << 20


def scratch(nverts, ntris, bins, entries, arrays):
    """Bytes of the frame's buffers with 8- or 16-pixel bins, to within 64 KB (descriptors, alignment)."""
    chunk = max(256, (-(-ntris // 900) + 255) // 256 * 256)
    return (34 * nverts + (8 + 4 + 12) * ntris + 4 * -(-ntris // chunk) * bins + 8 * bins + 4 * arrays * bins +
            4 * entries + 4 * (32 * ntris + 4096))


def quads(n):
    """n screen-filling pairs of triangles, one behind another."""
    pos = [(x, y, 0.9 - 0.2 * k) for k in range(n) for x, y in [(-1.5, -1.5), (-1.5, 1.5), (1.5, 1.5), (1.5, -1.5)]]
    return pos, [t for k in range(n) for t in [(4 * k, 4 * k + 1, 4 * k + 2), (4 * k, 4 * k + 2, 4 * k + 3)]]


def scattered(n):
    """n triangles over 600 places of a few pixels, some across the view's edges."""
    rng = np.random.default_rng(4)
    c = rng.uniform(-1.0, 1.0, (600, 1, 2))
    xy = c + rng.uniform(-0.002, 0.002, (600, 3, 2))
    pos = np.concatenate([xy, rng.uniform(-0.9, 0.9, (600, 3, 1))], 2).reshape(-1, 3)
    return pos, np.arange(1800).reshape(-1, 3)[rng.integers(0, 600, n)]


def check(w, h, tile, mesh, first, last):
    """`first`, `last`: arrays that fit for the first estimate of the bins and for what the frame needs."""
    torch = pytest.importorskip("torch")
    pos, idx = mesh
    scene = _ndc_scene(w, h, pos, idx, "queue")
    ref, st, r = renderer.render_scene(scene, tile=tile)
    r.close()
    assert st == _lib.OK and (ref != 0xFF191919).any()
    bins, nt = -(-w // tile) * -(-h // tile), len(idx)
    need = [4 * nt + bins + 1024]
    if last is not None:  # the box of either half of a quad is the whole image
        need.append(int(1.25 * nt * bins))
    for entries, arrays in zip(need, (first, last)):
        six, one = (scratch(len(pos), nt, bins, entries, a) for a in (6, 1))
        assert one < LIMIT - 65536 and (six < LIMIT - 65536 if arrays == 6 else six > LIMIT)
    out = torch.zeros(h * w, dtype=torch.int32, device="cuda")
    for _ in range(2):
        out.fill_(0)
        assert _noalloc(torch, scene, out, tile=tile) == _lib.OK
        assert (out.cpu().numpy().view(np.uint32).reshape(h, w) == ref).all()


def test_one_array_from_the_first_attempt():
    check(8192, 7168, 8, quads(1), 1, 1)


def test_one_array_after_regrowth():
    check(8192, 6250, 8, quads(2), 6, 1)


def test_one_array_with_many_triangles():
    check(4000, 3040, 8, scattered(9000), 1, None)

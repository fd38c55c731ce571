"""The texture filter that shades fragments (tex_argb, op 11 of rast_debug_kat) against the oracle's
Texture::sample and Color::to_argb (src/texture.rs:47-83, src/color.rs:15-29), the packed colour with its
alpha and the reads past the texture, bit for bit: every byte value in every channel, coordinates at 0, at 1, on texel
centres and one step either side, negative, above 1, infinite and NaN, one-texel-wide textures, and
sides of 65 535 and 65 536, on both sides of the range where texel indices are computed in 32 bits."""
import ctypes

import numpy as np
import pytest

import oracle
from rusterizer_gb300 import _lib

pytestmark = pytest.mark.gpu


def gpu(tex, uv):
    h, w = tex.shape[:2]
    n = len(uv)
    inp = np.concatenate([np.array([w, h, n, 0], np.int32), uv.astype(np.float32).reshape(-1).view(np.int32),
                          np.ascontiguousarray(tex).reshape(-1).view(np.int32)])
    out = np.zeros(2 * n, np.uint32)
    assert _lib.load().rast_debug_kat(11, inp.ctypes.data_as(ctypes.c_void_p), inp.nbytes,
                                      out.ctypes.data_as(ctypes.c_void_p), out.nbytes) == _lib.OK
    return out[:n], out[n:] != 0


def ref(tex, uv):
    tex = np.ascontiguousarray(tex)
    h, w = tex.shape[:2]
    L, c = oracle.lib(), np.zeros(4, np.float32)
    p, cp = tex.ctypes.data_as(oracle._u8p), oracle.fptr(c)
    argb, oob = np.zeros(len(uv), np.uint32), np.zeros(len(uv), bool)
    for i, (u, v) in enumerate(uv):
        oob[i] = bool(L.oracle_kat_tex_sample(p, w, h, u, v, cp))
        argb[i] = L.oracle_kat_to_argb(cp)
    return argb, oob


def around(n):
    """Coordinates of an n-texel side's centres (at most 260 of them) and the floats next to them."""
    k = np.unique(np.linspace(0, n - 1, min(n, 260)).astype(np.int64))
    c = (k / np.float64(max(n - 1, 1))).astype(np.float32)
    mid = ((k[:-1] + 0.5) / np.float64(max(n - 1, 1))).astype(np.float32)
    return np.concatenate([c, np.nextafter(c, np.float32(2)), np.nextafter(c, np.float32(-1)), mid])


SPECIAL = np.array([0.0, -0.0, 1.0, 1e-45, -1e-45, 1e-30, 0.5, 0.25, np.nextafter(np.float32(1), np.float32(2)),
                    np.nextafter(np.float32(1), np.float32(0)), 1.5, 2.0, -0.25, -3.0, 1e9, 1e30, -1e30, np.inf, -np.inf,
                    np.nan], np.float32)


def coordinates(w, h, seed):
    rng = np.random.default_rng(seed)
    u, v = around(w), around(h)
    pairs = [np.stack([u, rng.choice(v, len(u))], 1), np.stack([rng.choice(u, len(v)), v], 1),
             np.stack(np.meshgrid(SPECIAL, SPECIAL), -1).reshape(-1, 2), rng.random((600, 2)),
             np.stack([rng.choice(SPECIAL, 100), rng.random(100)], 1), np.stack([rng.random(100), rng.choice(SPECIAL, 100)], 1)]
    return np.concatenate(pairs).astype(np.float32)


def check(tex, uv):
    g, goob = gpu(tex, uv)
    r, roob = ref(tex, uv)
    bad = np.nonzero((g != r) | (goob != roob))[0]
    assert len(bad) == 0, (len(bad), uv[bad[0]], hex(g[bad[0]]), hex(r[bad[0]]), goob[bad[0]], roob[bad[0]])


@pytest.mark.parametrize("w,h", [(256, 1), (1, 256), (16, 16)])
def test_every_byte_in_every_channel(w, h):
    i = np.arange(256)
    t = np.stack([i, 255 - i, (i * 7) & 255, (i * 13 + 5) & 255], 1).astype(np.uint8).reshape(h, w, 4)
    uv = np.stack([np.tile(np.arange(w) / max(w - 1, 1), h), np.repeat(np.arange(h) / max(h - 1, 1), w)], 1)
    check(t, uv.astype(np.float32))  # each texel alone
    check(t, coordinates(w, h, w))


@pytest.mark.parametrize("w,h", [(1, 1), (2, 1), (1, 3), (2, 2), (5, 7), (64, 64), (100, 33), (65535, 1), (1, 65535),
                                 (65536, 1), (1, 65536), (65537, 2), (65535, 3)])
def test_sizes(w, h):
    check(np.random.default_rng(w * 31 + h).integers(0, 256, (h, w, 4), dtype=np.uint8), coordinates(w, h, w + h))

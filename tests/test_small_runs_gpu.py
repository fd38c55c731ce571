"""Runs of several small frames (k_front): four triangles per warp up to 16 384 triangles in the run, ten
beyond. Frames whose triangle counts leave every remainder of a warp and of a chunk, with straddlers
in all of a warp's places, in a short run and in a long one; every image equals the oracle's."""
import numpy as np
import pytest

import oracle
from rusterizer_gb300.batch import BatchRenderer
from test_small_frame_clipping_gpu import INSIDE, STRADDLES, scene

pytestmark = pytest.mark.gpu

SIZES = [1, 3, 4, 9, 10, 11, 31, 39, 40, 41, 79, 80, 81, 95, 161, 1003]


def frames(more):
    out = [scene([STRADDLES] * n if n % 2 else list(np.random.default_rng(n).integers(0, 4, n)), n) for n in SIZES]
    # each place of a warp's ten triangles alone
    out += [scene([STRADDLES if t == k else INSIDE for t in range(10)], 50 + k) for k in range(10)]
    return out + [scene(list(np.random.default_rng(n).integers(0, 4, n)), n) for n in more]


# in all 1 788 triangles, then 16 383, 16 384, 16 385 and 24 427
@pytest.mark.parametrize("more", [[], [8160, 6435], [8160, 6436], [8160, 6437], [8160, 8160, 6319]])
def test_run(more):
    sc = frames(more)
    assert sum(len(s["draws"][0]["idx"]) for s in sc) == 1788 + sum(more)
    br = BatchRenderer()
    for s in sc:
        br.add_scene(s)
    imgs = [np.zeros((s["height"], s["width"]), np.uint32) for s in sc]
    br.render(imgs)
    br.close()
    for k, s in enumerate(sc):
        assert (imgs[k] == oracle.render_scene(s, nthreads=4)[0]).all(), k

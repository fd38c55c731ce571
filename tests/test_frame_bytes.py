"""What the render server charges a request against its memory budget (frame_bytes in rast_types.h):
at least the scratch that a run reserves for the frame and its image, summed here from the HBM
layout, and no more than the fixed allowance above it. On the GPU: a budget of exactly that admits the request, one byte
less refuses it."""
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "rusterizer_gb300", "csrc")
CASES = [(nv, nt, w, h, ts, bins)
         for nv, nt in [(3, 1), (24, 12), (6000, 2000), (300_000, 100_000), (1_002_001, 2_000_000), (100, 200_000)]
         for w, h in [(1, 1), (33, 17), (1920, 1080), (16384, 16384)] for ts in (8, 16, 32) for bins in (0, 5_000_000)]


def reserved(nverts, ntris, w, h, ts, bins):
    """Bytes of the run's buffers for the frame, from their element sizes."""
    tiles = -(-w // ts) * -(-h // ts)
    chunk = min(8192, max(256, (-(-ntris // 900) + 255) // 256 * 256))
    cap = max(bins, 4 * ntris + tiles + 1024)
    return {"vbin": 16 * nverts, "vscr": 16 * nverts, "tri_rect": 8 * ntris, "tri_aux": 4 * ntris,
            "clip_list": 12 * ntris, "counts": 4 * -(-ntris // chunk) * tiles, "tile_start": 4 * tiles,
            "tile_count": 4 * tiles, "tile_order": 6 * 4 * tiles, "bins": 4 * cap, "qbins": 16 * cap * (ts == 32),
            "qcount": 16 * tiles * (ts == 32), "clip_store": 4 * (32 * ntris + 4096), "image": 4 * w * h}


@pytest.fixture(scope="module")
def frame_bytes(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("layout") / "layout")
    subprocess.run(["g++", "-O1", "-std=c++17", "-I", CSRC, os.path.join(HERE, "c", "layout.cpp"), "-o", exe], check=True)

    def run(cases):
        text = "".join(" ".join(str(v) for v in c) + "\n" for c in cases)
        return [int(x) for x in subprocess.run([exe], input=text, capture_output=True, text=True, check=True).stdout.split()]
    return run


def test_charge_covers_what_a_run_reserves(frame_bytes):
    for case, got in zip(CASES, frame_bytes(CASES)):
        need = sum(reserved(*case).values())
        assert need <= got <= need + 65536, (case, need, got)


@pytest.mark.gpu
@pytest.mark.parametrize("tile", [8, 32])
def test_admission_at_the_budget(frame_bytes, tile):
    torch = pytest.importorskip("torch")
    from rusterizer_gb300 import _lib, scenes
    from rusterizer_gb300.batch import BatchRenderer
    from rusterizer_gb300.server import RenderServer
    w, h, n = 1920, 1080, 500
    s = scenes.soup_scene(n, w, h, 4, np.random.default_rng(1), 32)
    br = BatchRenderer()
    br.add_scene(s, tile=tile)
    out = torch.zeros(w * h, dtype=torch.int32, device="cuda")
    size = frame_bytes([(3 * n, n, w, h, tile, 0)])[0]
    srv = RenderServer(br, budget_bytes=size - 1)
    with pytest.raises(_lib.RastError) as e:
        srv.submit(0, out.data_ptr())
    assert e.value.status == _lib.ADMISSION_REFUSED
    srv.close()
    srv = RenderServer(br, budget_bytes=size)
    assert srv.wait(srv.submit(0, out.data_ptr()), timeout_ms=60000)[0] == _lib.OK
    srv.close()
    ref = np.zeros((h, w), np.uint32)
    br.render([ref])
    br.close()
    assert (out.cpu().numpy().view(np.uint32).reshape(h, w) == ref).all()

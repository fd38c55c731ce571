"""Asynchronous mesh updates while asynchronous frames are in flight: an update's copies wait for
the last frame that reads the mesh, whichever of its draws that is, and only the next frame that draws
it waits for them. Frames and updates of three meshes are enqueued without a wait between them, far ahead of the
device, into an image each; every image shows the data that its meshes held when it was enqueued, as the
oracle draws it. (The reference borrows the mesh afresh on every render call, src/render.rs:98-114.)"""
import numpy as np
import pytest

import oracle
from rusterizer_gb300 import renderer, scenes

pytestmark = pytest.mark.gpu

W, H, NTRIS, DATA = 960, 540, 60_000, 6

# ("update", mesh, data) or ("frame", meshes): meshes by name, data by index
CASES = {
    # two meshes in turn, each updated while the frame before reads the other, then without a turn
    "in_turn": ([("update", "a", 0), ("frame", "a"), ("update", "b", 1), ("frame", "b")] +
                [("update", "a", 2), ("frame", "a"), ("update", "b", 3), ("frame", "b")] +
                [("update", "a", 4), ("frame", "a"), ("update", "a", 5), ("frame", "a"), ("update", "a", 0), ("frame", "a")]),
    # a frame of several meshes, each of which is then updated at once
    "several": [("update", "a", 1), ("update", "b", 2), ("frame", "ab"), ("update", "b", 3), ("update", "a", 4),
                ("frame", "ba"), ("frame", "c"), ("update", "a", 5), ("frame", "cab"), ("update", "c", 0),
                ("update", "b", 1), ("frame", "abc"), ("frame", "b")],
    # meshes drawn (the last draw of a frame, and alone) before their first update
    "first": [("frame", "a"), ("update", "a", 3), ("frame", "bc"), ("frame", "a"), ("update", "c", 4), ("update", "b", 5),
              ("frame", "cb"), ("update", "b", 0), ("frame", "a"), ("frame", "b")],
    # two updates with no frame between them, and a frame of another mesh between an update and its frame
    "twice": [("update", "a", 1), ("update", "a", 2), ("frame", "a"), ("update", "a", 3), ("update", "a", 4), ("frame", "b"),
              ("frame", "a"), ("update", "b", 5), ("frame", "a"), ("frame", "b")],
}
START = {"a": 0, "b": 1, "c": 2}


@pytest.fixture(scope="module")
def data():
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(12)
    base = scenes.soup_scene(NTRIS, W, H, 4, rng, 64)
    draws = [scenes.soup(NTRIS, W, H, rng, min_px=1.0, max_px=24.0) for _ in range(DATA)]
    pinned = [[torch.from_numpy(np.ascontiguousarray(d[k]).view(t)).pin_memory()
               for k, t in (("pos", np.float32), ("uv", np.float32), ("idx", np.int32))] for d in draws]
    return base, draws, pinned, {}


def expected(data, held):
    base, draws, _, seen = data
    if held not in seen:
        ds = [dict(draws[k], world=base["draws"][0]["world"], fs=0) for k in held]
        seen[held] = oracle.render_scene(dict(base, draws=ds), nthreads=8)[0]
    return seen[held]


@pytest.mark.parametrize("case", sorted(CASES))
def test_updates_between_frames_in_flight(case, data):
    torch = pytest.importorskip("torch")
    base, draws, pinned, _ = data
    r = renderer.Renderer(W, H, 4)
    r.uniforms().bind_texture(0, renderer.Texture(base["textures"][0]))
    blk = r.uniforms().write_block()
    blk.view, blk.projection, blk.world = base["view"], base["proj"], base["draws"][0]["world"]
    mesh = {n: renderer.Mesh(draws[k]["pos"], draws[k]["uv"], draws[k]["idx"]) for n, k in START.items()}
    steps = CASES[case]
    frames = [s[1] for s in steps if s[0] == "frame"]
    outs = [torch.zeros((H, W), dtype=torch.int32, device="cuda") for _ in frames]

    def draw(names):
        for n in names:
            r.render(mesh[n], renderer.VS_MVP, 0)

    for _ in range(2):  # sizes the context's buffers for every combination of this case
        for names in sorted(set(frames), key=len):
            draw(names)
            r.framebuffer()
    torch.cuda.synchronize()
    held, want, k = dict(START), [], 0
    for s in steps:
        if s[0] == "update":
            r.update_async(mesh[s[1]], pinned[s[2]][0], pinned[s[2]][1], pinned[s[2]][2])
            held[s[1]] = s[2]
        else:
            draw(s[1])
            r.framebuffer_async(outs[k])
            want.append(tuple(held[n] for n in s[1]))
            k += 1
    torch.cuda.synchronize()
    got = [o.cpu().numpy().view(np.uint32) for o in outs]
    r.close()
    for k, w in enumerate(want):
        assert (got[k] == expected(data, w)).all(), (case, k, frames[k], w)
    assert len({g.tobytes() for g in got}) > 1

"""Terrain frames on several streams, from several threads and from a graph
beside direct calls: each launch claims its pixels from its own cursor, so
every frame is the one that it is alone."""
import threading

import pytest
import torch

import rayengine_b200 as rb

pytestmark = pytest.mark.gpu

SIZES = [(320, 180), (64, 36), (300, 170), (17, 33)]


def _frames():
    out = []
    for i, (w, h) in enumerate(SIZES):
        tc = rb.configs.TerrainConfig(seed=50 + i, width=w, height=h)
        out.append((tc.params(), tc.camera(), w, h, rb.sdf_shade_params()))
    return out


def _buffers(frame):
    n = frame[2] * frame[3]
    return (torch.full((n, 8), -1, dtype=torch.int32, device="cuda"),
            torch.full((n,), -1, dtype=torch.int32, device="cuda"))


def _render(frame, hits, rgba, stream=None):
    field, cam, w, h, shade = frame
    rb.render_sdf_frame(field, shade, cam, w, h, hits, rgba, stream=stream)


def _serial(frames):
    want = []
    for f in frames:
        hits, rgba = _buffers(f)
        _render(f, hits, rgba)
        torch.cuda.synchronize()
        want.append((hits, rgba))
    return want


@pytest.mark.parametrize("threads", [False, True])
def test_streams_side_by_side(cuda, threads):
    frames = _frames()
    want = _serial(frames)
    streams = [torch.cuda.Stream() for _ in frames]
    got = [[_buffers(f) for _ in range(6)] for f in frames]
    torch.cuda.synchronize()

    def run(i, k):
        _render(frames[i], *got[i][k], stream=streams[i])

    if threads:
        def work(i):
            for k in range(6):
                run(i, k)

        pool = [threading.Thread(target=work, args=(i,)) for i in range(len(frames))]
        for t in pool:
            t.start()
        for t in pool:
            t.join()
    else:
        for k in range(6):
            for i in range(len(frames)):
                run(i, k)
    torch.cuda.synchronize()
    for i, w in enumerate(want):
        for hits, rgba in got[i]:
            assert torch.equal(hits, w[0]) and torch.equal(rgba, w[1]), SIZES[i]


def test_graph_beside_direct_calls(cuda):
    """Two captured frames, replayed on one stream while the stream that they
    were captured on renders directly."""
    frames = _frames()
    want = _serial(frames)
    capture, other = torch.cuda.Stream(), torch.cuda.Stream()
    graphs, bufs = [], []
    for i in (0, 1):
        b = _buffers(frames[i])
        torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=capture):
            _render(frames[i], *b, stream=capture)
        graphs.append(g)
        bufs.append(b)
    direct = [_buffers(frames[2]) for _ in range(8)]
    torch.cuda.synchronize()
    for d in direct:
        with torch.cuda.stream(other):
            graphs[0].replay()
            graphs[1].replay()
        _render(frames[2], *d, stream=capture)
    torch.cuda.synchronize()
    for i in (0, 1):
        assert torch.equal(bufs[i][0], want[i][0]) and torch.equal(bufs[i][1], want[i][1])
    for hits, rgba in direct:
        assert torch.equal(hits, want[2][0]) and torch.equal(rgba, want[2][1])
    graphs.clear()


def test_more_streams_than_slots(cuda):
    """The cursors of streams that may be gone are used again."""
    frame = _frames()[3]
    want = _serial([frame])[0]
    import ctypes
    rt = ctypes.CDLL("libcudart.so.12")
    hits, rgba = _buffers(frame)
    for _ in range(1100):
        s = ctypes.c_void_p()
        assert rt.cudaStreamCreateWithFlags(ctypes.byref(s), 1) == 0
        _render(frame, hits, rgba, stream=s.value)
        assert rt.cudaStreamDestroy(s) == 0
    torch.cuda.synchronize()
    assert torch.equal(hits, want[0]) and torch.equal(rgba, want[1])


_FIRST = """
import torch
import rayengine_b200 as rb

tc = rb.configs.TerrainConfig(width=64, height=36)
n = 64 * 36
hits = torch.full((n, 8), -1, dtype=torch.int32, device="cuda")
rgba = torch.full((n,), -1, dtype=torch.int32, device="cuda")
shade = rb.sdf_shade_params()
s = torch.cuda.Stream()
torch.cuda.synchronize()
g = torch.cuda.CUDAGraph()
with torch.cuda.graph(g, stream=s):
    rb.render_sdf_frame(tc.params(), shade, tc.camera(), 64, 36, hits, rgba, stream=s)
g.replay()
torch.cuda.synchronize()
want = rb.render_sdf_frame(tc.params(), shade, tc.camera(), 64, 36)
assert torch.equal(rgba, want[0]) and torch.equal(hits, want[1])
for _ in range(40):  # graphs that come and go
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        rb.render_sdf_frame(tc.params(), shade, tc.camera(), 64, 36, hits, rgba, stream=s)
    g.replay()
    del g
torch.cuda.synchronize()
assert torch.equal(rgba, want[0]) and torch.equal(hits, want[1])
print("ok")
"""


def test_first_call_of_a_process_is_captured(cuda):
    import os
    import subprocess
    import sys

    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    out = subprocess.run([sys.executable, "-c", _FIRST], capture_output=True, text=True,
                         timeout=200, cwd=root)
    assert out.returncode == 0 and out.stdout.strip() == "ok", out.stderr[-2000:]

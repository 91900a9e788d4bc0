"""Scenes' memory on the device: scenes destroyed beside another thread's stream
capture, adds that fail, what the pool keeps and gives back, scenes of two
threads.
"""
import ctypes as C
import threading

import numpy as np
import pytest
import torch

from ascent_gb300 import _native as N
from ascent_gb300 import scene as S
from ascent_gb300 import volume as V
from ascent_gb300 import workloads as W

pytestmark = pytest.mark.gpu

GLOBAL, THREAD_LOCAL, RELAXED = 0, 1, 2


class Capture:
    """An (empty) capture of this thread on a stream of its own."""

    def __init__(self, mode):
        self.cu = C.CDLL("libcuda.so.1")
        self.stream = C.c_void_p()
        torch.cuda.current_stream().synchronize()
        assert self.cu.cuStreamCreate(C.byref(self.stream), 1) == 0
        assert self.cu.cuStreamBeginCapture_v2(self.stream, mode) == 0

    def end(self):
        """Whether the capture was left whole."""
        graph = C.c_void_p()
        rc = self.cu.cuStreamEndCapture(self.stream, C.byref(graph))
        if graph:
            self.cu.cuGraphDestroy(graph)
        self.cu.cuStreamDestroy_v2(self.stream)
        return rc == 0


def in_thread(fn):
    out = []
    t = threading.Thread(target=lambda: out.append(fn()))
    t.start()
    t.join()
    return out[0]


def free_bytes():
    torch.cuda.synchronize()
    N.scratch_trim(0, 0)
    return torch.cuda.mem_get_info(0)[0]


def make(wl):
    sc = S.Scene(0)
    V.load_workload(sc, wl)
    return sc


def two_domains():
    """More bytes than the blocks a pool takes from the system; rendered and
    captured once, so that everything that is made at first use is there."""
    wl = W.plain_small(n=224, width=96, height=80, parts=(2, 1, 1))
    cam, p = V.workload_camera(wl), V.workload_params(wl)
    sc = make(wl)
    sc.render(cam, p)
    sc.close()
    assert Capture(THREAD_LOCAL).end()
    torch.zeros(1, device="cuda")
    return wl, cam, p, free_bytes()


@pytest.mark.parametrize("mode", [THREAD_LOCAL, RELAXED])
def test_destroy_beside_capture(mode):
    wl, cam, p, before = two_domains()
    a, b = make(wl), make(wl)
    image = a.render(cam, p)[0]
    cap = Capture(mode)
    in_thread(a.close)
    assert cap.end()
    assert np.array_equal(b.render(cam, p)[0], image)
    b.close()
    assert free_bytes() == before


def test_destroy_beside_refusing_capture():
    """A capture in global mode refuses the wait of every thread: the scene's
    memory is left to a later one and no error stays behind."""
    wl, cam, p, before = two_domains()
    a, b = make(wl), make(wl)
    image = a.render(cam, p)[0]
    cap = Capture(GLOBAL)
    in_thread(a.close)
    cap.end()
    assert np.array_equal(b.render(cam, p)[0], image)
    b.close()
    assert free_bytes() == before


def crowded_mesh(n=3000):
    """n hexahedra around one node: too many for a bucket, so the faces are sorted."""
    a = np.linspace(0.0, 2.0 * np.pi, n + 1)[:-1]
    ring = lambda r, z: np.stack([r * np.cos(a), r * np.sin(a), np.full(n, z)], 1)
    pts = np.concatenate([[[0, 0, 0], [0, 0, 1]], ring(0.5, 0.0), ring(0.5, 1.0), ring(1.0, 0.0), ring(1.0, 1.0)])
    i = np.arange(n)
    j = (i + 1) % n
    node = lambda k, q: 2 + k * n + q
    conn = np.stack([np.zeros(n, int), node(0, i), node(2, i), node(0, j),
                     np.ones(n, int), node(1, i), node(3, i), node(1, j)], 1)
    return pts, conn


def hex_scene(pts, conn):
    sc = S.Scene(0)
    sc.add_hex(*[np.ascontiguousarray(pts[:, k]) for k in range(3)], conn, pts[:, 2] + pts[:, 0])
    return sc


def test_failed_adds_give_their_memory_back():
    """Refused fields and meshes leave nothing behind, and the scene as it was."""
    pts, conn = crowded_mesh()
    hex_scene(pts, conn).close()
    wl, cam, p, before = two_domains()
    sc = make(wl)
    image = sc.render(cam, p)[0]
    n = 160
    bad = np.zeros((n, n, n), np.float32)
    bad[-1, -1, -1] = np.nan
    missing = conn.copy()
    missing[-1, -1] = len(pts)
    for _ in range(3):
        for assoc in (N.ASSOC_VERTEX, N.ASSOC_ELEMENT):
            with pytest.raises(N.GvrError):
                sc.add_uniform(bad, (0, 0, 0), (1, 1, 1), association=assoc)
            with pytest.raises(N.GvrError):
                grid = [np.linspace(0.0, 1.0, n + (assoc == N.ASSOC_ELEMENT))] * 3
                sc.add_rectilinear(bad, *grid, association=assoc)
        with pytest.raises(N.GvrError):
            sc.add_hex(*[np.ascontiguousarray(pts[:, k]) for k in range(3)], missing, pts[:, 2])
        hex_scene(pts, conn).close()
    assert np.array_equal(sc.render(cam, p)[0], image)
    sc.close()
    assert free_bytes() == before


def available():
    return torch.cuda.mem_get_info(0)[0]


def test_pool_is_bounded_and_given_back():
    """Scenes that come and go take the same memory again; at most 4 GiB stay
    reserved when one is gone, and a trim gives that back too, with no wait in
    between."""
    wl, cam, p, before = two_domains()
    scenes = []
    for _ in range(6):
        sc = make(wl)
        sc.render(cam, p)
        sc.close()
        scenes.append(before - available())
    assert scenes[0] > 0 and max(scenes) == scenes[0], scenes
    cells = torch.zeros((1300, 1100, 1100), device="cuda")      # 6.3 GB
    held = available()
    with S.Scene(0) as sc:
        sc.add_uniform(cells, (0, 0, 0), (1, 1, 1), association=N.ASSOC_ELEMENT)
        assert held - available() > 5 << 30
    assert held + scenes[0] - available() <= (4 << 30) + (64 << 20)
    N.scratch_trim(0, 0)
    assert available() == held + scenes[0]
    del cells
    torch.cuda.empty_cache()


def test_scenes_of_two_threads():
    """Threads that make, render and destroy scenes get their own images."""
    wls = [W.plain_small(n=n, width=96, height=80, parts=(2, 1, 1)) for n in (40, 72)]

    def images(wl, turns):
        cam, p = V.workload_camera(wl), V.workload_params(wl)
        out = []
        for _ in range(turns):
            sc = make(wl)
            out.append(sc.render(cam, p)[0])
            sc.close()
        return out

    want = [images(wl, 1)[0] for wl in wls]
    got = [None, None]

    def work(k):
        got[k] = images(wls[k], 25)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for k in range(2):
        assert all(np.array_equal(g, want[k]) for g in got[k])

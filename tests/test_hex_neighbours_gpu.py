"""The face-neighbour table against a numpy restatement of its rule (faces
ordered by their three smallest node ids, then by number; each takes the cell of
the next face with its triple, else of the one before), bit for bit: one cell,
grids whose faces fill odd numbers of blocks, shuffled node numbers and cells,
triples shared by more than two faces, and nodes with fewer and more faces than
a bucket may hold (256), where the table is sorted instead.
"""
import numpy as np
import pytest

from ascent_gb300 import scene as S
from ascent_gb300 import workloads as W

pytestmark = pytest.mark.gpu

FACES = np.array([[0, 3, 7, 4], [1, 2, 6, 5], [0, 1, 5, 4], [3, 2, 6, 7], [0, 1, 2, 3], [4, 5, 6, 7]])


def neighbours(conn):
    t = np.sort(conn[:, FACES].reshape(-1, 4), axis=1)[:, :3]
    order = np.lexsort((np.arange(len(t)), t[:, 2], t[:, 1], t[:, 0]))
    s = t[order]
    same = np.concatenate([(s[1:] == s[:-1]).all(axis=1), [False]])
    out = np.full(len(t), -1, np.int64)
    before = np.concatenate([[False], same[:-1]])
    out[order[1:]] = np.where(before[1:], order[:-1] // 6, -1)
    out[order[:-1]] = np.where(same[:-1], order[1:] // 6, out[order[:-1]])
    return out.reshape(-1, 6)


def grid(n, rng, shuffle):
    m = n + 1
    g = np.arange(m) / n
    z, y, x = np.meshgrid(g, g, g, indexing="ij")
    pts = np.stack([x.ravel(), y.ravel(), z.ravel()], 1)
    conn = W.hex_grid_connectivity(n)
    if shuffle:
        perm = rng.permutation(len(pts))
        moved = np.empty_like(pts)
        moved[perm] = pts
        pts, conn = moved, perm[conn].astype(np.int32)[rng.permutation(len(conn))]
    return pts, np.ascontiguousarray(conn)


def check(pts, conn):
    x, y, z = (np.ascontiguousarray(pts[:, a], dtype=np.float32) for a in range(3))
    with S.Scene(0) as sc:
        did = sc.add_hex(x, y, z, conn, np.ascontiguousarray(x + y))
        got, _ = sc.hex_neighbors(did)
    np.testing.assert_array_equal(got, neighbours(conn))


@pytest.mark.parametrize("n", [1, 2, 7, 11, 24])
@pytest.mark.parametrize("shuffle", [False, True])
def test_grids(n, shuffle):
    check(*grid(n, np.random.default_rng(n), shuffle))


def test_triples_of_many_faces():
    pts, conn = grid(4, np.random.default_rng(1), True)
    check(pts, np.ascontiguousarray(np.concatenate([conn, conn[5:9], conn[5:7]])))


@pytest.mark.parametrize("cells", [40, 85, 86, 300])
def test_crowded_node(cells):
    """Every cell holds node 0, in three of its faces: 85 cells are 255 faces in
    its bucket, 86 are 258."""
    rng = np.random.default_rng(cells)
    pts = rng.uniform(0, 1, (60, 3))
    conn = np.stack([np.concatenate([[0], 1 + rng.permutation(59)[:7]]) for _ in range(cells)]).astype(np.int32)
    check(pts, conn)


@pytest.mark.parametrize("cells", [2, 3, 255, 256, 257, 511, 1000, 3000])
def test_refit(cells):
    """The tree's boxes, whose nodes are joined in shared memory where their
    leaves belong to one block of 256, against boxes joined from the leaves up
    in numpy; and every point at a cell's middle is found through them."""
    rng = np.random.default_rng(cells)
    pts, conn = grid(int(np.ceil(cells ** (1 / 3))), rng, True)
    conn = np.ascontiguousarray(conn[:cells])
    x, y, z = (np.ascontiguousarray(pts[:, a], dtype=np.float32) for a in range(3))
    with S.Scene(0) as sc:
        did = sc.add_hex(x, y, z, conn, x)
        t = sc.hex_bvh(did)
        mid = np.stack([v[conn].mean(axis=1) for v in (x, y, z)], 1)
        found, _ = sc.hex_locate(did, mid)
    np.testing.assert_array_equal(found, np.arange(cells))
    xyz = np.stack([x, y, z], 1)
    n_inner = cells - 1
    box = np.zeros((2 * cells - 1, 6), np.float32)
    box[n_inner:, :3] = xyz[conn[t["ids"]]].min(axis=1)
    box[n_inner:, 3:] = xyz[conn[t["ids"]]].max(axis=1)
    done = np.zeros(2 * cells - 1, bool)
    done[n_inner:] = True
    while not done.all():
        for i in np.nonzero(~done)[0]:
            l, r = t["left"][i], t["right"][i]
            if done[l] and done[r]:
                box[i, :3], box[i, 3:] = np.minimum(box[l, :3], box[r, :3]), np.maximum(box[l, 3:], box[r, 3:])
                done[i] = True
    np.testing.assert_array_equal(t["inner_box"][:n_inner], box[:n_inner])

"""What a volume-plot user has the renderer do, as cases to be timed.

Every case is one call, or one in-situ step, through the package's public entry
points: frames of structured and hexahedral scenes, Cinema sweeps, field
publishes followed by a frame, new meshes followed by a frame, compositing of
partials and of opaque canvases, and a training step of the differentiable
render. `exact` restates each computed image or gradient in float64 with plain
torch, from the stepping rule alone.
"""
import math

import numpy as np
import torch

from ascent_gb300 import _native as N
from ascent_gb300 import compositing as CP
from ascent_gb300 import diff as D
from ascent_gb300 import scene as S
from ascent_gb300 import volume as V

FOV = 30.0
CULL, EARLY = 0.001, 0.99


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------

def listed():
    return [
        # a thumbnail of a small single-task run: latency and launches are all there is
        frame("thumbnail", (32, 28, 40), (1, 1, 1), 160, 120, 96, "ramp", field="noise"),
        # one task's 64^3 grid at the usual window size, half-cell samples
        frame("plain64", (63, 63, 63), (1, 1, 1), 512, 512, 218, "ramp", field="noise"),
        # the headline view: 512^3 cells in 8 domains, half-cell samples, float LUT
        frame("plain512", (512, 512, 512), (2, 2, 2), 1024, 1024, 1774, "ramp", field="turbulence"),
        # a stretched rectilinear grid of odd extents at a ragged window
        frame("rectilinear", (241, 199, 173), (1, 1, 1), 901, 677, 640, "ramp", mesh="rectilinear"),
        # a mixed scene: opaque surfaces Z-composited, then a cell-centred field over them
        {"name": "element_over_surfaces", "kind": "over", "nx": 160, "ny": 144, "nz": 121, "px": 2, "py": 2,
         "pz": 1, "mesh": "uniform", "assoc": "element", "field": "blobs", "tf": "ramp", "lut8": False,
         "width": 1280, "height": 720, "samples": 420, "az": 30.0, "el": 20.0, "canvases": 3},
        # 8M hexahedra with moved nodes, half-cell samples
        {"name": "hex200", "kind": "hex", "nx": 200, "ny": 200, "nz": 200, "width": 1024, "height": 1024,
         "samples": 693, "tf": "ramp", "az": 30.0, "el": 20.0, "assoc": "vertex", "new_mesh": False},
        # a Cinema database: 8 x 8 views of 37 uneven domains in one call
        {"name": "cinema64", "kind": "cinema", "cells": 256, "domains": 37, "views_phi": 8, "views_theta": 8,
         "width": 512, "height": 512, "samples": 887, "tf": "ramp"},
        # one in-situ step of a GPU code: 8 resident float32 fields published, a frame at the
        # default number of samples with a transfer function that hides the low values
        {"name": "step_device", "kind": "step", "nx": 512, "ny": 512, "nz": 512, "px": 2, "py": 2, "pz": 2,
         "mesh": "uniform", "assoc": "vertex", "dtype": "float32", "host": False, "field": "turbulence",
         "tf": "hidden", "lut8": True, "width": 1024, "height": 1024, "samples": 100, "az": 30.0, "el": 20.0},
        # one in-situ step of a CPU code as the front end takes it: new scene, float64 host
        # arrays of odd extents, a frame back to the host
        {"name": "step_host", "kind": "step", "nx": 185, "ny": 151, "nz": 97, "px": 2, "py": 2, "pz": 1,
         "mesh": "uniform", "assoc": "vertex", "dtype": "float64", "host": True, "field": "blobs",
         "tf": "hidden", "lut8": True, "width": 800, "height": 600, "samples": 100, "az": 40.0, "el": 25.0},
        # one in-situ step of an unstructured GPU code whose mesh changes: 1M new hexahedra, a frame
        {"name": "step_hex", "kind": "hex", "nx": 100, "ny": 100, "nz": 100, "width": 512, "height": 512,
         "samples": 100, "tf": "hidden", "az": 30.0, "el": 20.0, "assoc": "vertex", "new_mesh": True},
        # the partials of 8 ranks at 1024^2, 80% covered, pixel range known
        {"name": "partials", "kind": "partials", "images": 8, "width": 1024, "height": 1024, "cover": 0.8,
         "known_range": True},
        # a training step: 128^3 field and 256-entry transfer function, 16 views at 256^2
        {"name": "train", "kind": "train", "n": 128, "views": 16, "width": 256, "height": 256, "lut": 256,
         "samples": 440},
    ]


def frame(name, cells, parts, width, height, samples, tf, mesh="uniform", assoc="vertex", field="blobs",
          lut8=False, az=30.0, el=20.0):
    return {"name": name, "kind": "frame", "nx": cells[0], "ny": cells[1], "nz": cells[2], "px": parts[0],
            "py": parts[1], "pz": parts[2], "mesh": mesh, "assoc": assoc, "field": field, "tf": tf, "lut8": lut8,
            "width": width, "height": height, "samples": samples, "az": az, "el": el}


def draw(rng):
    def log(a, b):
        return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))

    kind = rng.choice(["frame", "frame", "frame", "over", "hex", "cinema", "step", "step", "hexstep", "partials",
                       "train"])
    az, el = round(rng.uniform(-180.0, 180.0), 1), round(rng.uniform(-70.0, 70.0), 1)
    view = {"width": log(120, 1100), "height": log(100, 1000), "az": az, "el": el}
    if kind in ("frame", "over", "step"):
        host = kind == "step" and rng.random() < 0.4
        top = 220 if host else 420
        cells = {a: log(24, top) for a in ("nx", "ny", "nz")}
        if rng.random() < 0.35:
            parts = {"px": 1, "py": 1, "pz": 1}
        else:
            parts = {a: rng.randint(1, 3) for a in ("px", "py", "pz")}
        single = parts["px"] * parts["py"] * parts["pz"] == 1
        coarse = kind == "step" or rng.random() < 0.3
        samples = log(60, 200) if coarse else int(1.0 + 2.0 * math.sqrt(sum(c * c for c in cells.values())))
        c = {"kind": kind, **cells, **parts, **view, "samples": samples,
             "mesh": "rectilinear" if rng.random() < 0.3 else "uniform",
             "assoc": "element" if rng.random() < (0.6 if kind == "over" else 0.25) else "vertex",
             "field": rng.choice(["blobs", "turbulence", "noise"]), "tf": rng.choice(["ramp", "hidden"]),
             "lut8": coarse and not single}
        if kind == "over":
            c["canvases"] = rng.randint(1, 6)
        if kind == "step":
            c["dtype"] = rng.choice(["float32", "float64"])
            c["host"] = host
        return c
    if kind in ("hex", "hexstep"):
        n = {a: log(12, 150) for a in ("nx", "ny", "nz")}
        fine = kind == "hex"
        samples = int(1.0 + 2.0 * math.sqrt(sum(c * c for c in n.values()))) if fine else log(60, 200)
        return {"kind": "hex", **n, **view, "samples": samples, "tf": rng.choice(["ramp", "hidden"]),
                "assoc": "element" if rng.random() < 0.25 else "vertex", "new_mesh": not fine}
    if kind == "cinema":
        cells = rng.choice([96, 128, 192, 256])
        return {"kind": "cinema", "cells": cells, "domains": rng.randint(2, 8) if cells < 192 else rng.randint(4, 37),
                "views_phi": rng.randint(2, 8), "views_theta": rng.randint(1, 7), "width": log(100, 512),
                "height": log(100, 512), "samples": int(math.sqrt(3.0) * cells * 2) + 1,
                "tf": rng.choice(["ramp", "hidden"])}
    if kind == "partials":
        return {"kind": "partials", "images": log(1, 12), "width": log(64, 1024), "height": log(64, 1024),
                "cover": round(rng.uniform(0.05, 0.95), 3), "known_range": rng.random() < 0.5}
    n = log(24, 120)
    return {"kind": "train", "n": n, "views": log(1, 16), "width": log(48, 256), "height": log(48, 256),
            "lut": log(32, 512), "samples": int(math.sqrt(3.0) * n * 2)}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------

def transfer_function(name):
    if name == "ramp":     # 256 points, colour (x, .5, 1 - x), opacity 0 -> 0.3
        x = np.linspace(0.0, 1.0, 256)
        return x, np.stack([x, np.full_like(x, 0.5), 1.0 - x], axis=1), x.copy(), 0.3 * x
    # five colours, nothing below a fifth of the range
    return (np.array([0.0, 0.25, 0.5, 0.75, 1.0]),
            np.array([[0.2, 0.25, 0.6], [0.3, 0.7, 0.8], [0.9, 0.9, 0.6], [0.95, 0.6, 0.2], [0.7, 0.1, 0.1]]),
            np.array([0.0, 0.2, 0.6, 1.0]), np.array([0.0, 0.0, 0.35, 0.8]))


def cuts(n, p):
    return [round(i * n / p) for i in range(p + 1)]


def boxes_of(c):
    """The domains of a structured case, each as (x0, y0, z0, x1, y1, z1) in cells of the whole grid."""
    if c["kind"] == "cinema":
        rng = np.random.default_rng(c["domains"] * 1000 + c["cells"])
        edges = [e for e in (8, 16, 24, 32, 48, 64, 96, 128, 160, 192, 224) if e < c["cells"]]
        boxes = [(0, 0, 0) + (c["cells"],) * 3]
        while len(boxes) < c["domains"]:
            for i in sorted(range(len(boxes)), key=lambda j: -np.prod([boxes[j][3 + a] - boxes[j][a] for a in range(3)])):
                b = boxes[i]
                a = int(rng.integers(3))
                fit = [e for e in edges if e < b[3 + a] - b[a]]
                if fit:
                    e = int(rng.choice(fit))
                    boxes[i:i + 1] = [b[:3 + a] + (b[a] + e,) + b[4 + a:], b[:a] + (b[a] + e,) + b[a + 1:]]
                    break
        return boxes
    xs, ys, zs = cuts(c["nx"], c["px"]), cuts(c["ny"], c["py"]), cuts(c["nz"], c["pz"])
    return [(xs[i], ys[j], zs[k], xs[i + 1], ys[j + 1], zs[k + 1])
            for k in range(c["pz"]) for j in range(c["py"]) for i in range(c["px"])]


def blobs(x, y, z, rng):
    """Eight separable Gaussians on the grid x, y, z: float32 (nz, ny, nx)."""
    centre, sigma, amp = rng.uniform(0.2, 0.8, (8, 3)), rng.uniform(0.05, 0.15, 8), rng.uniform(0.5, 1.0, 8)
    f = torch.zeros((len(z), len(y), len(x)), dtype=torch.float32, device="cuda")
    for c, s, a in zip(centre, sigma, amp):
        gx, gy, gz = (torch.exp(-((v - float(m)) ** 2) / (2 * s * s)).float() for v, m in zip((x, y, z), c))
        f += (float(a) * gz)[:, None, None] * (gy[:, None] * gx[None, :])
    return f


def structured(c, seed):
    """The grid of a structured case: spacing, coordinates and the whole field on the GPU."""
    rng = np.random.default_rng([seed, 1])
    cells = (c["cells"],) * 3 if c["kind"] == "cinema" else (c["nx"], c["ny"], c["nz"])
    h = 1.0 / max(cells)
    coords = [np.arange(n + 1) * h for n in cells]
    if c.get("mesh") == "rectilinear":   # stretched, and uneven from cell to cell
        for a in range(3):
            w = 1.0 + 0.6 * np.sin(np.linspace(0.0, 3.0, cells[a]) + a) + rng.uniform(-0.2, 0.2, cells[a])
            coords[a] = np.concatenate([[0.0], np.cumsum(w)]) * (cells[a] * h / w.sum())
    at = [torch.from_numpy(v).cuda() for v in coords]
    if c.get("assoc") == "element":
        at = [0.5 * (v[1:] + v[:-1]) for v in at]
    f = blobs(*at, rng)
    if c.get("field") == "turbulence":
        for o in range(3):
            ph, k = rng.uniform(0.0, 1.0, 3), 4.0 * math.pi * 2 ** o
            sx, sy, sz = (torch.sin(k * (v + float(q))).float() for v, q in zip(at, ph))
            f += (0.2 * 0.5 ** o * sz)[:, None, None] * (sy[:, None] * sx[None, :])
    elif c.get("field") == "noise":
        g = torch.Generator(device="cuda").manual_seed(seed)
        f += 0.01 * torch.randn(f.shape, generator=g, device="cuda")
    return h, coords, f


def parts_of(c, coords, f, h):
    """(field, box, origin, axes) of every domain."""
    cell = 1 if c.get("assoc") == "element" else 0
    out = []
    for b in boxes_of(c):
        sub = f[b[2]:b[5] + 1 - cell, b[1]:b[4] + 1 - cell, b[0]:b[3] + 1 - cell].contiguous()
        out.append((sub, b, (b[0] * h, b[1] * h, b[2] * h), [coords[a][b[a]:b[3 + a] + 1] for a in range(3)]))
    return out


def hexahedra(c, seed):
    """Nodes moved by up to a fifth of a cell, connectivity, and a field: GPU tensors."""
    rng = np.random.default_rng([seed, 2])
    n = (c["nx"], c["ny"], c["nz"])
    h = 1.0 / max(n)
    gen = torch.Generator(device="cuda").manual_seed(seed)
    z, y, x = torch.meshgrid(*[torch.arange(n[a] + 1, device="cuda", dtype=torch.float64) * h for a in (2, 1, 0)],
                             indexing="ij")
    pts = [(p + 0.4 * h * (torch.rand(p.shape, generator=gen, device="cuda", dtype=torch.float64) - 0.5)).float()
           for p in (x, y, z)]
    centre, sigma, amp = rng.uniform(0.2, 0.8, (8, 3)), rng.uniform(0.05, 0.15, 8), rng.uniform(0.5, 1.0, 8)
    f = torch.zeros_like(pts[0])
    for m, s, a in zip(centre, sigma, amp):
        f += float(a) * torch.exp(-sum((p - float(q)) ** 2 for p, q in zip(pts, m)) / (2 * s * s))
    m0, m1 = n[0] + 1, (n[0] + 1) * (n[1] + 1)
    k, j, i = torch.meshgrid(*[torch.arange(n[a], device="cuda") for a in (2, 1, 0)], indexing="ij")
    base = (k * m1 + j * m0 + i).reshape(-1, 1)
    off = torch.tensor([0, 1, m0 + 1, m0, m1, m1 + 1, m1 + m0 + 1, m1 + m0], device="cuda")
    if c["assoc"] == "element":
        f = 0.125 * sum(f[dz:n[2] + dz, dy:n[1] + dy, dx:n[0] + dx] for dz in (0, 1) for dy in (0, 1) for dx in (0, 1))
    return [p.reshape(-1) for p in pts], (base + off).int(), f.reshape(-1).contiguous()


def eye_of(bounds, az, el):
    """Camera position, target and up of a view that holds the bounds."""
    b = np.asarray(bounds, dtype=np.float64)
    mid, diag = 0.5 * (b[0::2] + b[1::2]), float(np.linalg.norm(b[1::2] - b[0::2]))
    dist = 0.5 * diag / math.tan(math.radians(0.5 * FOV))
    a, e = math.radians(az), math.radians(el)
    pos = mid + dist * np.array([math.sin(a) * math.cos(e), math.sin(e), math.cos(a) * math.cos(e)])
    return {"pos": pos.astype(np.float32), "at": mid.astype(np.float32), "up": np.array([0, 1, 0], np.float32),
            "near": np.float32(0.01 * diag), "far": np.float32(100 * diag)}


def orbit(bounds, n_phi, n_theta):
    """The cameras of a Cinema sweep."""
    b = np.asarray(bounds, dtype=np.float64)
    mid, diag = 0.5 * (b[0::2] + b[1::2]), float(np.linalg.norm(b[1::2] - b[0::2]))
    out = []
    for i in range(n_phi):
        for j in range(n_theta):
            p, t = math.radians(-180.0 + i * 360.0 / n_phi), math.radians(3.0 + j * 180.0 / n_theta)
            up = np.array([-math.sin(p) * math.cos(t), math.cos(p) * math.cos(t), math.sin(t)])
            pos = mid + 1.25 * diag * np.array([math.sin(p) * math.sin(t), -math.cos(p) * math.sin(t), math.cos(t)])
            out.append({"pos": pos.astype(np.float32), "at": mid.astype(np.float32), "up": up.astype(np.float32),
                        "near": np.float32(0.01 * diag), "far": np.float32(100 * diag)})
    return out


def camera(eye):
    c = N.Camera()
    for a in range(3):
        c.position[a], c.look_at[a], c.up[a] = float(eye["pos"][a]), float(eye["at"][a]), float(eye["up"][a])
    c.fov_y, c.zoom, c.near_plane, c.far_plane = FOV, 1.0, float(eye["near"]), float(eye["far"])
    return c


def plot(c, bounds, data_range, single):
    """Render parameters of the case's plot, as the front end sets them up."""
    vr = V.VolumeRenderer()
    vr.set_num_samples(c["samples"])
    vr.set_color_table(V.TransferFunction(*transfer_function(c["tf"])))
    return vr.params(c["width"], c["height"], bounds, data_range, single,
                     lut=None if c.get("lut8") or single else vr.lut(True))


def add_parts(sc, c, parts, h):
    assoc = N.ASSOC_ELEMENT if c.get("assoc") == "element" else N.ASSOC_VERTEX
    for f, _, origin, axes in parts:
        if c.get("mesh") == "rectilinear":
            sc.add_rectilinear(f, *axes, association=assoc)
        else:
            sc.add_uniform(f, origin, (h, h, h), association=assoc)


def canvases(c, seed):
    """Opaque surface renders: spheres in front of and behind the volume's middle."""
    rng = np.random.default_rng([seed, 3])
    y, x = torch.meshgrid(torch.linspace(-1, 1, c["height"], device="cuda"),
                          torch.linspace(-1, 1, c["width"], device="cuda"), indexing="ij")
    cols, deps = [], []
    for _ in range(c["canvases"]):
        u, v, r = rng.uniform(-0.5, 0.5), rng.uniform(-0.5, 0.5), rng.uniform(0.2, 0.5)
        d2 = 1.0 - ((x - float(u)) ** 2 + (y - float(v)) ** 2) / float(r * r)
        hit = d2 > 0
        shade = torch.where(hit, torch.sqrt(d2.clamp_min(0)), torch.zeros_like(d2))
        rgb = torch.tensor(rng.uniform(0.2, 1.0, 3), device="cuda", dtype=torch.float32)
        cols.append(torch.cat([shade[..., None] * rgb, hit[..., None].float()], dim=-1).contiguous())
        # image depths of distances around the volume's middle
        far = float(rng.uniform(0.994, 0.9965))
        deps.append(torch.where(hit, far - 0.001 * shade, torch.ones_like(shade)).contiguous())
    return cols, deps


def partials(c, seed):
    """One record per covered pixel of every image: (n, 6) int32 with the floats' bits. Which pixels
    an image covers is the case's, what it holds there the seed's."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    px = c["width"] * c["height"]
    cover = torch.Generator(device="cuda").manual_seed(px + c["images"])
    out = []
    for _ in range(c["images"]):
        pid = torch.nonzero(torch.rand(px, generator=cover, device="cuda") < c["cover"]).reshape(-1).int()
        a = torch.rand(len(pid), generator=g, device="cuda") * 0.9 + 0.01
        rgb = torch.rand((len(pid), 3), generator=g, device="cuda") * a[:, None]
        dep = torch.rand(len(pid), generator=g, device="cuda") * 4.0 + 1.0
        out.append(torch.cat([pid[:, None], torch.cat([dep[:, None], rgb, a[:, None]], 1).contiguous().view(torch.int32)], 1))
    return torch.cat(out).contiguous()


def train_inputs(c, seed):
    """Field, transfer function, cameras and target images of a training step."""
    n, rng = c["n"], np.random.default_rng([seed, 4])
    v = torch.linspace(0.0, 1.0, n, dtype=torch.float64, device="cuda")
    f = blobs(v, v, v, rng)
    lo, hi = float(f.min()), float(f.max())
    x = np.linspace(0.0, 1.0, c["lut"])
    lut = torch.from_numpy(np.stack([x, np.full_like(x, 0.5), 1.0 - x, 1.0 - (1.0 - 0.3 * x) ** (10.0 / c["samples"])],
                                    1).astype(np.float32)).cuda()
    h = 1.0 / (n - 1)
    bounds = np.array([0.0, np.float32((n - 1) * float(np.float32(h)))] * 3)
    phi = max(1, int(math.sqrt(c["views"])))
    eyes = orbit(bounds, phi, -(-c["views"] // phi))[:c["views"]]
    dt = float(np.float32(np.linalg.norm(bounds[1::2] - bounds[0::2]) / c["samples"]))
    g = torch.Generator(device="cuda").manual_seed(seed)
    noisy = f + 0.05 * torch.randn(f.shape, generator=g, device="cuda")
    target, _ = train_forward(noisy, lut, eyes, c, h, dt, (lo, hi), torch.float32)
    return f, lut, eyes, h, dt, (lo, hi), target


# ---------------------------------------------------------------------------
# prepare and run
# ---------------------------------------------------------------------------

def prepare(case, seed):
    c = case
    st = {"case": c}
    if c["kind"] == "partials":
        p = partials(c, seed)
        st.update(p=p, lo=0, hi=c["width"] * c["height"] - 1)
        if c["known_range"]:
            st.update(out=torch.zeros_like(p), n=torch.zeros(1, dtype=torch.int64, device="cuda"))
        return st
    if c["kind"] == "train":
        f, lut, eyes, h, dt, rng, target = train_inputs(c, seed)
        st.update(f=f.requires_grad_(True), lut=lut.requires_grad_(True), cams=[camera(e) for e in eyes], h=h, dt=dt,
                  range=rng, target=target)
        return st
    if c["kind"] == "hex":
        pts, conn, f = hexahedra(c, seed)
        if c["new_mesh"]:
            st.update(pts=pts, conn=conn, f=f)
            return st
        sc = S.Scene(0)
        sc.add_hex(*pts, conn, f, association=N.ASSOC_ELEMENT if c["assoc"] == "element" else N.ASSOC_VERTEX)
        b = sc.bounds()
        st.update(sc=sc, cam=camera(eye_of(b, c["az"], c["el"])), p=plot(c, b, sc.scalar_range(), False))
        return st
    h, coords, f = structured(c, seed)
    parts = parts_of(c, coords, f, h)
    del f
    if c["kind"] == "step":
        t = torch.float64 if c["dtype"] == "float64" else torch.float32
        parts = [(p[0].to(t).cpu().numpy() if c["host"] else p[0].to(t),) + p[1:] for p in parts]
        if c["host"]:
            st.update(parts=parts, h=h)
            return st
    sc = S.Scene(0)
    add_parts(sc, c, parts, h)
    b = sc.bounds()
    single = len(parts) == 1
    st.update(sc=sc, p=plot(c, b, sc.scalar_range(), single))
    if c["kind"] == "cinema":
        st["cams"] = [camera(e) for e in orbit(b, c["views_phi"], c["views_theta"])]
    else:
        st["cam"] = camera(eye_of(b, c["az"], c["el"]))
    if c["kind"] == "step":
        st.update(fields=[p[0] for p in parts], bounds=b)
    if c["kind"] == "over":
        st["cols"], st["deps"] = canvases(c, seed)
    return st


def run(state):
    c = state["case"]
    if c["kind"] == "frame":
        return state["sc"].render(state["cam"], state["p"], device_out=True)
    if c["kind"] == "cinema":
        return state["sc"].render_batch(state["cams"], state["p"], device_out=True)
    if c["kind"] == "over":
        rgba, depth = CP.zbuffer_composite(state["cols"], state["deps"])
        return state["sc"].render_over(state["cam"], state["p"], rgba, depth)
    if c["kind"] == "partials":
        if c["known_range"]:
            return CP.composite_partials_device_async(state["p"], state["lo"], state["hi"], out=state["out"],
                                                      n_out=state["n"])
        return CP.composite_partials_device(state["p"])
    if c["kind"] == "train":
        f, lut = state["f"], state["lut"]
        img = D.render(f, lut, state["cams"], (0.0, 0.0, 0.0), (state["h"],) * 3, c["width"], c["height"],
                       state["dt"], state["range"])
        loss = (img - state["target"]).square().sum()
        gf, gl = torch.autograd.grad(loss, (f, lut))
        return img.detach(), gf, gl
    if c["kind"] == "hex":
        if not c["new_mesh"]:
            return state["sc"].render(state["cam"], state["p"], device_out=True)
        with S.Scene(0) as sc:
            sc.add_hex(*state["pts"], state["conn"], state["f"],
                       association=N.ASSOC_ELEMENT if c["assoc"] == "element" else N.ASSOC_VERTEX)
            b = sc.bounds()
            return sc.render(camera(eye_of(b, c["az"], c["el"])), plot(c, b, sc.scalar_range(), False),
                             device_out=True)
    if c["host"]:
        with S.Scene(0) as sc:
            add_parts(sc, c, state["parts"], state["h"])
            b = sc.bounds()
            return sc.render(camera(eye_of(b, c["az"], c["el"])),
                             plot(c, b, sc.scalar_range(), len(state["parts"]) == 1))
    sc = state["sc"]
    sc.update_fields(range(len(state["fields"])), state["fields"], stream=torch.cuda.current_stream())
    lo, hi = sc.scalar_range()
    p = state["p"]
    p.scalar_min, p.scalar_max = float(lo), float(hi)
    return sc.render(state["cam"], p, device_out=True) + (float(lo), float(hi))


def work(case):
    """Every input value read once and every output value written once; about 40 operations a structured
    sample and 200 a hexahedral one, over the samples of a view of the whole box."""
    c = case
    if c["kind"] == "partials":
        n, px = c["images"] * c["width"] * c["height"] * c["cover"], c["width"] * c["height"]
        return {"bytes": 24 * n + 24 * px * (1 - (1 - c["cover"]) ** c["images"]), "flops": 8 * n}
    if c["kind"] == "train":
        px, nf = c["views"] * c["width"] * c["height"], c["n"] ** 3
        # orbit() stands 1.25 diagonals away: the box covers this many samples
        s = samples_of((1.0, 1.0, 1.0), 1.25 * math.sqrt(3.0), c["width"], c["height"], math.sqrt(3.0) / c["samples"])
        return {"bytes": 8.0 * nf + 16.0 * px * 3, "flops": 120.0 * s * c["views"]}
    px = c["width"] * c["height"]
    if c["kind"] == "hex":
        n = (c["nx"], c["ny"], c["nz"])
        cells = n[0] * n[1] * n[2]
        nodes = (n[0] + 1) * (n[1] + 1) * (n[2] + 1)
        ext = [v / max(n) for v in n]
        s = samples_of(ext, None, c["width"], c["height"], float(np.linalg.norm(ext)) / c["samples"])
        field = 4.0 * (cells if c["assoc"] == "element" else nodes)
        return {"bytes": 32.0 * cells + 12.0 * nodes + field + 20.0 * px, "flops": 200.0 * s}
    n = (c["cells"],) * 3 if c["kind"] == "cinema" else (c["nx"], c["ny"], c["nz"])
    node = 0 if c.get("assoc") == "element" else 1
    field = float((n[0] + node) * (n[1] + node) * (n[2] + node))
    ext = [v / max(n) for v in n]
    views = c["views_phi"] * c["views_theta"] if c["kind"] == "cinema" else 1
    dist = 1.25 * float(np.linalg.norm(ext)) if c["kind"] == "cinema" else None
    s = samples_of(ext, dist, c["width"], c["height"], float(np.linalg.norm(ext)) / c["samples"])
    size = 8 if c.get("dtype") == "float64" else 4
    extra = 20.0 * px * c["canvases"] if c["kind"] == "over" else 0.0
    return {"bytes": size * field + 20.0 * px * views + extra, "flops": 40.0 * s * views}


def samples_of(ext, dist, width, height, dt):
    """Samples of a view: the box's volume over a pixel's footprint at its middle, by the step."""
    if dist is None:
        dist = 0.5 * float(np.linalg.norm(ext)) / math.tan(math.radians(0.5 * FOV))
    pixel = 2.0 * math.tan(math.radians(0.5 * FOV)) * dist / height
    return float(np.prod(ext)) / (pixel * pixel * dt)


# ---------------------------------------------------------------------------
# the same in float64
# ---------------------------------------------------------------------------

F64 = torch.float64


def dev(a):
    return torch.as_tensor(np.asarray(a, dtype=np.float64), device="cuda")


def unit(v):
    return v / np.linalg.norm(v)


class View64:
    """The pinhole rays of one camera, and its projection."""

    def __init__(self, eye, width, height, dtype=F64):
        o, at, up = (np.asarray(eye[k], np.float64) for k in ("pos", "at", "up"))
        self.look = unit(at - o)
        self.ru = unit(np.cross(self.look, up))
        self.rv = unit(np.cross(self.ru, self.look))
        ty = math.tan(math.radians(0.5 * FOV))
        self.sx, self.sy = 2 * ty * width / height / width, 2 * ty / height
        self.w, self.h, self.dtype = width, height, dtype
        n, f = float(eye["near"]), float(eye["far"])
        s = unit(np.cross(self.look, up))
        u = np.cross(s, self.look)
        view = np.array([[*s, -s @ o], [*u, -u @ o], [*-self.look, self.look @ o], [0, 0, 0, 1.0]])
        ff = 1.0 / ty
        proj = np.array([[ff * height / width, 0, 0, 0], [0, ff, 0, 0], [0, 0, (f + n) / (n - f), 2 * f * n / (n - f)],
                         [0, 0, -1, 0]])
        self.m = (proj @ view).tolist()
        self.o, self.look, self.ru, self.rv = o.tolist(), self.look.tolist(), self.ru.tolist(), self.rv.tolist()

    def rays(self, fy_along=None):
        """Unit directions (3 tensors over the flat image)."""
        y, x = torch.meshgrid(torch.arange(self.h, device="cuda", dtype=self.dtype),
                              torch.arange(self.w, device="cuda", dtype=self.dtype), indexing="ij")
        fx, fy = self.sx * (x - 0.5 * self.w).reshape(-1), self.sy * (y - 0.5 * self.h).reshape(-1)
        along = self.rv if fy_along is None else fy_along
        d = [self.look[a] + self.ru[a] * fx + along[a] * fy for a in range(3)]
        n = torch.sqrt(d[0] ** 2 + d[1] ** 2 + d[2] ** 2)
        return [v / n for v in d]

    def image_depth(self, dist):
        d = self.rays(fy_along=self.ru)
        p = [self.o[a] + dist * d[a] for a in range(3)]
        z, w = (m[0] * p[0] + m[1] * p[1] + m[2] * p[2] + m[3] for m in self.m[2:])
        return 0.5 * (z / w) + 0.49

    def distance(self, depth):
        """Distance along each pixel's ray of an image depth."""
        i = np.linalg.inv(np.array(self.m)).tolist()
        y, x = torch.meshgrid(torch.arange(self.h, device="cuda", dtype=F64),
                              torch.arange(self.w, device="cuda", dtype=F64), indexing="ij")
        v = [2 * x.reshape(-1) / self.w - 1, 2 * y.reshape(-1) / self.h - 1, 2 * depth - 1]
        p = [r[0] * v[0] + r[1] * v[1] + r[2] * v[2] + r[3] for r in i]
        return torch.sqrt(sum((p[a] / p[3] - self.o[a]) ** 2 for a in range(3)))


def slab(o, d, lo, hi):
    lo, hi = [float(v) for v in lo], [float(v) for v in hi]
    t0, t1 = torch.zeros_like(d[0]), torch.full_like(d[0], 3e38)
    for a in range(3):
        ta, tb = (lo[a] - o[a]) / d[a], (hi[a] - o[a]) / d[a]
        t0, t1 = torch.maximum(t0, torch.minimum(ta, tb)), torch.minimum(t1, torch.maximum(ta, tb))
    return t0, t1


def lut64(c, single):
    px, rgb, ax, al = transfer_function(c["tf"])
    x = np.arange(1024) / 1023.0
    al = 1.0 - (1.0 - al) ** float(np.float32(10.0) / np.float32(c["samples"]))
    t = np.stack([np.interp(x, px, rgb[:, k]) for k in range(3)] + [np.interp(x, ax, al)], axis=1)
    if c.get("lut8") and not single:
        t = np.floor(np.clip(t, 0, 1) * 255.0 + 0.5) / 255.0
    return dev(t)


def step64(bounds, samples):
    e = (bounds[1::2] - bounds[0::2]).astype(np.float32)
    return float(np.sqrt((e * e).sum(dtype=np.float32)) / np.float32(samples))


def walk(t0, t1, thr, dt, lut, rng, value, act):
    """March rays `act` from t0 to t1: (colour and opacity) of the partial of each."""
    acc = torch.zeros((len(t0), 4), dtype=F64, device="cuda")
    live = act
    k = 0
    lo, inv = rng[0], 1.0 / (rng[1] - rng[0]) if rng[1] > rng[0] else 0.0
    top = float(lut.shape[0] - 1)
    while len(live):
        a0, b1, th = t0[live], t1[live], thr[live]
        got = acc[live]
        for _ in range(16):
            t = a0 + k * dt
            on = (t < b1) & (got[:, 3] < th)
            v, seen = value(live, torch.where(on, t, a0))
            s = ((v - lo) * inv).clamp(0.0, 1.0)
            col = lut[(s * top).long()]
            w = torch.where(on if seen is None else on & seen, (1.0 - got[:, 3]) * col[:, 3], 0.0)
            got = torch.cat([got[:, :3] + w[:, None] * col[:, :3], (got[:, 3] + w)[:, None]], 1)
            k += 1
        acc[live] = got
        live = live[(a0 + k * dt < b1) & (got[:, 3] < th)]
    return acc


def image64(view, doms, dt, lut, rng, value_of, quantize, canvas=None):
    """One view: domains (lo, hi) in order of entry, each marched by value_of(domain of each ray, ray, t)."""
    d = view.rays()
    n = len(d[0])
    spans = [slab(view.o, d, lo, hi) for lo, hi in doms]
    t0s, t1s = torch.stack([s[0] for s in spans]), torch.stack([s[1] for s in spans])
    order = torch.sort(torch.where(t1s > t0s, t0s, 3e38), dim=0, stable=True)[1]
    tmax = torch.full((n,), 3e38, dtype=F64, device="cuda")
    if canvas is not None:
        tmax = view.distance(canvas[1])
    rgb, ca = torch.zeros((n, 3), dtype=F64, device="cuda"), torch.zeros(n, dtype=F64, device="cuda")
    depth = torch.zeros(n, dtype=F64, device="cuda")
    have = torch.zeros(n, dtype=torch.bool, device="cuda")
    covered = torch.full((n,), -3e38, dtype=F64, device="cuda")
    for p in range(len(doms)):
        dom = order[p]
        e0, e1 = t0s.gather(0, dom[None])[0], t1s.gather(0, dom[None])[0]
        hit = (e1 > e0) & (ca < EARLY)
        if not bool(hit.any()):
            break
        b0, b1 = torch.maximum(e0, covered), torch.minimum(e1, tmax)
        covered = torch.where(hit, torch.maximum(covered, b1), covered)
        thr = (EARLY - ca) / (1.0 - ca)
        acc = walk(b0, b1, thr, dt, lut, rng, value_of(view, d, dom), torch.nonzero(hit & (b0 < b1)).reshape(-1))
        keep = hit & ~(acc[:, 3] < CULL)
        first, more = keep & ~have, keep & have & (ca < 1.0)
        op = torch.where(first, 1.0, torch.where(more, 1.0 - ca, 0.0))
        rgb = rgb + op[:, None] * acc[:, :3]
        ca = torch.where(first | more, torch.clamp(ca + op * acc[:, 3], max=1.0), ca)
        depth = torch.where(first, b1, depth)
        have |= keep
    cin = torch.zeros((n, 4), dtype=F64, device="cuda") if canvas is None else canvas[0]
    din = torch.ones(n, dtype=F64, device="cuda") if canvas is None else canvas[1]
    om = (1.0 - ca)[:, None]
    out = torch.where(have[:, None], torch.cat([rgb, ca[:, None]], 1) + cin * om, cin)
    dep = torch.where(have, view.image_depth(depth), din)
    if quantize:
        out, dep = torch.floor((out * 255.0).clamp(0.0, 255.0)) / 255.0, dep.abs()
    return out.reshape(view.h, view.w, 4), dep.reshape(view.h, view.w)


def structured_value(c, boxes, h, coords, f):
    """value_of for a structured grid: the whole field, each ray clamped to its domain's cells."""
    first = torch.tensor([b[:3] for b in boxes], device="cuda")
    cells = torch.tensor([[b[3 + a] - b[a] for a in range(3)] for b in boxes], device="cuda")
    flat = f.reshape(-1)
    nz, ny, nx = f.shape
    org = dev(np.array([[np.float32(b[a] * h) for a in range(3)] for b in boxes]))
    inv = float(np.float32(1.0) / np.float32(h))
    axes = [dev(np.asarray(v, np.float32)) for v in coords]

    def value_of(view, d, dom):
        def value(live, t):
            dm = dom[live]
            i, w = [], []
            for a in range(3):
                p = view.o[a] + t * d[a][live]
                s, n = first[:, a][dm], cells[:, a][dm]
                if c.get("mesh") == "rectilinear":
                    ca = torch.searchsorted(axes[a], p, right=True) - 1
                    ca = torch.minimum(torch.maximum(ca, s), s + n - 1)
                    x0, x1 = axes[a][ca], axes[a][ca + 1]
                    w.append(((p - x0) / (x1 - x0)).clamp(0.0, 1.0))
                    i.append(ca)
                else:
                    g = (p - org[:, a][dm]) * inv
                    ca = torch.minimum(g.long().clamp(min=0), n - 1)
                    w.append(g - ca)
                    i.append(ca + s)
            at = (i[2] * ny + i[1]) * nx + i[0]
            if c.get("assoc") == "element":
                return flat[at].double(), None
            v = [flat[at + dz * ny * nx + dy * nx + dx].double() for dz in (0, 1) for dy in (0, 1) for dx in (0, 1)]
            v = [v[2 * k] + w[0] * (v[2 * k + 1] - v[2 * k]) for k in range(4)]
            v = [v[2 * k] + w[1] * (v[2 * k + 1] - v[2 * k]) for k in range(2)]
            return v[0] + w[2] * (v[1] - v[0]), None
        return value
    return value_of


def hex_value(c, pts, f):
    """value_of for the moved grid of hexahedra: the cell is found by Newton steps from the grid's own."""
    n = (c["nx"], c["ny"], c["nz"])
    h = 1.0 / max(n)
    m0, m1 = n[0] + 1, (n[0] + 1) * (n[1] + 1)
    off = [dz * m1 + dy * m0 + dx for dz in (0, 1) for dy in (0, 1) for dx in (0, 1)]
    P = torch.stack(pts, 1)

    def tri(v, r):
        v = [v[2 * k] + r[0][..., None] * (v[2 * k + 1] - v[2 * k]) for k in range(4)]
        v = [v[2 * k] + r[1][..., None] * (v[2 * k + 1] - v[2 * k]) for k in range(2)]
        return v[0] + r[2][..., None] * (v[1] - v[0])

    def value_of(view, d, dom):
        def value(live, t):
            p = torch.stack([view.o[a] + t * d[a][live] for a in range(3)], 1)
            cell = [(p[:, a] / h).long().clamp(0, n[a] - 1) for a in range(3)]
            for hop in range(4):
                base = cell[2] * m1 + cell[1] * m0 + cell[0]
                v = [P[base + o].double() for o in off]
                r = [(p[:, a] / h - cell[a]).clamp(0.0, 1.0) for a in range(3)]
                for _ in range(4):
                    x = tri(v, r)
                    e = [[v[4 * k + 2 * j + 1] - v[4 * k + 2 * j] for j in (0, 1)] for k in (0, 1)]
                    jr = (e[0][0] * (1 - r[1])[:, None] + e[0][1] * r[1][:, None]) * (1 - r[2])[:, None] \
                        + (e[1][0] * (1 - r[1])[:, None] + e[1][1] * r[1][:, None]) * r[2][:, None]
                    q = [v[2 * k] + r[0][:, None] * (v[2 * k + 1] - v[2 * k]) for k in range(4)]
                    js = (q[1] - q[0]) * (1 - r[2])[:, None] + (q[3] - q[2]) * r[2][:, None]
                    jt = (q[2] - q[0]) * (1 - r[1])[:, None] + (q[3] - q[1]) * r[1][:, None]
                    b = p - x
                    det = (jr * torch.linalg.cross(js, jt)).sum(1)
                    r = [r[0] + (b * torch.linalg.cross(js, jt)).sum(1) / det,
                         r[1] + (b * torch.linalg.cross(jt, jr)).sum(1) / det,
                         r[2] + (b * torch.linalg.cross(jr, js)).sum(1) / det]
                out = sum(((r[a] < 0.0) | (r[a] > 1.0)).int() for a in range(3)) > 0
                if hop == 3 or not bool(out.any()):
                    break
                cell = [torch.where(out, (cell[a] + torch.floor(r[a]).clamp(-1, 1).long()).clamp(0, n[a] - 1), cell[a])
                        for a in range(3)]
            seen = ((r[0] >= -2e-4) & (r[0] <= 1 + 2e-4) & (r[1] >= -2e-4) & (r[1] <= 1 + 2e-4)
                    & (r[2] >= -2e-4) & (r[2] <= 1 + 2e-4))
            if c["assoc"] == "element":
                return f[(cell[2] * n[1] + cell[1]) * n[0] + cell[0]].double(), seen
            base = cell[2] * m1 + cell[1] * m0 + cell[0]
            return tri([f[base + o].double()[:, None] for o in off], [x.clamp(0.0, 1.0) for x in r])[:, 0], seen
        return value
    return value_of


def zbuffer64(cols, deps):
    d, win = deps[0].abs().double(), torch.zeros_like(deps[0], dtype=torch.long)
    for k in range(1, len(deps)):
        dk = deps[k].abs().double()
        take = ~((dk > 1.0) | (d < dk))
        d, win = torch.where(take, dk, d), torch.where(take, k, win)
    # the 8-bit image is the float product truncated
    u = torch.floor((torch.stack(cols) * 255.0).clamp(0.0, 255.0)).double() / 255.0
    return torch.gather(u, 0, win[None, :, :, None].expand(1, *win.shape, 4))[0].reshape(-1, 4), d.reshape(-1)


def exact(case, seed):
    c = case
    if c["kind"] == "partials":
        return None      # the records are compared bit for bit
    if c["kind"] == "train":
        f, lut, eyes, h, dt, rng, target = train_inputs(c, seed)
        return train64(f, lut, eyes, c, h, dt, rng, target)
    if c["kind"] == "hex":
        pts, _, f = hexahedra(c, seed)
        b = np.array([float(v) for p in pts for v in (p.min(), p.max())])
        doms, single, value_of = [(b[0::2], b[1::2])], False, hex_value(c, pts, f)
    else:
        h, coords, f = structured(c, seed)
        boxes = boxes_of(c)
        single = len(boxes) == 1
        if c.get("mesh") == "rectilinear":
            ax = [np.asarray(v, np.float32).astype(np.float64) for v in coords]
            doms = [([ax[a][q[a]] for a in range(3)], [ax[a][q[3 + a]] for a in range(3)]) for q in boxes]
        else:
            lo = [[np.float64(np.float32(q[a] * h)) for a in range(3)] for q in boxes]
            doms = [(l, [np.float64(np.float32(l[a] + (q[3 + a] - q[a]) * np.float64(np.float32(h)))) for a in range(3)])
                    for l, q in zip(lo, boxes)]
        value_of = structured_value(c, boxes, h, coords, f)
        b = np.array([v for a in range(3) for v in (min(l[a] for l, _ in doms), max(u[a] for _, u in doms))])
    rng = (float(f.min()), float(f.max()))
    lut, dt = lut64(c, single), step64(b, c["samples"])
    if c["kind"] == "cinema":
        if c["views_phi"] * c["views_theta"] > 12:
            return None      # a view takes a second or two
        imgs = [image64(View64(e, c["width"], c["height"]), doms, dt, lut, rng, value_of, single)
                for e in orbit(b, c["views_phi"], c["views_theta"])]
        return torch.stack([i[0] for i in imgs]), torch.stack([i[1] for i in imgs])
    canvas = zbuffer64(*canvases(c, seed)) if c["kind"] == "over" else None
    out = image64(View64(eye_of(b, c["az"], c["el"]), c["width"], c["height"]), doms, dt, lut, rng, value_of, single,
                  canvas)
    if c["kind"] == "step" and not c["host"]:
        return out + (rng[0], rng[1])
    return out


def train_samples(view, c, h, dt, dtype):
    """Entry distance, sample count and grid coordinates' coefficients of every ray of a view."""
    n = c["n"]
    hf = float(np.float32(h))
    top = float(np.float32((n - 1) * hf))
    d = view.rays()
    t0, t1 = slab(view.o, d, [0.0] * 3, [top] * 3)
    inv = float(np.float32(1.0) / np.float32(h))
    return d, t0, t1, [(view.o[a] * inv, d[a] * inv) for a in range(3)]


def train_scalar(flat, n, ab, t):
    i, w = [], []
    for a in range(3):
        g = ab[a][0] + t * ab[a][1]
        ca = g.long().clamp(0, n - 2)
        i.append(ca)
        w.append(g - ca)
    at = (i[2] * n + i[1]) * n + i[0]
    v = [flat[at + dz * n * n + dy * n + dx] for dz in (0, 1) for dy in (0, 1) for dx in (0, 1)]
    v = [v[2 * k] + w[0] * (v[2 * k + 1] - v[2 * k]) for k in range(4)]
    v = [v[2 * k] + w[1] * (v[2 * k + 1] - v[2 * k]) for k in range(2)]
    return v[0] + w[2] * (v[1] - v[0]), at, w


def train_lookup(lut, v, rng):
    s = (v - rng[0]) / (rng[1] - rng[0])
    x = s.clamp(0.0, 1.0) * (lut.shape[0] - 1)
    i = x.long().clamp(max=lut.shape[0] - 2)
    wl = (x - i)[:, None]
    return lut[i] + wl * (lut[i + 1] - lut[i]), i, wl[:, 0], (s > 0) & (s < 1)


def train_forward(f, lut, eyes, c, h, dt, rng, dtype):
    """Images of every view, and the transmittance and scalar at each sample when in float64."""
    views = [View64(e, c["width"], c["height"], dtype) for e in eyes]
    parts = [train_samples(v, c, h, dt, dtype) for v in views]
    t0, t1 = torch.cat([p[1] for p in parts]), torch.cat([p[2] for p in parts])
    ab = [(torch.cat([torch.full_like(p[1], float(p[3][a][0])) for p in parts]), torch.cat([p[3][a][1] for p in parts]))
          for a in range(3)]
    flat, lu = f.detach().reshape(-1).to(dtype), lut.detach().to(dtype)
    rgb = torch.zeros((len(t0), 3), dtype=dtype, device="cuda")
    tr = torch.ones(len(t0), dtype=dtype, device="cuda")
    kept = []
    n = int(((t1 - t0).max() / dt).item()) + 2
    for k in range(n):
        t = t0 + k * dt
        on = t < t1
        v, _, _ = train_scalar(flat, c["n"], ab, torch.where(on, t, t0))
        col, _, _, _ = train_lookup(lu, v, rng)
        if dtype == F64:
            kept.append((tr, v))
        a = torch.where(on, col[:, 3], 0.0)
        rgb = rgb + (tr * a)[:, None] * col[:, :3]
        tr = tr * (1.0 - a)
    img = torch.cat([rgb, (1.0 - tr)[:, None]], 1).reshape(len(eyes), c["height"], c["width"], 4)
    return img, (t0, t1, ab, kept)


def train64(f, lut, eyes, c, h, dt, rng, target):
    img, (t0, t1, ab, kept) = train_forward(f, lut, eyes, c, h, dt, rng, F64)
    n, m = c["n"], lut.shape[0]
    lu, flat = lut.double(), f.reshape(-1).double()
    g = (2.0 * (img - target.double())).reshape(-1, 4)
    gf = torch.zeros(n ** 3, dtype=F64, device="cuda")
    spread = 512       # copies of the transfer function's gradient, so that sums do not queue
    gl = torch.zeros((m * spread, 4), dtype=F64, device="cuda")
    lane = torch.arange(len(t0), device="cuda") % spread
    R = torch.zeros((len(t0), 4), dtype=F64, device="cuda")
    for k in range(len(kept) - 1, -1, -1):
        tr, v = kept[k]
        kept[k] = None
        t = t0 + k * dt
        on = t < t1
        _, at, w = train_scalar(flat, n, ab, torch.where(on, t, t0))
        col, i, wl, inner = train_lookup(lu, v, rng)
        a = torch.where(on, col[:, 3], 0.0)
        dc = (tr * a)[:, None] * g[:, :3]
        da = torch.where(on, tr * ((g[:, :3] * (col[:, :3] - R[:, :3])).sum(1) + g[:, 3] * (1.0 - R[:, 3])), 0.0)
        R = a[:, None] * torch.cat([col[:, :3], torch.ones_like(a)[:, None]], 1) + (1.0 - a)[:, None] * R
        dl = torch.cat([dc, da[:, None]], 1)
        gl.index_add_(0, i * spread + lane, dl * (1.0 - wl)[:, None])
        gl.index_add_(0, (i + 1) * spread + lane, dl * wl[:, None])
        dv = torch.where(on & inner, (dl * (lu[i + 1] - lu[i])).sum(1) * (m - 1) / (rng[1] - rng[0]), 0.0)
        for q in range(8):
            b = (q & 1, q >> 1 & 1, q >> 2)
            wt = dv
            for x in range(3):
                wt = wt * (w[x] if b[x] else 1.0 - w[x])
            gf.index_add_(0, at + b[2] * n * n + b[1] * n + b[0], wt)
    return img, gf.reshape(n, n, n), gl.reshape(m, spread, 4).sum(1)

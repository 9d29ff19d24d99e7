"""The workloads the framework is timed on, each through its public entry points.

A case names one kind of call and its sizes:

  frame   a flat world drawn and read back into pinned memory: one blocking frame (``clip`` 0), or
          a camera path of ``clip`` frames captured one behind the draw, as an exporter or a
          streaming viewer runs it
  lod     a LOD world drawn and read back
  batch   many views of one world submitted together, images read
  served  a burst of requests for several resident scenes through the server
  sort    the standalone argsort over device memory (``noalloc``: the fixed-workspace entry point)

Scenes have the shapes and distributions of ``splatkit_b200.synthetic`` and of the benchmark
(positions in a 20 m cube, log-scales N(-3, 0.5), opacity sigmoid(N(0, 1)), harmonics N(0, 0.1);
LOD scenes of 2000 anisotropic clusters in a 200 m box), drawn on the GPU from the seed.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "splatkit-ios_b200"))

import splatkit_b200 as sk  # noqa: E402
from splatkit_b200 import camera  # noqa: E402

FOV = math.radians(60.0)
NEAR, FAR = 0.05, 200.0
VIEW_SIZES = [(256, 256), (320, 240), (400, 300), (512, 384), (640, 480)]
SERVE_SIZES = [(640, 480), (1280, 720), (1920, 1080), (2560, 1440), (3840, 2160)]


def listed():
    return [
        # a thumbnail of a small object: launches and latency are all there is
        dict(name="frame_thumbnail", kind="frame", splats=4_000, degree=0, width=160, height=120,
             bits=16, float_image=False, ranges=1, clip=0),
        # a small tiled scene (several resident ranges) rendered to floats for an offline user, odd sizes
        dict(name="frame_tiles_f32", kind="frame", splats=30_011, degree=2, width=517, height=389,
             bits=32, float_image=True, ranges=3, clip=0),
        # the plain frame at small size: 100k splats without harmonics, 720p, 32-bit keys
        dict(name="frame_100k_720p", kind="frame", splats=100_000, degree=0, width=1280, height=720,
             bits=32, float_image=False, ranges=1, clip=0),
        # the headline scene, one blocking frame, 32-bit keys
        dict(name="frame_1m_1080p_k32", kind="frame", splats=1_000_000, degree=3, width=1920, height=1080,
             bits=32, float_image=False, ranges=1, clip=0),
        # the headline scene on its orbit, frames captured while the next one draws, 16-bit keys
        dict(name="clip_1m_1080p_k16", kind="frame", splats=1_000_000, degree=3, width=1920, height=1080,
             bits=16, float_image=False, ranges=1, clip=8),
        # the largest target that serving mixes in, on a large scene
        dict(name="frame_3m_4k", kind="frame", splats=3_000_000, degree=3, width=3840, height=2160,
             bits=16, float_image=False, ranges=1, clip=0),
        # the LOD walk: cut at 1.5 px, 1080p
        dict(name="lod_2m_1080p", kind="lod", leaves=2_000_000, width=1920, height=1080, limit=0),
        # many small views of one world at once (a view set for a viewer grid or for evaluation)
        dict(name="batch_24_views", kind="batch", splats=500_000, degree=3, views=24, graphs=True),
        # requests of mixed scenes and sizes arriving together at the server
        dict(name="served_burst", kind="served", splats=1_200_000, scenes=4, requests=16, degree=3),
        # a small argsort between other work, without any allocation
        dict(name="sort_20k_k32", kind="sort", keys=20_011, bits=32, noalloc=True),
        # an ordinary argsort: a million 16-bit depth keys
        dict(name="sort_1m_k16", kind="sort", keys=1_000_003, bits=16, noalloc=False),
        # the large argsort, 32-bit keys
        dict(name="sort_40m_k32", kind="sort", keys=40_000_000, bits=32, noalloc=False),
    ]


def _log_int(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(["frame", "frame", "frame", "frame", "lod", "batch", "served", "sort", "sort"])
    if kind == "frame":
        width = _log_int(rng, 130, 3840)
        height = max(90, min(2160, int(width * rng.uniform(0.5, 0.8)) + rng.randrange(3)))
        splats = _log_int(rng, 3_000, 2_500_000)
        clip = rng.choice([0, 0, 3, 6]) if splats <= 1_000_000 and width <= 1920 else 0
        return dict(kind="frame", splats=splats, degree=rng.randrange(4), width=width, height=height,
                    bits=rng.choice([16, 16, 32]), float_image=rng.random() < 0.2,
                    ranges=rng.choice([1, 1, 1, 2, 5]), clip=clip)
    if kind == "lod":
        return dict(kind="lod", leaves=_log_int(rng, 30_000, 1_900_000), width=_log_int(rng, 400, 1920),
                    height=_log_int(rng, 300, 1080), limit=rng.choice([0, 0, 200_000]))
    if kind == "batch":
        return dict(kind="batch", splats=_log_int(rng, 20_000, 480_000), degree=rng.randrange(4),
                    views=rng.randrange(2, 25), graphs=rng.random() < 0.5)
    if kind == "served":
        return dict(kind="served", splats=_log_int(rng, 60_000, 1_100_000), scenes=rng.randrange(1, 5),
                    requests=rng.randrange(3, 17), degree=rng.randrange(4))
    noalloc = rng.random() < 0.4
    return dict(kind="sort", keys=_log_int(rng, 3_000, 1_048_576 if noalloc else 39_000_000),
                bits=rng.choice([16, 32]), noalloc=noalloc)


# ---- inputs ----------------------------------------------------------------------------------
def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _host(t):
    return t.cpu().numpy()


def _attributes(g, n, degree):
    """Covariances, colours, opacities and harmonics of n splats (device tensors)."""
    scale = torch.exp(torch.randn((n, 3), generator=g, device="cuda") * 0.5 - 3.0)
    q = torch.nn.functional.normalize(torch.randn((n, 4), generator=g, device="cuda"), dim=1)
    x, y, z, w = q.unbind(1)
    rows = [[1 - 2 * (y * y + z * z), 2 * (x * y - w * z), 2 * (x * z + w * y)],
            [2 * (x * y + w * z), 1 - 2 * (x * x + z * z), 2 * (y * z - w * x)],
            [2 * (x * z - w * y), 2 * (y * z + w * x), 1 - 2 * (x * x + y * y)]]
    m = [torch.stack(r, 1) * scale for r in rows]
    cov = torch.stack([(m[i] * m[j]).sum(1) for i, j in ((0, 0), (0, 1), (0, 2), (1, 1), (1, 2), (2, 2))], 1)
    colors = torch.rand((n, 3), generator=g, device="cuda")
    alphas = torch.sigmoid(torch.randn((n,), generator=g, device="cuda"))
    sh = None
    if degree > 0:
        sh = torch.randn((n, 3 * sk.sh_coefficients(degree)), generator=g, device="cuda") * 0.1
    return cov, colors, alphas, sh


def _cloud(seed, n, degree):
    g = _generator(seed)
    pos = torch.rand((n, 3), generator=g, device="cuda") * 20.0 - 10.0
    cov, colors, alphas, sh = _attributes(g, n, degree)
    return sk.Cloud(_host(pos), _host(cov), _host(colors), _host(alphas), degree,
                    None if sh is None else _host(sh))


def _clustered(seed, leaves, degree):
    g = _generator(seed)
    clusters = max(8, min(2000, leaves // 64))
    centres = torch.rand((clusters, 3), generator=g, device="cuda") * 200.0 - 100.0
    axes = torch.exp(torch.randn((clusters, 3, 3), generator=g, device="cuda") * 0.3)
    axes *= 2.0 / axes.square().sum((1, 2), keepdim=True).sqrt()  # offsets of 2 m RMS
    of = torch.arange(leaves, device="cuda") % clusters
    offsets = torch.randn((leaves, 1, 3), generator=g, device="cuda")
    signs = torch.where(torch.rand((clusters, 3, 3), generator=g, device="cuda") < 0.5, -1.0, 1.0)
    pos = centres[of] + ((axes * signs)[of] * offsets).sum(2)
    cov, colors, alphas, sh = _attributes(g, leaves, degree)
    host = _host(pos)
    return sk.Cloud(host, _host(cov), _host(colors), _host(alphas), degree, None if sh is None else _host(sh),
                    host.min(axis=0), host.max(axis=0))


def _orbit(degrees, width, height, ranges, degree, radius=15.0):
    view, eye = camera.orbit_view(1, radius, degrees)
    return sk.Frame(view, camera.perspective(FOV, width / height, NEAR, FAR), eye, ranges, degree)


def _ranges(n, count):
    """`count` ranges that cover the world but for a gap between neighbours (tiles not drawn)."""
    if count == 1:
        return [(0, n)]
    edge = [n * i // count for i in range(count + 1)]
    return [(a, b - a - (b - a) // 16) for a, b in zip(edge, edge[1:])]


def _angle(seed):
    return float((int(seed) * 37) % 360)


def _pinned(width, height, float_image):
    return torch.empty((height, width, 4), dtype=torch.float32 if float_image else torch.uint8,
                       pin_memory=True).numpy()


class _Held(np.ndarray):
    """A server image's array that keeps its pinned buffer."""


def prepare(case, seed):
    kind = case["kind"]
    if kind == "frame":
        w, h, n, d = case["width"], case["height"], case["splats"], case["degree"]
        r = sk.Renderer(w, h, image_format=sk.FORMAT_RGBA32F if case["float_image"] else sk.FORMAT_RGBA8,
                        time_stages=False)
        r.apply_render_policy(sk.Policy(sort_depth_bits=case["bits"]))
        r.upload_world(_cloud(seed, n, d), d)
        shots = max(1, case["clip"])
        # a small object is seen from near by, as it is framed in use
        radius = 15.0 if n >= 20_000 else 12.0
        frames = [_orbit(_angle(seed) + 3.0 * i, w, h, _ranges(n, case["ranges"]), d, radius) for i in range(shots)]
        return dict(kind=kind, clip=case["clip"], renderer=r, frames=frames,
                    images=[_pinned(w, h, case["float_image"]) for _ in range(shots)])
    if kind == "lod":
        w, h = case["width"], case["height"]
        tree = sk.build_lod_tree(_clustered(seed, case["leaves"], 0))
        r = sk.Renderer(w, h, time_stages=False)
        r.apply_render_policy(sk.Policy(lod_error_pixels=1.5, lod_splat_limit=case["limit"]))
        r.upload_lod_world(tree, 0, 4_000_000)
        x = -90.0 + float((int(seed) * 53) % 181)
        eye = np.array([x, 1.7, 0.0], np.float32)
        frame = sk.Frame(camera.look_at_view(eye, (x + 10.0, 1.7, 0.0)),
                         camera.perspective(FOV, w / h, NEAR, 400.0), eye, [], 0)
        return dict(kind=kind, renderer=r, frame=frame, image=_pinned(w, h, False))
    if kind == "batch":
        n, d = case["splats"], case["degree"]
        r = sk.Renderer(64, 64, time_stages=False)
        r.upload_world(_cloud(seed, n, d), d)
        views, images = [], []
        for i in range(case["views"]):
            w, h = VIEW_SIZES[(i * 7) % len(VIEW_SIZES)]
            frame = _orbit(_angle(seed) + 360.0 * i / case["views"], w, h, [(0, n)], d)
            views.append(sk.BatchView(r, frame, w, h))
            images.append(np.empty((h, w, 4), np.uint8))
        batch = sk.Batch(lanes=2, max_views=64, use_graphs=case["graphs"])
        return dict(kind=kind, renderer=r, batch=batch, views=views, images=images)
    if kind == "served":
        d = case["degree"]
        server = sk.Server(lanes=2, max_batch_views=16, max_batch_splats=24_000_000)
        sizes = [max(1000, case["splats"] * (i + 1) // case["scenes"]) for i in range(case["scenes"])]
        for i, n in enumerate(sizes):
            r = sk.Renderer(64, 64, time_stages=False)
            r.upload_world(_cloud(seed * 16 + i, n, d), d)
            server.add_scene(r)
        requests, images = [], []
        for i in range(case["requests"]):
            w, h = SERVE_SIZES[(i * 3) % len(SERVE_SIZES)]
            scene = i % case["scenes"]
            frame = _orbit(_angle(seed) + 41.0 * i, w, h, [(0, sizes[scene])], d)
            image = sk.HostImage(w, h)
            held = image.array.view(_Held)
            held.owner = image
            requests.append(sk.Request(scene, frame, w, h, image))
            images.append(held)
        return dict(kind=kind, server=server, requests=requests, images=images)
    n = case["keys"]
    g = _generator(seed)
    # depth keys as the cull writes them: bits of distances between the near plane and the far end
    depth = 0.05 + 40.0 * torch.rand((n,), generator=g, device="cuda")
    keys = depth.view(torch.int32)
    if case["bits"] == 16:
        near = int(np.array([NEAR], np.float32).view(np.int32)[0])
        keys = ((keys - near).clamp_(min=0) >> 11).clamp_(max=65535)
    state = dict(kind=kind, noalloc=case["noalloc"], n=n, bits=case["bits"], keys=keys.contiguous(),
                 count=torch.tensor([n], dtype=torch.int32, device="cuda"),
                 order=torch.empty((n,), dtype=torch.int32, device="cuda"),
                 error=torch.zeros((1,), dtype=torch.int32, device="cuda"))
    if not case["noalloc"]:
        state["workspace"] = torch.empty((sk.sort_workspace_bytes(n),), dtype=torch.uint8, device="cuda")
    return state


# ---- one pass --------------------------------------------------------------------------------
def run(state):
    kind = state["kind"]
    if kind == "frame":
        r, images = state["renderer"], state["images"]
        if state["clip"] == 0:
            r.draw(state["frames"][0])
            return r.read_image(out=images[0])
        waiting = None
        for frame, image in zip(state["frames"], images):
            ticket = r.capture_next_frame(image)
            r.draw(frame)
            if waiting is not None:
                r.wait_capture(waiting)
            waiting = ticket
        r.wait_capture(waiting)
        return images
    if kind == "lod":
        state["renderer"].draw(state["frame"])
        return state["renderer"].read_image(out=state["image"])
    if kind == "batch":
        batch = state["batch"]
        ticket = batch.submit(state["views"])
        batch.wait(ticket)
        return [batch.read_image(ticket, i, out=image) for i, image in enumerate(state["images"])]
    if kind == "served":
        server = state["server"]
        for request in state["requests"]:
            server.submit(request)
        server.drain()
        done = sorted(server.take_completions(), key=lambda c: c["id"])
        return {"images": state["images"], "visible": [c["visible"] for c in done],
                "status": [c["status"] for c in done]}
    stream = torch.cuda.current_stream().cuda_stream
    keys, count, order, error = (state[k].data_ptr() for k in ("keys", "count", "order", "error"))
    if state["noalloc"]:
        sk.radix_argsort_noalloc(keys, count, state["n"], state["bits"], order, error, stream)
    else:
        sk.radix_argsort_device(keys, count, state["n"], state["bits"], order, state["workspace"].data_ptr(),
                                state["workspace"].numel(), error, stream)
    return state["order"]


# ---- what a pass cannot do without ---------------------------------------------------------------
def _frame_work(n, degree, pixels, pixel_bytes):
    """Every record is read (32 bytes) and the survivors' harmonics (about three in four splats of
    these orbits are in view) and the image is written. Operations: about 400 per projected splat
    and 20 per blended fragment, of which a pixel of these scenes takes some 20 per 100k splats
    drawn, up to the depth at which it saturates (about 40)."""
    sh = 2 * 3 * sk.sh_coefficients(degree)
    return dict(bytes=32.0 * n + 0.75 * sh * n + float(pixel_bytes) * pixels,
                flops=400.0 * n + 20.0 * pixels * min(40.0, n / 5_000.0))


def _sum(works):
    return dict(bytes=sum(w["bytes"] for w in works), flops=sum(w["flops"] for w in works))


def work(case):
    kind = case["kind"]
    if kind == "frame":
        one = _frame_work(case["splats"], case["degree"], case["width"] * case["height"],
                          16 if case["float_image"] else 4)
        return _sum([one] * max(1, case["clip"]))
    if kind == "lod":
        # the cut holds about a sixth of the leaves; a cluster (64 bytes) per four of them is tested
        cut = case["leaves"] / 6.0
        w = _frame_work(cut, 0, case["width"] * case["height"], 4)
        return dict(bytes=w["bytes"] + 16.0 * cut, flops=w["flops"] + 20.0 * cut)
    if kind == "batch":
        # the world is read once for all views; every view projects its survivors and writes its image
        sizes = [VIEW_SIZES[(i * 7) % len(VIEW_SIZES)] for i in range(case["views"])]
        works = [_frame_work(case["splats"], case["degree"], w * h, 4) for w, h in sizes]
        world = _frame_work(case["splats"], case["degree"], 0, 0)["bytes"]
        return dict(bytes=world + sum(4.0 * w * h for w, h in sizes), flops=_sum(works)["flops"])
    if kind == "served":
        n = [max(1000, case["splats"] * (i + 1) // case["scenes"]) for i in range(case["scenes"])]
        bytes_, flops = 0.0, 0.0
        for i in range(case["requests"]):
            w, h = SERVE_SIZES[(i * 3) % len(SERVE_SIZES)]
            one = _frame_work(n[i % len(n)], case["degree"], w * h, 4)
            flops += one["flops"]
            bytes_ += 4.0 * w * h + (one["bytes"] - 4.0 * w * h if i < len(n) else 0.0)
        return dict(bytes=bytes_, flops=flops)
    return dict(bytes=8.0 * case["keys"], flops=0.0)


# ---- the same frame in 64 bits -------------------------------------------------------------------
def exact(case, seed):
    """A float frame of up to 60k splats as numpy gives it in 64 bits from the stored world (8-bit
    colours, binary16 covariances and harmonics): projection, harmonics, depth order and blending."""
    if case["kind"] != "frame" or not case["float_image"] or case["splats"] > 60_000 or case["clip"]:
        return None
    w, h, n, d = case["width"], case["height"], case["splats"], case["degree"]
    if w * h > 600_000:
        return None
    cloud = _cloud(seed, n, d)
    pick = np.concatenate([np.arange(o, o + c) for o, c in _ranges(n, case["ranges"])])
    radius = 15.0 if n >= 20_000 else 12.0
    frame = _orbit(_angle(seed), w, h, [], d, radius)
    V = np.asarray(frame.view, np.float64).reshape(4, 4).T
    P = np.asarray(frame.proj, np.float64).reshape(4, 4).T
    pos = cloud.positions[pick].astype(np.float64)
    cov = cloud.covariances[pick].astype(np.float16).astype(np.float64)
    rgb = np.rint(cloud.colors[pick].astype(np.float64) * 255) / 255
    alpha = np.rint(cloud.alphas[pick].astype(np.float64) * 255) / 255
    v = pos @ V[:3, :3].T + V[:3, 3]
    clip = np.concatenate([v, np.ones((len(v), 1))], 1) @ P.T
    z = v[:, 2]
    keep = (alpha >= 2 / 255) & (z < 0) & (clip[:, 2] >= 0) & (clip[:, 2] <= clip[:, 3]) & (clip[:, 3] > NEAR)
    fx, fy = w * P[0, 0] / 2, h * P[1, 1] / 2
    limx, limy = 1.3 / P[0, 0], 1.3 / P[1, 1]
    with np.errstate(all="ignore"):
        vx, vy = np.clip(v[:, 0] / z, -limx, limx) * z, np.clip(v[:, 1] / z, -limy, limy) * z
        t0 = (fx / z)[:, None] * V[0, :3] + (-fx * vx / z ** 2)[:, None] * V[2, :3]
        t1 = (fy / z)[:, None] * V[1, :3] + (-fy * vy / z ** 2)[:, None] * V[2, :3]
        S = cov[:, [0, 1, 2, 1, 3, 4, 2, 4, 5]].reshape(-1, 3, 3)
        a = np.einsum("ni,nij,nj->n", t0, S, t0) + 0.3
        b = np.einsum("ni,nij,nj->n", t1, S, t0)
        c = np.einsum("ni,nij,nj->n", t1, S, t1) + 0.3
        mean = (a + c) / 2
        dist = np.maximum(0.1, np.sqrt(np.maximum(mean * mean - (a * c - b * b), 0)))
        l1, l2 = mean + dist, mean - dist
        nx, ny = b, c - l2
        ln = np.hypot(nx, ny)
        wide = (a > c).astype(np.float64)
        ex, ey = np.where(b == 0, wide, nx / ln), np.where(b == 0, 1 - wide, ny / ln)
        s1, s2 = np.sqrt(l1), np.sqrt(np.maximum(l2, 0))
        reach = np.minimum(2.5, np.sqrt(2 * np.log(np.maximum(alpha * 127.5, 1))))
        reach = np.minimum(reach, 512 / np.maximum(np.maximum(s1, s2), 1e-6))
        half = (a - c) / 2
        source = mean + np.sqrt(half * half + b * b) - 0.3
        keep &= np.sqrt(np.maximum(source, 0)) * reach >= 1.0
    if d:
        sh = cloud.sh[pick].astype(np.float16).astype(np.float64).reshape(len(pick), -1, 3)
        dirs = pos - np.asarray(frame.camera_position, np.float64)
        x, y, zz_ = (dirs / np.linalg.norm(dirs, axis=1, keepdims=True)).T
        basis = [-0.4886025119 * y, 0.4886025119 * zz_, -0.4886025119 * x]
        if d >= 2:
            basis += [1.0925484306 * x * y, -1.0925484306 * y * zz_,
                      0.3153915653 * (2 * zz_ * zz_ - x * x - y * y), -1.0925484306 * x * zz_,
                      0.5462742153 * (x * x - y * y)]
        if d >= 3:
            basis += [-0.5900435899 * y * (3 * x * x - y * y), 2.8906114426 * x * y * zz_,
                      -0.4570457995 * y * (4 * zz_ * zz_ - x * x - y * y),
                      0.3731763326 * zz_ * (2 * zz_ * zz_ - 3 * x * x - 3 * y * y),
                      -0.4570457995 * x * (4 * zz_ * zz_ - x * x - y * y),
                      1.4453057213 * zz_ * (x * x - y * y), -0.5900435899 * x * (x * x - 3 * y * y)]
        rgb = np.maximum(rgb + np.einsum("kn,nkc->nc", np.stack(basis), sh), 0)
    cx, cy = (clip[:, 0] / clip[:, 3] + 1) * w / 2, (clip[:, 1] / clip[:, 3] + 1) * h / 2
    depth = (-z).astype(np.float32)  # the 32-bit key
    if case["bits"] == 16:
        depth = np.minimum((np.maximum(depth, np.float32(NEAR)).view(np.int32)
                            - np.array([NEAR], np.float32).view(np.int32)[0]) >> 11, 65535)
    order = np.argsort(depth, kind="stable")
    color, T = np.zeros((h, w, 3)), np.ones((h, w))
    for i in order[keep[order]]:
        a1, a2, r = (ex[i] * s1[i], ey[i] * s1[i]), (ey[i] * s2[i], -ex[i] * s2[i]), reach[i]
        rx, ry = r * (abs(a1[0]) + abs(a2[0])), r * (abs(a1[1]) + abs(a2[1]))
        x0, x1 = max(0, int(cx[i] - rx - 1)), min(w, int(cx[i] + rx + 2))
        y0, y1 = max(0, int(h - cy[i] - ry - 1)), min(h, int(h - cy[i] + ry + 2))
        if x0 >= x1 or y0 >= y1:
            continue
        dx = np.arange(x0, x1) + 0.5 - cx[i]
        dy = (h - (np.arange(y0, y1) + 0.5) - cy[i])[:, None]
        det = a1[0] * a2[1] - a2[0] * a1[1]
        u, t = (a2[1] * dx - a2[0] * dy) / det, (a1[0] * dy - a1[1] * dx) / det
        q = u * u + t * t
        Tw = T[y0:y1, x0:x1]
        take = (Tw >= 1e-4) & (np.abs(u) <= r) & (np.abs(t) <= r) & (q <= 2 * np.log(255 * alpha[i]))
        weight = Tw * np.where(take, np.minimum(1, alpha[i] * np.exp(-q / 2)), 0)
        color[y0:y1, x0:x1] += weight[:, :, None] * rgb[i]
        T[y0:y1, x0:x1] = Tw - weight
    out = np.ones((h, w, 4))
    out[:, :, :3] = np.clip(color + T[:, :, None] * np.array([0.05, 0.05, 0.08]), 0, 1)
    return out

"""The depth pipeline's performance cases: what a program that uses this package has it do.

A case names a kind of call and its sizes:

  node      one camera through the Depthmap facade, as a ROS node runs it: a frame in, the fused
            depth map and the debug map out, pageable host memory
  batch     several cameras through BatchDepthmap: pinned frames in, fused depth maps out, with or
            without the semi-dense tracker
  nodes     quadtree levels and the matching cost volume of one keyframe on the GPU
  bp        belief propagation and depth extraction from a cost volume, the messages kept (they
            hold each node's beliefs, from which a caller reads its confidence)
  upsample  the edge-aware upsampling of sparse node depths
  fuse      the Bayesian fusion of a depth map with the previous seeds
  fit       one keyframe of the parameter fitting: forward, L1 loss, backward to the penalties and
            the per-pixel edge weights

Images are ray-cast views of a textured room with boxes along a closed camera path, 8-bit, with
smooth and detailed regions, so that every quadtree level occurs; all inputs follow from the seed.
"""
import math

import numpy as np
import torch

from open_quadtree_mapping_b200 import diff, stages
from open_quadtree_mapping_b200.depthmap import BatchDepthmap, Depthmap
from open_quadtree_mapping_b200.params import Params

PATH = 24  # poses of the closed camera path (about 10 cm apart)
WARM = 32  # frames a stream has seen before it is measured: fusion has converged at most pixels
TAU = 0.05
HYPS = (32, 48, 64, 96, 128)


def listed():
    return [
        # the smallest camera, one frame at a time: launches and host work count
        dict(name="node_160x128", kind="node", W=160, H=128, D=64, F=5, streams=1),
        # the reference's own configuration, live: one camera at frame rate
        dict(name="node_752x480", kind="node", W=752, H=480, D=64, F=5, streams=1),
        # one HD video camera with more measurement frames
        dict(name="video_1280x720", kind="batch", W=1280, H=720, D=64, F=10, streams=1,
             tracker=False, mixed=False),
        # a server of many cameras, the measured configuration
        dict(name="batch_32x752x480", kind="batch", W=752, H=480, D=64, F=5, streams=32,
             tracker=False, mixed=False),
        # cameras of different sizes, hypothesis and slot counts in one batch, with the tracker
        dict(name="mixed_9_tracker", kind="batch", W=752, H=480, D=64, F=7, streams=9,
             tracker=True, mixed=True),
        # the largest: full HD, many hypotheses and measurement frames
        dict(name="batch_8x1920x1080", kind="batch", W=1920, H=1080, D=128, F=20, streams=8,
             tracker=False, mixed=False),
        # an odd-sized keyframe through the first two stages
        dict(name="nodes_1241x376", kind="nodes", W=1241, H=376, D=96, F=4),
        # belief propagation alone, at a hypothesis count that is no power of two
        dict(name="bp_640x480x48", kind="bp", W=640, H=480, D=48),
        # the upsampling of a full-HD map
        dict(name="upsample_1920x1080", kind="upsample", W=1920, H=1080),
        # fusion alone
        dict(name="fuse_1280x720", kind="fuse", W=1280, H=720),
        # parameter fitting: the resolution that is fitted on, and a small one
        dict(name="fit_752x480", kind="fit", W=752, H=480, D=64),
        dict(name="fit_160x128", kind="fit", W=160, H=128, D=32),
    ]


def draw(rng):
    def size(lo, hi, wm, hm):
        w = math.exp(rng.uniform(math.log(lo), math.log(hi)))
        h = w * rng.uniform(0.5, 0.85)
        return max(wm, int(w / wm) * wm), max(hm, int(h / hm) * hm)

    kind = rng.choice(["node", "batch", "batch", "nodes", "bp", "upsample", "fuse", "fit"])
    D = rng.choice(HYPS)
    if kind == "node":
        W, H = size(160, 1280, 16, 8)
        return dict(kind=kind, W=W, H=H, D=D, F=5, streams=1)
    if kind == "batch":
        W, H = size(160, 1920, 16, 8)
        most = max(1, min(32, int(12e6 * 64 / (W * H * D))))
        return dict(kind=kind, W=W, H=min(H, 1080), D=D, F=rng.randint(1, 10),
                    streams=rng.randint(1, most), tracker=rng.random() < 0.3,
                    mixed=rng.random() < 0.3)
    if kind == "nodes":
        W, H = size(97, 1920, 1, 1)
        return dict(kind=kind, W=W, H=min(H, 1080), D=D, F=rng.randint(1, 12))
    if kind == "bp":
        W, H = size(97, 1920, 1, 1)
        return dict(kind=kind, W=W, H=min(H, 1080), D=D)
    W, H = size(160, 1920 if kind != "fit" else 960, 16, 8)
    case = dict(kind=kind, W=W, H=min(H, 1080))
    if kind == "fit":
        case["D"] = rng.choice(HYPS[:4])
    return case


# ---------------------------------------------------------------- scenes


def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


class _Room:
    """A 10 x 6 x 4 m room with boxes, seen along a closed path; every face shows a piece of one
    noise texture whose fine octaves come and go."""

    def __init__(self, seed):
        dev = _dev()
        r = np.random.default_rng(seed)
        g = torch.Generator(device="cpu").manual_seed(int(r.integers(1 << 31)))
        n = 1024
        noise = lambda k: torch.nn.functional.interpolate(  # noqa: E731
            torch.rand((1, 1, k, k), generator=g).to(dev), size=(n, n), mode="bilinear",
            align_corners=False)
        detail = ((noise(12) - 0.5) * 4.0).clamp(0.0, 1.0)
        tex = 0.9 * (noise(6) - 0.5) + 0.3 * (noise(20) - 0.5)
        for k, a in ((96, 0.5), (192, 0.4), (384, 0.3)):
            tex = tex + a * detail * (noise(k) - 0.5)
        self.tex = (0.5 + tex).clamp(0.0, 1.0)
        size = r.uniform([0.4, 0.4, 0.4], [1.6, 1.6, 1.8], (6, 3))
        lo = r.uniform([4.0, 0.3, 0.0], [8.2, 4.5, 1.2], (6, 3))
        self.boxes = torch.tensor(np.stack([lo, lo + size]), dtype=torch.float32, device=dev)
        self.shift = torch.tensor(r.uniform(0, 1, (42, 2)), dtype=torch.float32, device=dev)
        self.path = []
        phase, c = r.uniform(0, 2 * math.pi, 4), np.array([1.7, r.uniform(2.4, 3.6), 1.6])
        for i in range(PATH):
            th = 2 * math.pi * i / PATH
            pos = c + [0.38 * math.cos(th + phase[0]), 0.42 * math.sin(th + phase[0]),
                       0.12 * math.sin(2 * th + phase[1])]
            yaw, pitch = 0.06 * math.sin(th + phase[2]), 0.03 * math.sin(th + phase[3])
            cy, sy, cp, sp = math.cos(yaw), math.sin(yaw), math.cos(pitch), math.sin(pitch)
            R0 = np.array([[0.0, 0.0, 1.0], [-1.0, 0.0, 0.0], [0.0, -1.0, 0.0]])
            R = (np.array([[cy, -sy, 0], [sy, cy, 0], [0, 0, 1]])
                 @ np.array([[cp, 0, sp], [0, 1, 0], [-sp, 0, cp]]) @ R0)
            T = np.eye(4)
            T[:3, :3], T[:3, 3] = R, pos
            self.path.append(T)

    def view(self, i, W, H, f):
        """(8-bit image, Euclidean depth) from pose i of the path."""
        dev, T = _dev(), torch.tensor(self.path[i % PATH], dtype=torch.float32, device=_dev())
        x = (torch.arange(W, device=dev, dtype=torch.float32) - W / 2.0) / f
        y = (torch.arange(H, device=dev, dtype=torch.float32) - H / 2.0) / f
        d = torch.stack([x[None].expand(H, W), y[:, None].expand(H, W), torch.ones(H, W, device=dev)])
        d = d / d.square().sum(0).sqrt()
        d = (T[:3, :3, None, None] * d[None]).sum(1)
        o = T[:3, 3, None, None]
        inv = 1.0 / torch.where(d.abs() < 1e-9, 1e-9, d)
        ends = torch.tensor([10.0, 6.0, 4.0], device=dev)[:, None, None]
        t0, t1 = -o * inv, (ends - o) * inv
        t, axis = torch.maximum(t0, t1).min(0)
        face = 2 * axis + (t1 > t0).gather(0, axis[None])[0].long()
        for b in range(self.boxes.shape[1]):
            u, v = (self.boxes[k, b][:, None, None] - o for k in (0, 1))
            u, v = u * inv, v * inv
            tn, ax = torch.minimum(u, v).max(0)
            hit = (tn <= torch.maximum(u, v).amin(0)) & (tn > 0.2) & (tn < t)
            side = (u > v).gather(0, ax[None])[0].long()
            t, axis = torch.where(hit, tn, t), torch.where(hit, ax, axis)
            face = torch.where(hit, 6 + 6 * b + 2 * ax + side, face)
        P = o + d * t
        st = torch.stack([torch.where(axis == 0, P[1], P[0]), torch.where(axis == 2, P[1], P[2])], -1)
        st = (st / 4.0 + self.shift[face]).remainder(1.0) * 2.0 - 1.0
        img = torch.nn.functional.grid_sample(self.tex, st[None], align_corners=False)[0, 0]
        return (img * 255.0).round().clamp(0, 255).to(torch.uint8), t


def _inv(T):
    out = np.eye(4)
    out[:3, :3], out[:3, 3] = T[:3, :3].T, -T[:3, :3].T @ T[:3, 3]
    return out


def _focal(W):
    return 460.0 * W / 752.0


def _cam(W, H):
    return (_focal(W), _focal(W), W / 2.0, H / 2.0)


def _params(case):
    return Params.for_range(case.get("D", 64), 0.5, 50.0,
                            qt_max_level=5 if case["W"] * case["H"] > 1500000 else 4)


def _streams(case):
    """Sizes, hypotheses and slots of every stream of a batch."""
    W, H, D, F, n = case["W"], case["H"], case["D"], case["F"], case["streams"]
    out = []
    for i in range(n):
        if case["mixed"]:  # a third smaller, a third larger where the range allows
            k = (1.0, 0.85, min(1.7, 1920.0 / W))[i % 3]
            w, h = max(160, int(W * k) // 16 * 16), min(1080, max(128, int(H * k) // 8 * 8))
            d = (D, HYPS[max(0, HYPS.index(D) - 1)], HYPS[min(4, HYPS.index(D) + 1)])[i // 3 % 3]
            out.append((w, h, d, 1 + (F - 1 + 2 * i) % 10))
        else:
            out.append((W, H, D, F))
    return out


def _slots(room, F, W, H):
    """The keyframe at pose F of the path and the F views before it, with their relative poses."""
    f = _focal(W)
    ref, gt = room.view(F, W, H, f)
    meas = [room.view(F - 1 - k, W, H, f)[0] for k in range(F)]
    T = [(_inv(room.path[(F - 1 - k) % PATH]) @ room.path[F % PATH])[:3, :4].reshape(-1)
         for k in range(F)]
    return ref, gt, meas, np.array(T, dtype=np.float32)


# ---------------------------------------------------------------- prepare and run


def prepare(case, seed):
    kind, W, H = case["kind"], case["W"], case["H"]
    dev, p = _dev(), _params(case)
    if kind == "node":
        room = _Room(seed)
        dm = Depthmap(W, H, _focal(W), W / 2.0, _focal(W), H / 2.0, params=p)
        frames = [room.view(i, W, H, _focal(W))[0].cpu().numpy() for i in range(PATH)]
        poses = [np.float32(_inv(T)[:3, :4].reshape(12)) for T in room.path]
        for i in range(WARM):
            dm.add_frames(frames[i % PATH], poses[i % PATH])
        return dict(kind=kind, dm=dm, frames=frames, poses=poses, i=WARM)
    if kind == "batch":
        shapes = _streams(case)
        b = BatchDepthmap([dict(width=w, height=h, fx=_focal(w), fy=_focal(w), cx=w / 2.0,
                                cy=h / 2.0, num_hyp=d, num_slots=s) for w, h, d, s in shapes],
                          params=p)
        if case["tracker"]:
            b.set_semidense(True)
        rooms = [_Room(seed * 4 + k) for k in range(min(4, len(shapes)))]
        shown = {}
        for i, (w, h, _, _) in enumerate(shapes):
            for k in range(PATH):
                key = (i % len(rooms), w, h, k)
                if key not in shown:
                    t = torch.empty((h, w), dtype=torch.uint8, pin_memory=True)
                    t.copy_(rooms[key[0]].view(k, w, h, _focal(w))[0])
                    shown[key] = t.numpy()
        frames = [[shown[(i % len(rooms), w, h, k)] for i, (w, h, _, _) in enumerate(shapes)]
                  for k in range(PATH)]
        poses = [[np.float32(_inv(rooms[i % len(rooms)].path[k])[:3, :4].reshape(12))
                  for i in range(len(shapes))] for k in range(PATH)]
        outs = [torch.empty((h, w), dtype=torch.float32, pin_memory=True).numpy()
                for w, h, _, _ in shapes]
        for i in range(WARM):
            b.add_frames(frames[i % PATH], poses[i % PATH])
        return dict(kind=kind, b=b, frames=frames, poses=poses, outs=outs, i=WARM)
    s = _inputs(case, seed)
    if kind == "fit":
        s["kf"] = diff.Keyframe(ref=s["ref"], slots=s["meas"], T_slot_ref=s["T"],
                                cam=_cam(W, H), seeds=s["seeds"], T_fuse=s["T_fuse"], gt=s["gt"],
                                levels=s["levels"], cost=s["cost"])
        s["pen"] = torch.tensor([p.P1, p.P2], dtype=torch.float64, requires_grad=True)
        s["omega"] = s["omega0"].clone().requires_grad_(True)
    s.update(kind=kind, W=W, H=H, p=p, cam=_cam(W, H))
    return s


def _inputs(case, seed):
    """GPU inputs of the stage calls."""
    kind, W, H, dev, p = case["kind"], case["W"], case["H"], _dev(), _params(case)
    room = _Room(seed)
    g = torch.Generator(device="cpu").manual_seed(int(seed) + 77)
    normal = lambda *n: torch.randn(n, generator=g).to(dev)  # noqa: E731
    uniform = lambda a, b, *n: (a + (b - a) * torch.rand(n, generator=g)).to(dev)  # noqa: E731
    ref, gt, meas, T = _slots(room, case.get("F", 5), W, H)
    s = dict(ref=ref, meas=meas, T=T, gt=gt)
    if kind in ("bp", "upsample", "fit"):
        s["levels"] = _levels(ref, p)
    if kind in ("bp", "fit"):
        s["cost"] = _cost(ref, s["levels"], meas, T, _cam(W, H), p).float().contiguous()
    if kind == "upsample":  # depths at the node pixels, some of them missing
        node = _node_cells(s["levels"], H, W)
        node &= uniform(0, 1, *node.shape) > 0.02
        s["sparse"] = torch.zeros((H, W), device=dev)
        y, x = torch.nonzero(node, as_tuple=True)
        s["sparse"][4 * y, 4 * x] = gt[4 * y, 4 * x] * (1.0 + 0.02 * normal(len(y)))
    if kind in ("fuse", "fit"):
        # seeds of the previous keyframe: most have seen a dozen updates, some none
        prev = room.view(4, W, H, _focal(W))[1]
        seeds = torch.stack([uniform(8, 40, H, W), uniform(3, 12, H, W),
                             prev * (1.0 + 0.04 * normal(H, W)), uniform(0.05, 5, H, W)], -1)
        seeds[uniform(0, 1, H, W) < 0.08] = torch.tensor([10.0, 10.0, 3.0, 2500.0], device=dev)
        s["seeds"] = seeds.contiguous()
        s["T_fuse"] = np.float32((_inv(room.path[5]) @ room.path[4])[:3, :4].reshape(12))
    if kind == "fuse":
        s["depth"] = (gt * (1.0 + 0.03 * normal(H, W))).contiguous()
    if kind == "fit":
        s["omega0"] = uniform(0.6, 1.4, H, W)
    return s


def run(s):
    kind = s["kind"]
    if kind == "node":
        k = s["i"] % PATH
        s["i"] += 1
        has = s["dm"].add_frames(s["frames"][k], s["poses"][k])
        return dict(has=has, depth=s["dm"].getDepthmap(), debug=s["dm"].getDebugmap())
    if kind == "batch":
        k = s["i"] % PATH
        s["i"] += 1
        has = s["b"].submit(s["frames"][k], s["poses"][k], outs=s["outs"])
        s["b"].wait()
        return dict(has=sum(has), depth=s["outs"])
    p = s["p"]
    if kind == "nodes":
        levels = stages.quadtree(s["ref"], p)
        return dict(levels=levels, cost=stages.cost_volume(s["ref"], levels, s["meas"], s["T"],
                                                           s["cam"], p))
    if kind == "bp":
        sparse, labels, messages = stages.bp_extract(s["cost"], s["W"], s["H"], s["levels"], p,
                                                     want_messages=True)
        return dict(sparse=sparse, labels=labels, messages=messages)
    if kind == "upsample":
        return dict(dense=stages.upsample(s["sparse"], s["ref"], p))
    if kind == "fuse":
        fused, _, seeds, table = stages.fuse(s["depth"], s["seeds"], s["T_fuse"], s["cam"], p)
        return dict(fused=fused, seeds=seeds, table=table)
    s["pen"].grad = s["omega"].grad = None
    loss = diff.batch_loss([s["kf"]], s["pen"], [s["omega"]], p, TAU)
    loss.backward()
    return dict(loss=loss, pen=s["pen"].grad, omega=s["omega"].grad)


def work(case):
    """Inputs read once and outputs written once; operations of the algorithm on all cells."""
    kind, W, H, D = case["kind"], case["W"], case["H"], case.get("D", 64)

    def sweeps(w, h, iters=(4, 10, 10, 10)):  # cell updates of one BP run
        n = 0
        for it in iters:
            n += it * w * h / 2.0
            w, h = (w + 1) // 2, (h + 1) // 2
        return n

    def cost(w, h, d, f):
        return w * h / 16.0 * d * f * 60.0

    def bp(w, h, d):
        return sweeps(w // 4, h // 4) * d * 40.0

    P, cells = W * H, (W // 4) * (H // 4)
    if kind in ("node", "batch"):
        shapes = _streams(case) if kind == "batch" else [(W, H, D, case["F"])]
        b = sum(w * h * (1 + f + 4 + 32) for w, h, _, f in shapes)
        fl = sum(cost(w, h, d, f) + bp(w, h, d) + 150.0 * w * h for w, h, d, f in shapes)
        if case.get("tracker"):
            b += sum(w * h * (1 + 64 + 4) for w, h, _, _ in shapes)
            fl += sum(500.0 * w * h for w, h, _, _ in shapes)
        return dict(bytes=b, flops=fl)
    if kind == "nodes":
        return dict(bytes=P * (2 + case["F"]) + 4 * cells * D, flops=cost(W, H, D, case["F"]))
    if kind == "bp":
        return dict(bytes=5 * 4 * cells * D + P * 5 + 4 * cells, flops=bp(W, H, D))
    if kind == "upsample":
        return dict(bytes=P * 9, flops=P * 60.0)
    if kind == "fuse":
        return dict(bytes=P * (4 + 16 + 4 + 16 + 4), flops=P * 120.0)
    return dict(bytes=4 * cells * D + P * (1 + 1 + 16 + 4 + 4 + 4),
                flops=4 * bp(W, H, D) + P * 600.0)


# ---------------------------------------------------------------- the same in 64 bits


def _levels(img, p):
    """Quadtree levels: the largest approved power-of-two block around each pixel."""
    H, W = img.shape
    T = 1 << p.qt_max_level
    ph, pw = -(-H // T) * T, -(-W // T) * T
    v = torch.zeros((ph, pw), dtype=torch.float64, device=img.device)
    v[:H, :W] = img.double()
    ok = torch.zeros((ph, pw), dtype=torch.bool, device=img.device)
    ok[:H, :W] = True
    level = torch.zeros((ph, pw), dtype=torch.int64, device=img.device)
    total, hi, lo = v, v, v
    quad = lambda t: torch.stack([t[j::2, i::2] for j in (0, 1) for i in (0, 1)])  # noqa: E731
    for i in range(1, p.qt_max_level + 1):
        total, hi, lo, ok = quad(total).sum(0), quad(hi).amax(0), quad(lo).amin(0), quad(ok).all(0)
        mean = total / 4.0 ** i
        ok = ok & (hi - mean <= p.qt_threshold) & (mean - lo <= p.qt_threshold)
        level += ok.repeat_interleave(1 << i, 0).repeat_interleave(1 << i, 1).long()
    return level[:H, :W].clamp(min=p.qt_min_level).to(torch.uint8).contiguous()


def _node_cells(levels, H, W):
    """Cells (4 x 4 pixels) whose corner pixel is the origin of its quadtree block."""
    y = 4 * torch.arange(H // 4, device=levels.device)
    x = 4 * torch.arange(W // 4, device=levels.device)
    size = 1 << levels[y][:, x].long()
    return (y[:, None] % size == 0) & (x[None] % size == 0)


def _cost(ref, levels, meas, T, cam, p):
    H, W = ref.shape
    dev, (fx, fy, cx, cy), D = ref.device, cam, p.num_hyp
    node = _node_cells(levels, H, W)
    yy, xx = torch.nonzero(node, as_tuple=True)
    yy, xx = 4 * yy, 4 * xx
    inner = (xx > 0) & (yy > 0) & (xx < W - 1) & (yy < H - 1)
    yy, xx = yy[inner], xx[inner]
    ray = torch.stack([(xx - cx) / fx, (yy - cy) / fy, torch.ones_like(xx)]).double()
    ray = ray / ray.square().sum(0).sqrt()
    d = torch.arange(D, device=dev, dtype=torch.float64)
    pts = ray[:, :, None] * (1.0 / (p.inv_depth_step * d + p.min_inv_depth))
    sad = torch.zeros(pts.shape[1:], dtype=torch.float64, device=dev)
    seen = torch.zeros_like(sad)
    flat = ref.double().reshape(-1)
    for img, t in zip(meas, np.asarray(T, np.float64).reshape(-1, 3, 4)):
        q = [sum(t[r, k] * pts[k] for k in range(3)) + t[r, 3] for r in range(3)]
        u, v = fx * q[0] / q[2] + cx, fy * q[1] / q[2] + cy
        ok = (u >= 1.5) & (u < W - 2.5) & (v >= 1.5) & (v < H - 2.5)
        u, v = torch.where(ok, u, 2.0), torch.where(ok, v, 2.0)
        m = img.double().reshape(-1)
        one = torch.zeros_like(sad)
        for j in (-1, 0, 1):
            for i in (-1, 0, 1):
                px = (u + t[0, 0] * i + t[0, 1] * j + 0.5).floor().long()
                py = (v + t[1, 0] * i + t[1, 1] * j + 0.5).floor().long()
                one += (m[py * W + px] - flat[(yy + j) * W + xx + i][:, None]).abs()
        sad += torch.where(ok, one, 0.0)
        seen += ok
    c = torch.where(seen > 0, sad / seen.clamp(min=1.0) / 255.0, 100.0) / D
    out = torch.zeros((H // 4, W // 4, D), dtype=torch.float64, device=dev)
    out[yy // 4, xx // 4] = c
    return out


def _messages(cost, levels, p, P1, P2):
    """Level-0 messages (to the upper, lower, left and right neighbour) of the hierarchical
    min-sum belief propagation."""
    H, W = levels.shape
    dev, data = cost.device, [cost]
    for _ in range(1, p.bp_levels):
        a = torch.nn.functional.pad(data[-1], (0, 0, 0, data[-1].shape[1] % 2, 0,
                                               data[-1].shape[0] % 2))
        data.append(a[0::2, 0::2] + a[1::2, 0::2] + a[0::2, 1::2] + a[1::2, 1::2])
    msg = None
    for lev in range(p.bp_levels - 1, -1, -1):
        c = data[lev]
        h, w = c.shape[:2]
        ys, xs = torch.arange(h, device=dev), torch.arange(w, device=dev)
        m = ([torch.zeros_like(c)] * 4 if msg is None
             else [q[ys // 2][:, xs // 2] for q in msg])
        size = 1 << (lev + 2)
        keep = torch.ones((h, w), dtype=torch.bool, device=dev)
        if lev + 2 <= p.qt_max_level:
            sx, sy = (xs // 2 * size).clamp(max=W - 1), (ys * size).clamp(max=H - 1)
            keep = levels[sy][:, sx] <= lev + 2
        far = torch.full_like(c[..., :1], math.inf)
        for it in range(p.bp_iters[lev]):
            now = (keep & ((xs[None] + ys[:, None] + it) % 2 == 0))[..., None]
            got = _incoming(m)
            new = []
            for k in range(4):
                hv = c + sum(g for n, g in enumerate(got) if n != k)
                best = torch.minimum(hv, hv.amin(-1, keepdim=True) + P2)
                best = torch.minimum(best, torch.cat([far, hv[..., :-1]], -1) + P1)
                best = torch.minimum(best, torch.cat([hv[..., 1:], far], -1) + P1)
                new.append(best - best.mean(-1, keepdim=True))
            m = [torch.where(now, n, o) for n, o in zip(new, m)]
        msg = m
    return msg


def _incoming(m):
    """What each cell receives from its upper, lower, left and right neighbour."""
    pad = torch.nn.functional.pad
    return [pad(m[1][:-1], (0, 0, 0, 0, 1, 0)), pad(m[0][1:], (0, 0, 0, 0, 0, 1)),
            pad(m[3][:, :-1], (0, 0, 1, 0)), pad(m[2][:, 1:], (0, 0, 0, 1))]


def _at_nodes(depth, levels):
    H, W = levels.shape
    out = torch.zeros((H, W), dtype=depth.dtype, device=depth.device)
    y, x = torch.nonzero(_node_cells(levels, H, W), as_tuple=True)
    return out.index_put((4 * y, 4 * x), depth[y, x])


def _solve(rhs, w, lam):
    """(I + lam L) s = rhs down the first axis; w[k] is the weight of the edge (k - 1, k)."""
    n = rhs.shape[0]
    c, d = [], []
    for k in range(n):
        left = lam * w[k]
        den = 1.0 + left + lam * w[k + 1] + (left * c[-1] if k else 0.0)
        c.append(-lam * w[k + 1] / den)
        d.append((rhs[k] + (left * d[-1] if k else 0.0)) / den)
    out = [d[-1]]
    for k in range(n - 2, -1, -1):
        out.append(d[k] - c[k] * out[-1])
    return torch.stack(out[::-1])


def _smooth(sparse, img, p, omega=None):
    I, lam = img.double(), p.up_lambda
    H, W = img.shape
    om = torch.ones_like(I) if omega is None else omega
    both = torch.stack([sparse, (sparse > 0).double()], -1)
    ww = om[:, 1:] * torch.exp(-(I[:, 1:] - I[:, :-1]).square() / p.up_sigma)
    end = torch.zeros_like(I[:, :1])
    ww = torch.cat([end, ww, end + (W % 16 != 0)], 1).T[..., None]
    both = _solve(both.transpose(0, 1), ww, lam).transpose(0, 1)
    wh = om[1:] * torch.exp(-(I[1:] - I[:-1]).square() / p.up_sigma)
    end = torch.zeros_like(I[:1])
    wh = torch.cat([end, wh, end + (H % 16 != 0)])[..., None]
    both = _solve(both, wh, lam)
    return both[..., 0] / both[..., 1]


def _fuse(depth, seeds, T, cam, p):
    """(fused depth, new seeds); differentiable in depth."""
    H, W = depth.shape
    dev, (fx, fy, cx, cy) = depth.device, cam
    T = torch.tensor(np.asarray(T, np.float64).reshape(3, 4), device=dev)
    a, b, mu, s2 = seeds.double().reshape(-1, 4).unbind(-1)
    idx = torch.arange(H * W, device=dev)
    ray = torch.stack([(idx % W - cx) / fx, (idx // W - cy) / fy, torch.ones_like(idx)]).double()
    q = T[:, :3] @ (ray / ray.square().sum(0).sqrt() * mu) + T[:, 3:]
    far = q.square().sum(0).sqrt()
    tx = (fx * q[0] / q[2] + cx + 0.5).trunc().nan_to_num(-9.0).clamp(-9, W + 9).long()
    ty = (fy * q[1] / q[2] + cy + 0.5).trunc().nan_to_num(-9.0).clamp(-9, H + 9).long()
    ok = (a >= 0.001) & (a / (a + b) >= 0.45) & (far > 0.5) & (tx >= 0) & (tx < W) & (ty >= 0) & (ty < H)
    mu, s2 = torch.where(ok, far, mu), torch.where(ok, s2 + 0.01 * far, s2)
    ok = ok & (idx != 0)
    to = torch.where(ok, ty * W + tx, 0)
    near = torch.full((H * W,), math.inf, dtype=torch.float64, device=dev)
    near = near.scatter_reduce(0, to[ok], far[ok], "amin")
    first = ok & (far == near[to])
    src = torch.full((H * W,), H * W, device=dev)
    src = src.scatter_reduce(0, to[first], idx[first], "amin").reshape(H, W)
    near = near.reshape(H, W)
    # an empty pixel takes the nearest of the filled pixels around it
    gives = torch.zeros((H, W), dtype=torch.bool, device=dev)
    gives[2:H - 1, 2:W - 1] = True
    pad = torch.nn.functional.pad
    wn = pad(torch.where(gives, near, math.inf), (1, 1, 1, 1), value=math.inf)
    ws = pad(src, (1, 1, 1, 1), value=H * W)
    around = torch.stack([wn[j:j + H, i:i + W] for j in range(3) for i in range(3)]).min(0)
    fill = torch.stack([ws[j:j + H, i:i + W] for j in range(3) for i in range(3)])
    fill = fill.gather(0, around.indices[None])[0]
    src = torch.where(near.isfinite(), src, torch.where(around.values.isfinite(), fill, 0))
    src = torch.where(src == H * W, 0, src)
    dep = depth.double()
    unc = torch.where(dep <= 0.0, 1e9, (dep * 0.2).clamp(min=0.5).square())
    has = src > 0
    a, b = torch.where(has, a[src], 10.0), torch.where(has, b[src], 10.0)
    mu, s2 = torch.where(has, mu[src], dep), torch.where(has, s2[src], 2500.0)
    off = (dep - mu).square() > unc + s2
    a, b = torch.where(off, 10.0, a), torch.where(off, 10.0, b)
    mu, s2 = torch.where(off, dep, mu), torch.where(off, 2500.0, s2)
    var = unc + s2
    new_mu, new_s2 = (dep * s2 + mu * unc) / var, unc * s2 / var
    c1 = a / (a + b) * torch.exp(-(dep - mu).square() / (2.0 * var)) / (2.0 * math.pi * var).sqrt()
    c2 = b / (a + b) / 50.0
    c1, c2 = c1 / (c1 + c2), c2 / (c1 + c2)
    f = c1 * (a + 1) / (a + b + 1) + c2 * a / (a + b + 1)
    e = (c1 * (a + 1) * (a + 2) + c2 * a * (a + 1)) / ((a + b + 1) * (a + b + 2))
    m = c1 * new_mu + c2 * mu
    v = c1 * (new_s2 + new_mu.square()) + c2 * (s2 + mu.square()) - m.square()
    an = (e - f) / (f - e / f)
    return (torch.where(a / (a + b) > 0.60, m, -1.0),
            torch.stack([an, an * (1.0 - f) / f, m, v], -1))


def exact(case, seed):
    """None for the whole calls: some forty dense passes over the frames before (and an epipolar
    search per pixel) take plain torch far longer than the time allowed; their stages are here."""
    kind, p = case["kind"], _params(case)
    if kind in ("node", "batch"):
        return None
    s, cam = _inputs(case, seed), _cam(case["W"], case["H"])
    if kind == "nodes":
        lv = _levels(s["ref"], p)
        return dict(levels=None, cost=_cost(s["ref"], lv, s["meas"], s["T"], cam, p))
    if kind == "bp":
        # a depth follows the winning label, which rounding decides where a region has no
        # texture: the messages have a value in 64 bits, the depths have none
        m = _messages(s["cost"].double(), s["levels"], p, float(np.float32(p.P1)),
                      float(np.float32(p.P2)))
        return dict(sparse=None, labels=None, messages=torch.stack(m))
    if kind == "upsample":
        return dict(dense=_smooth(s["sparse"].double(), s["ref"], p))
    if kind == "fuse":
        fused, seeds = _fuse(s["depth"], s["seeds"], s["T_fuse"], cam, p)
        return dict(fused=fused, seeds=seeds, table=None)
    P1, P2 = (torch.tensor(float(np.float32(x)), dtype=torch.float64, device=_dev(),
                           requires_grad=True) for x in (p.P1, p.P2))
    omega = s["omega0"].double().requires_grad_(True)
    cost = s["cost"].double()
    b = cost + sum(_incoming(_messages(cost, s["levels"], p, P1, P2)))
    disp = (torch.softmax(-b / TAU, -1) * torch.arange(p.num_hyp, device=b.device)).sum(-1)
    sparse = _at_nodes(1.0 / (p.inv_depth_step * disp + p.min_inv_depth), s["levels"])
    fused, _ = _fuse(_smooth(sparse, s["ref"], p, omega), s["seeds"], s["T_fuse"], cam, p)
    gt = s["gt"].double()
    mask = ((fused > 0) & (gt > 0)).double()
    loss = ((fused - gt).abs() * mask).sum() / mask.sum().clamp(min=1.0)
    loss.backward()
    return dict(loss=loss.detach(), pen=torch.stack([P1.grad, P2.grad]), omega=omega.grad)

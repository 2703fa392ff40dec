"""The work a user of this framework has it do, as cases that can be timed.

A case is a dict of plain values; `listed()` gives the standing ones, `draw`
one more of the same ranges.  `prepare` makes what a program holds before the
call (rendered frames, a map that already holds the start of the scan, a
network and its training batch), `run` is one pass through the public entry
points, `work` the bytes and operations the pass cannot do without, `exact`
the results of the confidence network's passes in 64 bits.

Kinds of pass:

  live     the viewer's loop: one host frame in (addMap), the mesh updated, the
           whole mesh out to host memory (getMeshInterleavedMarchingCubes)
  single   frames already on the GPU, one call per frame (addMapDevice), then
           one mesh update; the mesh stays on the GPU
  sequence the same frames in one call (addMapSequenceDevice), then one mesh
           update; with `weight` "learned" every frame runs the confidence
           network first
  maps     several independent maps of mixed image and voxel size, one frame of
           each per call (add_maps_device), then every map's mesh update
  session  a whole scan on an empty map: create it, fuse all frames in steps of
           10 from page-locked host memory, a mesh update after each step, the
           final mesh to host memory, close it
  raycast  depth of the fused surface along every pixel's ray (the training
           targets of the confidence network, ConfidenceNet examples)
  infer    depth images to per-pixel confidence (ConfidenceNet.features, forward)
  train    one step of the confidence network (ConfidenceNet.train_step): forward,
           loss, backward, Adam

A fusing pass takes the next frames of the state's trajectory and starts over
when they are used up, as a camera that comes back does.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

from fastfusion_b200 import confidence, fusion, scene

SCALING, MAXCAM = 1.0 / 5000.0, 4.0


def listed():
    return [
        # the smallest call: a low-resolution live preview, where launches and latency are all there is
        dict(name="live_160x120", kind="live", width=160, height=120, frames=1, voxel=0.005, storage="fp32"),
        # the viewer's loop at the sensor's resolution, meshed every frame, host images in and host mesh out
        dict(name="live_640x480", kind="live", width=640, height=480, frames=1, voxel=0.005, storage="fp32"),
        # the benchmark's step, one call per frame: 10 device frames, one mesh update
        dict(name="single_640x480", kind="single", width=640, height=480, frames=10, voxel=0.005, storage="fp32"),
        # the benchmark's step through the several-frames call
        dict(name="sequence_640x480", kind="sequence", width=640, height=480, frames=10, voxel=0.005,
             storage="fp32", weight="plain"),
        # the large-map configuration's frames: 1280x960 with FP16 storage
        dict(name="sequence_1280x960_fp16", kind="sequence", width=1280, height=960, frames=10, voxel=0.005,
             storage="fp16", weight="plain"),
        # the learned weight: the confidence network runs on every frame
        dict(name="learned_640x480", kind="sequence", width=640, height=480, frames=10, voxel=0.005,
             storage="fp32", weight="learned"),
        # independent maps of uneven size in one call per frame set
        dict(name="maps_8", kind="maps", maps=8, frames=4, voxel=0.006, storage="fp32"),
        # a scan from nothing: almost every brick and mesh cell is new
        dict(name="session_640x480", kind="session", width=640, height=480, frames=60, voxel=0.005, storage="fp32"),
        # training targets of the confidence network
        dict(name="raycast_640x480", kind="raycast", width=640, height=480, voxel=0.005, storage="fp32"),
        # confidence of one sensor frame
        dict(name="infer_640x480", kind="infer", width=640, height=480, images=1),
        # a training step at the trainer's batch of 4 sensor images
        dict(name="train_4x640x480", kind="train", width=640, height=480, images=4),
        # a training step on odd, ragged images
        dict(name="train_3x333x251", kind="train", width=333, height=251, images=3),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["live", "single", "sequence", "sequence", "maps", "session", "raycast", "infer", "train"])
    width = _log(rng, 150, 1280)
    height = max(100, int(width * rng.uniform(0.6, 0.8)))
    voxel = round(rng.uniform(0.004, 0.010), 4)
    storage = rng.choice(["fp32", "fp16"])
    if kind == "live":
        return dict(kind=kind, width=min(width, 800), height=min(height, 600), frames=1, voxel=voxel, storage=storage)
    if kind in ("single", "sequence"):
        c = dict(kind=kind, width=width, height=height, frames=rng.randint(2, 16 if width < 800 else 10),
                 voxel=voxel, storage=storage)
        if kind == "sequence":
            c["weight"] = rng.choice(["plain", "learned"])
        return c
    if kind == "maps":
        return dict(kind=kind, maps=rng.randint(2, 8), frames=rng.randint(1, 4), voxel=max(voxel, 0.005),
                    storage=storage)
    if kind == "session":
        return dict(kind=kind, width=min(width, 640), height=min(height, 480), frames=10 * rng.randint(1, 6),
                    voxel=max(voxel, 0.005), storage=storage)
    if kind == "raycast":
        return dict(kind=kind, width=min(width, 640), height=min(height, 480), voxel=voxel, storage=storage)
    pixels = 4 * 640 * 480 if kind == "train" else 8 * 640 * 480
    images = rng.randint(1, max(1, min(8, pixels // (width * height))))
    if images * width * height > pixels:
        width, height, images = 640, 480, 1
    return dict(kind=kind, width=width, height=height, images=images)


# ------------------------------------------------------------------ inputs

_RING = {"live": 24, "single": 40, "sequence": 40, "maps": 12, "raycast": 1}
_WARM = {"live": 12, "single": 20, "sequence": 20, "maps": 8, "raycast": 12}


def _walk(seed, n, width, height, room=(8.0, 8.0, 3.0), prims=80):
    return scene.room_walk_sequence(int(seed), n_frames=n, width=width, height=height, n_prims=prims, room=room)


def _frames(seq, ks, learned=False):
    """The frames on the GPU: depth int16 bit patterns [n, H, W], BGR uint8 [n, H, W, 3], cameras."""
    noise = dict(noise_k=confidence.NOISE_K, flying_frac=confidence.FLYING) if learned else {}
    d = torch.empty((len(ks), seq.height, seq.width), dtype=torch.int16, device="cuda")
    c = torch.empty((len(ks), seq.height, seq.width, 3), dtype=torch.uint8, device="cuda")
    cams = []
    for i, k in enumerate(ks):
        R, t = seq.poses[k]
        dk, ck = scene.render_torch(seq.scene, R, t, seq.width, seq.height, seq.K, seq.seed, k, cull_m=MAXCAM + 1.0,
                                    **noise)
        d[i].copy_(dk)
        c[i].copy_(ck)
        cams.append(fusion.CameraInfo(seq.K, R, t))
    return d, c, cams


def _map(case, voxel=None, leaves=60000, rcp="host"):
    v = voxel or case["voxel"]
    f = fusion.FusionMipMapCPU(0, 0, 0, v, 2 * v, 0, True, leaves_max=leaves, branches_max=1 << 21,
                               storage=case["storage"], rcp=rcp)
    f.set_stream(torch.cuda.current_stream().cuda_stream)
    return f


def _pointers(d, c, ks):
    return [d[k].data_ptr() for k in ks], [c[k].data_ptr() for k in ks]


def _pinned(t):
    return t.cpu().pin_memory()


# The vertex and face buffers a program draws from: of fixed size, filled from the front.
_NV, _NF = 600000, 800000


class _Device:
    """An array in the map's device memory, for torch.as_tensor."""

    def __init__(self, ptr, shape, typestr):
        self.__cuda_array_interface__ = dict(shape=shape, typestr=typestr, data=(ptr, False), version=2)


def _device_buffers(nv=_NV, nf=_NF):
    return [torch.zeros((n, 3), dtype=t, device="cuda")
            for n, t in ((nv, torch.float32), (nv, torch.uint8), (nf, torch.int32))]


def _device_mesh(f, out):
    """The map's mesh (ff_get_mesh_counts, ff_get_mesh_device) into device buffers: sizes, vertices, colours, faces."""
    L = fusion.load_library()
    nv, nf = ctypes.c_uint64(), ctypes.c_uint64()
    p = [ctypes.c_void_p() for _ in range(3)]
    if L.ff_get_mesh_counts(f._h, ctypes.byref(nv), ctypes.byref(nf)) or \
            L.ff_get_mesh_device(f._h, *[ctypes.byref(x) for x in p]):
        raise RuntimeError("no mesh")
    for x, n, ty, o in zip(p, (nv.value, nv.value, nf.value), ("<f4", "|u1", "<i4"), out):
        n = min(n, o.shape[0])
        if n:
            o[:n].copy_(torch.as_tensor(_Device(x.value, (n, 3), ty), device="cuda"))
    return [np.array([nv.value, nf.value], np.int64), *out]


class _Held(np.ndarray):
    """A view of a MeshBuffer's memory that keeps the buffer."""


def _host_buffers():
    """A MeshBuffer and its whole memory as arrays (zero until filled)."""
    out = fusion.MeshBuffer(_NV, _NF)
    arrays = []
    for key, dtype, n in (("xyz", np.float32, _NV), ("rgb", np.uint8, _NV), ("faces", np.int32, _NF)):
        v = out.view(key, dtype, (n, 3)).view(_Held)
        v.owner = out
        v[:] = 0
        arrays.append(v)
    return out, arrays


def _host_mesh(f, buffers):
    out, arrays = buffers
    m = f.getMeshInterleavedMarchingCubes(out)
    return [np.array([len(m.vertices), len(m.faces)], np.int64), *arrays]


def _batch(case, seed):
    """Depth images [n, H, W] on the GPU and the intrinsics, of a noisy walk."""
    n, w, h = case["images"], case["width"], case["height"]
    seq = _walk(seed, 10 * n, w, h)
    d, _, _ = _frames(seq, list(range(0, 10 * n, 10)), learned=True)
    return d, seq.K


def _train_inputs(case, seed):
    """A training step's inputs: features (with the library's own kernel), targets (cm, -1 where there is no
    label) and the optimiser's state some hundred steps into a training."""
    d, K = _batch(case, seed)
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) + 5)
    shape = (case["images"], case["height"], case["width"])
    t = torch.rand(shape, generator=g, device="cuda").pow(3) * confidence.CAP_CM
    t = torch.where((d == 0) | (torch.rand(shape, generator=g, device="cuda") < 0.02), torch.full_like(t, -1.0), t)
    p = confidence.init_params(int(seed) % 1000)
    m = torch.randn(confidence.N_PARAMS, generator=g, device="cuda") * 0.05
    v = torch.rand(confidence.N_PARAMS, generator=g, device="cuda") * 0.02 + 0.001
    return d, K, t, p, m, v


_LR, _STEP = 2e-3, 200


_STREAM = None


def _stream():
    """The program's own stream: all work, and what reads a map's mesh, is ordered on it."""
    global _STREAM
    if _STREAM is None:
        _STREAM = torch.cuda.Stream()
    return torch.cuda.stream(_STREAM)


def prepare(case, seed):
    with _stream():
        return _prepare(case, seed)


def _prepare(case, seed):
    kind = case["kind"]
    if kind in ("infer", "train"):
        if kind == "infer":
            d, K = _batch(case, seed)
            params, tau = confidence.load_weights()
            return dict(kind=kind, net=confidence.ConfidenceNet(params), depth=d, K=K, tau=tau)
        d, K, t, p, m, v = _train_inputs(case, seed)
        net = confidence.ConfidenceNet(p)
        net.m.copy_(m)
        net.v.copy_(v)
        net.step_no = _STEP
        return dict(kind=kind, net=net, feat=net.features(d, K), target=t, inv=1.0 / max(1, int((t >= 0).sum())))
    if kind == "session":
        seq = _walk(seed, case["frames"], case["width"], case["height"])
        d, c, cams = _frames(seq, range(case["frames"]))
        return dict(kind=kind, case=dict(case), depth=[x.numpy().view(np.uint16) for x in _pinned(d)],
                    bgr=[x.numpy() for x in _pinned(c)], cams=cams, out=_host_buffers())
    warm, ring = _WARM[kind], _RING[kind]
    if kind == "maps":
        sizes = ((320, 240), (640, 480), (1280, 960), (640, 480))
        s = dict(kind=kind, frames=case["frames"], next=0, ring=ring, maps=[], data=[],
                 out=[_device_buffers() for _ in range(case["maps"])])
        for i in range(case["maps"]):
            w, h = sizes[i % 4]
            side = (4.0, 6.0, 9.0, 12.0, 5.0)[i % 5]
            seq = _walk(int(seed) * 64 + i, warm + ring, w, h, room=(side, side, 3.0), prims=10 + 20 * (i % 7))
            f = _map(case, voxel=case["voxel"] * (1.0 + 0.1 * (i % 5)), leaves=40000)
            d, c, cams = _frames(seq, range(warm + ring))
            f.addMapSequenceDevice(*_pointers(d, c, range(warm)), w, h, cams[:warm], SCALING, MAXCAM)
            f.updateMeshes()
            s["maps"].append(f)
            s["data"].append((d[warm:].clone(), c[warm:].clone(), cams[warm:], w, h))
        return s
    learned = case.get("weight") == "learned"
    if case["width"] > 800:
        ring = min(ring, 20)
    seq = _walk(seed, warm + ring, case["width"], case["height"])
    d, c, cams = _frames(seq, range(warm + ring), learned)
    f = _map(case)
    if learned:
        params, tau = confidence.load_weights()
        f.set_confidence(params, tau)
    f.addMapSequenceDevice(*_pointers(d, c, range(warm)), seq.width, seq.height, cams[:warm], SCALING, MAXCAM)
    f.updateMeshes()
    f.sync()
    s = dict(kind=kind, map=f, frames=case.get("frames", 1), next=0, ring=ring, width=seq.width, height=seq.height,
             cams=cams[warm:])
    if kind == "live":
        s.update(depth=[x.numpy().view(np.uint16) for x in _pinned(d[warm:])],
                 bgr=[x.numpy() for x in _pinned(c[warm:])], out=_host_buffers())
    else:
        s.update(depth=d[warm:].clone(), bgr=c[warm:].clone(), out=_device_buffers())
    if kind == "raycast":
        s["out"] = torch.empty((seq.height, seq.width), dtype=torch.float32, device="cuda")
    return s


def run(state):
    with _stream():
        return _run(state)


def _run(state):
    kind = state["kind"]
    if kind == "infer":
        net = state["net"]
        feat = net.features(state["depth"], state["K"])
        return dict(features=feat, confidence=net.forward(feat, state["tau"]))
    if kind == "train":
        net = state["net"]
        net.train_step(state["feat"], state["target"], state["inv"], _LR)
        return dict(loss=net.loss, prediction=net.bufs(*state["target"].shape)["pred"], weights=net.master, m=net.m, v=net.v)
    if kind == "session":
        f = _map(state["case"], leaves=30000, rcp="exact")
        counts = []
        for i in range(0, len(state["cams"]), 10):
            counts += f.addMapSequence(state["depth"][i:i + 10], state["cams"][i:i + 10], state["bgr"][i:i + 10],
                                       SCALING, MAXCAM)
            f.updateMeshes()
        mesh = _host_mesh(f, state["out"])
        f.close()
        return dict(queued=np.array(counts, np.int32), mesh=mesh)
    if kind == "raycast":
        state["map"].raycast_depth(state["depth"][0].data_ptr(), state["width"], state["height"], state["cams"][0],
                                   state["out"].data_ptr(), SCALING, confidence.CAP_CM * confidence.UNIT_M,
                                   0.5 * confidence.VOXEL_M)
        return state["out"]
    ks = [(state["next"] + i) % state["ring"] for i in range(state["frames"])]
    state["next"] = (ks[-1] + 1) % state["ring"]
    if kind == "maps":
        counts = []
        for k in ks:
            data = state["data"]
            counts.append(fusion.add_maps_device(
                state["maps"], [x[0][k].data_ptr() for x in data], [x[1][k].data_ptr() for x in data],
                [x[3] for x in data], [x[4] for x in data], [x[2][k] for x in data], SCALING, MAXCAM))
        meshes = []
        for f in state["maps"]:
            f.updateMeshes()
            meshes.append(_device_mesh(f, state["out"][len(meshes)]))
        return dict(queued=np.array(counts, np.int32), meshes=meshes)
    f, cams = state["map"], [state["cams"][k] for k in ks]
    if kind == "live":
        n = f.addMap(state["depth"][ks[0]], cams[0], state["bgr"][ks[0]], SCALING, MAXCAM)
        f.updateMeshes()
        return dict(queued=n, mesh=_host_mesh(f, state["out"]))
    dd, cc = _pointers(state["depth"], state["bgr"], ks)
    if kind == "sequence":
        counts = f.addMapSequenceDevice(dd, cc, state["width"], state["height"], cams, SCALING, MAXCAM)
    else:
        counts = [f.addMapDevice(a, b, state["width"], state["height"], cam, SCALING, MAXCAM)
                  for a, b, cam in zip(dd, cc, cams)]
    f.updateMeshes()
    return dict(queued=np.array(counts, np.int32), mesh=_device_mesh(f, state["out"]))


# ------------------------------------------------- what a pass cannot do without

# The walk in the 8x8 m room: surface bricks one frame sees at 5 mm (about 800,
# scaling with 1 / voxel^2), those that each further frame of a step adds, and
# the mesh of a brick's surface.
_BRICKS, _MORE, _VERTS, _FACES = 800, 35, 80, 103


def _fusion_bytes(frames, width, height, voxel, storage, mesh_bricks=None):
    bricks = (_BRICKS + _MORE * (frames - 1)) * (0.005 / voxel) ** 2
    pixels = 5 * frames * width * height
    state = bricks * 512 * 2 * ((4 if storage == "fp16" else 8) + 6)
    return pixels + state + (bricks if mesh_bricks is None else mesh_bricks) * (15 * _VERTS + 12 * _FACES)


def work(case):
    kind = case["kind"]
    if kind in ("infer", "train"):
        px = case["images"] * case["width"] * case["height"]
        macs = 16 * 5 * 25 + 16 * 16 * 25 + 16 * 25
        if kind == "infer":
            return dict(bytes=px * (2 + 16 + 4), flops=2.0 * px * macs)
        # forward, the weight gradients, and the input gradients of layers 3 and 2
        return dict(bytes=px * (16 + 4) + 8833 * 4 * 8, flops=2.0 * px * (2 * macs + 16 * 16 * 25 + 16 * 25))
    if kind == "raycast":
        px = case["width"] * case["height"]
        return dict(bytes=px * 6 + _BRICKS * 512 * 8, flops=px * 120 * 60.0)
    if kind == "maps":
        sizes = ((320, 240), (640, 480), (1280, 960), (640, 480))
        b = sum(_fusion_bytes(case["frames"], *sizes[i % 4], case["voxel"] * (1.0 + 0.1 * (i % 5)), case["storage"])
                for i in range(case["maps"]))
        return dict(bytes=b, flops=0)
    return dict(bytes=_fusion_bytes(case["frames"], case["width"], case["height"], case["voxel"], case["storage"]),
                flops=0)


# --------------------------------------------------------------- 64 bits

def _bf16(x):
    """A value as the network stores it (the gradient passes through)."""
    return x + (x.detach().float().to(torch.bfloat16).double() - x.detach())


def _features64(d, K):
    """Depth, unit normal from central differences and validity, in 64 bits (stored as BF16 by the network)."""
    z = (d.to(torch.int32) & 0xFFFF).double() * float(np.float32(SCALING))
    n, H, W = z.shape
    fx, fy, cx, cy = (float(np.float32(v)) for v in K)
    p = torch.nn.functional.pad(z, (1, 1, 1, 1))
    zl, zr, zu, zd = p[:, 1:-1, :-2], p[:, 1:-1, 2:], p[:, :-2, 1:-1], p[:, 2:, 1:-1]
    x = torch.arange(W, dtype=torch.float64, device=d.device)[None, None, :]
    y = torch.arange(H, dtype=torch.float64, device=d.device)[None, :, None]
    a = torch.stack([((x + 1 - cx) * zr - (x - 1 - cx) * zl) / fx, (y - cy) * (zr - zl) / fy, zr - zl])
    b = torch.stack([(x - cx) * (zd - zu) / fx, ((y + 1 - cy) * zd - (y - 1 - cy) * zu) / fy, zd - zu])
    nrm = torch.linalg.cross(b, a, dim=0)
    length = nrm.norm(dim=0, keepdim=True)
    ok = ((z > 0) & (zl > 0) & (zr > 0) & (zu > 0) & (zd > 0))[None] & (length > 0)
    nrm = torch.where(ok, nrm / torch.where(ok, length, torch.ones_like(length)), torch.zeros_like(nrm))
    f = torch.zeros((n, H, W, 8), dtype=torch.float64, device=d.device)
    f[..., 0] = z
    f[..., 1:4] = nrm.permute(1, 2, 3, 0)
    f[..., 4] = (z > 0).double()
    return f


def _net64(feat, params):
    """The three layers from stored features [n, H, W, 8]: the prediction (cm) [n, H, W]."""
    conv = torch.nn.functional.conv2d
    q = _bf16(params)
    part = [q[o:o + k] for o, k in confidence.LAYOUT]
    x = feat[..., :5].permute(0, 3, 1, 2)
    with torch.backends.cudnn.flags(enabled=False):
        x = _bf16(torch.relu(conv(x, part[0].view(16, 5, 5, 5), part[1], padding=2)))
        x = _bf16(torch.relu(conv(x, part[2].view(16, 16, 5, 5), part[3], padding=2)))
        return conv(x, part[4].view(1, 16, 5, 5), part[5], padding=2)[:, 0]


def exact(case, seed):
    """The confidence network's passes in 64 bits: stored features, activations and weights are BF16 by the
    network's definition, everything between them is not rounded.  The fused maps have none: which bricks a frame
    touches follows from a recurrence over its pixels in raster order and from the reference's float arithmetic,
    and a plain program takes minutes for it."""
    kind = case["kind"]
    if kind == "infer":
        d, K = _batch(case, seed)
        params, tau = confidence.load_weights()
        f = _features64(d, K)
        with torch.no_grad():
            out = torch.cat([_net64(_bf16(f[i:i + 1]), torch.as_tensor(params, dtype=torch.float64, device="cuda"))
                             for i in range(f.shape[0])])
            c = torch.clamp(1.0 - torch.relu(out) / (tau / confidence.UNIT_M), min=0.0)
            return dict(features=f, confidence=c * c)
    if kind == "train":
        d, K, target, p, m, v = _train_inputs(case, seed)
        inv = 1.0 / max(1, int((target >= 0).sum()))
        w = torch.as_tensor(p, dtype=torch.float64, device="cuda").requires_grad_()
        loss = torch.zeros((), dtype=torch.float64, device="cuda")
        preds = []
        for i in range(case["images"]):
            pred = _net64(_bf16(_features64(d[i:i + 1], K)), w)
            t = target[i:i + 1].double()
            part = (torch.where(t >= 0, pred - t, torch.zeros_like(t)) ** 2).sum() * inv
            part.backward()
            preds.append(pred.detach())
            loss = loss + part.detach()
        g, m, v, step = w.grad, m.double(), v.double(), _STEP + 1
        m = 0.9 * m + 0.1 * g
        v = 0.999 * v + 0.001 * g * g
        new = w.detach() - _LR * (m / (1 - 0.9 ** step)) / (torch.sqrt(v / (1 - 0.999 ** step)) + 1e-8)
        return dict(loss=loss.reshape(1), prediction=torch.cat(preds), weights=new, m=m, v=v)
    return None

"""The calls a user of the engine makes, at the sizes they are made at.

``listed()`` are the fixed cases and ``draw(rng)`` gives more of the same ranges; ``prepare``
makes what a program holds before the call (images, POI queues, an engine), ``run`` is one pass
through the public entry points, ``work`` the bytes and operations the result cannot do without,
and ``exact`` the same result in 64 bits by plain torch.

Images are seeded speckle: a sum of Gaussian spots, rendered for the reference as it is and for
a target at the material point each pixel shows (so the target is exact, not resampled), plus
sensor noise.  The displacement is a translation, a small affine strain and a sine whose local
strain is about 1 %.  POI queues are the solvers' grids (margin radius + 2).

Outputs are the queue's result fields: the six deformation parameters of every POI and its
result record (seed u0, v0, zncc, iteration, convergence, feature).
"""
import math
import random

import numpy as np
import torch

import fasticgn_gb300 as dic
from fasticgn_gb300 import _lib
from fasticgn_gb300.proposal import WEIGHTS, ProposalNet

_DTYPES = {"u8": (torch.uint8, _lib.DIC_U8, 255), "u16": (torch.uint16, _lib.DIC_U16, 4095),
           "f32": (torch.float32, _lib.DIC_F32, 255)}
_FRAMES = 6          # a stream's frames: two solved by prepare, the other four by each pass
_BATCH = ("1536x1120:15:4 384x512:10:3 1024x768:20:5 640x900:30:6 2048x512:12:5 333x451:15:2 "
          "256x256:20:4 1200x800:10:4")


def listed():
    return [
        # one small pair handed over in host memory and its results read back: latency of the
        # whole call counts (a 512 x 512 camera crop on a coarse grid)
        {"name": "host_pair_512", "call": "host", "w": 512, "h": 512, "radius": 15, "step": 10, "dtype": "u8"},
        # the dense full-frame pair: FFTCC seed and IC-GN on a quarter million POIs
        {"name": "pair_2048_r15", "call": "pair", "w": 2048, "h": 2048, "radius": 15, "step": 4, "dtype": "u8"},
        # full field, one POI per pixel, small subsets on a wide low frame
        {"name": "pair_1036x186_r7", "call": "pair", "w": 1036, "h": 186, "radius": 7, "step": 1, "dtype": "u8"},
        # wide subsets (coarse speckle) on an odd-width 12-bit frame
        {"name": "pair_1023x771_r20", "call": "pair", "w": 1023, "h": 771, "radius": 20, "step": 5, "dtype": "u16"},
        {"name": "pair_1024_r30", "call": "pair", "w": 1024, "h": 1024, "radius": 30, "step": 5, "dtype": "u8"},
        # the 63 x 63 subsets of the accuracy gate, float images
        {"name": "pair_700x500_r31", "call": "pair", "w": 700, "h": 500, "radius": 31, "step": 6, "dtype": "f32"},
        # a camera stream: every frame seeded from the one before, results read back
        {"name": "stream_2048_r15", "call": "stream", "w": 2048, "h": 2048, "radius": 15, "step": 5, "dtype": "u16"},
        {"name": "stream_1036x186_r7", "call": "stream", "w": 1036, "h": 186, "radius": 7, "step": 1, "dtype": "u8"},
        # pairs of different sizes, radii and POI counts solved together
        {"name": "batch_8_pairs", "call": "batch", "jobs": _BATCH, "dtype": "u8"},
        # seeds from the proposal network, FFTCC where they fail
        {"name": "learned_1024_r15", "call": "learned", "w": 1024, "h": 1024, "radius": 15, "step": 4, "dtype": "u8"},
        # the proposal network's training: forward, loss and backward of one mini-batch
        {"name": "train_4096", "call": "train", "batch": 4096},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_frame(rng, radius, most):
    """A frame size and a step that give up to about ``most`` POIs of this radius."""
    lo = max(160, 4 * radius + 40)
    w, h = _log_int(rng, lo, 2048), _log_int(rng, lo, 2048)
    m = 2 * (radius + 2)
    pois = _log_int(rng, 1000, most)
    step = max(1, math.ceil(math.sqrt((w - m) * (h - m) / pois)))
    return w, h, step


def draw(rng):
    call = rng.choice(["host", "pair", "pair", "pair", "pair", "stream", "batch", "learned", "train"])
    if call == "train":
        return {"call": call, "batch": _log_int(rng, 256, 6000)}
    dtype = rng.choice(["u8", "u8", "u16", "f32"])
    if call == "batch":
        jobs = []
        for _ in range(rng.randint(3, 10)):
            r = rng.choice([10, 12, 15, 20, 30])
            w, h, step = _draw_frame(rng, r, 40_000 if r <= 15 else 15_000)
            jobs.append("%dx%d:%d:%d" % (w, h, r, step))
        return {"call": call, "jobs": " ".join(jobs), "dtype": dtype}
    r = 15 if call == "learned" else rng.randint(7, 31)
    w, h, step = _draw_frame(rng, r, {"host": 20_000, "learned": 60_000}.get(call, 120_000 if r <= 15 else 25_000))
    return {"call": call, "w": w, "h": h, "radius": r, "step": step, "dtype": dtype}


# ------------------------------------------------------------------------------------ images

def _cuda():
    return torch.device("cuda", 0)


class _Scene:
    """Speckle and displacement of one image pair (or stream), from a seed."""

    def __init__(self, seed, w, h, radius, max_value):
        rng = np.random.default_rng(seed)
        self.w, self.h, self.max_value = w, h, max_value
        pad, fine = 28.0, radius < 10            # small subsets are used with fine speckle
        n = int((3000.0 / 512**2) * (2.0 if fine else 1.0) * (w + 2 * pad) * (h + 2 * pad))
        sigma = rng.uniform(1.0, 2.0, n) if fine else rng.uniform(1.5, 3.0, n)
        scale = max_value / 255.0
        host = np.stack([rng.uniform(-pad, w + pad, n), rng.uniform(-pad, h + pad, n), sigma,
                         rng.uniform(80.0, 200.0, n) * scale])
        self.x, self.y, self.sigma, self.peak = torch.from_numpy(host).to(_cuda())
        self.background, self.noise = 40.0 * scale, rng.uniform(1.0, 2.0) * scale
        most = min(8.0, 0.3 * radius)
        sign = rng.choice([-1.0, 1.0], 2)
        self.shift = sign * rng.uniform(0.2, 0.5, 2) * most
        self.strain = rng.uniform(-0.2, 0.2, 4) * most / max(w, h)
        self.amp, self.wave = 0.2 * most, 400.0 * most / 4.5
        self.phase = rng.uniform(0.0, 2 * math.pi, 2)
        self.gen = torch.Generator(device=_cuda())
        self.gen.manual_seed(int(seed) * 7919 + 13)

    def field(self, x, y, part):
        k = 2 * math.pi / self.wave
        cx, cy = x - 0.5 * self.w, y - 0.5 * self.h
        s = self.strain
        u = self.shift[0] + s[0] * cx + s[1] * cy + self.amp * torch.sin(k * x + self.phase[0])
        v = self.shift[1] + s[2] * cx + s[3] * cy + self.amp * torch.sin(k * y + self.phase[1])
        return part * u, part * v

    def gradients(self, x, y, part):
        k = 2 * math.pi / self.wave
        s = self.strain
        ux = s[0] + self.amp * k * torch.cos(k * x + self.phase[0])
        vy = s[3] + self.amp * k * torch.cos(k * y + self.phase[1])
        return part * ux, part * s[1] + 0 * ux, part * s[2] + 0 * ux, part * vy

    def image(self, part, dtype):
        """The frame that shows ``part`` of the displacement (0: the reference)."""
        dev = _cuda()
        yy, xx = torch.meshgrid(torch.arange(self.h, dtype=torch.float64, device=dev),
                                torch.arange(self.w, dtype=torch.float64, device=dev), indexing="ij")
        bx, by, fx, fy = xx, yy, self.x, self.y
        if part:
            for _ in range(6):
                u, v = self.field(bx, by, part)
                bx, by = xx - u, yy - v
            u, v = self.field(self.x, self.y, part)
            fx, fy = self.x + u, self.y + v
        reach = int(math.ceil(4.0 * float(self.sigma.max())))
        off = torch.arange(-reach, reach + 1, device=dev)
        oy, ox = (o.reshape(-1) for o in torch.meshgrid(off, off, indexing="ij"))
        bx, by = bx.reshape(-1), by.reshape(-1)
        acc = torch.zeros(self.h * self.w, dtype=torch.int64, device=dev)   # fixed point: any order, same sum
        for a in range(0, len(fx), 1 << 14):
            b = a + (1 << 14)
            px = fx[a:b].round().long()[:, None] + ox
            py = fy[a:b].round().long()[:, None] + oy
            inside = (px >= 0) & (px < self.w) & (py >= 0) & (py < self.h)
            at = torch.where(inside, py * self.w + px, 0)
            d2 = (bx[at] - self.x[a:b, None]) ** 2 + (by[at] - self.y[a:b, None]) ** 2
            val = self.peak[a:b, None] * torch.exp(-d2 / (2.0 * self.sigma[a:b, None] ** 2))
            acc.index_add_(0, at.reshape(-1), (torch.where(inside, val, 0.0) * 2.0**32).round().long().reshape(-1))
        img = self.background + acc.reshape(self.h, self.w).double() * 2.0**-32
        img = img + self.noise * torch.randn((self.h, self.w), generator=self.gen, device=dev)
        img = img.clamp(0, self.max_value)
        if dtype == torch.float32:
            return img.float().contiguous()
        return img.round().to(torch.int32).to(dtype).contiguous()


def _pair(seed, w, h, radius, dtype, parts=(1.0,)):
    tt, _, top = _DTYPES[dtype]
    s = _Scene(seed, w, h, radius, top)
    return s, s.image(0.0, tt), [s.image(p, tt) for p in parts]


def _parts(case):
    return [0.55 + 0.05 * k for k in range(_FRAMES)] if case["call"] == "stream" else [1.0]


def _jobs(case):
    out = []
    for text in case["jobs"].split():
        size, r, step = text.split(":")
        w, h = size.split("x")
        out.append((int(w), int(h), int(r), int(step)))
    return out


def _device_queue(w, h, radius, step):
    q = dic.grid_queue(w, h, radius, step)
    return torch.from_numpy(q.view(np.uint8).copy()).to(_cuda())


def _host_image(t):
    return t.to(torch.int32).cpu().numpy().astype(np.uint16) if t.dtype == torch.uint16 else t.cpu().numpy()


def _fields(records):
    """Deformation and result fields of queue records (a float view, one row of 14 per POI)."""
    return {"deformation": records[:, 2:8], "result": records[:, 8:14]}


# ------------------------------------------------------------------------------ prepare and run

def prepare(case, seed):
    call = case["call"]
    if call == "train":
        x0, target = _samples(case["batch"], seed)
        return {"call": call, "net": ProposalNet(0, _init_params(seed)), "x0": x0, "target": target}
    if call == "batch":
        jobs = []
        for k, (w, h, r, step) in enumerate(_jobs(case)):
            _, ref, tars = _pair(seed * 101 + k, w, h, r, case["dtype"])
            tmpl = _device_queue(w, h, r, step)
            jobs.append((ref, tars[0], r, tmpl, torch.empty_like(tmpl)))
        return {"call": call, "engine": dic.Engine(15), "jobs": jobs}
    w, h, r, step = case["w"], case["h"], case["radius"], case["step"]
    _, ref, tars = _pair(seed, w, h, r, case["dtype"], _parts(case))
    e = dic.Engine(r)
    state = {"call": call, "engine": e, "dtype": _DTYPES[case["dtype"]][1], "w": w, "h": h}
    if call == "host":
        state |= {"ref": _host_image(ref), "tar": _host_image(tars[0]), "template": dic.grid_queue(w, h, r, step)}
        return state
    stride = w * ref.element_size()
    state |= {"ref": ref, "tars": tars, "stride": stride}
    if call == "stream":
        tmpl = dic.grid_queue(w, h, r, step)
        torch.cuda.synchronize()
        e.set_ref_device(ref.data_ptr(), w, h, stride, state["dtype"])
        e.sequence_begin(tmpl)
        for t in tars[:2]:
            e.sequence_frame(None, device_ptr=t.data_ptr(), width=w, height=h, dtype=state["dtype"], report=False)
        # page-locked result buffers, one per frame in flight
        pinned = [torch.empty(len(tmpl) * 14, dtype=torch.float32, pin_memory=True) for _ in range(_FRAMES - 2)]
        state |= {"pinned": pinned, "results": [p.numpy().view(dic.POI_DTYPE) for p in pinned]}
        e.sequence_fetch(state["results"][0], report=False)
        return state
    if call == "learned":
        tmpl = dic.grid_queue(w, h, r, step)
        pinned = torch.empty(len(tmpl) * 14, dtype=torch.float32, pin_memory=True)
        state |= {"net": ProposalNet.load(), "template": tmpl, "pinned": pinned,
                  "queue": pinned.numpy().view(dic.POI_DTYPE)}
        e.set_proposal(state["net"])
        return state
    tmpl = _device_queue(w, h, r, step)
    state |= {"template": tmpl, "queue": torch.empty_like(tmpl), "n": tmpl.numel() // dic.POI_DTYPE.itemsize,
              "stream": torch.cuda.ExternalStream(e.stream)}
    return state


def run(state):
    call = state["call"]
    if call == "train":
        loss, grad = state["net"].gradient(state["x0"], state["target"])
        return {"gradient": grad, "loss": float(loss)}
    e = state["engine"]
    if call == "batch":
        for _, _, _, tmpl, q in state["jobs"]:
            q.copy_(tmpl)
        e.batch_process_device([(ref, tar, r, q) for ref, tar, r, _, q in state["jobs"]])
        return [_fields(q.view(torch.float32).view(-1, 14)) for _, _, _, _, q in state["jobs"]]
    if call == "host":
        q = state["template"].copy()
        e.set_ref(state["ref"])
        e.set_tar(state["tar"])
        e.process_pair(q)
        return _fields(q.view(np.float32).reshape(-1, 14))
    w, h, dt = state["w"], state["h"], state["dtype"]
    if call == "stream":
        # the next frame is enqueued before the one before it is read
        res = state["results"]
        for k, t in enumerate(state["tars"][2:]):
            e.sequence_frame(None, device_ptr=t.data_ptr(), width=w, height=h, dtype=dt, report=False)
            if k:
                e.sequence_fetch(res[k - 1], report=False, frames_back=1)
        e.sequence_fetch(res[-1], report=False)
        return [_fields(r.view(np.float32).reshape(-1, 14)) for r in res]
    e.set_ref_device(state["ref"].data_ptr(), w, h, state["stride"], dt)
    e.set_tar_device(state["tars"][0].data_ptr(), w, h, state["stride"], dt)
    q = state["queue"]
    if call == "learned":
        np.copyto(q, state["template"])
        e.process_pair_learned(q)
        return _fields(q.view(np.float32).reshape(-1, 14))
    with torch.cuda.stream(state["stream"]):
        q.copy_(state["template"])
    e.run_device(q.data_ptr(), state["n"], _lib.DIC_RUN_FFTCC | _lib.DIC_RUN_ICGN | _lib.DIC_RUN_PREPARE)
    return _fields(q.view(torch.float32).view(-1, 14))


# ---------------------------------------------------------------------------------------- work

_NET_FLOPS = 2 * (256 * 32 * 18 + (64 + 16 + 4) * 32 * 288 + 128 * 256 + 256 * 6)


def _pois(w, h, r, step):
    m = r + 2
    return len(range(m, w - m, step)) * len(range(m, h - m, step))


def _solve_work(w, h, r, step, dtype, iterations, fftcc, images=2):
    n, es = _pois(w, h, r, step), {"u8": 1, "u16": 2, "f32": 4}[dtype]
    m = 2 * r
    flops = n * (2 * r + 1) ** 2 * (75.0 * iterations + 40.0)     # 75 per sample and iteration, 40 for its reference data
    if fftcc:
        flops += n * 2 * 5.0 * m * m * math.log2(m * m)           # one packed transform each way
    return {"bytes": float(images * w * h * es + 2 * 56 * n), "flops": flops}


def work(case):
    call = case["call"]
    if call == "train":
        n = case["batch"]
        return {"bytes": n * (31 * 31 * 2 * 2 + 24.0) + 4.0 * 62918 * 2, "flops": 3.0 * n * _NET_FLOPS}
    if call == "batch":
        each = [_solve_work(w, h, r, s, case["dtype"], 3, True) for w, h, r, s in _jobs(case)]
        return {k: sum(x[k] for x in each) for k in ("bytes", "flops")}
    a = case["w"], case["h"], case["radius"], case["step"], case["dtype"]
    if call == "stream":
        one = _solve_work(*a, 2, False, 1)
        return {k: (_FRAMES - 2) * v for k, v in one.items()}
    if call == "learned":
        one = _solve_work(*a, 2, False)
        one["flops"] += _pois(*a[:4]) * float(_NET_FLOPS)
        return one
    return _solve_work(*a, 3, True)


# --------------------------------------------------------------------------- the proposal network

_NET_SIZES = [("w", 32 * 18, 18), ("b", 32, 0)] + 3 * [("w", 32 * 288, 288), ("b", 32, 0)] + \
    [("w", 256 * 128, 128), ("b", 256, 0), ("w", 6 * 256, 256), ("b", 6, 0)]


def _init_params(seed):
    rng = np.random.default_rng(seed + 77)
    return np.concatenate([np.zeros(n, np.float32) if kind == "b" else
                           rng.normal(0.0, math.sqrt(2.0 / fan) * (0.5 if i == 10 else 1.0), n).astype(np.float32)
                           for i, (kind, n, fan) in enumerate(_NET_SIZES)])


def _windows(img, x, y):
    """31 x 31 windows at integer positions, each of zero mean and unit variance (edges repeat)."""
    h, w = img.shape
    o = torch.arange(-15, 16, device=img.device)
    xs, ys = (x[:, None] + o).clamp(0, w - 1), (y[:, None] + o).clamp(0, h - 1)
    win = img[ys[:, :, None], xs[:, None, :]]
    win = win - win.mean((1, 2), keepdim=True)
    return win / win.square().mean((1, 2), keepdim=True).sqrt()


def _samples(batch, seed):
    s, ref, (tar,) = _pair(seed, 1024, 1024, 15, "u8")
    g = torch.Generator(device=_cuda())
    g.manual_seed(int(seed) + 5)
    x, y = torch.randint(20, 1004, (2, batch), generator=g, device=_cuda())
    x0 = torch.stack([_windows(ref.double(), x, y), _windows(tar.double(), x, y)], dim=3)
    u, v = s.field(x.double(), y.double(), 1.0)
    ux, uy, vx, vy = s.gradients(x.double(), y.double(), 1.0)
    return x0.to(torch.bfloat16).contiguous(), torch.stack([u, v, ux, uy, vx, vy], dim=1).float().contiguous()


def _network(params, x0):
    """The network in 64 bits: x0 [n, 31, 31, 2] to (u, v, 100 ux, 100 uy, 100 vx, 100 vy)."""
    p = torch.split(params, [n for _, n, _ in _NET_SIZES])
    a = x0
    for layer in range(4):
        n, s, _, c = a.shape
        so = (s + 1) // 2
        a = torch.nn.functional.pad(a, (0, 0, 1, 1, 1, 1))
        cols = torch.cat([a[:, ky:ky + 2 * so - 1:2, kx:kx + 2 * so - 1:2] for ky in range(3) for kx in range(3)], dim=3)
        a = torch.relu(cols @ p[2 * layer].reshape(32, 9 * c).T + p[2 * layer + 1])
    a = torch.relu(a.reshape(len(a), 128) @ p[8].reshape(256, 128).T + p[9])
    return a @ p[10].reshape(6, 256).T + p[11]


# --------------------------------------------------------------------------------------- exact

_BC = torch.tensor([[-144.0, 384.0, -384.0, 144.0], [342.0, -702.0, 450.0, -90.0], [-198.0, -18.0, 270.0, -54.0],
                    [0.0, 336.0, 0.0, 0.0]], dtype=torch.float64) / 336.0
_CHUNK = 6_000_000     # samples handled together


def _grid64(w, h, r, step):
    m = r + 2
    xs = torch.arange(m, w - m, step, dtype=torch.float64, device=_cuda())
    ys = torch.arange(m, h - m, step, dtype=torch.float64, device=_cuda())
    y, x = torch.meshgrid(ys, xs, indexing="ij")
    return x.reshape(-1), y.reshape(-1)


def _fftcc64(ref, tar, x, y, r):
    """Whole-pixel displacement of every POI: the peak of the circular cross-correlation."""
    h, w = ref.shape
    m = 2 * r
    o = torch.arange(-r, r, device=ref.device)
    u, v = torch.zeros_like(x), torch.zeros_like(x)
    per = max(1, _CHUNK // (m * m))
    for a in range(0, len(x), per):
        s = slice(a, a + per)
        at = (y[s].long()[:, None, None] + o[:, None]) * w + x[s].long()[:, None, None] + o
        f, g = ref.reshape(-1)[at], tar.reshape(-1)[at]
        f, g = f - f.mean((1, 2), keepdim=True), g - g.mean((1, 2), keepdim=True)
        c = torch.fft.irfft2(torch.fft.rfft2(f).conj() * torch.fft.rfft2(g), s=(m, m)).reshape(len(f), -1)
        k = c.argmax(1)
        lu, lv = k % m, k // m
        u[s], v[s] = torch.where(lu > r, lu - m, lu).double(), torch.where(lv > r, lv - m, lv).double()
    return u, v


def _gradient64(img):
    gx, gy = torch.zeros_like(img), torch.zeros_like(img)
    gx[:, 2:-2] = (img[:, :-4] - img[:, 4:]) / 12 + (img[:, 3:-1] - img[:, 1:-3]) * (2 / 3)
    gy[2:-2] = (img[:-4] - img[4:]) / 12 + (img[3:-1] - img[1:-3]) * (2 / 3)
    return gx, gy


def _interpolate64(tar, x, y):
    """Bicubic B-spline value at (x, y): weights of the 4 x 4 pixels around each point."""
    h, w = tar.shape
    fx, fy = x.floor(), y.floor()
    at = (fy.long() - 1) * w + fx.long() - 1
    flat = tar.reshape(-1)

    def weights(d):
        return [_BC[3, m].item() + d * (_BC[2, m].item() + d * (_BC[1, m].item() + d * _BC[0, m].item()))
                for m in range(4)]
    wx, wy = weights(x - fx), weights(y - fy)
    out = torch.zeros_like(x)
    for n in range(4):
        row = wx[0] * flat[at + n * w]
        for m in range(1, 4):
            row += wx[m] * flat[at + n * w + m]
        out += wy[n] * row
    return out


def _icgn64(ref, tar, x, y, p, r, max_iteration=10, conv=1e-3):
    """First-order IC-GN from p [n, 6] = (u, ux, uy, v, vx, vy): (p, zncc, iterations, last step)."""
    h, w = ref.shape
    gx, gy = _gradient64(ref)
    ly, lx = (o.reshape(-1).double() for o in torch.meshgrid(*(2 * [torch.arange(-r, r + 1, device=ref.device)]),
                                                             indexing="ij"))
    span = torch.tensor([1.0, r, r, 1.0, r, r], dtype=torch.float64, device=ref.device)
    out = p.clone()
    zncc, iters, step = (torch.zeros_like(x) for _ in range(3))
    per = max(1, _CHUNK // len(lx))
    for a in range(0, len(x), per):
        s = slice(a, a + per)
        at = (y[s, None] + ly).long() * w + (x[s, None] + lx).long()
        f = ref.reshape(-1)[at]
        f = f - f.mean(1, keepdim=True)
        nf = f.norm(dim=1)
        g, q = gx.reshape(-1)[at], gy.reshape(-1)[at]
        sd = torch.stack([g, g * lx, g * ly, q, q * lx, q * ly], dim=1)
        hess = sd @ sd.transpose(1, 2)
        warp = torch.eye(3, dtype=torch.float64, device=ref.device).repeat(len(f), 1, 1)
        warp[:, 0, 0] += p[s, 1]; warp[:, 0, 1] = p[s, 2]; warp[:, 0, 2] = p[s, 0]
        warp[:, 1, 0] = p[s, 4]; warp[:, 1, 1] += p[s, 5]; warp[:, 1, 2] = p[s, 3]
        live = torch.arange(len(f), device=ref.device)
        px, py = x[s], y[s]
        for it in range(1, max_iteration + 1):
            W = warp[live]
            wx = px[live, None] + W[:, 0, 0, None] * lx + W[:, 0, 1, None] * ly + W[:, 0, 2, None]
            wy = py[live, None] + W[:, 1, 0, None] * lx + W[:, 1, 1, None] * ly + W[:, 1, 2, None]
            ok = ((wx >= 1) & (wy >= 1) & (wx < w - 2) & (wy < h - 2)).all(1)
            if not bool(ok.all()):
                zncc[a + live[~ok]] = -3.0
                live, wx, wy, W = live[ok], wx[ok], wy[ok], W[ok]
            if not len(live):
                break
            t = _interpolate64(tar, wx, wy)
            t = t - t.mean(1, keepdim=True)
            e = t * (nf[live] / t.norm(dim=1))[:, None] - f[live]
            z = e.square().sum(1) / nf[live].square()
            dp = torch.linalg.solve(hess[live], (sd[live] @ e[:, :, None]))[:, :, 0]
            d = torch.eye(3, dtype=torch.float64, device=ref.device).repeat(len(live), 1, 1)
            d[:, 0, 0] += dp[:, 1]; d[:, 0, 1] = dp[:, 2]; d[:, 0, 2] = dp[:, 0]
            d[:, 1, 0] = dp[:, 4]; d[:, 1, 1] += dp[:, 5]; d[:, 1, 2] = dp[:, 3]
            W = W @ torch.linalg.inv(d)
            warp[live] = W
            norm = (dp * span).norm(dim=1)
            end = (norm < conv) if it < max_iteration else torch.ones_like(norm, dtype=torch.bool)
            to = a + live[end]
            E = W[end]
            out[to] = torch.stack([E[:, 0, 2], E[:, 0, 0] - 1, E[:, 0, 1], E[:, 1, 2], E[:, 1, 0], E[:, 1, 1] - 1], dim=1)
            zncc[to] = torch.where(norm[end] < conv, 0.5 * (2 - z[end]), -4.0)
            iters[to], step[to] = float(it), norm[end]
            live = live[~end]
            if not len(live):
                break
    return out, zncc, iters, step


def _records64(seed_p, solved, u0, v0):
    p, zncc, iters, step = solved
    lost = zncc == -3.0                       # out of range: the seed stays, with the seeding step's own u0, v0
    u = torch.where(lost, u0, seed_p[:, 0])
    v = torch.where(lost, v0, seed_p[:, 3])
    return {"deformation": p, "result": torch.stack([u, v, zncc, iters, step, torch.zeros_like(u)], dim=1)}


def _from_fftcc64(ref, tar, x, y, r):
    u, v = _fftcc64(ref, tar, x, y, r)
    o = torch.zeros_like(u)
    p = torch.stack([u, o, o, v, o, o], dim=1)
    return _records64(p, _icgn64(ref, tar, x, y, p, r), o, o)


def _pair64(ref, tar, w, h, r, step):
    return _from_fftcc64(ref.double(), tar.double(), *_grid64(w, h, r, step), r)


def _wide(t):
    return t.to(torch.int32) if t.dtype == torch.uint16 else t


def exact(case, seed):
    call = case["call"]
    if call == "train":
        x0, target = _samples(case["batch"], seed)
        params = torch.from_numpy(_init_params(seed)).to(_cuda()).double().requires_grad_(True)
        scale = torch.tensor([1.0, 1.0, 100.0, 100.0, 100.0, 100.0], dtype=torch.float64, device=_cuda())
        loss = (_network(params, x0.double()) - target.double() * scale).square().mean()
        loss.backward()
        return {"gradient": params.grad.detach(), "loss": float(loss)}
    if call == "batch":
        out = []
        for k, (w, h, r, step) in enumerate(_jobs(case)):
            _, ref, tars = _pair(seed * 101 + k, w, h, r, case["dtype"])
            out.append(_pair64(_wide(ref), _wide(tars[0]), w, h, r, step))
        return out
    w, h, r, step = case["w"], case["h"], case["radius"], case["step"]
    _, ref, tars = _pair(seed, w, h, r, case["dtype"], _parts(case))
    ref, tars = _wide(ref), [_wide(t) for t in tars]
    if call in ("host", "pair"):
        return _pair64(ref, tars[0], w, h, r, step)
    ref, x, y = ref.double(), *_grid64(w, h, r, step)
    o = torch.zeros_like(x)
    if call == "stream":
        out = [_pair64(ref, tars[0], w, h, r, step)]
        for t in tars[1:]:
            # seeded from the frame before where that was solved, else from zero; then POIs that
            # came out bad (below 0.8, not -3) are solved again from FFTCC and the better one kept
            t, z0 = t.double(), out[-1]["result"][:, 2]
            p = torch.where((z0 >= 0)[:, None], out[-1]["deformation"], 0.0)
            got = _records64(p, _icgn64(ref, t, x, y, p, r), o, o)
            z = got["result"][:, 2]
            bad = ((z < 0.8) & (z != -3) & ((z < 0) | (z0 >= 0.8))).nonzero()[:, 0]
            if len(bad):
                again = _from_fftcc64(ref, t, x[bad], y[bad], r)
                fz = again["result"][:, 2]
                take = (fz != -3) & (fz >= z[bad])
                for name, value in again.items():
                    got[name][bad[take]] = value[take]
            out.append(got)
        return out[2:]
    tar = tars[0].double()
    params = torch.from_numpy(np.load(WEIGHTS)["params"]).to(_cuda()).double()
    net = []
    for a in range(0, len(x), 4096):
        xi, yi = x[a:a + 4096].long(), y[a:a + 4096].long()
        net.append(_network(params, torch.stack([_windows(ref, xi, yi), _windows(tar, xi, yi)], dim=3)))
    net = torch.cat(net)
    p = torch.stack([net[:, 0], net[:, 2] / 100, net[:, 3] / 100, net[:, 1], net[:, 4] / 100, net[:, 5] / 100], dim=1)
    got = _records64(p, _icgn64(ref, tar, x, y, p, r, max_iteration=6), o, o)
    bad = (got["result"][:, 2] < 0.9).nonzero()[:, 0]
    if len(bad):                                 # FFTCC and the full budget where the proposal did not hold
        for name, value in _from_fftcc64(ref, tar, x[bad], y[bad], r).items():
            got[name][bad] = value
    return got


if __name__ == "__main__":
    for c in listed() + [draw(random.Random(k)) for k in range(12)]:
        print(c, work(c))

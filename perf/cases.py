"""The encode work that this framework is timed on, through its public entry
points (mav1cu.Stream and mav1cu.Session).

Three kinds of case, each as a caller runs it:

  clip     planned frames of one or several clips through device-resident
           streams: every source frame comes from page-locked host memory and
           every frame's writer inputs (and shown reconstruction) leave by the
           compact export into page-locked images, as the encoder driver does
           it frame by frame. Outputs: the images.
  core     one frame through the backend's frame_core hook (motion search,
           analysis, edge types, reconstruction) against references that the
           same backend coded. Outputs: motion vectors, block records,
           superblock table, levels, reconstruction.
  filters  the post-reconstruction hooks of one frame: filter info,
           deblocking, CDEF and its choice. Outputs: filter info,
           reconstruction, choices.
  lr       the loop-restoration search and its application to one frame.
           Outputs: units, frame parameters (the chosen types), picture.

Every output is whole numbers, decided by integer rules (and by double
precision in a fixed order in the loop-restoration search): there is no
nearby value that would also do, so exact() has none to give.

Sizes, quantizers and tool sets are the repository's own: the 352x288,
1920x1080 and 3840x2160 clips with their flags, the batching workload's
frame sizes and quantizers, odd sizes as in the parity tests. The content
follows the synthetic clips' recipe (blurred noise panned with sub-pixel
steps, moving flat rectangles, sensor noise), made on the GPU from the seed.
"""
import os
import sys

# several streams per encoder: as many hardware queues as the driver offers
# (read when the CUDA context is created; the integration notes ask for it)
os.environ.setdefault("CUDA_DEVICE_MAX_CONNECTIONS", "32")
sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mav1-encoder_b200"))

import torch  # noqa: E402

import mav1cu  # noqa: E402

# tool sets by name: flags of the command line encoder
TOOLS = {
    # the real-time set: deblocking and CDEF on, loop restoration off
    "turbo": dict(turbo=1, keyint=60),
    # every tool: transform search, transform depth, dual filter, compound, loop restoration
    "full": dict(altref=16, golden=1, me_range=64),
    "full_altref4": dict(altref=4, golden=1, me_range=64),
    # one frame at a time without hidden frames, LAST and GOLDEN
    "lowdelay": dict(golden=1, keyint=0),
    # Walsh-Hadamard 4x4 everywhere (the quantizer index has to be 0)
    "lossless": dict(fast=1),
}


def listed():
    return [
        # the smallest everyday call: a short CIF clip, where launches and latency count
        dict(name="clip_cif_turbo", kind="clip", tools="turbo", w=352, h=288, frames=5, q=125, tiles=0, streams=1),
        # the headline workload: 1080p turbo, a key frame and eight hidden / leaf pairs
        dict(name="clip_1080p_turbo", kind="clip", tools="turbo", w=1920, h=1080, frames=17, q=125, tiles=2, streams=1),
        # batching: four small clips at once on one GPU
        dict(name="batch_360p_turbo", kind="clip", tools="turbo", w=640, h=360, frames=9, q=170, tiles=2, streams=4),
        # the quality workload: 3840x2160 with every tool, key frame and one inter frame
        dict(name="clip_2160p_full", kind="clip", tools="full", w=3840, h=2160, frames=2, q=90, tiles=3, streams=1),
        # every tool on a small picture with hidden and compound frames
        dict(name="clip_360p_full", kind="clip", tools="full_altref4", w=640, h=360, frames=5, q=90, tiles=1, streams=1),
        # low delay, odd size: nothing is a multiple of a block
        dict(name="clip_odd_lowdelay", kind="clip", tools="lowdelay", w=363, h=241, frames=4, q=120, tiles=1, streams=1),
        # lossless archiving of a small clip
        dict(name="clip_cif_lossless", kind="clip", tools="lossless", w=352, h=288, frames=3, q=0, tiles=1, streams=1),
        # one key frame at the batching workload's largest size (stream start, scene cut)
        dict(name="core_key_1440p", kind="core", frame="key", w=2560, h=1440, q=125, tiles=2),
        # one hidden ALTREF frame of the headline clip (one reference, inter and intra blocks)
        dict(name="core_altref_1080p", kind="core", frame="altref", w=1920, h=1080, q=125, tiles=2),
        # one leaf frame at 4K (two references, compound prediction)
        dict(name="core_leaf_2160p", kind="core", frame="leaf", w=3840, h=2160, q=170, tiles=2),
        # the loop filters of a 1080p key frame
        dict(name="filters_1080p", kind="filters", w=1920, h=1080, q=125, tiles=2),
        # loop restoration of a 720p frame
        dict(name="lr_720p", kind="lr", w=1280, h=720, q=90, tiles=1),
    ]


def draw(rng):
    def size(lo, hi):
        """Width and height of about 16:9, 4:3 or a tall picture, widths spread over their logarithm, odd ones among them."""
        w = int(round(lo * (hi / lo) ** rng.random()))
        h = max(64, int(round(w / rng.choice((16 / 9, 4 / 3, 1.0)))))
        return (w, h) if rng.random() < 0.5 else (w + w % 2, h + h % 2)

    kind = rng.choice(("turbo", "turbo", "full", "lowdelay", "lossless", "key", "altref", "leaf", "filters", "lr"))
    q = rng.choice((60, 80, 90, 125, 170, 200))
    tiles = rng.randrange(4)
    if kind == "turbo":
        w, h = size(96, 1920)
        streams = rng.choice((1, 1, 2, 4)) if w <= 1280 else 1
        return dict(kind="clip", tools="turbo", w=w, h=h, frames=rng.randrange(2, 12), q=q, tiles=tiles, streams=streams)
    if kind in ("full", "lowdelay"):
        w, h = size(96, 960)
        tools = "lowdelay" if kind == "lowdelay" else rng.choice(("full", "full_altref4"))
        return dict(kind="clip", tools=tools, w=w, h=h, frames=rng.randrange(1, 6), q=q, tiles=tiles, streams=1)
    if kind == "lossless":
        w, h = size(96, 640)
        return dict(kind="clip", tools="lossless", w=w, h=h, frames=rng.randrange(1, 5), q=0, tiles=tiles, streams=1)
    if kind in ("key", "altref", "leaf"):
        w, h = size(96, 2560)
        return dict(kind="core", frame=kind, w=w, h=h, q=q, tiles=tiles)
    w, h = size(96, 2560 if kind == "filters" else 1280)
    return dict(kind=kind, w=w, h=h, q=q, tiles=tiles)


# ---- content ---------------------------------------------------------------------------


def _blur(img, sigma):
    """Gaussian blur with a periodic border."""
    r = int(3 * sigma + 0.999)
    k = torch.exp(-0.5 * (torch.arange(-r, r + 1, device=img.device, dtype=torch.float32) / sigma) ** 2)
    k = k / k.sum()
    x = torch.nn.functional.pad(img[None, None], (r, r, r, r), mode="circular")
    x = torch.nn.functional.conv2d(x, k.view(1, 1, 1, -1))
    return torch.nn.functional.conv2d(x, k.view(1, 1, -1, 1))[0, 0]


def _clip(w, h, frames, seed):
    """Packed I420 frames [frames, bytes] on the GPU: a panned texture with moving rectangles and noise."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    s = max(1.0, w / 352.0)
    pan = (1.25 * min(s, 4.0), -0.5 * min(s, 4.0))
    n = int(round(4 * min(s, 6.0)))
    rnd = torch.rand(8, n, generator=g, device="cuda").tolist()
    lo, hi = int(24 * s) // 2 + 4, int(64 * s)
    rects = [(lo + int(a * (hi - lo)), lo + int(b * (hi - lo)), int(c * w) - lo // 2, int(d * h) - lo // 2,
              int(e * 9) - 4, int(f * 9) - 4, 30 + int(v * 190), 30 + int(u * 190)) for a, b, c, d, e, f, v, u in zip(*rnd)]
    size = w * h + 2 * ((w + 1) // 2) * ((h + 1) // 2)
    out = torch.empty(frames, size, dtype=torch.uint8, device="cuda")
    off = 0
    for p in range(3):
        div = 2 if p else 1
        pw, ph = (w + div - 1) // div, (h + div - 1) // div
        tex = _blur(torch.rand(ph + 64, pw + 64, generator=g, device="cuda") * 255, 5.0 if p else 3.0)
        th, tw = tex.shape
        for t in range(frames):
            oy, ox = pan[1] * t / div, pan[0] * t / div
            y0, x0 = int(oy // 1), int(ox // 1)
            fy, fx = oy - y0, ox - x0
            win = torch.roll(tex, (-y0, -x0), (0, 1))
            win = win + fx * (torch.roll(win, -1, 1) - win)
            win = win + fy * (torch.roll(win, -1, 0) - win)
            img = win[:ph, :pw].clone()
            for rw, rh, rx, ry, vx, vy, val, cval in rects:
                x, y = (rx + vx * t) // div, (ry + vy * t) // div
                img[max(y, 0):max(y + rh // div, 0), max(x, 0):max(x + rw // div, 0)] = (cval + 40 * p) % 256 if p else val
            img += 2.0 * torch.randn(ph, pw, generator=g, device="cuda")
            out[t, off:off + pw * ph] = img.round().clamp(0, 255).to(torch.uint8).reshape(-1)
        off += pw * ph
    return out


# ---- what a caller holds ------------------------------------------------------------------


class _Memory:
    """Device memory of a session buffer, for torch.as_tensor: a tensor made from it keeps the session alive."""

    def __init__(self, session, ptr, count, typestr):
        self.session = session
        self.__cuda_array_interface__ = dict(shape=(count,), typestr=typestr, data=(ptr, False), version=3)


def _view(session, name, dtype="|u1"):
    n = session.size(name) // int(dtype[2:])
    return torch.as_tensor(_Memory(session, session.device_ptr(name), n, dtype), device="cuda")


def _config(case):
    # only the full tool set restores
    tools = TOOLS[case.get("tools", "full" if case["kind"] == "lr" else "turbo")]
    return mav1cu.cli_config(case["w"], case["h"], q=case["q"], tiles=case["tiles"], **tools)


class _Clip:
    """Streams with their plans, sources in page-locked memory and an image for every frame."""

    def __init__(self, case, seed):
        cfg = _config(case)
        self.streams = [mav1cu.Stream(cfg) for _ in range(case["streams"])]
        jobs = mav1cu.plan(cfg, case["frames"])
        cap = (self.streams[0].engines[0].export_capacity() + 255) // 256 * 256  # every image starts aligned
        self.sources, self.images, self.steps = [], [], []
        for k in range(case["streams"]):
            dev = _clip(case["w"], case["h"], case["frames"], seed * 64 + k)
            src = torch.empty(dev.shape, dtype=torch.uint8, pin_memory=True)
            src.copy_(dev)
            self.sources.append(src)
            self.images.append(torch.zeros(len(jobs), cap, dtype=torch.uint8, pin_memory=True))
        for j, job in enumerate(jobs):  # the streams take turns, a frame each
            for k, st in enumerate(self.streams):
                self.steps.append((st, job, self.sources[k][job["disp"]].data_ptr(), self.images[k][j].data_ptr(), cap,
                                   not job["hidden"]))


def _padded(session, i420, name):
    """Loads a packed I420 picture into a session buffer, edges replicated to whole superblocks."""
    g = session.geom
    buf = _view(session, name)
    off = 0
    for p in range(3):
        pw, ph = ((g["w"] + 1) // 2, (g["h"] + 1) // 2) if p else (g["w"], g["h"])
        img = i420[off:off + pw * ph].view(1, 1, ph, pw).float()
        off += pw * ph
        img = torch.nn.functional.pad(img, (0, g["stride"][p] - pw, 0, g["plane_h"][p] - ph), mode="replicate")
        buf[g["offset"][p]:g["offset"][p] + img.numel()] = img.to(torch.uint8).view(-1)
    torch.cuda.synchronize()


class _Frame:
    """A session holding one frame's inputs: source, references and parameters."""

    def __init__(self, case, seed):
        cfg = _config(case)
        self.s = s = mav1cu.Session(case["w"], case["h"])
        clip = _clip(case["w"], case["h"], 3, seed)
        key, altref, leaf = mav1cu.plan(cfg, 3)[:3]
        frame = case.get("frame", "key")
        for disp, name in ((0, "REF"), (2, "GOLD")) if frame != "key" else ():
            params, presets = mav1cu.frame_params(cfg, key)
            _padded(s, clip[disp], "SRC")
            s.set_params(params)
            s.frame_core()
            s.filter_info()
            s.filter(presets)
            s.cdef_select(presets)
            s.copy(name, "REC")
            s.synchronize()
        job = dict(key=key, altref=altref, leaf=leaf)[frame]
        params, self.presets = mav1cu.frame_params(cfg, job)
        _padded(s, clip[int(job["disp"])], "SRC")
        s.set_params(params)
        s.synchronize()


class _Core(_Frame):
    def __init__(self, case, seed):
        super().__init__(case, seed)
        s = self.s
        self.out = dict(blocks=_view(s, "BLOCKS", "<i4"), sbs=_view(s, "SBS", "<i4"), levels=_view(s, "COEFS", "<i4"),
                        rec=_view(s, "REC"))
        if case["frame"] != "key":
            self.out.update(mv=_view(s, "MVFIELD", "<i4"), mv2=_view(s, "MVGOLD", "<i4"))

    def run(self):
        self.s.frame_core()
        return self.out


class _Filters(_Frame):
    def __init__(self, case, seed):
        super().__init__(case, seed)
        s = self.s
        s.frame_core()
        s.copy("LROUT", "REC")  # the unfiltered reconstruction
        s.synchronize()
        self.out = dict(rec=_view(s, "REC"), mask=_view(s, "LFMASK"), choice=_view(s, "CDEF_CHOICE"))

    def run(self):
        s = self.s
        s.copy("REC", "LROUT")
        s.filter_info()
        s.filter(self.presets)
        s.cdef_select(self.presets)
        return self.out


class _Restoration(_Frame):
    def __init__(self, case, seed):
        super().__init__(case, seed)
        s = self.s
        s.frame_core()
        s.filter_info()
        s.filter(self.presets)
        s.copy("DBK", "REC")
        s.cdef_select(self.presets)
        s.synchronize()
        self.out = dict(units=_view(s, "LRUNITS", "<i4"), params=_view(s, "PARAMS", "<i4"), picture=_view(s, "LROUT"))

    def run(self):
        s = self.s
        s.lr_search()
        s.copy("LROUT", "REC")
        s.restore()
        return self.out


def prepare(case, seed):
    kind = dict(clip=_Clip, core=_Core, filters=_Filters, lr=_Restoration)[case["kind"]]
    state = kind(case, seed)
    torch.cuda.synchronize()
    return state


def run(state):
    if not isinstance(state, _Clip):
        return state.run()
    for stream, job, source, image, cap, shown in state.steps:
        stream.encode(job, source, False).export(image, cap, rec=shown)
    return state.images


def work(case):
    """Each frame's source and references read once, its reconstruction and superblock records written once."""
    g = mav1cu.geometry(case["w"], case["h"])
    picture = case["w"] * case["h"] + 2 * ((case["w"] + 1) // 2) * ((case["h"] + 1) // 2)
    records = g["num_sbs"] * (mav1cu.SB_DTYPE.itemsize + mav1cu.BLOCK_DTYPE.itemsize)
    if case["kind"] == "clip":
        jobs = mav1cu.plan(_config(case), case["frames"])
        refs = sum((int(j["last_slot"]) >= 0) + (int(j["arf_slot"]) >= 0) for j in jobs)
        return dict(bytes=case["streams"] * (len(jobs) * (2 * picture + records) + refs * picture), flops=0)
    if case["kind"] == "core":
        refs = dict(key=0, altref=1, leaf=2)[case["frame"]]
        return dict(bytes=(2 + refs) * picture + records, flops=0)
    # the unfiltered picture (for loop restoration also the deblocked one) and the source read, the result written
    return dict(bytes=(3 if case["kind"] == "filters" else 4) * picture, flops=0)


def exact(case, seed):
    return None

"""The spot finder's timed cases: what a user of this framework has it do, through the package's public
calls, over the range of detectors, batch sizes, pixel widths, kernels and scenes that its benchmark,
tests and configurations use.

listed() names the cases, draw(rng) gives more of the same ranges, prepare(case, seed) makes what a
program holds before the call, run(state) is one pass, work(case) the bytes a pass cannot do without,
and exact(case, seed) the outputs that are computed numbers, in 64 bits by plain torch.

Frames are synthetic and made on the GPU: a Poisson background (flat, or falling from the beam centre to
the edge, with diffuse rings in the dense scene), Gaussian spots whose rocking curves span a few frames,
module gaps or masked bands and hot pixels as the masked value, and overloads in the dense scene.
"""
import importlib
import math

import numpy as np
import torch

# The package folder's name is no identifier; it is found through sys.path like any other.
_PKG = "dials-metal_gb300.sfgb"
api = importlib.import_module(_PKG + ".api")
labeller = importlib.import_module(_PKG + ".labeller")
synth = importlib.import_module(_PKG + ".synth")

# Detector shapes (height, width): EIGER2 1M, 4M, 9M and 16M.
SHAPES = {"1m": (1065, 1030), "4m": (2162, 2068), "9m": (3262, 3108), "16m": (4362, 4148)}

# Scenes: background at the edge and the centre, spots visible on a frame for each megapixel of it, spot
# widths, the masked pattern, rings and overloads, and the list capacity as a divisor of the pixel count.
SCENES = {
    # A small plain sweep: flat background, a masked band each way, a few hot pixels.
    "plain": dict(edge=0.5, centre=0.5, spots=190.0, sxy=(1.2, 1.2), sz=(0.8, 0.8), gaps="bands", hot=20, cap=16),
    # A rotation sweep on a module detector: low background falling with radius, gaps masked.
    "eiger": dict(edge=0.3, centre=1.5, spots=166.0, sxy=(1.0, 1.5), sz=(0.5, 1.0), gaps="modules", hot=20, cap=16),
    # Frames for batched thresholding: flat background of one count, wider spots, no gaps.
    "batch": dict(edge=1.0, centre=1.0, spots=250.0, sxy=(1.0, 2.0), sz=(0.8, 0.8), gaps=None, hot=0, cap=16),
    # High background with rings, many spots, 2% of the pixels overloaded.
    "dense": dict(edge=20.0, centre=20.0, spots=1105.0, sxy=(1.0, 1.5), sz=(0.8, 0.8), gaps="modules", hot=500,
                  rings=3, overload=0.02, cap=4),
}
OVERLOAD = 1_000_000
PEAKS = (50.0, 2000.0)


def _case(name, call, shape, frames, scene, bits=32, kernel=3, algorithm="extended"):
    h, w = SHAPES.get(shape, shape) if isinstance(shape, str) else shape
    return {"name": name, "call": call, "height": h, "width": w, "frames": frames, "scene": scene, "bits": bits,
            "kernel": kernel, "algorithm": algorithm}


def listed():
    return [
        # One frame of the smallest detector as it arrives (its rows are not whole 16-byte pieces): the
        # latency of a live display or of a data-collection loop.
        _case("frame_1m", "device", "1m", 1, "plain"),
        # One frame of the largest detector on the plain per-frame path.
        _case("frame_16m", "device", "16m", 1, "eiger"),
        # The throughput form: a detector loop's buffers through a plan, launched as one batch.
        _case("batch_16m", "plan", "16m", 32, "eiger"),
        # The batched form's other kernel sizes on the middle detectors.
        _case("batch_4m_k2", "plan", "4m", 32, "batch", kernel=2),
        _case("batch_9m_k4", "plan", "9m", 16, "batch", kernel=4),
        # The plain dispersion threshold, batched.
        _case("batch_9m_dispersion", "batch", "9m", 16, "batch", algorithm="dispersion"),
        # 16-bit detectors (and 32-bit ones read as 16-bit), batched.
        _case("batch_16m_u16", "batch", "16m", 16, "eiger", bits=16),
        # The dense stress: high background, rings, many spots and overloads.
        _case("dense_16m", "batch", "16m", 4, "dense"),
        # Several detectors served together: four frames of each in one launch sequence.
        _case("mixed_served", "mixed", "16m", 16, "eiger"),
        # A detector file's chunk: bitshuffle+LZ4 from host memory, decoded and thresholded, list to the host.
        _case("chunk_16m", "chunk", "16m", 1, "eiger"),
        # 3-D labelling of a sweep's lists: a labeller opened, fed in calls of 16 frames, finished and read.
        _case("label_16m", "label", "16m", 32, "eiger"),
        # A whole small sweep: dispersion threshold in batches of 50, labelled, spots read back.
        _case("sweep_1m_dispersion", "sweep", (1024, 1024), 100, "plain", algorithm="dispersion"),
    ]


def draw(rng):
    """One more case of the listed ranges: any detector size between 256 x 256 and the 16M one, odd sizes
    among them, 1 to 64 frames a call, both pixel widths, every kernel and algorithm, every call."""
    call = rng.choice(["device", "device", "plan", "plan", "batch", "batch", "mixed", "chunk", "label", "sweep"])
    h = int(round(math.exp(rng.uniform(math.log(256), math.log(4362)))))
    w = int(round(math.exp(rng.uniform(math.log(256), math.log(4148)))))
    if rng.random() < 0.6:  # most detectors' rows are whole pieces of 4 pixels
        w -= w % 4
    scene = rng.choice(["plain", "eiger", "batch", "batch", "dense"])
    algorithm = rng.choice(["extended", "extended", "extended", "dispersion"])
    kernel = rng.choice([3, 3, 3, 2, 4])
    bits = 16 if call in ("device", "batch") and rng.random() < 0.3 else 32
    if call in ("label", "sweep"):
        scene = rng.choice(["plain", "eiger"])  # one pool of the default size holds these sweeps
        kernel = 3
    if call == "chunk":
        bits = rng.choice([32, 32, 16])
    most = 64
    if scene == "dense" or algorithm == "dispersion" or bits == 16 or kernel != 3:
        most = 8
    most = max(1, min(most, int(150e6 // (h * w))))
    frames = int(round(math.exp(rng.uniform(0.0, math.log(most))))) if most > 1 else 1
    if call in ("device", "chunk"):
        frames = 1
    return {"call": call, "height": h, "width": w, "frames": frames, "scene": scene, "bits": bits,
            "kernel": kernel, "algorithm": algorithm}


def _shapes(case):
    """The frames' shapes: all alike, or for a mixed call cycling through the detector and three smaller
    ones (the served detectors' proportions)."""
    h, w, n = case["height"], case["width"], case["frames"]
    if case["call"] != "mixed":
        return [(h, w)] * n
    if (h, w) == SHAPES["16m"]:
        four = [SHAPES[k] for k in ("16m", "9m", "4m", "1m")]
    else:
        four = [(max(16, int(h * s)), max(16, int(w * s))) for s in (1.0, 0.75, 0.5, 0.25)]
    return [four[j % 4] for j in range(n)]


def _params(case):
    alg = api.DISPERSION if case["algorithm"] == "dispersion" else api.DISPERSION_EXTENDED
    return api.Params(algorithm=alg, kernel_x=case["kernel"], kernel_y=case["kernel"])


class _Sweep:
    """Frames z = 0 .. n - 1 of one seeded sweep of a scene, made on the GPU."""

    def __init__(self, scene, h, w, n, seed):
        s = SCENES[scene]
        self.s, self.h, self.w = s, h, w
        g = torch.Generator(device="cuda")
        g.manual_seed(int(seed) * 7919 + h * 31 + w)
        self.g = g

        def uniform(k):
            return torch.rand(k, generator=g, device="cuda", dtype=torch.float64)

        span = max(1.0, 2.5 * sum(s["sz"]))
        margin = 3.0 * s["sz"][1] + 1.0
        total = int(round(s["spots"] * h * w / 1e6 * (n + 2 * margin) / span)) + 1
        self.z = uniform(total) * (n + 2 * margin) - margin
        self.x = 3.0 + (w - 6.0) * uniform(total)
        self.y = 3.0 + (h - 6.0) * uniform(total)
        self.sxy = s["sxy"][0] + (s["sxy"][1] - s["sxy"][0]) * uniform(total)
        self.sz = s["sz"][0] + (s["sz"][1] - s["sz"][0]) * uniform(total)
        self.peak = PEAKS[0] * torch.exp(math.log(PEAKS[1] / PEAKS[0]) * uniform(total))
        yy = torch.arange(h, device="cuda", dtype=torch.float32)[:, None] + 0.5 - 0.5 * h
        xx = torch.arange(w, device="cuda", dtype=torch.float32)[None, :] + 0.5 - 0.5 * w
        r = torch.sqrt(yy * yy + xx * xx) / (0.5 * math.hypot(h, w))
        rate = s["centre"] + (s["edge"] - s["centre"]) * r
        for k in range(s.get("rings", 0)):
            d = (r - (k + 1.0) / (s["rings"] + 1.0)) / 0.01
            rate = rate + 15.0 * torch.exp(-0.5 * d * d)
        self.rate = rate
        row = torch.arange(h, device="cuda")[:, None]
        col = torch.arange(w, device="cuda")[None, :]
        masked = torch.zeros(h, w, dtype=torch.bool, device="cuda")
        if s["gaps"] == "modules":
            masked |= (row % 550 >= 512) | (col % 1040 >= 1028)
        elif s["gaps"] == "bands":
            masked |= ((row >= h // 2) & (row < h // 2 + 8)) | ((col >= w // 3) & (col < w // 3 + 8))
        if s["hot"]:
            masked.view(-1)[torch.randint(h * w, (s["hot"],), generator=g, device="cuda")] = True
        self.masked = masked

    def _share(self, f):
        k = 0.7071067811865476 / self.sz
        return 0.5 * (torch.erf((f + 1.0 - self.z) * k) - torch.erf((f - self.z) * k))

    def frame(self, z, bits):
        s, h, w = self.s, self.h, self.w
        share = self._share(float(z)) / self._share(torch.floor(self.z)).clamp_min(1e-12)
        amp = self.peak * share
        live = torch.nonzero((amp >= 0.05) & ((self.z - z).abs() < 4.0 * s["sz"][1] + 2.0)).view(-1)
        rate = self.rate.clone().view(-1)
        if live.numel():
            rad = int(math.ceil(3.5 * s["sxy"][1]))
            d = torch.arange(-rad, rad + 1, device="cuda")
            py = torch.floor(self.y[live])[:, None] + d[None, :]
            px = torch.floor(self.x[live])[:, None] + d[None, :]
            sig2 = 2.0 * self.sxy[live] ** 2
            ey = torch.exp(-(py + 0.5 - self.y[live][:, None]) ** 2 / sig2[:, None])
            ex = torch.exp(-(px + 0.5 - self.x[live][:, None]) ** 2 / sig2[:, None])
            val = (amp[live][:, None, None] * ey[:, :, None] * ex[:, None, :])
            inside = ((py >= 0) & (py < h))[:, :, None] & ((px >= 0) & (px < w))[:, None, :]
            at = (py.clamp(0, h - 1) * w)[:, :, None] + px.clamp(0, w - 1)[:, None, :]
            # Added in whole millionths, so that the sums do not depend on the order of the additions.
            add = torch.zeros(h * w, dtype=torch.int64, device="cuda")
            add.index_add_(0, at.long().view(-1), torch.where(inside, val * 1e6, 0.0).round().long().view(-1))
            rate += (add.double() * 1e-6).float()
        v = torch.poisson(rate, generator=self.g).view(h, w).to(torch.int32)
        if s.get("overload"):
            hit = torch.rand(h, w, generator=self.g, device="cuda") < s["overload"]
            v = torch.where(hit, torch.full_like(v, OVERLOAD), v)
        if bits == 16:
            v = v.clamp_max(65533)
        v[self.masked] = -1
        return v.to(torch.int16) if bits == 16 else v


def _frames(case, seed):
    shapes = _shapes(case)
    if case["call"] == "mixed":
        kinds = sorted(set(shapes))
        sweeps = {k: _Sweep(case["scene"], k[0], k[1], shapes.count(k), seed + 101 * i) for i, k in enumerate(kinds)}
        seen = dict.fromkeys(kinds, 0)
        out = []
        for k in shapes:
            out.append(sweeps[k].frame(seen[k], case["bits"]))
            seen[k] += 1
        return out
    s = _Sweep(case["scene"], case["height"], case["width"], case["frames"], seed)
    return [s.frame(z, case["bits"]) for z in range(case["frames"])]


class _View:
    """A plan's device memory, for torch.as_tensor: the tensor keeps this object, and so the plan, alive."""

    def __init__(self, plan, ptr, n, typestr="<i4"):
        self.plan = plan
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": typestr, "data": (ptr, False), "version": 3}


def _capacity(case):
    h, w = case["height"], case["width"]
    return max(64, h * w // SCENES[case["scene"]]["cap"])


def _lists(out, n, cap):
    """The fields of n signal lists of cap 16-byte records each (views, nothing is copied)."""
    r = out.view(torch.int32).view(-1, cap, 4)[:n]
    return {"index": r[..., 0], "value": r[..., 1], "background": r[..., 2].view(torch.float32), "population": r[..., 3]}


def prepare(case, seed):
    call, h, w = case["call"], case["height"], case["width"]
    p, cap = _params(case), _capacity(case)
    frames = _frames(case, seed)
    st = {"call": call, "case": case, "frames": frames, "cap": cap}
    if call == "device":
        t = st["threshold"] = api.DeviceThreshold(h, w, capacity=cap, params=p)
        t.out.zero_()
    elif call == "batch":
        t = st["threshold"] = api.DeviceBatch(h, w, len(frames), capacity=cap, params=p)
        t.out.zero_()
    elif call == "mixed":
        t = st["threshold"] = api.MixedBatch([tuple(f.shape) for f in frames], capacity=cap, params=p)
        t.out.zero_()
        t.bits.zero_()
    elif call == "plan":
        n = len(frames)
        t = st["threshold"] = api.Plan(h, w, n, capacity=cap, params=p)
        L = api.lib()
        st["out"] = torch.as_tensor(_View(t, t.lists_ptr, n * cap * 4), device="cuda")
        st["bits"] = torch.as_tensor(_View(t, L.sf_plan_masks(t._p), n * t.words), device="cuda")
        st["counts"] = torch.as_tensor(_View(t, t.counts_ptr, n), device="cuda")
        st["out"].zero_()
    elif call == "chunk":
        host = frames[0].cpu().numpy().view(np.uint16 if case["bits"] == 16 else np.uint32)
        st["chunk"] = synth.chunk(host, "bslz4").copy()
        st["params"] = p
        st["frames"] = None
        st["list"] = np.zeros(cap, api.SIGNAL_DTYPE)
    elif call in ("label", "sweep"):
        mpix = len(frames) * h * w / 1e6
        st["spots"] = np.zeros(int(150 * mpix) + 4096, labeller.SPOT_DTYPE)
        st["pixels"] = np.zeros(int(9000 * mpix) + 65536, labeller.PIXEL_DTYPE)
        st["label_counts"] = np.zeros(6, np.uint64)
        step = 16 if call == "label" else 50
        step = min(step, len(frames))
        st["step"] = step
        st["threshold"] = [api.DeviceBatch(h, w, min(step, len(frames) - j), capacity=cap, params=p)
                           for j in range(0, len(frames), step if call == "label" else len(frames))]
        if call == "label":
            for k, t in enumerate(st["threshold"]):
                t(frames[k * step: k * step + t.n])
            torch.cuda.synchronize()
            for t in st["threshold"]:
                t.workspace = t.bits = None
            st["frames"] = None
    return st


def _signed(a):
    """Unsigned whole numbers seen as signed ones of their width (torch indexes no others on the CPU)."""
    return a.view(a.dtype.str.replace("u", "i")) if a.dtype.kind == "u" else a


def _read(st, lab):
    """The labeller's spots, kept pixels and counts into the program's own arrays, by the C calls that
    fill a caller's buffers."""
    L, spots, pixels, counts = api.lib(), st["spots"], st["pixels"], st["label_counts"]
    for rc in (L.sf_label_finish(lab._h), L.sf_label_spots(lab._h, spots.ctypes.data, len(spots)),
               L.sf_label_pixels(lab._h, pixels.ctypes.data, len(pixels))):
        if rc != 0:
            raise RuntimeError(f"reading the labelling: {api.last_error()} ({rc})")
    L.sf_label_counts(lab._h, counts.ctypes.data)
    return {"n_spots": L.sf_label_n_spots(lab._h), "n_pixels": L.sf_label_n_pixels(lab._h), "counts": counts,
            "spots": {k: _signed(spots[k]) for k in spots.dtype.names},
            "pixels": {k: _signed(pixels[k]) for k in pixels.dtype.names}}


def run(st):
    call, t, frames, cap = st["call"], st.get("threshold"), st["frames"], st["cap"]
    if call == "device":
        t(frames[0])
        return {"bits": t.bits, "counts": t.count, **_lists(t.out, 1, cap)}
    if call in ("batch", "mixed"):
        t(frames)
        return {"bits": t.bits, "counts": t.counts, **_lists(t.out, len(frames), cap)}
    if call == "plan":
        t(frames)
        return {"bits": st["bits"], "counts": st["counts"], **_lists(st["out"], len(frames), cap)}
    case = st["case"]
    h, w = case["height"], case["width"]
    if call == "chunk":
        r = api.find_compressed(st["chunk"], "bslz4", case["bits"], h, w, params=st["params"])
        out = st["list"]
        out[:len(r)] = r
        return {"n": len(r), **{k: out[k] for k in ("index", "value", "background", "population")}}
    lab = labeller.DeviceLabeller(h, w)
    try:
        if call == "label":
            z = 0
            for b in t:
                lab.add_device(list(range(z, z + b.n)), b.out.data_ptr(), cap, b.counts.data_ptr())
                z += b.n
        else:
            b = t[0]
            for z in range(0, len(frames), st["step"]):
                part = frames[z: z + st["step"]]
                b(part)
                lab.add_device(list(range(z, z + len(part))), b.out.data_ptr(), cap, b.counts.data_ptr())
        return _read(st, lab)
    finally:
        lab.close()


def work(case):
    """Each input read once, each output written once: the pixels (a chunk: about a twelfth of them, and
    the frame once), the strong-pixel mask, and 16 bytes a strong pixel, about 20 of those a spot; for a
    labelling the lists in, the spots (112 bytes) and kept pixels (12 bytes) out."""
    s = SCENES[case["scene"]]
    total = 0.0
    for h, w in _shapes(case):
        strong = 20.0 * s["spots"] * h * w / 1e6
        spots = s["spots"] * h * w / 1e6 / max(1.0, 2.5 * sum(s["sz"]))
        pixels = h * w * case["bits"] / 8
        mask = (w + 31) // 32 * 4 * h
        labels = 12.0 * strong + 112.0 * spots
        if case["call"] == "label":
            total += 16.0 * strong + labels
        elif case["call"] == "sweep":
            total += pixels + labels
        elif case["call"] == "chunk":
            total += pixels / 12 + 16.0 * strong
        else:
            total += pixels + mask + 16.0 * strong
    return {"bytes": total, "flops": 0}


def _box(a, k):
    """Sums of a (int64, h x w) over the clipped (2k + 1)-square windows."""
    for dim in (0, 1):
        n = a.shape[dim]
        c = torch.cumsum(a, dim)
        c = torch.cat([torch.zeros_like(c.narrow(dim, 0, 1)), c], dim)
        i = torch.arange(n, device=a.device)
        a = c.index_select(dim, (i + k + 1).clamp_max(n)) - c.index_select(dim, (i - k).clamp_min(0))
    return a


def _strong(frame, case):
    """The strong pixels of a 32-bit frame and their backgrounds, in 64 bits: (indexes, backgrounds)."""
    k, (h, w) = case["kernel"], frame.shape
    valid = frame != -1
    v = torch.where(valid, frame, 0).long()
    m, s, q = _box(valid.long(), k).double(), _box(v, k).double(), _box(v * v, k).double()
    root = torch.sqrt(2.0 * (m - 1.0))
    signal = (m >= 2) & ((m * q - s * s - s * (m - 1.0)) > s * 6.0 * root)
    if case["algorithm"] == "dispersion":
        keep = valid & signal & (v > 0) & ((m * v.double() - s) > 3.0 * torch.sqrt(s * m))
        mean = s / m
    else:
        clear = (~(signal | ~valid)).long()
        eroded = ~valid | (_box(clear, k - 1) == 0)
        bg = valid & ~eroded
        bm, bs = _box(bg.long(), k + 2).double(), _box(torch.where(bg, v, 0), k + 2).double()
        mean = torch.where(bm >= 2, bs / bm, torch.zeros_like(bs))
        keep = valid & eroded & (v > 0) & (v.double() >= mean + 3.0 * torch.sqrt(mean))
    at = torch.nonzero(keep.view(-1)).view(-1)
    return at, mean.view(-1)[at]


def exact(case, seed):
    """The backgrounds, the outputs that are computed numbers; the others are whole numbers. None where
    the reference itself decides in 32 bits (16-bit pixels), or a labelling takes too long in plain numpy."""
    if case["bits"] == 16 or case["call"] in ("label", "sweep"):
        return None
    cap = _capacity(case)
    frames = _frames(case, seed)
    out = torch.zeros(len(frames), cap, dtype=torch.float64, device="cuda")
    for j, f in enumerate(frames):
        at, mean = _strong(f, case)
        n = min(cap, at.numel())
        out[j, :n] = mean[:n]
    if case["call"] == "chunk":
        return {"n": None, "index": None, "value": None, "background": out[0], "population": None}
    return {"bits": None, "counts": None, "index": None, "value": None, "background": out, "population": None}

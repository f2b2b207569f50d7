"""Performance cases of the library: what its users have it do, through the C ABI (include/bm3d_b200.h).

A case is one request for frames: colour conversion, a Basic or Final estimate, or a V-BM3D
estimate, at a profile, sample format, frame size and precision.  `listed` gives the named ones,
`draw` one more of the same ranges, `prepare` the filter handles and frames a caller has in hand,
`run` the calls themselves, `work` the bytes and operations a request cannot do without, and
`exact` the same result in 64-bit arithmetic, restated in plain torch.

The Basic and the Final estimate are separate cases, the Final one on a ref clip made here: its
match lists follow its ref, so behind a Basic estimate, whose sums are atomics in any order, a
last-bit difference swaps near-equal matches and the outputs of two runs could not be compared.
Integer clips take the conversion kernels and then the same path as float ones.  They appear where
two runs differ in enough of the rounded pixels to be told from a fault: 16-bit Basic and V-BM3D
requests, whose sums differ in thousands of pixels from run to run; 8-bit outputs and Final's
16-bit ones differ in none to a few dozen.  Conversions are exact and are drawn in every format.
"""
import ctypes as C
import math
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "vapoursynth-bm3d_b200"))
from bm3d_b200 import _capi as capi  # noqa: E402

# families a clip can have: "OPP" is YUV without subsampling in the opponent colour space
FAMILY = {"GRAY": capi.GRAY, "RGB": capi.RGB, "YUV": capi.YUV, "OPP": capi.YUV}
DTYPE = {"u8": torch.uint8, "u16": torch.uint16, "f32": torch.float32}
BITS = {"u8": 8, "u16": 16, "f32": 32}


def _case(name, kind, family, fmt, width, height, frames, profile="", sigma=10.0, precision="fp32", host=False, out=""):
    c = dict(kind=kind, family=family, format=fmt, width=width, height=height, frames=frames, profile=profile,
             sigma=sigma, precision=precision, host=host, out=out)
    return dict(c, name=name) if name else c


def listed():
    return [
        # one small gray picture at every default (profile "fast"): launch and host latency
        _case("basic_fast_cif", "basic", "GRAY", "f32", 352, 288, 1, "fast", 10.0),
        # a standard-definition frame, refined in the default profile
        _case("final_fast_sd", "final", "YUV", "f32", 720, 480, 1, "fast", 10.0),
        # a VapourSynth script: one 16-bit frame in host memory in, the estimate in host memory out
        _case("basic_lc_hd_host_u16", "basic", "YUV", "u16", 1280, 720, 1, "lc", 10.0, host=True),
        # one 1080p frame on the GPU, refined at the normal profile
        _case("final_np_1080p", "final", "OPP", "f32", 1920, 1080, 1, "np", 10.0),
        # the two halves of the full RGB pipeline on a batch of 1080p frames: RGB -> OPP -> filter -> RGB
        _case("rgb_basic_np_1080p_x8", "rgb_basic", "RGB", "f32", 1920, 1080, 8, "np", 10.0),
        _case("rgb_final_np_1080p_x8", "rgb_final", "RGB", "f32", 1920, 1080, 8, "np", 10.0),
        # the same refinement on the tensor cores
        _case("rgb_final_np_1080p_x4_tf32", "rgb_final", "RGB", "f32", 1920, 1080, 4, "np", 10.0, "tf32"),
        # highest quality, odd size, RGB straight into the filter (its own conversion to OPP)
        _case("final_high_odd", "final", "RGB", "f32", 1279, 719, 1, "high", 15.0),
        # very noisy material: profile "vn" (11 x 11 blocks in Final)
        _case("final_vn_720p", "final", "GRAY", "f32", 1280, 720, 1, "vn", 40.0),
        # V-BM3D on a 16-bit clip: stacked estimate, then VAggregate to 16 bits
        _case("vbasic_fast_1080p_u16", "vbasic", "YUV", "u16", 1920, 1080, 5, "fast", 15.0, out="stacked16"),
        # V-BM3D refinement at the normal profile (radius 3), aggregated on the device, float out
        _case("vfinal_np_720p", "vfinal", "YUV", "u16", 1280, 720, 7, "np", 15.0, out="aggregate32"),
        # conversion alone: 16-bit RGB to float OPP and back to 16-bit RGB
        _case("convert_u16_1080p_x4", "convert", "RGB", "u16", 1920, 1080, 4),
    ]


def draw(rng):
    kind = rng.choice(["basic", "basic", "final", "final", "final", "rgb_basic", "rgb_final", "vbasic", "vfinal", "convert"])
    # pixels of the request: CIF to two (filters) or eight (conversion) 1080p frames, by their logarithm
    pixels = math.exp(rng.uniform(math.log(1e5), math.log(1.6e7 if kind == "convert" else 4e6)))
    frames = 1
    if kind in ("vbasic", "vfinal"):
        frames = rng.randint(3, 8)
    elif pixels > 8e5:
        frames = rng.randint(1, 4)
    aspect = rng.uniform(1.0, 1.9)
    height = max(96, int(math.sqrt(pixels / frames / aspect)))
    width = max(128, int(height * aspect))
    if rng.random() < 0.5:      # frame sizes are even more often than not, and multiples of 16 often
        height, width = height // 2 * 2, width // 2 * 2
    if rng.random() < 0.3:
        height, width = height // 16 * 16, width // 16 * 16
    sigma = rng.choice([5.0, 10.0, 10.0, 15.0, 25.0])
    if kind == "convert":
        return _case("", kind, "RGB", rng.choice(["u8", "u16", "f32"]), width, height, frames)
    if kind in ("rgb_basic", "rgb_final"):
        precision = rng.choice(["fp32", "fp32", "tf32_match" if kind == "rgb_basic" else "tf32"])
        return _case("", kind, "RGB", "f32", width, height, frames, rng.choice(["lc", "np", "np", "high"]), sigma, precision)
    if kind in ("vbasic", "vfinal"):
        return _case("", kind, rng.choice(["GRAY", "YUV", "OPP"]), rng.choice(["u16", "u16", "f32"]), width, height, frames,
                     rng.choice(["fast", "lc", "np"]), sigma, out=rng.choice(["stacked16", "aggregate16", "aggregate32"]))
    profile = rng.choice(["fast", "fast", "lc", "np", "np", "high", "vn"])
    return _case("", kind, rng.choice(["GRAY", "YUV", "OPP", "RGB"]), rng.choice(["u16", "f32"] if kind == "basic" else ["f32"]), width, height,
                 frames, profile, 40.0 if profile == "vn" else sigma, host=rng.random() < 0.2)


# ---- clips ---------------------------------------------------------------------------------------

def _clean(height, width, r):
    """A gray picture in about [0.1, 0.9]: gradient, rectangles and patches of texture."""
    yy = torch.arange(height, device="cuda", dtype=torch.float32)[:, None]
    xx = torch.arange(width, device="cuda", dtype=torch.float32)[None, :]
    a = r.uniform(0, 2 * math.pi)
    t = xx / width * math.cos(a) + yy / height * math.sin(a)
    canvas = torch.full((height, width), 0.5, device="cuda")
    for _ in range(40):
        y0, y1 = sorted(r.randint(0, height) for _ in range(2))
        x0, x1 = sorted(r.randint(0, width) for _ in range(2))
        canvas[y0:y1, x0:x1] = r.uniform(0.1, 0.9)
    img = 0.5 * canvas + 0.25 + 0.15 * t
    for _ in range(6):
        h, w = r.randint(height // 8, height // 2), r.randint(width // 8, width // 2)
        y0, x0 = r.randint(0, height - h), r.randint(0, width - w)
        period, ang = r.uniform(4, 16), r.uniform(0, math.pi)
        wave = torch.sin((xx[:, x0:x0 + w] * math.cos(ang) + yy[y0:y0 + h] * math.sin(ang)) * (2 * math.pi / period))
        img[y0:y0 + h, x0:x0 + w] += 0.1 * wave
    return img.clamp_(0.02, 0.98)


def _clip(case, seed):
    """Noisy frames and the ref clip (close to the clean picture), each [frames][planes][H][W] in the
    case's sample format."""
    r = random.Random(seed)
    g = torch.Generator(device="cuda").manual_seed(seed)
    planes, h, w, fmt = (1 if case["family"] == "GRAY" else 3), case["height"], case["width"], case["format"]
    chroma = case["family"] in ("YUV", "OPP")
    shared = _clean(h, w, r)
    base = [shared]
    for _ in range(planes - 1):
        own = _clean(h, w, r)
        base.append(0.4 * (own - 0.5) if chroma else 0.6 * shared + 0.4 * own)
    base = torch.stack(base)
    src, ref = [], []
    for k in range(case["frames"]):
        pic = torch.roll(base, (k * r.randint(-2, 2), k * r.randint(-2, 2)), (1, 2))
        for clip, s in ((src, case["sigma"]), (ref, 0.15 * case["sigma"])):
            clip.append(pic + torch.randn(pic.shape, generator=g, device="cuda") * (s / 255.0))
    out = []
    for clip in (torch.stack(src), torch.stack(ref)):
        if fmt != "f32":
            top = (1 << BITS[fmt]) - 1
            if chroma:
                clip[:, 1:] += 0.5
            clip = (clip * top + 0.5).clamp_(0, top).to(torch.int32).to(DTYPE[fmt])
        out.append(clip.contiguous())
    return out


# ---- filters and frames over the C ABI --------------------------------------------------------------

class Filter:
    """A filter handle on a stream of the program's own."""

    def __init__(self, name, stream, **args):
        L = capi.lib()
        m = L.bm3d_map_create()
        for k, v in args.items():
            key = k.encode()
            if isinstance(v, capi.VideoInfo):
                L.bm3d_map_set_clip(m, key, C.byref(v))
            elif isinstance(v, str):
                L.bm3d_map_set_data(m, key, v.encode())
            elif isinstance(v, float):
                L.bm3d_map_set_float(m, key, v)
            else:
                L.bm3d_map_set_int(m, key, v)
        self.handle = C.c_void_p()
        rc = L.bm3d_create(name.encode(), m, C.byref(self.handle))
        L.bm3d_map_free(m)
        if rc:
            raise RuntimeError(capi.last_error())
        self.info = capi.VideoInfo()
        L.bm3d_output_info(self.handle, C.byref(self.info))
        L.bm3d_set_stream(self.handle, C.c_void_p(stream.cuda_stream))

    def __del__(self):
        if self.handle:
            capi.lib().bm3d_free(self.handle)
            self.handle = None


class Frames:
    """The frames of a clip, [frames][planes][H][W] (torch on the GPU, numpy in host memory), as the
    library takes them."""

    def __init__(self, data, props=None):
        self.data = data
        self.structs = []
        host = isinstance(data, np.ndarray)
        for f in data:
            s = capi.Frame()
            for p in range(f.shape[0]):
                s.data[p] = f[p].ctypes.data if host else f[p].data_ptr()
                s.stride[p] = f[p].strides[0] if host else f[p].stride(0) * f.element_size()
            s.memory = capi.MEM_HOST if host else capi.MEM_DEVICE
            s.prop_bm3d_opp = s.prop_range = s.prop_matrix = s.prop_v_radius = s.prop_v_process_count = -1
            for k, v in (props or {}).items():
                setattr(s, k, v)
            self.structs.append(s)
        self.table = (C.POINTER(capi.Frame) * len(self.structs))(*[C.pointer(s) for s in self.structs])


def _empty(info, frames, host):
    planes = 1 if info.color_family == capi.GRAY else 3
    dt = torch.float32 if info.sample_type == capi.FLOAT else torch.uint8 if info.bits_per_sample <= 8 else torch.uint16
    if host:
        return Frames(np.zeros((frames, planes, info.height, info.width), str(dt).replace("torch.", "")))
    return Frames(torch.empty((frames, planes, info.height, info.width), dtype=dt, device="cuda"))


def prepare(case, seed):
    """Filter handles (made once per clip), input frames and output buffers of a request for every
    frame of the clip."""
    src, ref = _clip(case, seed)
    kind, nf, host, family = case["kind"], case["frames"], case["host"], case["family"]
    stream = torch.cuda.Stream()
    vi = capi.VideoInfo(FAMILY[family], capi.FLOAT if case["format"] == "f32" else capi.INTEGER, BITS[case["format"]], 0, 0,
                        case["width"], case["height"], nf)
    props = {"prop_bm3d_opp": 1} if family == "OPP" else None
    if host:
        src, ref = src.cpu().numpy(), ref.cpu().numpy()
    src, ref = Frames(src, props), Frames(ref, props)
    calls = []          # (filter, input frames, ref frames, output frames)

    def add(name, inp, rf=None, **args):
        f = Filter(name, stream, **args)
        dst = _empty(f.info, nf, host)
        calls.append((f, inp, rf, dst))
        return f, dst

    common = {}
    if kind != "convert":
        common = {"profile": case["profile"], "sigma": case["sigma"]}
        if case["precision"] != "fp32":
            common["precision"] = case["precision"]
        if family == "OPP" or kind.startswith("rgb_"):
            common["matrix"] = 100
    if kind == "convert":
        f, opp = add("RGB2OPP", src, input=vi, sample=1)
        add("OPP2RGB", opp, input=f.info, sample=0)
    elif kind in ("rgb_basic", "rgb_final"):
        f, opp = add("RGB2OPP", src, input=vi, sample=1)
        if kind == "rgb_final":
            g, oref = add("RGB2OPP", ref, input=vi, sample=1)
            b, est = add("Final", opp, oref, input=f.info, ref=g.info, **common)
        else:
            b, est = add("Basic", opp, input=f.info, **common)
        add("OPP2RGB", est, input=b.info, sample=1)
    elif kind == "basic":
        add("Basic", src, input=vi, **common)
    elif kind == "final":
        add("Final", src, ref, input=vi, ref=vi, **common)
    else:
        name = "VBasic" if kind == "vbasic" else "VFinal"
        rf = ref if kind == "vfinal" else None
        if rf is not None:
            common["ref"] = vi
        if case["out"] == "stacked16":
            f, st = add(name, src, rf, input=vi, **common)
            add("VAggregate", st, input=f.info, radius=_v_params(case)["radius"], sample=0)
        else:
            add(name, src, rf, input=vi, aggregate=1, sample=1 if case["out"] == "aggregate32" else 0, **common)
    torch.cuda.synchronize()
    return {"calls": calls, "frames": nf, "host": host, "stream": stream}


def run(state):
    """One request: every filter of the chain for all frames.  Frames on the GPU are queued on the
    program's stream, frames in host memory come back before the call returns."""
    L = capi.lib()
    fn = L.bm3d_get_frames if state["host"] else L.bm3d_get_frames_async
    for f, src, ref, dst in state["calls"]:
        if fn(f.handle, 0, state["frames"], src.table, ref.table if ref else None, dst.table):
            raise RuntimeError(capi.last_error())
    out = state["calls"][-1][3].data
    if not state["host"] and out.dtype == torch.uint16:
        out = out.view(torch.int16)         # the same bits, in a type that torch can index
    return [out[k, p] for k in range(out.shape[0]) for p in range(out.shape[1])]


# ---- parameters of a profile -------------------------------------------------------------------------

def _params(case, wiener):
    p = {"B": 8, "R": 16, "step": 3 if wiener else 4, "G": 32 if wiener else 16, "lam": 2.7}
    prof = case["profile"]
    if prof == "fast":
        p.update(R=9, G=8, step=7 if wiener else 8)
    elif prof == "lc":
        p.update(R=9, step=5, G=16) if wiener else p.update(R=9, step=6)
    elif prof == "high":
        p.update(step=2 if wiener else 3)
    elif prof == "vn":
        p.update(B=11, step=6) if wiener else p.update(G=32, lam=2.8)
    s = case["sigma"]
    if wiener:
        p["thmse"] = 400 + s * 40 if prof == "vn" else 200 + s * 10
    else:
        p["thmse"] = 1000 + s * 150 if prof == "vn" else 400 + s * 80
    return p


def _v_params(case):
    w = case["kind"] == "vfinal"
    p = dict(_params(case, w), radius=3, G=8, R=12, ps_num=2, ps_range=6 if w else 5)
    prof = case["profile"]
    if prof == "fast":
        p.update(radius=1, R=7, ps_range=5 if w else 4)
    elif prof == "lc":
        p.update(radius=2, R=9, ps_range=5 if w else 4)
    elif prof == "high":
        p.update(radius=4, R=16, ps_range=8 if w else 7)
    elif prof == "vn":
        p.update(radius=4, G=16)
    return p


def _scan(extent, block, step):
    last = extent - block
    return list(range(0, last, step)) + [last]


def work(case):
    """Bytes: every input plane read once, every output plane written once.  Operations: subtract,
    multiply and add per pixel of every matching candidate, and 2 N log2 N per transform of length
    N (a fast transform) over the rows, columns and depth of every group; 30 per pixel converted."""
    w, h, nf, kind = case["width"], case["height"], case["frames"], case["kind"]
    planes = 1 if case["family"] == "GRAY" else 3
    px = w * h * nf * planes
    size = BITS[case["format"]] // 8
    if kind == "convert":
        return {"bytes": px * (size + 2.0), "flops": 10.0 * px}
    wiener = kind in ("final", "rgb_final", "vfinal")
    video = kind in ("vbasic", "vfinal")
    p = _v_params(case) if video else _params(case, wiener)
    b, g = p["B"], p["G"]
    ys, xs = _scan(h, b, p["step"]), _scan(w, b, p["step"])
    span = lambda pos, lim: min(lim, pos + p["R"]) - max(0, pos - p["R"]) + 1  # noqa: E731
    groups = len(ys) * len(xs) * nf
    cand = sum(span(y, h - b) for y in ys) * sum(span(x, w - b) for x in xs) * nf
    if video:
        others = sum(min(nf - 1, k + p["radius"]) - max(0, k - p["radius"]) for k in range(nf))
        cand += len(ys) * len(xs) * others * (2 * p["ps_range"] + 1) ** 2
    one = 2 * (g * 2 * b * b * math.log2(b) + b * b * g * math.log2(g))
    flops = 3.0 * b * b * cand + one * (3 if wiener else 2) * planes * groups
    out = {"stacked16": 2, "aggregate16": 2, "aggregate32": 4}.get(case["out"], size)
    return {"bytes": float(px * (size * (2 if wiener else 1) + out)), "flops": flops}


# ---- the same in 64 bits -------------------------------------------------------------------------------

def _opp(rgb):
    r, g, b = rgb[:, 0], rgb[:, 1], rgb[:, 2]
    return torch.stack([(r + g + b) / 3, (r - b) / 2, (r - 2 * g + b) / 4], 1)


def _rgb(opp):
    y, u, v = opp[:, 0], opp[:, 1], opp[:, 2]
    return torch.stack([y + u + v * 2 / 3, y - v * 4 / 3, y - u + v * 2 / 3], 1)


def _norms(case):
    if case["family"] in ("OPP", "RGB"):
        m = [[1 / 3] * 3, [.5, 0, -.5], [.25, -.5, .25]]
    else:
        w, h = case["width"], case["height"]
        kr, kg, kb = ((.2627, .6780, .0593) if w > 2048 or h > 1536 else (.2126, .7152, .0722) if w > 1024 or h > 576
                      else (.299, .587, .114))
        m = [[kr, kg, kb], [-kr / 2 / (1 - kb), -kg / 2 / (1 - kb), .5], [.5, -kg / 2 / (1 - kr), -kb / 2 / (1 - kr)]]
    return [math.sqrt(sum(v * v for v in row)) for row in m]


def _dct(n, inverse):
    """Rows of the unnormalised DCT-II (REDFT10) or its inverse's (REDFT01) matrix."""
    k = torch.arange(n, dtype=torch.float64, device="cuda")
    if not inverse:
        return 2 * torch.cos(math.pi * (2 * k[None] + 1) * k[:, None] / (2 * n))
    m = 2 * torch.cos(math.pi * k[None] * (2 * k[:, None] + 1) / (2 * n))
    m[:, 0] = 1
    return m


def _blocks(plane, ys, xs, b):
    """Blocks of b x b at (ys, xs) of a flat plane stack: plane [.., H, W] contiguous, ys already holding
    the row offset of the frame."""
    w = plane.shape[-1]
    k = torch.arange(b, device="cuda")
    return plane.reshape(-1)[(ys[..., None, None] + k[:, None]) * w + xs[..., None, None] + k]


def _full_search(plane, p, th, limit):
    """Match lists of one plane: (y, x, distance) [blocks][limit], distance inf past the end.  The
    reference block first, then the nearest; a last candidate at (0, 0) is always in the list."""
    h, w = plane.shape
    b, r = p["B"], p["R"]
    sy, sx = (torch.tensor(_scan(e, b, p["step"]), device="cuda") for e in (h, w))
    ny, nx = len(sy), len(sx)
    pad = torch.nn.functional.pad(plane[None, None], (r, r, r, r))[0, 0]
    dist = torch.full(((2 * r + 1) ** 2 + 1, ny * nx), math.inf, dtype=torch.float64, device="cuda")
    for dy in range(-r, r + 1):
        oky = (sy + dy >= 0) & (sy + dy <= h - b)
        for dx in range(-r, r + 1):
            if dy == 0 and dx == 0:
                continue
            d = (plane - pad[r + dy:r + dy + h, r + dx:r + dx + w]).square_()
            d = sum(d[:, sx + k] for k in range(b))
            d = sum(d[sy + k] for k in range(b))
            okx = (sx + dx >= 0) & (sx + dx <= w - b)
            dist[(dy + r) * (2 * r + 1) + dx + r] = torch.where(oky[:, None] & okx[None], d, math.inf).reshape(-1)
    ry, rx = sy[:, None].expand(ny, nx).reshape(-1), sx[None].expand(ny, nx).reshape(-1)
    dist[-1] = (_blocks(plane, ry, rx, b) - plane[:b, :b]).square_().sum((1, 2))
    dist[(dist > th) | (dist == 0)] = math.inf
    val, idx = torch.topk(dist.t().contiguous(), limit - 1, 1, largest=False, sorted=True)
    last = idx == dist.shape[0] - 1
    y = torch.where(last, 0, ry[:, None] + idx // (2 * r + 1) - r)
    x = torch.where(last, 0, rx[:, None] + idx % (2 * r + 1) - r)
    return torch.cat([ry[:, None], y], 1), torch.cat([rx[:, None], x], 1), torch.cat([torch.zeros_like(val[:, :1]), val], 1)


def _predictive(plane, blocks, cy, cx, cd, p, th):
    """The best matches in another frame around the centres (cy, cx) (cd inf: no centre)."""
    h, w = plane.shape
    b, r, g = p["B"], p["ps_range"], p["G"]
    k = torch.arange(-r, r + 1, device="cuda")
    ys = (cy[:, :, None, None] + k[:, None]).expand(-1, -1, 2 * r + 1, 2 * r + 1)
    xs = (cx[:, :, None, None] + k).expand_as(ys)
    ok = (ys >= 0) & (ys <= h - b) & (xs >= 0) & (xs <= w - b) & torch.isfinite(cd)[:, :, None, None]
    for s in range(1, cy.shape[1]):
        for t in range(s):      # positions that an earlier centre's window holds already
            near = ((ys[:, s] - cy[:, t, None, None]).abs() <= r) & ((xs[:, s] - cx[:, t, None, None]).abs() <= r)
            ok[:, s] &= ~(near & torch.isfinite(cd[:, t])[:, None, None])
    n = ys.shape[0]
    ys, xs, ok = ys.reshape(n, -1), xs.reshape(n, -1), ok.reshape(n, -1)
    d = torch.full(ys.shape, math.inf, dtype=torch.float64, device="cuda")
    for i in range(0, n, 8192):
        s = slice(i, i + 8192)
        v = (_blocks(plane, ys[s] * ok[s], xs[s] * ok[s], b) - blocks[s, None]).square_().sum((2, 3))
        d[s] = torch.where(ok[s] & (v <= th) & (v > 0), v, math.inf)
    val, idx = torch.topk(d, g, 1, largest=False, sorted=True)
    return ys.gather(1, idx), xs.gather(1, idx), val


def _video_lists(luma, f, p, th):
    """Lists (frame, y, x, count) of the reference blocks of frame f over its temporal window."""
    g, r = p["G"], p["radius"]
    y, x, d = _full_search(luma[f], p, th, g)
    blocks = _blocks(luma[f], y[:, 0], x[:, 0], p["B"])
    lists = [(torch.full_like(y, f), y, x, d)]
    for way in (-1, 1):
        cy, cx, cd = (t[:, :p["ps_num"]] for t in (y, x, d))
        z = f + way
        while 0 <= z < luma.shape[0] and abs(z - f) <= r:
            py, px, pd = _predictive(luma[z], blocks, cy, cx, cd, p, th)
            lists.append((torch.full_like(py, z), py, px, pd))
            cy, cx, cd = (t[:, :p["ps_num"]] for t in (py, px, pd))
            z += way
    z, y, x, d = (torch.cat(t, 1) for t in zip(*lists))
    count = torch.isfinite(d).sum(1)
    # more than g: the nearest g in order; else as they were found
    place = torch.arange(d.shape[1], device="cuda", dtype=torch.float64).expand_as(d)
    key = torch.where(torch.isfinite(d), torch.where(count[:, None] > g, d, place), math.inf)
    order = torch.argsort(key, dim=1, stable=True)[:, :g]
    return z.gather(1, order), y.gather(1, order), x.gather(1, order), count.clamp(max=g)


def _filter(src, ref, num, den, z, y, x, count, p, sigma):
    """Collaborative filtering of the groups of one plane stack [frames][H][W], added to num and den."""
    h, w = src.shape[-2:]
    b = p["B"]
    cf, ci = _dct(b, False), _dct(b, True)
    k = torch.arange(b, device="cuda")
    for n in count.unique().tolist():
        rows = (count == n).nonzero()[:, 0]
        zf, zi = _dct(n, False), _dct(n, True)
        amp = 2.0 * n * 2 * b * 2 * b
        fwd = lambda t: torch.einsum("kz,gzuv->gkuv", zf, cf @ t @ cf.t())  # noqa: E731
        for sel in rows.split(max(1, (1 << 24) // (n * b * b))):
            yy, xx = z[sel, :n] * h + y[sel, :n], x[sel, :n]
            c = fwd(_blocks(src, yy, xx, b))
            if ref is None:
                flag = ((torch.arange(n, device="cuda") == 0).int()[:, None, None] + (k == 0).int()[:, None] + (k == 0).int())
                keep = c.abs() > sigma * p["lam"] * math.sqrt(amp) * torch.sqrt(2.0 ** flag.double())
                c *= keep
                wgt = 1.0 / keep.sum((1, 2, 3)).clamp(min=1).double()
            else:
                r2 = fwd(_blocks(ref, yy, xx, b)).square_()
                r2 /= r2 + max(sigma * sigma * amp, 2.0 ** -126)
                c *= r2
                wgt = 1.0 / r2.square_().sum((1, 2, 3)).clamp(min=2.0 ** -23)
            v = ci @ torch.einsum("kz,gzuv->gkuv", zi, c) @ ci.t()
            v *= (wgt / amp)[:, None, None, None]
            at = ((yy[..., None, None] + k[:, None]) * w + xx[..., None, None] + k).reshape(-1)
            num.view(-1).index_add_(0, at, v.reshape(-1))
            den.view(-1).index_add_(0, at, wgt[:, None, None, None].expand_as(v).reshape(-1))


def exact(case, seed):
    """What run returns, in 64 bits; None where the outputs are whole numbers."""
    if case["format"] != "f32" and case["out"] != "aggregate32" or case["kind"] == "convert" or case["out"].endswith("16"):
        return None
    src, ref = (t.to(torch.int32).double() if case["format"] != "f32" else t.double() for t in _clip(case, seed))
    kind, family = case["kind"], case["family"]
    if case["format"] != "f32":
        top = (1 << BITS[case["format"]]) - 1
        for t in (src, ref):
            if family != "GRAY":
                t[:, 1:] -= 1 << (BITS[case["format"]] - 1)
            t /= top
            if family != "GRAY":
                t[:, 1:].clamp_(-.5, .5)
    if family == "RGB":
        src, ref = _opp(src), _opp(ref)
    wiener = kind in ("final", "rgb_final", "vfinal")
    video = kind in ("vbasic", "vfinal")
    p = _v_params(case) if video else _params(case, wiener)
    norms = _norms(case)
    th = p["thmse"] * norms[0] * p["B"] ** 2 / 255 ** 2
    src, ref = src.transpose(0, 1).contiguous(), ref.transpose(0, 1).contiguous()       # [planes][frames][H][W]
    num, den = torch.zeros_like(src), torch.zeros_like(src)
    match = ref[0] if wiener else src[0]
    for f in range(case["frames"]):
        if video:
            z, y, x, count = _video_lists(match, f, p, th)
        else:
            y, x, d = _full_search(match[f], p, th, p["G"])
            z, count = torch.full_like(y, f), torch.isfinite(d).sum(1)
        for c in range(src.shape[0]):
            _filter(src[c], ref[c] if wiener else None, num[c], den[c], z, y, x, count, p, case["sigma"] / 255 * norms[c])
    out = (num / den).transpose(0, 1)
    if family == "RGB":
        out = _rgb(out)
    out = out.cpu()
    return [out[k, c] for k in range(out.shape[0]) for c in range(out.shape[1])]

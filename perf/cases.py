"""The work that programs give this engine, as measurable cases.

Each case is one call pattern of a program that uses the engine through its public entry points:

  resident  an image whose coefficients stay on the device, reconstructed into a device surface
  batch     many images of uneven sizes and formats, reconstructed by one captured launch sequence
  requests  a batch of full, region and thumbnail decodes of resident images, as a server submits them
  host      one call from an entropy decoder's arena in host memory to pixels in host memory
  orient    the presentation orientation of a decoded surface
  analyze   the encoder's front half: sample planes to quantized coefficients

Images are the generator's seeded content (`jxr_b200.synth`), coded by the forward half of the codec, so the
coefficients have the values and distributions of coded photographs.  A case's sizes and options come from
the case alone, its content from the seed.  Every output is whole numbers or bytes (binary32 surfaces are
exact widenings), so there is no value in 64 bits to compare them with.
"""
import math
import os
import random

import torch

import jxr_b200 as J
from jxr_b200 import api

THREADS = min(os.cpu_count() or 8, 16)
ROTATE90 = api.ORIENTATION["ROTATE90"]

# coded format -> blocks of each plane's macroblock, and bytes of an output pixel
FORMATS = {
    "rgb444": ((16, 16, 16), 3),
    "rgb420": ((16, 4, 4), 3),
    "rgb422": ((16, 8, 8), 3),
    "gray16": ((16,), 2),
    "rgba": ((16, 16, 16, 16), 4),
    "hdr": ((16, 16, 16, 16), 16),      # half floats and a separate alpha plane, to binary32 channel planes
}
CODED = ("format", "width", "height", "quality", "overlap", "tile", "hard")


def coded(fmt, width, height, quality=85, overlap=1, tile=16, hard=0):
    return {"format": fmt, "width": width, "height": height, "quality": quality, "overlap": overlap, "tile": tile,
            "hard": hard}


def listed():
    return [
        # the smallest call: one small picture of a web page, host memory to host memory, where latency counts
        dict(name="host_small", kind="host", **coded("rgb420", 192, 144, quality=75)),
        # the large photograph decode: 8-bit RGB, two-level overlap, 256 x 256 soft tiles
        dict(name="photo_4096", kind="resident", **coded("rgb444", 4096, 4096, quality=90, overlap=2)),
        # the HDR texture with alpha: the largest output a pixel, binary32 channel planes for a network or renderer
        dict(name="hdr_alpha_3072", kind="resident", **coded("hdr", 3072, 3072, quality=0, overlap=2, tile=32)),
        # a camera's 4:2:0 photograph whose sides are no multiple of a macroblock: rows start at odd bytes
        dict(name="photo420_3999x2999", kind="resident", **coded("rgb420", 3999, 2999, quality=75)),
        # a 4:2:2 video frame
        dict(name="frame422_1920x1080", kind="resident", **coded("rgb422", 1920, 1080, quality=85)),
        # a zoomable scan with independently decodable (hard) tiles
        dict(name="hard_tiles_2500x1900", kind="resident", **coded("rgb444", 2500, 1900, overlap=2, hard=1)),
        # a 16-bit lossless radiograph
        dict(name="gray16_2047x1535", kind="resident", **coded("gray16", 2047, 1535, quality=100, overlap=0, tile=32)),
        # a data loader's batch: half 4:2:0 photographs, gray scans and RGBA pictures, one captured launch
        dict(name="batch_mixed", kind="batch", images=32, low=64, high=2048, pick=4),
        # a server's batch: full decodes, regions of interest and thumbnails of resident images
        dict(name="requests_mixed", kind="requests", images=12, low=128, high=2048, pick=5, requests=24, regions=0.3,
             reduced=0.2),
        # a gallery page: quarter and sixteenth resolution thumbnails only
        dict(name="requests_thumbnails", kind="requests", images=8, low=512, high=2048, pick=6, requests=16, regions=0.0,
             reduced=1.0),
        # a camera's portrait picture, turned after its decode
        dict(name="orient_rgb8_3999x2999", kind="orient", width=3999, height=2999, pixel_bytes=3, orientation=ROTATE90),
        # the encoder's analysis of a 4:2:0 photograph
        dict(name="analyze420_2048x1536", kind="analyze", width=2048, height=1536, subsampled=True, overlap=1, hard=0),
    ]


def _between(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(("host", "resident", "resident", "resident", "resident", "batch", "requests", "orient", "analyze"))
    if kind in ("host", "resident"):
        fmt = rng.choice(tuple(FORMATS))
        low, high = (64, 768) if kind == "host" else (128, 2048) if fmt == "hdr" else (128, 3072)
        overlap = rng.choice((0, 1, 2))
        quality = 0 if fmt == "hdr" else 100 if fmt == "gray16" else rng.choice((50, 75, 85, 90, 95))
        return dict(kind=kind, **coded(fmt, _between(rng, low, high), _between(rng, low, high), quality=quality,
                                       overlap=overlap, tile=rng.choice((8, 16, 32)), hard=int(rng.random() < 0.25)))
    if kind == "batch":
        return dict(kind=kind, images=rng.randint(2, 32), low=64, high=_between(rng, 128, 1536), pick=rng.randrange(1 << 20))
    if kind == "requests":
        return dict(kind=kind, images=rng.randint(1, 8), low=128, high=_between(rng, 256, 1536), pick=rng.randrange(1 << 20),
                    requests=_between(rng, 1, 32), regions=rng.choice((0.0, 0.3, 0.6)), reduced=rng.choice((0.0, 0.2, 0.4)))
    if kind == "orient":
        return dict(kind=kind, width=_between(rng, 64, 4096), height=_between(rng, 64, 4096),
                    pixel_bytes=rng.choice((1, 2, 3, 4, 6, 8, 16)), orientation=rng.randrange(1, 8))
    return dict(kind=kind, width=32 * max(1, _between(rng, 64, 2048) // 32), height=32 * max(1, _between(rng, 64, 2048) // 32),
                subsampled=rng.random() < 0.5, overlap=rng.choice((0, 1, 2)), hard=int(rng.random() < 0.25))


# ---------------------------------------------------------------------------
# the pictures of a case
# ---------------------------------------------------------------------------
def _pool(case):
    """The coded pictures of a batch or a server: half 4:2:0 photographs with one overlap level, three in ten
    lossless 16-bit gray without overlap, the rest RGBA with two levels; sides log-uniform, tiles of 128 to
    512 samples."""
    rng = random.Random(case["pick"])
    out = []
    for _ in range(case["images"]):
        w, h = _between(rng, case["low"], case["high"]), _between(rng, case["low"], case["high"])
        tile, u = rng.randint(8, 32), rng.random()
        out.append(coded("rgb420", w, h, quality=75, overlap=1, tile=tile) if u < 0.5 else
                   coded("gray16", w, h, quality=100, overlap=0, tile=tile) if u < 0.8 else
                   coded("rgba", w, h, quality=85, overlap=2, tile=tile))
    return out


def _wanted(case, pool):
    """The requests of a server's batch as (picture, (x, y, w, h), denominator): regions hold a tenth to a half of
    the picture, reduced decodes the whole picture at a quarter or a sixteenth of the resolution."""
    rng = random.Random(case["pick"] + 1)
    out = []
    for _ in range(case["requests"]):
        i = rng.randrange(len(pool))
        W, H = pool[i]["width"], pool[i]["height"]
        box, denominator, u = (0, 0, W, H), 1, rng.random()
        if u < case["regions"]:
            f, aspect = rng.uniform(0.1, 0.5), math.exp(rng.uniform(-0.7, 0.7))
            w = min(W, max(1, round(math.sqrt(f * W * H * aspect))))
            h = min(H, max(1, round(f * W * H / w)))
            box = (rng.randint(0, W - w), rng.randint(0, H - h), w, h)
        elif u < case["regions"] + case["reduced"]:
            denominator = rng.choice((4, 4, 16))
        out.append((i, box, denominator))
    return out


def _image(c, seed):
    C, A = J.COLOR, J.ALPHA
    more = dict(overlap=c["overlap"], tile_width=c["tile"], tile_height=c["tile"], hard_tiles=c["hard"], seed=seed,
                threads=THREADS)
    if c["format"] == "gray16":
        more.update(content=J.CONTENT["GRAY16"], color_format=C["LUMA"], quality=c["quality"], scaled=0)
    elif c["format"] == "hdr":
        more.update(content=J.CONTENT["HDR_HALF"], alpha_mode=A["SEPARATE"], scaled=0, quality=0, qp=(4, 8, 16),
                    alpha_overlap=0)
    elif c["format"] == "rgba":
        more.update(alpha_mode=A["INTEGRATED"], quality=c["quality"], alpha_overlap=c["overlap"], alpha_qp=(8, 8, 8))
    else:
        more.update(color_format=C[{"rgb444": "YUV444", "rgb420": "YUV420", "rgb422": "YUV422"}[c["format"]]],
                    quality=c["quality"])
    return J.synth(c["width"], c["height"], **more)


def _output(c, box=None):
    C, D, S, L = J.COLOR, J.DEPTH, J.STORE, J.LAYOUT
    x, y, w, h = box or (0, 0, c["width"], c["height"])
    if c["format"] == "gray16":
        return J.OutputFormat(C["LUMA"], D["U16"], S["U16"], L["LUMA"], w, h, crop_x=x, crop_y=y)
    if c["format"] == "hdr":
        return J.OutputFormat(C["RGB"], D["F16"], S["F16"], L["RGBA"], w, h, crop_x=x, crop_y=y,
                              alpha_bit_depth=D["F16"], nchw=1, widen_f16=1)
    if c["format"] == "rgba":
        return J.OutputFormat(C["RGB"], D["U8"], S["U8"], L["RGBA"], w, h, crop_x=x, crop_y=y, alpha_bit_depth=D["U8"])
    return J.OutputFormat(C["RGB"], D["U8"], S["U8"], L["RGB"], w, h, crop_x=x, crop_y=y)


_session = None


def _decoder():
    """The one session that a program keeps."""
    global _session
    if _session is None:
        _session = J.CudaDecoderSession(0)
    return _session


# ---------------------------------------------------------------------------
# one case
# ---------------------------------------------------------------------------
def prepare(case, seed):
    return {"host": _prepare_host, "resident": _prepare_resident, "batch": _prepare_resident,
            "requests": _prepare_requests, "orient": _prepare_orient, "analyze": _prepare_analyze}[case["kind"]](case, seed)


def run(state):
    return state["run"](state)


def _prepare_host(case, seed):
    img = _image(case, seed)
    return dict(run=_run_host, session=_decoder(),
                plan=J.CudaDecodePlan(img.arena, img.geometry, _output(case), img.alpha_arena))


def _run_host(state):
    return state["session"].decode_to_host(state["plan"])


def _prepare_resident(case, seed):
    pool = _pool(case) if case["kind"] == "batch" else [{k: case[k] for k in CODED}]
    images = [_image(c, seed * 1009 + i) for i, c in enumerate(pool)]
    plans = [J.CudaDecodePlan(im.arena, im.geometry, _output(c), im.alpha_arena) for c, im in zip(pool, images)]
    res = _decoder().resident(plans)
    out = torch.zeros(res.output_bytes(), dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    stream = torch.cuda.Stream()
    if case["kind"] == "batch":
        res.capture(out.data_ptr(), out.numel())
        return dict(run=_run_batch, res=res, out=out, stream=stream)
    view = {"gray16": torch.int16, "hdr": torch.float32}.get(case["format"], torch.uint8)
    return dict(run=_run_resident, res=res, out=out, stream=stream, pixels=out.view(view))


def _run_resident(state):
    state["res"].run(state["out"].data_ptr(), state["out"].numel(), stream=state["stream"].cuda_stream)
    return state["pixels"]


def _run_batch(state):
    state["res"].replay(state["stream"].cuda_stream)
    return state["out"]


def _prepare_requests(case, seed):
    pool, session = _pool(case), _decoder()
    images = []
    for i, c in enumerate(pool):
        img = _image(c, seed * 1013 + i)
        images.append(session.upload(img.arena, img.geometry, img.alpha_arena))
    wanted = [(images[i], _output(pool[i], box), d) for i, box, d in _wanted(case, pool)]
    made = [im.request(o, d) for im, o, d in wanted]
    size = sum((r.output_bytes() + 255) // 256 * 256 for r in made)
    out = torch.zeros(size, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    return dict(run=_run_requests, session=session, wanted=wanted, out=out)


def _run_requests(state):
    requests = [im.request(o, d) for im, o, d in state["wanted"]]
    sub = state["session"].submit_requests(requests, state["out"].data_ptr(), state["out"].numel())
    sub.wait()
    sub.close()
    for r in requests:
        r.close()
    return state["out"]


def _prepare_orient(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    w, h, n = case["width"], case["height"], case["pixel_bytes"]
    src = torch.randint(0, 256, (w * h * n,), dtype=torch.uint8, device="cuda", generator=g)
    return dict(run=_run_orient, src=src, dst=torch.zeros_like(src), args=(w, h, n, case["orientation"]))


def _run_orient(state):
    api.orient(state["src"].data_ptr(), state["dst"].data_ptr(), *state["args"],
               stream=torch.cuda.current_stream().cuda_stream)
    return state["dst"]


def _prepare_analyze(case, seed):
    """Luma and two chroma planes of a photograph-like picture, in the codec's scaled samples."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    fresh, planes = [], []
    for k in range(3):
        half = 2 if case["subsampled"] and k else 1
        w, h, b = case["width"] // half, case["height"] // half, 4 // half
        coarse = torch.randn((1, 1, h // 16 + 2, w // 16 + 2), device="cuda", generator=g)
        smooth = torch.nn.functional.interpolate(coarse, size=(h, w), mode="bicubic")[0, 0]
        noise = torch.randn((h, w), device="cuda", generator=g)
        s = ((smooth * (40 if k == 0 else 16) + noise * 6).clamp(-128, 127).round() * 8).to(torch.int32)
        mx, my = w // (4 * b), h // (4 * b)
        fresh.append(s)
        planes.append(api.AnalysisPlane(torch.empty_like(s), b, b, 1, case["overlap"], (24, 28, 36),
                                        list(range(0, mx, 16)) + [mx], list(range(0, my, 16)) + [my], case["hard"]))
    return dict(run=_run_analyze, fresh=fresh, planes=planes)


def _run_analyze(state):
    # the picture's samples into the planes, which the analysis filters in place
    for s, p in zip(state["fresh"], state["planes"]):
        p.samples.copy_(s)
    coefficients = api.analyze(state["planes"], stream=torch.cuda.current_stream().cuda_stream)
    return [coefficients, [p.samples for p in state["planes"]]]


def exact(case, seed):
    return None


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def _coded_bytes(c, width=None, height=None, low_pass_only=False, out_pixels=None):
    """Coefficients and macroblock tables read once, the surface written once."""
    blocks, pixel = FORMATS[c["format"]]
    w, h = width or c["width"], height or c["height"]
    mbs = -(-w // 16) * -(-h // 16)
    read = sum(mbs * (4 * (b if low_pass_only else 16 * b) + 16) for b in blocks)
    return read + pixel * (w * h if out_pixels is None else out_pixels)


def work(case):
    kind = case["kind"]
    if kind in ("host", "resident"):
        n = _coded_bytes(case)
    elif kind == "batch":
        n = sum(_coded_bytes(c) for c in _pool(case))
    elif kind == "requests":
        pool, n = _pool(case), 0
        for i, (_, _, w, h), d in _wanted(case, pool):
            c, s = pool[i], {1: 1, 4: 4, 16: 16}[d]
            n += _coded_bytes(c, w, h, low_pass_only=d != 1, out_pixels=-(-w // s) * -(-h // s))
    elif kind == "orient":
        n = 2 * case["width"] * case["height"] * case["pixel_bytes"]
    else:
        n = 0
        for k in range(3):
            half = 2 if case["subsampled"] and k else 1
            w, h = case["width"] // half, case["height"] // half
            mbs = (w * half // 16) * (h * half // 16)
            n += w * h * 4 * 2 + mbs * (16 + 256) * 4
    return {"bytes": n, "flops": 0}

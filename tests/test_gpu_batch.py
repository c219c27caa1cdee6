"""The batched paths against the oracle: one persistent launch sequence over
a mixed batch, one launch sequence per image, CUDA-graph replay, and every
launch shape the autotuner may choose -- all bit-exact."""
import numpy as np
import pytest

import jxr_b200 as J
from jxr_b200 import autotune, workloads as W
from tests._bridge import decode_synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def session():
    if not J.CudaDecoderSession.is_available():
        pytest.fail("no B200 visible: the GPU tests need the CUDA engine")
    s = J.CudaDecoderSession(0)
    yield s
    s.close()


@pytest.fixture(scope="module")
def batch():
    items = W.mixed_batch(count=14, seed=7, lo=64, hi=720, threads=8)
    refs = []
    for it in items:
        rc, ref = decode_synth(it.image, it.output, threads=8)
        assert rc == 0
        refs.append(ref)
    return items, W.plans_of(items), refs


def split(buf, plans):
    out, at = [], 0
    for p in plans:
        at = (at + 255) // 256 * 256
        out.append(buf[at:at + p.output_bytes()])
        at += p.output_bytes()
    return out


def check_all(buf, plans, refs):
    for i, (got, ref) in enumerate(zip(split(buf, plans), refs)):
        assert np.array_equal(got, ref), f"image {i} differs"


def test_mix_covers_all_kinds(batch):
    items, _, _ = batch
    assert {it.kind for it in items} == {"rgb420", "gray16", "rgba"}


def test_batched_per_image_and_graph(session, batch):
    import torch
    items, plans, refs = batch
    res = session.resident(plans)
    n = res.output_bytes()
    stream = torch.cuda.Stream()
    for batched in (True, False):
        dst = torch.full((n,), 0x33, dtype=torch.uint8, device="cuda")
        res.run(dst.data_ptr(), n, batched, stream.cuda_stream)
        stream.synchronize()
        assert res.status() == 0
        check_all(dst.cpu().numpy(), plans, refs)
    for batched in (True, False):
        dst = torch.full((n,), 0x44, dtype=torch.uint8, device="cuda")
        res.capture(dst.data_ptr(), n, batched)
        for _ in range(2):
            res.replay(stream.cuda_stream)
        stream.synchronize()
        check_all(dst.cpu().numpy(), plans, refs)
    res.close()


@pytest.mark.parametrize("blocks,side", autotune.candidates()[::3])
def test_every_launch_shape_is_exact(session, batch, blocks, side):
    import torch
    _, plans, refs = batch
    res = session.resident(plans)
    n = res.output_bytes()
    res.set_tuning(blocks, side)
    dst = torch.zeros(n, dtype=torch.uint8, device="cuda")
    res.run(dst.data_ptr(), n, True, 0)
    torch.cuda.synchronize()
    check_all(dst.cpu().numpy(), plans, refs)
    res.close()


def test_autotuner_picks_a_candidate(session, batch, tmp_path, monkeypatch):
    import torch
    monkeypatch.setenv("JXRB_TUNING_CACHE", str(tmp_path / "tuning.json"))
    _, plans, refs = batch
    res = session.resident(plans)
    n = res.output_bytes()
    dst = torch.zeros(n, dtype=torch.uint8, device="cuda")
    stream = torch.cuda.Stream()
    first = autotune.tune(res, plans, dst.data_ptr(), n, stream, reps=3)
    assert first["source"] == "measured"
    assert (tuple(first["blocks_per_sm"]), first["side_stream"]) in set(autotune.candidates())
    again = autotune.tune(res, plans, dst.data_ptr(), n, stream, reps=3)
    assert again["source"] == "cache" and again["blocks_per_sm"] == first["blocks_per_sm"]
    res.run(dst.data_ptr(), n, True, stream.cuda_stream)
    stream.synchronize()
    check_all(dst.cpu().numpy(), plans, refs)
    res.close()


@pytest.mark.parametrize("fmt", ["RGB", "YUV420", "YUV422", "GRAY", "RGBA"])
@pytest.mark.parametrize("hard", [0, 1])
def test_few_tiles_of_a_kind_and_more(session, fmt, hard):
    """Sets with interior and edge tiles of one kind around the count at which
    the two stop sharing a kernel (128 tiles): 32, 128, 160 and 32 tiles beside
    another kind's."""
    C, D, S, L = J.COLOR, J.DEPTH, J.STORE, J.LAYOUT
    kw = dict(overlap=1, tile_width=9, tile_height=10, hard_tiles=hard)
    w, h = 256, 512
    if fmt == "GRAY":
        im = J.synth(w, h, content=J.CONTENT["GRAY16"], color_format=C["LUMA"], quality=100, scaled=0, seed=3, **kw)
        out = J.OutputFormat(C["LUMA"], D["U16"], S["U16"], L["LUMA"], w, h)
    elif fmt == "RGBA":
        im = J.synth(w, h, alpha_mode=J.ALPHA["INTEGRATED"], quality=80, alpha_overlap=1, seed=4, **kw)
        out = J.OutputFormat(C["RGB"], D["U8"], S["U8"], L["RGBA"], w, h, alpha_bit_depth=D["U8"])
    else:
        colour = C["YUV444" if fmt == "RGB" else fmt]
        im = J.synth(w, h, color_format=colour, quality=80, seed=5, **kw)
        out = J.OutputFormat(C["RGB"], D["U8"], S["U8"], L["RGB"], w, h)
    other = J.synth(w, h, content=J.CONTENT["GRAY16"] if fmt != "GRAY" else J.CONTENT["PHOTO_RGB8"],
                    color_format=C["LUMA" if fmt != "GRAY" else "YUV444"], quality=100 if fmt != "GRAY" else 80,
                    scaled=int(fmt == "GRAY"), seed=6, **kw)
    other_out = (J.OutputFormat(C["LUMA"], D["U16"], S["U16"], L["LUMA"], w, h) if fmt != "GRAY" else
                 J.OutputFormat(C["RGB"], D["U8"], S["U8"], L["RGB"], w, h))
    rc, ref = decode_synth(im, out, threads=8)
    rc2, ref2 = decode_synth(other, other_out, threads=8)
    assert rc == 0 and rc2 == 0
    plan = J.CudaDecodePlan(im.arena, im.geometry, out)
    plan2 = J.CudaDecodePlan(other.arena, other.geometry, other_out)
    for n, beside in ((1, 0), (4, 0), (5, 0), (1, 1)):
        sub = session.submit_batch([plan] * n + [plan2] * beside)
        sub.wait()
        for i in range(n):
            assert np.array_equal(sub.readback(i), ref), (n, i)
        for i in range(beside):
            assert np.array_equal(sub.readback(n + i), ref2)
        sub.close()


def test_submissions_in_flight_and_small_outputs(session):
    """More submissions at once than the session keeps upload buffers for, one
    whose descriptors fill more than a buffer, outputs around the size that
    comes back through page-locked memory, and callers on several threads."""
    from concurrent.futures import ThreadPoolExecutor
    C, D, S, L = J.COLOR, J.DEPTH, J.STORE, J.LAYOUT
    refs, plans = [], []
    for w, h in ((256, 256), (255, 256), (257, 256), (33, 17)):
        im = J.synth(w, h, quality=75, overlap=1, seed=50 + w)
        out = J.OutputFormat(C["RGB"], D["U8"], S["U8"], L["RGBX"], w, h)
        rc, ref = decode_synth(im, out, threads=8)
        assert rc == 0
        refs.append(ref)
        plans.append(J.CudaDecodePlan(im.arena, im.geometry, out))
    assert plans[0].output_bytes() == 256 << 10
    subs = [session.submit(plans[i % 4]) for i in range(40)]
    for i, sub in enumerate(subs):
        sub.wait()
        assert np.array_equal(sub.readback(), refs[i % 4])
        sub.close()
    many = session.submit_batch([plans[3]] * 600)
    many.wait()
    assert all(np.array_equal(many.readback(i), refs[3]) for i in (0, 1, 299, 598, 599))
    many.close()
    with ThreadPoolExecutor(8) as pool:
        got = list(pool.map(lambda i: session.decode_to_host(plans[i % 4]), range(64)))
    assert all(np.array_equal(g, refs[i % 4]) for i, g in enumerate(got))


@pytest.mark.parametrize("fmt,copies", [("YUV420", 39), ("YUV420", 40), ("YUV444", 1), ("YUV444", 25), ("YUV444", 26),
                                        ("YUV422", 1), ("YUV422", 2)])
def test_many_tiles_of_a_kind(session, fmt, copies):
    """Either side of the number of interior tiles from which the 4:2:0 kernel
    runs more CTAs an SM (64 of them in a picture of 640 x 640), and of the
    number of tiles from which three-plane edge tiles have a kernel of their own
    (100 in such a picture), or subsampled interior tiles."""
    img = J.synth(637, 640, color_format=J.COLOR[fmt], quality=80, overlap=1, tile_width=9, tile_height=7, seed=41,
                  threads=8)
    out = J.OutputFormat(J.COLOR["RGB"], J.DEPTH["U8"], J.STORE["U8"], J.LAYOUT["RGB"], 637, 640)
    rc, want = decode_synth(img, out, threads=8)
    assert rc == 0
    plan = J.CudaDecodePlan(img.arena, img.geometry, out)
    sub = session.submit_batch([plan] * copies)
    sub.wait()
    for k in range(copies):
        assert np.array_equal(sub.readback(k), want), k
    sub.close()


@pytest.mark.parametrize("copies", [25, 26])
def test_many_tiles_of_a_set(session, copies):
    """Either side of the number of tiles in a set, of any kind, from which the
    4:2:0 kernel runs more CTAs an SM (100 of them in a picture of 640 x 640)."""
    plans, wants = [], []
    for kw in (dict(color_format=J.COLOR["YUV420"], quality=80, overlap=1), dict(color_format=J.COLOR["YUV422"], quality=80)):
        img = J.synth(637, 640, tile_width=9, tile_height=7, seed=42, threads=8, **kw)
        out = J.OutputFormat(J.COLOR["RGB"], J.DEPTH["U8"], J.STORE["U8"], J.LAYOUT["RGB"], 637, 640)
        rc, want = decode_synth(img, out, threads=8)
        assert rc == 0
        plans.append(J.CudaDecodePlan(img.arena, img.geometry, out))
        wants.append(want)
    sub = session.submit_batch([plans[k % 2] for k in range(copies)])
    sub.wait()
    for k in range(copies):
        assert np.array_equal(sub.readback(k), wants[k % 2]), k
    sub.close()

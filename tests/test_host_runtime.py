"""The engine's host code (csrc/host.cpp) against a CUDA runtime on host memory
(tests/_fake_cuda.cpp): what it does when a call fails, in which order it queues
and waits, and what it leaves behind."""
import ctypes as C
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

import jxr_b200 as J
from jxr_b200 import api

ROOT = Path(__file__).resolve().parents[1]
CSRC = ROOT / "jxr_b200" / "csrc"
CUDA = next((p for p in (Path(shutil.which("nvcc") or "/x/x").resolve().parents[1] / "include",
                         Path("/usr/local/cuda/include")) if (p / "cuda_runtime.h").exists()), None)
STREAMS, EVENTS, DEVICE, PINNED = range(4)
C_, D, S, L = J.COLOR, J.DEPTH, J.STORE, J.LAYOUT


@pytest.fixture(scope="module")
def fake_lib(tmp_path_factory):
    out = tmp_path_factory.mktemp("fake_cuda") / "libjxr_fake.so"
    # its calls bind to the runtime built with it, not to one another library brought
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-Wl,-Bsymbolic", "-pthread", "-I", str(CUDA),
                    "-I", str(ROOT / "include"), "-I", str(CSRC), str(CSRC / "host.cpp"), str(CSRC / "sample_scale.cpp"),
                    str(ROOT / "tests" / "_fake_cuda.cpp"), "-o", str(out)], check=True)
    lib = C.CDLL(str(out))
    for name, (res, args) in api.EXPORTS.items():
        if hasattr(lib, name):
            fn = getattr(lib, name)
            fn.restype, fn.argtypes = res, args
    lib.fake_log.restype = C.c_char_p
    lib.fake_live.restype = C.c_long
    lib.fake_fail.argtypes = [C.c_char_p, C.c_int]
    return lib


@pytest.fixture
def fake(fake_lib, monkeypatch):
    monkeypatch.setenv("JXRB_STAGING_THREADS", "1")
    monkeypatch.setattr(api, "_lib", fake_lib)
    fake_lib.fake_reset()
    opened = []

    class Session(J.CudaDecoderSession):
        def __init__(self, *args, **kw):
            super().__init__(*args, **kw)
            opened.append(self)

    monkeypatch.setattr(J, "CudaDecoderSession", Session)
    yield fake_lib
    fake_lib.fake_reset()
    for s in opened:      # while the library is still this one
        s.close()


def live(lib):
    return [lib.fake_live(k) for k in (STREAMS, EVENTS, DEVICE, PINNED)]


def log(lib):
    return lib.fake_log().decode().splitlines()


def rgb_plan(w, h, **kw):
    img = J.synth(w, h, quality=70, overlap=1, seed=9, threads=4, **kw)
    return J.CudaDecodePlan(img.arena, img.geometry, J.OutputFormat(C_["RGB"], D["U8"], S["U8"], L["RGB"], w, h))


def one_kernel_plan():
    return rgb_plan(64, 64)


@pytest.mark.parametrize("call", ["cudaHostAlloc", "cudaEventCreateWithFlags"])
def test_uploads_survive_a_refused_buffer_or_event(fake, call):
    """One refused page-locked buffer or event fails at most its own
    submission: the session's next one uploads from pageable memory again."""
    plan = one_kernel_plan()
    refused = 0
    for after in range(12):
        session = J.CudaDecoderSession(0, streams=1)
        fake.fake_reset()
        fake.fake_fail(call.encode(), after)
        try:
            session.submit(plan).close()
        except J.CudaError as e:
            assert e.kind == "Driver"
            refused += 1
        fake.fake_reset()
        for _ in range(2):
            sub = session.submit(plan)
            sub.wait()
            sub.close()
        assert not any(line.startswith("bad") for line in log(fake)), (after, log(fake))
        session.close()
    assert refused > 0
    plan.close()


# 4:2:2 keeps its interior and edge tiles in kernels of their own, so the set
# takes a side stream
def two_kernel_plan():
    return rgb_plan(1024, 1024, color_format=C_["YUV422"])


@pytest.mark.parametrize("call", ["cudaStreamCreateWithFlags", "cudaEventCreateWithFlags"])
def test_side_streams_survive_a_refused_handle(fake, call):
    """One refused stream or event fails its submission alone: the session's
    next one finds each side stream with its event."""
    plan = two_kernel_plan()
    refused = 0
    for after in range(8):
        session = J.CudaDecoderSession(0, streams=1)
        fake.fake_reset()
        fake.fake_fail(call.encode(), after)
        try:
            session.submit(plan).close()
        except J.CudaError as e:
            assert e.kind == "Driver"
            refused += 1
        fake.fake_reset()
        for _ in range(2):
            sub = session.submit(plan)
            sub.wait()
            sub.close()
        assert any(line.startswith("launch on 2") for line in log(fake))
        assert not any(line.startswith("bad") for line in log(fake)), (after, log(fake))
        session.close()
    assert refused > 0
    plan.close()


def test_submissions_outlive_their_session(fake):
    """A submission released after its session still waits, reads back and
    frees its memory on a live stream; then nothing is left."""
    before = live(fake)
    plan, small = two_kernel_plan(), one_kernel_plan()
    session = J.CudaDecoderSession(0)
    subs = [session.submit(plan), session.submit(small), session.submit_batch([small, plan])]
    session.close()
    for k, sub in enumerate(subs):
        sub.wait()
        assert sub.is_complete()
        assert sub.readback(0).size == (plan, small, small)[k].output_bytes()
        assert sub.report()["selected"] == "Cuda"
        sub.close()
    assert not any(line.startswith("bad") for line in log(fake)), log(fake)
    assert live(fake) == before
    plan.close()
    small.close()


@pytest.mark.parametrize("call", ["cudaMallocAsync", "cudaMemcpyAsync", "cudaEventRecord", "cudaStreamWaitEvent", "launch_tiles"])
def test_failed_submissions_leave_nothing(fake, call):
    """A submission that fails at any of its calls gives back its memory,
    events and status word; so does one that is refused."""
    before = live(fake)
    plan = two_kernel_plan()
    refused = 0
    for after in range(8):
        session = J.CudaDecoderSession(0, streams=1)
        for _ in range(10):             # what a session makes once
            session.submit(plan).close()
        fake.fake_reset()
        kept = live(fake)
        fake.fake_fail(call.encode(), after)
        try:
            session.submit(plan).close()
        except J.CudaError as e:
            assert e.kind == "Driver"
            refused += 1
        fake.fake_reset()
        assert live(fake)[DEVICE] == kept[DEVICE] and live(fake)[EVENTS] == kept[EVENTS]
        buf = np.empty(16, np.uint8)
        with pytest.raises(J.CudaError) as e:
            session.submit_into(plan, buf.ctypes.data, 16)
        assert e.value.kind == "InvalidDestination"
        assert live(fake) == kept
        session.close()
        assert not any(line.startswith("bad") for line in log(fake))
    assert refused > 0
    assert live(fake) == before
    plan.close()


def test_small_outputs_are_queued_with_their_submission(fake):
    """decode_to_host of a small picture queues the copy of its pixels ahead of
    its own event and waits for that event alone: work that other callers queue
    on the stream afterwards is not waited for."""
    plan = one_kernel_plan()
    session = J.CudaDecoderSession(0, streams=1)
    session.decode_to_host(plan)
    fake.fake_reset()
    session.decode_to_host(plan)
    lines = log(fake)
    copy = next(k for k, line in enumerate(lines) if line.startswith(f"copy device to pinned {plan.output_bytes()} on"))
    done = next(k for k in range(len(lines) - 1, -1, -1) if lines[k].startswith("record"))
    assert copy < done, lines
    assert f"wait event {lines[done].split()[1]}" in lines[done:]
    assert not any(line.startswith("wait stream") for line in lines), lines
    assert session.diagnostics()["bytes_read_back"] == 2 * plan.output_bytes()
    session.close()
    plan.close()


@pytest.mark.parametrize("side", [64, 2048])
def test_staged_bytes_are_uploaded_bytes(fake, side):
    """bytes_staged is the part of bytes_uploaded that came from pageable
    memory: all of it for a pageable arena, whichever page-locked buffer the
    tables went through (2048 x 2048: more than one of the small ones holds),
    and the tables alone for a page-locked one."""
    img = J.synth(side, side, quality=70, overlap=1, seed=9, threads=4)
    out = J.OutputFormat(C_["RGB"], D["U8"], S["U8"], L["RGB"], side, side)
    session = J.CudaDecoderSession(0)
    plan = J.CudaDecodePlan(img.arena, img.geometry, out)
    for _ in range(2):
        before = session.diagnostics()
        session.decode_to_host(plan)
        after = session.diagnostics()
        uploaded = after["bytes_uploaded"] - before["bytes_uploaded"]
        assert after["bytes_staged"] - before["bytes_staged"] == uploaded > img.arena.coefficients.nbytes
    plan.close()
    # the same arena in page-locked memory
    a, p = img.arena, C.c_void_p()
    fake.cudaHostAlloc(C.byref(p), C.c_size_t(a.coefficients.nbytes), 0)
    pinned = np.ctypeslib.as_array(C.cast(p, C.POINTER(C.c_int32)), (a.coefficients.size,))
    pinned[:] = a.coefficients
    plan = J.CudaDecodePlan(J.Arena(pinned, a.coefficient_offsets, a.quantizers, a.bands, a.hp_predictions, a.coded_x, a.coded_y,
                                    a.planes), img.geometry, out)
    before = session.diagnostics()
    session.decode_to_host(plan)
    after = session.diagnostics()
    assert after["bytes_uploaded"] - before["bytes_uploaded"] == uploaded
    assert after["bytes_staged"] - before["bytes_staged"] == uploaded - pinned.nbytes
    session.close()
    plan.close()
    fake.cudaFreeHost(p)


@pytest.mark.parametrize("kind,size,launches", [
    (dict(color_format=C_["YUV444"]), (640, 640), 1),                       # 100 tiles: edge tiles folded
    (dict(color_format=C_["YUV444"]), (1600, 1200), 1),                     # 475
    (dict(color_format=C_["YUV444"]), (3264, 3200), 2),                     # 2550, and one picture more below
    (dict(color_format=C_["YUV444"], hard_tiles=1, tile_width=16, tile_height=16), (1600, 1200), 2),
    (dict(color_format=C_["YUV420"]), (640, 640), 1),                       # no more than 192: one kernel
    (dict(color_format=C_["YUV422"]), (1024, 704), 1),                      # 176, and 188
    (dict(color_format=C_["YUV420"]), (1600, 1200), 2),
    (dict(color_format=C_["LUMA"]), (1600, 1200), 1),
])
def test_launches_of_a_set(fake, kind, size, launches):
    """Which tiles share a kernel: one-plane edge tiles always run with the
    interior ones, three-plane ones in sets of fewer than 2560 tiles without
    hard boundaries, subsampled ones in sets of no more than 192."""
    w, h = size
    img = J.synth(w, h, quality=40, overlap=1, seed=9, threads=8, **kind)
    layout, colour = ("LUMA", "LUMA") if kind["color_format"] == C_["LUMA"] else ("RGB", "RGB")
    plan = J.CudaDecodePlan(img.arena, img.geometry, J.OutputFormat(C_[colour], D["U8"], S["U8"], L[layout], w, h))
    few = J.synth(64, 192, quality=40, overlap=1, seed=9, **kind)           # 3 tiles more
    more = J.CudaDecodePlan(few.arena, few.geometry, J.OutputFormat(C_[colour], D["U8"], S["U8"], L[layout], 64, 192))
    session = J.CudaDecoderSession(0)
    for plans in ([plan, more, more, more, more], [plan]):
        res = session.resident(plans)
        # 2550 tiles alone stay folded
        assert res.launches(True) == (1 if plans == [plan] and size == (3264, 3200) else launches)
        res.close()
    session.close()
    for p in (plan, more):
        p.close()

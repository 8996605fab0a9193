"""Public API behaviour on the GPU: batches, host pipelines, //!WHEN."""
import numpy as np
import pytest

from mpv_prescalers_gb300 import synth

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.fail("CUDA device required for -m gpu tests")
    yield


@pytest.mark.parametrize("name", ["ravu-lite-ar-r3", "ravu-r3-yuv", "nnedi3-nns32-win8x4"])
def test_host_pipeline_matches_device_calls(name):
    hm, _ = synth.model_for(name)
    C = hm.n_planes
    frames = torch.stack([torch.from_numpy(synth.frame(36, 52, 100 + i, hm.channels)) for i in range(5)])
    frames = frames.to(torch.float16).pin_memory()
    got = hm.upscale_host(frames)
    assert got.shape == (5, C, 72, 104)
    for i in range(5):
        ref = hm.upscale(frames[i].cuda()).cpu()
        assert torch.equal(got[i], ref)


def test_host_pipelines_of_two_models_overlap_and_match():
    """wait=False queues the work and returns an event: two models' host
    pipelines in flight together give the same frames as device calls."""
    a, _ = synth.model_for("ravu-lite-ar-r4")
    b, _ = synth.model_for("nnedi3-nns16-win8x4")
    frames = torch.stack([torch.from_numpy(synth.luma_plane(30, 44, 300 + i))[None] for i in range(4)])
    frames = frames.to(torch.float16).pin_memory()
    ya, ea = a.upscale_host(frames, precision="fast", wait=False)
    yb, eb = b.upscale_host(frames, precision="fast", wait=False)
    ea.synchronize()
    eb.synchronize()
    for i in range(4):
        assert torch.equal(ya[i], a.upscale(frames[i].cuda(), precision="fast").cpu())
        assert torch.equal(yb[i], b.upscale(frames[i].cuda(), precision="fast").cpu())


def test_host_pipelines_of_one_model_back_to_back_match():
    """Several wait=False calls of one model and frame size in flight
    together: each call gets a work buffer no queued call still uses (its
    copies start at once, on the library's copy streams), and finished
    buffers are handed out again."""
    hm, _ = synth.model_for("ravu-lite-ar-r3")
    sets = [torch.stack([torch.from_numpy(synth.luma_plane(192, 320, 500 + 10 * k + i))[None] for i in range(6)])
            .to(torch.float16).pin_memory() for k in range(3)]
    keys0 = set(hm._host_work)
    res = [hm.upscale_host(f, precision="fast", wait=False) for f in sets]
    for f, (y, ev) in zip(sets, res):
        ev.synchronize()
        for i in range(6):
            assert torch.equal(y[i], hm.upscale(f[i].cuda(), precision="fast").cpu())
    (key,) = set(hm._host_work) - keys0
    pool = hm._host_work[key]
    # one buffer per call still in flight when the next was queued (how many
    # overlapped depends on timing), never one buffer twice
    assert 1 <= len(pool) <= 3 and len({w.data_ptr() for _, w in pool}) == len(pool)
    n = len(pool)
    y = hm.upscale_host(sets[0], precision="fast")       # reuses a finished buffer
    assert len(hm._host_work[key]) == n
    assert torch.equal(y, res[0][0])


@pytest.mark.parametrize("shape", [(3, 240, 320), (2, 3, 120, 160)], ids=["planes", "batch"])
def test_upscale_on_a_side_stream(shape):
    """With ``stream=`` the results are allocated and gathered on that stream
    (the [C][H][W] result is one tensor whose planes the kernels write; a
    batch is stacked after its kernels), so they equal the default-stream run."""
    hm, _ = synth.model_for("ravu-r3-yuv")
    x = torch.from_numpy(np.stack([synth.frame(shape[-2], shape[-1], 700 + i, hm.channels)
                                   for i in range(shape[0] if len(shape) == 4 else 1)]))
    x = (x if len(shape) == 4 else x[0]).to("cuda", torch.float16)
    want = hm.upscale(x, precision="fast")
    torch.cuda.synchronize()
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    got = hm.upscale(x, precision="fast", stream=s)
    s.synchronize()
    assert got.shape == want.shape and got.is_contiguous()
    assert torch.equal(got, want)


def test_host_pipeline_c_abi_checks_work_and_layout():
    import ctypes
    from mpv_prescalers_gb300 import _ffi, PrescaleError
    hm, _ = synth.model_for("ravu-r3-yuv")
    frames = torch.from_numpy(synth.yuv_frame(20, 28, 5))[None].to(torch.float16).pin_memory()
    out = torch.empty((1, 3, 40, 56), dtype=torch.float16).pin_memory()
    o = _ffi.Opts()
    o.out_width, o.out_height = 56, 40
    L = _ffi.lib()
    h = hm.device_handle(0)
    need = L.pz_run_host_work_bytes(h, 28, 20, _ffi.PZ_F16, ctypes.byref(o))
    assert need >= 3 * (3 * 20 * 28 * 2 + 3 * 40 * 56 * 2) and need % 3 == 0
    work = torch.empty(need, dtype=torch.uint8, device="cuda")
    s = torch.cuda.current_stream()
    slot = need // 3   # one frame in flight: one of the three slots
    rc = L.pz_run_host(h, frames.data_ptr(), out.data_ptr(), 1, 28, 20, _ffi.PZ_F16, ctypes.byref(o),
                       work.data_ptr(), slot - 256, 0, s.cuda_stream)
    assert rc == _ffi.PZ_EINVAL and b"work" in L.pz_last_error()
    _ffi.check(L.pz_run_host(h, frames.data_ptr(), out.data_ptr(), 1, 28, 20, _ffi.PZ_F16, ctypes.byref(o),
                             work.data_ptr(), slot, 0, s.cuda_stream))
    s.synchronize()
    assert torch.equal(out[0], hm.upscale(frames[0].cuda()).cpu())
    with pytest.raises(ValueError, match="contiguous"):
        hm.upscale_host(frames.transpose(2, 3))


def test_host_pipeline_when_false_passes_frames_through():
    hm, _ = synth.model_for("ravu-lite-r3")
    frames = torch.rand((2, 1, 20, 30)).pin_memory()
    y = hm.upscale_host(frames, out_size=(33, 22))   # below the //!WHEN ratio
    assert torch.equal(y, frames)


def test_batch_of_frames_matches_frame_by_frame():
    hm, _ = synth.model_for("ravu-zoom-ar-r2-rgb")
    x = torch.stack([torch.from_numpy(synth.rgb_frame(30, 40, 7 + i)) for i in range(3)]).cuda()
    y = hm.upscale(x, out_size=(70, 51))
    assert y.shape == (3, 3, 51, 70)
    for i in range(3):
        assert torch.equal(y[i], hm.upscale(x[i], out_size=(70, 51)))


def test_when_false_leaves_planes_untouched():
    hm, _ = synth.model_for("ravu-lite-r3")
    x = torch.rand((40, 60), device="cuda")
    y = hm.upscale(x, out_size=(70, 50))  # 0.86x per axis: //!WHEN wants < 0.707
    assert torch.equal(y, x)
    nn, _ = synth.model_for("nnedi3-nns16-win8x4")
    y = nn.upscale(x, out_size=(60, 80))  # rows only
    assert y.shape == (80, 60)


@pytest.mark.parametrize("name,osz", [("ravu-lite-ar-r3", None), ("ravu-r3-yuv", None), ("ravu-r4-yuv", None),
                                      ("ravu-r4", None), ("ravu-3x-r2-rgb", None),
                                      ("ravu-zoom-ar-r2", (1440, 810)), ("nnedi3-nns32-win8x4", None)])
def test_one_call_for_a_tensor_gives_the_planes_pixels(name, osz):
    """A tensor on the current stream goes down in one native call; the same
    planes as a list, with ``out`` or on a stream of their own take the
    general path: the same pixels for whole tensors and for views (rows,
    planes and frames further apart than they are long), frame by frame."""
    hm, _ = synth.model_for(name)
    C, (W, H) = hm.n_planes, (960, 540) if osz else (203, 57)
    big = torch.rand((4, C + 1, H + 2, W + 5), device="cuda").to(torch.float16)
    for x in (big[:3, :C, :H, :W], big[1:4:2, 1:, 2:, 5:], big[:2, :C, :H, :W].contiguous()):
        y = hm.upscale(x, out_size=osz, precision="fast")
        assert y.is_contiguous() and y.shape[:2] == x.shape[:2]
        s = torch.cuda.Stream()
        s.wait_stream(torch.cuda.current_stream())
        z = hm.upscale(x, out_size=osz, precision="fast", stream=s)
        torch.cuda.synchronize()
        assert torch.equal(y, z)
        for f in range(x.shape[0]):
            want = hm.upscale(list(x[f].unbind(0)), out_size=osz, precision="fast")
            assert all(torch.equal(a, b) for a, b in zip(y[f], want))
            assert torch.equal(hm.upscale(x[f], out_size=osz, precision="fast"), y[f])
    if C == 1:
        assert torch.equal(hm.upscale(x[0, 0], out_size=osz, precision="fast"), y[0, 0])
    with pytest.raises(ValueError):
        hm.upscale(torch.rand((1, C + 1, H, W), device="cuda"), out_size=osz)
    with pytest.raises(ValueError):
        hm.upscale(big[:, :C].transpose(2, 3), out_size=osz)


@pytest.mark.parametrize("name", ["ravu-lite-ar-r4", "ravu-lite-r2", "ravu-r3", "ravu-r4-rgb", "ravu-3x-r3-yuv",
                                  "ravu-zoom-ar-r2"])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float16])
def test_tma_staging_gives_identical_pixels(name, dtype):
    """Interior tiles staged by TMA boxes, border tiles by clamped loads: the
    same pixels as clamped loads everywhere."""
    hm, _ = synth.model_for(name)
    x = torch.from_numpy(synth.frame(100, 216, 61, hm.channels)).to("cuda", dtype)
    osz = (400, 180) if hm.family == "zoom" else None
    a = hm.upscale(x, out_size=osz, staging="ldg")
    b = hm.upscale(x, out_size=osz, staging="tma")
    assert torch.equal(a, b)


@pytest.mark.parametrize("name", ["ravu-lite-ar-r4", "ravu-lite-r2", "ravu-r3", "ravu-r4-rgb", "ravu-3x-r3-yuv",
                                  "ravu-zoom-ar-r2-rgb"])
@pytest.mark.parametrize("rows", [4, 8, 16])
@pytest.mark.parametrize("prec,dtype", [("fast", torch.float16), ("fp32", torch.float32)], ids=["fast", "fp32"])
def test_tile_heights_give_identical_pixels(name, rows, prec, dtype):
    """4-, 8- and 16-row tiles (both stagings) give the pixels and keys of the
    default layout; 102 input rows (zoom: 181 output rows) leave a ragged
    last tile row at every height."""
    hm, _ = synth.model_for(name)
    x = torch.from_numpy(synth.frame(102, 216, 63, hm.channels)).to("cuda", dtype)
    osz = (400, 181) if hm.family == "zoom" else None
    want, wkeys = hm.upscale(x, out_size=osz, precision=prec, staging="ldg", return_keys=True)
    for st in ("ldg", "tma"):
        got, keys = hm.upscale(x, out_size=osz, precision=prec, staging=st, tile_rows=rows, return_keys=True)
        assert torch.equal(got, want), st
        assert torch.equal(keys, wkeys), st


def test_tile_rows_are_checked_by_the_library():
    import ctypes
    from mpv_prescalers_gb300 import _ffi
    from mpv_prescalers_gb300 import batch as B
    hm, _ = synth.model_for("ravu-lite-ar-r3")
    x = torch.rand((40, 64), device="cuda")
    y = torch.empty((80, 128), device="cuda")
    pin = (_ffi.Plane * 1)(_ffi.Plane(x.data_ptr(), 64, 40, 64, _ffi.PZ_F32))
    pout = (_ffi.Plane * 1)(_ffi.Plane(y.data_ptr(), 128, 80, 128, _ffi.PZ_F32))
    o = _ffi.Opts()
    L = _ffi.lib()
    for bad in (1, 2, 5, 12, 32, -8):
        o.tile_rows = bad
        assert L.pz_run(hm.device_handle(0), pin, 1, pout, 1, ctypes.byref(o), None) == _ffi.PZ_EINVAL
        assert b"tile_rows" in L.pz_last_error()
    o.tile_rows = 0
    for bad in (-1, 2, 7):
        o.staging = bad
        assert L.pz_run(hm.device_handle(0), pin, 1, pout, 1, ctypes.byref(o), None) == _ffi.PZ_EINVAL
        assert b"staging" in L.pz_last_error()
    assert B.Job.make(hm, x, tile_rows=16).to_c().opts.tile_rows == 16
    assert B.Job.make(hm, x).to_c().opts.tile_rows == 0


def test_tile_autotuner(tmp_path):
    from mpv_prescalers_gb300 import batch as B
    hm, _ = synth.model_for("ravu-r3")
    x = torch.rand((270, 480), device="cuda", dtype=torch.float16)
    cache = B.PlanCache(str(tmp_path / "p.json"))
    (st, rows), times = B.autotune_tiles(hm, x, precision="fast", cache=cache, reps=2)
    assert st in ("ldg", "tma") and rows in (4, 8, 16)
    assert set(times) == {f"{s}/{r}" for s, r in B.tile_layouts(hm)}
    assert B.autotune_tiles(hm, x, precision="fast", cache=cache)[0] == (st, rows)   # cached
    jobs = B.tune_tiles([B.Job.make(hm, x, precision="fast")], cache=cache)
    assert (jobs[0].staging, jobs[0].tile_rows) == (st, rows)


@pytest.mark.parametrize("name", ["ravu-zoom-r2", "ravu-zoom-ar-r2-rgb", "ravu-zoom-r3-yuv", "ravu-zoom-ar-r3"])
@pytest.mark.parametrize("osz", [(218, 101), (241, 131), (324, 150), (500, 101), (801, 367), (218, 370)],
                         ids=["1.0x", "1.1x", "1.5x", "2.3x1x", "3.7x", "1x3.7x"])
@pytest.mark.parametrize("prec,dtype", [("fast", torch.float16), ("fp32", torch.float32)], ids=["fast", "fp32"])
def test_zoom_tma_rectangles_give_identical_pixels(name, osz, prec, dtype):
    """ravu-zoom's input rectangles staged from TMA boxes fitted to the scale
    factor (interior rectangles; the others by clamped loads) give the
    clamped-load pixels at every scale, per axis, at every tile height."""
    hm, _ = synth.model_for(name)
    x = torch.from_numpy(synth.frame(100, 217, 64, hm.channels)).to("cuda", dtype)
    assert hm.enabled(217, 100, osz)
    want = hm.upscale(x, out_size=osz, precision=prec, staging="ldg")
    for rows in (4, 8, 16):
        assert torch.equal(hm.upscale(x, out_size=osz, precision=prec, staging="tma", tile_rows=rows), want), rows


@pytest.mark.parametrize("name", ["ravu-zoom-r2", "ravu-zoom-r3-yuv", "ravu-zoom-ar-r2-rgb", "ravu-zoom-ar-r3"])
@pytest.mark.parametrize("size,osz,table", [((721, 487), (1442, 974), True), ((720, 486), (1080, 729), True),
                                            ((640, 484), (1120, 847), True), ((960, 400), (1200, 800), True),
                                            ((640, 360), (960, 540), False), ((853, 479), (1501, 843), False)],
                         ids=["2x", "1.5x", "1.75x", "1.25x2x", "small", "no-ratio"])
@pytest.mark.parametrize("prec,dtype", [("fast", torch.float16), ("fp32", torch.float32), ("mpv", torch.float16)])
def test_zoom_phase_table_gives_identical_pixels(name, size, osz, table, prec, dtype):
    """With the scratch pz_scratch_wanted names, ravu-zoom takes its weights
    from a table of the scale's phases: the pixels and keys of the general
    path, at every tile height.  Small frames and scales of no simple ratio
    want none."""
    import ctypes
    from mpv_prescalers_gb300 import _ffi
    from mpv_prescalers_gb300.prescaler import PRECISIONS
    hm, _ = synth.model_for(name)
    W, H = size
    x = torch.rand((hm.n_planes, H, W), device="cuda").to(dtype)
    o = _ffi.Opts()
    o.precision = PRECISIONS[prec]
    o.out_width, o.out_height = osz
    n = _ffi.lib().pz_scratch_wanted(hm.device_handle(0), W, H, 0 if dtype == torch.float32 else 1, ctypes.byref(o))
    assert (n > 0) == table
    scratch = torch.empty(max(n, 16), dtype=torch.uint8, device="cuda")

    def run(**kw):
        y = torch.empty((hm.n_planes, osz[1], osz[0]), device="cuda", dtype=dtype)
        k = torch.empty(osz[::-1], device="cuda", dtype=torch.int32)
        hm.run_raw(list(x.unbind(0)), list(y.unbind(0)), osz, precision=prec, keys=k, **kw)
        return y, k

    want, wkeys = run()
    for rows in (None, 8, 16):
        got, keys = run(scratch=scratch, tile_rows=rows)
        assert torch.equal(got, want) and torch.equal(keys, wkeys), rows


def test_zoom_tma_box_larger_than_the_plane_falls_back():
    hm, _ = synth.model_for("ravu-zoom-ar-r2")
    x = torch.rand((6, 20), device="cuda", dtype=torch.float16)   # smaller than any box
    assert hm.enabled(20, 6, (37, 11))
    assert torch.equal(hm.upscale(x, out_size=(37, 11), staging="tma"), hm.upscale(x, out_size=(37, 11), staging="ldg"))


def test_tma_staging_falls_back_for_unaligned_pitch():
    hm, _ = synth.model_for("ravu-lite-ar-r3")
    big = torch.from_numpy(synth.luma_plane(90, 203, 62)).cuda()   # pitch 203 floats: not 16-byte rows
    view = big[:, :200]
    assert torch.equal(hm.upscale(view, staging="tma"), hm.upscale(view.contiguous(), staging="ldg"))


def test_staging_autotuner(tmp_path):
    from mpv_prescalers_gb300 import batch as B
    hm, _ = synth.model_for("ravu-lite-ar-r3")
    x = torch.rand((270, 480), device="cuda", dtype=torch.float16)
    best, times = B.autotune_staging(hm, x, cache=B.PlanCache(str(tmp_path / "p.json")), reps=2)
    assert best in ("ldg", "tma") and set(times) == {"ldg", "tma"}


@pytest.mark.parametrize("name,osz", [("ravu-lite-ar-r3", None), ("ravu-r3-yuv", None), ("ravu-3x-r2-rgb", None),
                                      ("ravu-zoom-ar-r2", (101, 77)), ("nnedi3-nns16-win8x4", None),
                                      ("nnedi3-nns16-win8x4", (40, 60)), ("nnedi3-nns16-win8x4", (80, 30))])
def test_query_matches_the_python_geometry(name, osz):
    import ctypes
    from mpv_prescalers_gb300 import _ffi
    hm, _ = synth.model_for(name)
    W, H = 40, 30
    o = _ffi.Opts()
    if osz is not None:
        o.out_width, o.out_height = osz
    if hm.family == "nnedi3":
        o.nnedi3_axes = hm.nnedi3_axes(W, H, osz)
    r = _ffi.QueryResult()
    _ffi.check(_ffi.lib().pz_query(hm.device_handle(0), W, H, _ffi.PZ_F16, ctypes.byref(o), ctypes.byref(r)))
    assert (r.out_width, r.out_height) == hm.output_size(W, H, osz)
    assert r.n_planes == hm.n_planes
    want_scratch = 2 * W * H * 2 if hm.family == "nnedi3" and o.nnedi3_axes == 3 else 0
    if hm.family == "ravu":   # the FP32 int11 plane between the two lattice launches
        want_scratch = hm.n_planes * W * H * 4
    assert r.scratch_bytes == want_scratch


@pytest.mark.parametrize("name,size,osz,precision", [
    ("ravu-r3", (203, 57), None, "fp32"), ("ravu-r4-yuv", (640, 360), None, "fast"),
    ("ravu-zoom-ar-r2", (960, 540), (1440, 810), "fast"), ("nnedi3-nns16-win8x4", (96, 40), None, "fp32"),
    ("nnedi3-nns64-win8x6", (320, 180), None, "fast")])
def test_chains_queued_back_to_back_and_captured(name, size, osz, precision):
    """A chain's second launch begins while its first still runs, waits for it,
    and a chain queued behind another one reuses its scratch: frames queued
    without a wait, and replayed from a graph, are the frames made one by one."""
    hm, _ = synth.model_for(name)
    (W, H), C = size, hm.n_planes
    xs = [torch.rand((C, H, W), device="cuda").to(torch.float16) for _ in range(6)]
    OW, OH = osz or (2 * W, 2 * H)
    scratch = torch.empty(16 << 20, dtype=torch.uint8, device="cuda")

    def run(x, out):
        hm.run_raw(list(x.unbind(0)), list(out.unbind(0)), (OW, OH), precision=precision, scratch=scratch)

    outs = [[torch.zeros((C, OH, OW), dtype=torch.float16, device="cuda") for _ in xs] for _ in range(3)]
    for x, o in zip(xs, outs[0]):
        run(x, o)
        torch.cuda.synchronize()
    for x, o in zip(xs, outs[1]):
        run(x, o)
    g = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(g):
        for x, o in zip(xs, outs[2]):
            run(x, o)
    g.replay()
    torch.cuda.synchronize()
    for a, b, c in zip(*outs):
        assert torch.equal(a, b) and torch.equal(a, c)


@pytest.mark.parametrize("name", ["ravu-r3", "ravu-r2-yuv", "nnedi3-nns32-win8x4"])
def test_frames_without_scratch_ignore_its_byte_count(name):
    """pz_run_frames without a scratch buffer has room for no frame, whatever
    byte count comes with the null pointer: it allocates for one frame at a
    time, and the frames are the same."""
    import ctypes
    from mpv_prescalers_gb300 import _ffi
    hm, _ = synth.model_for(name)
    n, C, H, W = 3, hm.n_planes, 40, 56
    x = torch.rand((n, C, H, W), device="cuda")
    y = torch.empty((n, C, 2 * H, 2 * W), device="cuda")
    o = _ffi.Opts()
    o.out_width, o.out_height = 2 * W, 2 * H
    _ffi.check(_ffi.lib().pz_run_frames(
        hm.device_handle(0), x.data_ptr(), C * H * W, H * W, W, y.data_ptr(), 4 * C * H * W, 4 * H * W, 2 * W, n, W, H,
        _ffi.PZ_F32, ctypes.byref(o), None, 1 << 30, torch.cuda.current_stream().cuda_stream))
    assert torch.equal(y, hm.upscale(x))


@pytest.mark.parametrize("name,size,osz", [("ravu-zoom-r2", (960, 540), (1440, 810)),
                                           ("ravu-zoom-ar-r3", (960, 540), (1920, 1080)),
                                           ("ravu-lite-r3", (96, 54), None), ("ravu-3x-r2", (96, 54), None)])
def test_scratch_that_a_chain_does_not_need_is_left_alone(name, size, osz):
    """pz_run does not write to the scratch of a chain for which
    pz_scratch_bytes says 0: a host may hand one buffer to all its calls."""
    hm, _ = synth.model_for(name)
    W, H = size
    x = torch.rand((H, W), device="cuda", dtype=torch.float16)
    OW, OH = hm.output_size(W, H, osz)
    y = torch.empty((OH, OW), device="cuda", dtype=torch.float16)
    scratch = torch.full((64 << 20,), 0x5A, dtype=torch.uint8, device="cuda")
    hm.run_raw([x], [y], (OW, OH), precision="fast", scratch=scratch)
    assert torch.equal(y, hm.upscale(x, out_size=osz, precision="fast"))
    assert bool((scratch == 0x5A).all())


@pytest.mark.parametrize("name", ["ravu-zoom-r2", "ravu-zoom-r3-yuv", "ravu-zoom-ar-r2-rgb", "ravu-zoom-ar-r3"])
@pytest.mark.parametrize("size,osz", [((721, 487), (1442, 974)), ((720, 486), (1080, 729)), ((960, 400), (1200, 800))],
                         ids=["2x", "1.5x", "1.25x2x"])
@pytest.mark.parametrize("prec,dtype", [("fast", torch.float16), ("fp32", torch.float32), ("mpv", torch.float16)])
def test_zoom_phase_table_in_a_calls_own_scratch(name, size, osz, prec, dtype):
    """Calls with scratch of their own (a list of planes, a tensor, with keys,
    into given outputs) take the weights from the phase table: the pixels and
    keys of the general path, at every tile height; queued behind one another
    in one scratch, and replayed from a graph."""
    import ctypes
    from mpv_prescalers_gb300 import _ffi
    from mpv_prescalers_gb300.prescaler import PRECISIONS
    hm, _ = synth.model_for(name)
    C, (W, H), (OW, OH) = hm.n_planes, size, osz
    xs = [torch.rand((C, H, W), device="cuda").to(dtype) for _ in range(3)]
    want = [torch.empty((C, OH, OW), device="cuda", dtype=dtype) for _ in xs]
    wkeys = torch.empty((OH, OW), device="cuda", dtype=torch.int32)
    for x, y in reversed(list(zip(xs, want))):
        hm.run_raw(list(x.unbind(0)), list(y.unbind(0)), osz, precision=prec, keys=wkeys)
    for rows in (None, 4, 8, 16):
        got, keys = hm.upscale(list(xs[0].unbind(0)), out_size=osz, precision=prec, tile_rows=rows, return_keys=True)
        assert all(torch.equal(a, b) for a, b in zip(got, want[0])) and torch.equal(keys, wkeys), rows
        assert torch.equal(hm.upscale(xs[0], out_size=osz, precision=prec, tile_rows=rows), want[0]), rows
    o = _ffi.Opts()
    o.precision = PRECISIONS[prec]
    o.out_width, o.out_height = osz
    n = _ffi.lib().pz_scratch_wanted(hm.device_handle(0), W, H, 0 if dtype == torch.float32 else 1, ctypes.byref(o))
    scratch = torch.zeros(n, dtype=torch.uint8, device="cuda")
    outs = [torch.zeros_like(y) for y in want]

    def queue():
        for x, y in zip(xs, outs):
            pin, pout, c = hm._planes(list(x.unbind(0)), list(y.unbind(0)))
            _ffi.check(_ffi.lib().pz_run_with_scratch(hm.device_handle(0), pin, c, pout, c, ctypes.byref(o),
                                                      scratch.data_ptr(), n, torch.cuda.current_stream().cuda_stream))

    queue()
    assert all(torch.equal(a, b) for a, b in zip(outs, want)) and bool((scratch != 0).any())
    for y in outs:
        y.zero_()
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        queue()
    g.replay()
    assert all(torch.equal(a, b) for a, b in zip(outs, want))


@pytest.mark.parametrize("size,osz,table", [((2624, 1476), (3840, 2160), 288 * 3600 * 21 * 16), ((2592, 1458), (3840, 2160), 1),
                                            ((4928, 2772), (7680, 4320), 0), ((5120, 2880), (7680, 4320), 1)])
def test_zoom_phase_table_is_bounded(size, osz, table):
    """Every 2160p output whose scale has few phases has room for its table;
    14400 phases of an 8K output do not (1.4 GB), 9 do."""
    import ctypes
    from mpv_prescalers_gb300 import _ffi
    hm, _ = synth.model_for("ravu-zoom-ar-r3")
    o = _ffi.Opts()
    o.out_width, o.out_height = osz
    n = _ffi.lib().pz_scratch_wanted(hm.device_handle(0), *size, _ffi.PZ_F16, ctypes.byref(o))
    assert n <= 512 << 20 and (n >= table if table else n == 0)


@pytest.mark.parametrize("name,osz", [("ravu-zoom-ar-r2", (1440, 810)), ("ravu-r3", None), ("nnedi3-nns16-win8x4", None)])
def test_upscale_without_room_for_scratch(name, osz, monkeypatch):
    """Scratch that the device has no room for is done without: a ravu-zoom
    interpolates per pixel, a batch runs frame by frame in scratch that the
    library allocates; as a tensor, a batch and a list."""
    hm, _ = synth.model_for(name)
    x = torch.rand((2, 1, 540, 960), device="cuda", dtype=torch.float16)
    want = hm.upscale(x, out_size=osz)
    empty = torch.empty

    def no_room(*args, **kw):
        if kw.get("dtype") is torch.uint8:
            raise torch.cuda.OutOfMemoryError("no room")
        return empty(*args, **kw)

    monkeypatch.setattr(torch, "empty", no_room)
    assert torch.equal(hm.upscale(x, out_size=osz), want)
    assert torch.equal(hm.upscale(x[0], out_size=osz), want[0])
    assert torch.equal(hm.upscale([x[1, 0]], out_size=osz)[0], want[1, 0])

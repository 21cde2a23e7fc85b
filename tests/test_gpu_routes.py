"""Launches that a kernel's geometry makes special, each frame's records and
mask against the oracle."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


def _spots(h, w, seed, mean=1.0):
    rng = np.random.default_rng(seed)
    f = rng.poisson(mean, (h, w)).astype(np.uint32)
    for _ in range(max(1, h * w // 500)):
        y, x = rng.integers(0, h), rng.integers(0, w)
        f[max(0, y - 1):y + 2, max(0, x - 1):x + 2] += rng.integers(20, 900, dtype=np.uint32)
    return f


def _device(f):
    import torch
    return torch.from_numpy(f.view(np.int32 if f.dtype == np.uint32 else np.int16)).cuda()


def _check(b, frames, p):
    for j, f in enumerate(frames):
        want, mask = O.dext(f, O.Params(**p), with_mask=True)
        assert b.result(j).tobytes() == want.tobytes(), (j, f.shape, p)
        assert np.array_equal(b.mask(j), mask.astype(bool)), (j, f.shape, p)


@pytest.mark.parametrize("algorithm", [0, 1])
@pytest.mark.parametrize("kernel", [2, 3, 4])
def test_blocks_without_rows(kernel, algorithm):
    # The grid is the tallest frame's: most blocks of the short frames have no
    # row, and their counts are still theirs to write.
    from sfgb import api
    p = dict(algorithm=algorithm, kernel_x=kernel, kernel_y=kernel)
    frames = [_spots(h, w, 10 * h + w) for h, w in [(4001, 90), (3, 5), (40, 33), (9, 90), (1, 1)]]
    b = api.MixedBatch([f.shape for f in frames], capacity=4001 * 90, params=api.Params(**p))
    for _ in range(4):
        b([_device(f) for f in frames])
        _check(b, frames, p)


# ---------------------------------------------------------------------------
# Kernel 3,3 above the pixel count where a launch takes the lattice (5,000,000):
# the frames of test_gpu_lattice.py, 32-bit ones beside a frame of that size and
# 16-bit ones as often as it takes.
# ---------------------------------------------------------------------------
LATTICE_PIXELS = 5_000_000


def _lattice_32(api, frames, what, params, offset=0):
    import torch
    filler = np.zeros((2300, 2300), np.uint32)
    filler[100:103, 200:203] = 500
    filler[2290:, 2290:] = 0xFFFFFFFF
    every = frames + [filler]
    b = api.MixedBatch([f.shape for f in every], capacity=max(f.size for f in every) // 8,
                       params=api.Params(**params), word_prefix=True)
    store = [torch.empty(f.size + 4, dtype=torch.int32, device="cuda") for f in every]
    views = [s[offset:offset + f.size].view(f.shape) for s, f in zip(store, every)]
    for v, f in zip(views, every):
        v.copy_(torch.from_numpy(f.view(np.int32)))
    b(views)
    for j, f in enumerate(every):
        want, mask = O.dext(f, O.Params(**params), with_mask=True)
        assert b.result(j).tobytes() == want.tobytes(), (what, j, f.shape, offset)
        assert np.array_equal(b.mask(j), mask.astype(bool)), (what, j, f.shape, offset)
        per = np.array([bin(int(x)).count("1") for x in b.words(j)])
        assert np.array_equal(b.words(j, b.word_prefix), np.cumsum(per) - per), (what, j)


def _lattice_16(api, frames, what, params):
    h, w = frames[0].shape
    reps = -(-(LATTICE_PIXELS + 1) // (64 * h * w))
    tall = [np.concatenate([f] * reps) for f in frames]
    dev = [_device(f) for f in tall]
    b = api.DeviceBatch(h * reps, w, 64, capacity=h * reps * w, params=api.Params(**params))
    b([dev[j % len(dev)] for j in range(64)])
    want = [O.dext(f, O.Params(**params), with_mask=True) for f in tall]
    for j in list(range(len(dev))) + [63]:
        records, mask = want[j % len(dev)]
        assert b.result(j).tobytes() == records.tobytes(), (what, j)
        assert np.array_equal(b.mask(j), mask.astype(bool)), (what, j)


@pytest.fixture
def large_launches(monkeypatch):
    """test_gpu_lattice with its comparisons in launches above the limit."""
    from sfgb import api
    import test_gpu_lattice as L

    def check(api, frames, what, params=None, also16=True):
        params = params or {}
        if frames[0].dtype == np.uint16:
            _lattice_16(api, frames, what, params)
            return
        _lattice_32(api, frames, what, params)
        _lattice_32(api, frames, what, params, offset=1)
        if also16 and frames[0].shape[1] % 4 == 0:
            _lattice_16(api, [L._as_u16(f) for f in frames], what, params)

    monkeypatch.setattr(L, "_check_batch", check)
    return api, L


@pytest.mark.parametrize("phase", [(0, 0), (2, 2), (1, 2), (2, 0)])
def test_lattice_masked_points(large_launches, phase):
    api, L = large_launches
    L.test_masked_pixels_on_lattice_points(api, phase)


@pytest.mark.parametrize("name", ["test_masked_bands_at_every_phase",
                                  "test_spots_on_tile_corners_and_last_columns",
                                  "test_saturated_and_wide_pixels_near_spots",
                                  "test_frame_of_signal_everywhere", "test_16bit_bright_values"])
def test_lattice_frames(large_launches, name):
    api, L = large_launches
    getattr(L, name)(api)


@pytest.mark.parametrize("params", [
    dict(gain=1.5), dict(gain=0.8, sigma_b=4.5, sigma_s=2.5), dict(min_local=5),
    dict(min_local=0), dict(global_threshold=40.5), dict(sigma_b=3.0, sigma_s=2.0)])
def test_lattice_16bit_parameters(large_launches, params):
    api, L = large_launches
    L.test_16bit_parameters(api, params)


def _boundary_frame(h, w):
    f = _spots(h, w, h * 1000 + w)
    rng = np.random.default_rng(h + 7 * w)
    f[rng.random((h, w)) < 0.01] = 0xFFFFFFFF
    return f


@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("params", [dict(), dict(min_local=20), dict(sigma_b=3.0, sigma_s=2.0),
                                    dict(sigma_b=0.0, sigma_s=0.0, min_local=0)])
def test_lattice_boundaries(params, offset):
    # Around the 360-column strips, the 28-column tiles, 8-row tiles and 3-row
    # triples; rows that are whole 16-byte pieces and rows that are not.
    from sfgb import api
    frames = [_boundary_frame(h, w) for h, w in [
        (1, 3), (2, 29), (7, 28), (8, 31), (9, 33), (17, 356), (31, 359), (33, 360), (40, 361),
        (23, 364), (12, 719), (25, 720), (19, 721), (16, 724), (130, 1030)]]
    _lattice_32(api, frames, "boundaries", params, offset)


@pytest.mark.parametrize("h,w", [(30, 4), (25, 28), (17, 32), (40, 356), (33, 360), (31, 364),
                                 (25, 720), (19, 724), (12, 1024)])
def test_lattice_16bit_boundaries(h, w):
    from sfgb import api
    frames = [_boundary_frame(h, w).astype(np.uint16) for _ in range(2)]
    frames[1][h // 2] = 0xFFFE
    _lattice_16(api, frames, f"{h} x {w}", {})


# ---------------------------------------------------------------------------
# Wide strips: 64 frames whose strips' rows are more than eight times the warps
# that a GB300 can hold (9728), which a launch of narrow ones never has.
# ---------------------------------------------------------------------------
WIDE_SHAPES = [(1220, 31), (1220, 360), (1217, 364), (1219, 361), (611, 724), (409, 1030),
               (613, 392)]


def _wide_strips(frames, p):
    from sfgb import api
    h, w = frames[0].shape
    assert 64 * h * ((w + 31) // 32 * 32 + 359) // 360 >= 8 * 64 * 152
    b = api.DeviceBatch(h, w, 64, capacity=h * w, params=api.Params(**p))
    dev = [_device(f) for f in frames]
    b([dev[j % len(dev)] for j in range(64)])
    for j, f in enumerate(frames):
        want, mask = O.dext(f, O.Params(**p), with_mask=True)
        assert b.result(j).tobytes() == want.tobytes(), (j, p)
        assert np.array_equal(b.mask(j), mask.astype(bool)), (j, p)


@pytest.mark.parametrize("algorithm", [0, 1])
@pytest.mark.parametrize("bits", [32, 16])
@pytest.mark.parametrize("kernel", [2, 3, 4])
@pytest.mark.parametrize("h,w", WIDE_SHAPES)
def test_wide_strips(h, w, kernel, bits, algorithm):
    from test_gpu_strips import _as16, _frames
    frames = _frames(h, w, h * 10000 + w)
    if bits == 16:
        frames = [_as16(f) for f in frames]
    for kw in (dict(), dict(gain=1.5, sigma_b=4.25, sigma_s=0.0, min_local=0),
               dict(sigma_b=1000.0, sigma_s=2.0), dict(sigma_b=2.5, gain=0.7),
               dict(gain=0.0, sigma_s=2.5, min_local=20, global_threshold=5.0)):
        _wide_strips(frames, dict(algorithm=algorithm, kernel_x=kernel, kernel_y=kernel, **kw))


@pytest.mark.parametrize("top", [7281, 9362, 13107, (1 << 20) - 1, 1 << 20, 1 << 22])
@pytest.mark.parametrize("algorithm", [0, 1])
@pytest.mark.parametrize("kernel", [2, 3, 4])
@pytest.mark.parametrize("h,w", [(1220, 84), (1219, 361), (613, 412)])
def test_wide_strips_large_counts(h, w, kernel, algorithm, top):
    # Rows that leave the strips' 32-bit sums, at 12 columns a lane.
    rng = np.random.default_rng(h + top)
    sparse = _spots(h, w, h + top, mean=3.0)
    hit = rng.random((h, w)) < 0.003
    sparse[hit] = top
    flat = rng.integers(top - 40, top + 1, (h, w)).astype(np.uint32)
    flat[h // 2:h // 2 + 3, w // 3:w // 3 + 3] = 5
    frames = [sparse, flat]
    for f in frames[:]:
        g = f.copy()
        g[rng.random((h, w)) < 0.03] = 0xFFFFFFFF
        g[:, w // 2:w // 2 + 4] = 0xFFFFFFFE
        frames.append(g)
    for kw in (dict(), dict(sigma_b=2.0, sigma_s=1.0, min_local=5), dict(gain=1.5, sigma_b=2.5)):
        _wide_strips(frames, dict(algorithm=algorithm, kernel_x=kernel, kernel_y=kernel, **kw))


# ---------------------------------------------------------------------------
# Settings that leave the streaming path for 32 x 32 tiles: a negative gain or
# sigma, and constants beyond the integer tests' range.
# ---------------------------------------------------------------------------
@pytest.mark.parametrize("algorithm", [0, 1])
@pytest.mark.parametrize("kernel", [2, 3, 4])
@pytest.mark.parametrize("params", [dict(gain=-1.0), dict(sigma_b=-2.0), dict(sigma_s=-1.5),
                                    dict(gain=1e6), dict(sigma_b=1e6),
                                    dict(gain=2e4, min_local=0, global_threshold=30.0)])
def test_tiles(params, kernel, algorithm):
    from sfgb import api
    p = dict(algorithm=algorithm, kernel_x=kernel, kernel_y=kernel, **params)
    frames = []
    for h, w in [(33, 31), (97, 130), (200, 333)]:
        f = _boundary_frame(h, w)
        f[h // 2, w // 2:w // 2 + 3] = [70000, 1 << 25, 0xFFFFFFFD]
        frames.append(f)
    b = api.MixedBatch([f.shape for f in frames], capacity=200 * 333, params=api.Params(**p))
    b([_device(f) for f in frames])
    _check(b, frames, p)


@pytest.mark.parametrize("h,w,kernel", [(1065, 1030, 3), (1065, 1030, 4), (2400, 2400, 3)])
def test_a_run_length_never_starves_a_small_launch(h, w, kernel):
    # A plan whose run length would leave most of the device without work takes
    # the default geometry: the same kernels in the same time (half again and the
    # best of many runs, against twice as long where the length was taken as given).
    import torch
    from sfgb import api
    frame = _device(_spots(h, w, 5))
    took = {}
    for rows in (0, 512):
        plan = api.Plan(h, w, 1, params=api.Params(kernel_x=kernel, kernel_y=kernel))
        plan.configure(rows)
        for _ in range(3):
            plan([frame])
        torch.cuda.synchronize()
        begin, end = (torch.cuda.Event(enable_timing=True) for _ in range(2))
        times = []
        for _ in range(20):
            begin.record()
            for _ in range(20):
                plan([frame])
            end.record()
            torch.cuda.synchronize()
            times.append(begin.elapsed_time(end))
        took[rows] = min(times)
        _check(plan, [frame.cpu().numpy().view(np.uint32)], dict(kernel_x=kernel, kernel_y=kernel))
        plan.close()
    assert took[512] < 1.5 * took[0], took


def test_profile_covers_frames_one_after_another():
    # A batch of the plain dispersion in a workspace for one frame runs frame by
    # frame; its profiled time is all frames' (eight here, against one's).
    import ctypes

    import torch
    from sfgb import api
    h, w, capacity = 1024, 1024, 1 << 16
    frame = _device(_spots(h, w, 9))
    p = api.Params(algorithm=1)
    L = api.lib()
    b = api.DeviceBatch(h, w, 8, capacity=capacity, params=p)
    small = L.sf_workspace_bytes(h, w, capacity)
    ptrs = (ctypes.c_void_p * 8)(*[frame.data_ptr()] * 8)

    def fused(n):
        best = 1e9
        for _ in range(10):
            rc = L.sf_threshold_u32_batch_device(
                ctypes.cast(ptrs, ctypes.c_void_p), n, h, w, ctypes.byref(b.params),
                b.out.data_ptr(), capacity, b.bits.data_ptr(), b.counts.data_ptr(), None,
                b.workspace.data_ptr(), small, torch.cuda.current_stream().cuda_stream)
            assert rc == 0, api.last_error()
            best = min(best, api.last_stage_times()["fused"])
        return best

    api.profile_stages(True)
    try:
        one, eight = fused(1), fused(8)
    finally:
        api.profile_stages(False)
    assert 0.0 < 1.8 * one < eight, (one, eight)
    want = O.dext(frame.cpu().numpy().view(np.uint32), O.Params(algorithm=1))
    for j in range(8):
        assert b.result(j).tobytes() == want.tobytes()

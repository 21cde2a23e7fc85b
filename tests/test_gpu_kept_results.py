"""Lists with little more room than their records: the results kept between the
decision and the record writer have a few places a 128-pixel run (none, one or
several), and pixels beyond them have their windows summed again. Spots stand
close together at the right end of a band's last rows, the runs a block takes
last, so that both algorithms meet runs and groups of runs with more strong
pixels than places. Whole records against the oracle."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


def _frame(h, w, seed, mean=1.0):
    rng = np.random.default_rng(seed)
    f = rng.poisson(mean, (h, w)).astype(np.uint32)
    scale = 1 if mean < 100.0 else 30
    bands = h // 8
    for b in range(seed % 3, bands, max(1, bands // 4)):
        for x in range(w // 5, w - 1, 8):
            f[8 * b + 5:8 * b + 8, x:x + 3] += scale * rng.integers(150, 900, dtype=np.uint32)
    f[h // 2:h // 2 + 2] = 0xFFFFFFFF
    f[:, w // 3] = 0xFFFFFFFE
    return f


# Runs of 128 pixels a row: 9, 25, 1 and 1; places a run: 11, 5, 1 and none.
@pytest.mark.parametrize("algorithm", [0, 1])
@pytest.mark.parametrize("bits", [32, 16])
@pytest.mark.parametrize("kernel", [2, 3, 4])
@pytest.mark.parametrize("h,w", [(1065, 1030), (1031, 3108), (60003, 40), (200000, 40)])
def test_more_strong_pixels_than_places(h, w, kernel, bits, algorithm):
    _check(h, w, kernel, bits, algorithm, 1.0)


# A background beyond the strips' saturation: every pixel is left to the decision
# of the plain dispersion, whole runs at a time.
@pytest.mark.parametrize("algorithm", [0, 1])
@pytest.mark.parametrize("bits", [32, 16])
@pytest.mark.parametrize("kernel", [2, 3, 4])
@pytest.mark.parametrize("h,w", [(1065, 1030), (131, 3109), (6003, 40)])
def test_candidates_everywhere(h, w, kernel, bits, algorithm):
    _check(h, w, kernel, bits, algorithm, 20000.0)


def _check(h, w, kernel, bits, algorithm, mean):
    import torch
    from sfgb import api
    frames = [_frame(h, w, seed, mean) for seed in (1, 2)]
    if bits == 16:
        frames = [f.astype(np.uint16) for f in frames]  # (the markers keep their low bits)
    p = dict(algorithm=algorithm, kernel_x=kernel, kernel_y=kernel)
    want = [O.dext(f, O.Params(**p)) for f in frames]
    capacity = max(len(r) for r in want) + 1
    view = np.int32 if bits == 32 else np.int16
    dev = [torch.from_numpy(f.view(view)).cuda() for f in frames]
    for n in (1, 2):
        b = api.DeviceBatch(h, w, n, capacity=capacity, params=api.Params(**p))
        b(dev[:n])
        for j in range(n):
            assert b.result(j).tobytes() == want[j].tobytes(), (n, j, p)

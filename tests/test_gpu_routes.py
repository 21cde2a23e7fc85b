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

"""Both algorithms' strips against the oracle, bit for bit: widths around a
strip's 360 columns and a mask word's 32, rows that are whole aligned pieces of
4 pixels and rows that are not, heights around a run's rows, values at and
beyond the strips' saturation and 2^32, masked bands, and parameters that leave
the integer decisions."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


def _frames(h, w, seed):
    rng = np.random.default_rng(seed)
    base = rng.poisson(1.0, (h, w)).astype(np.uint32)
    for _ in range(max(2, h * w // 600)):
        y, x = rng.integers(0, h), rng.integers(0, w)
        k = int(rng.integers(1, 4))
        base[max(0, y - k):y + k, max(0, x - k):x + k] += rng.integers(2, 2000, dtype=np.uint32)
    masked = base.copy()
    masked[h // 3:h // 3 + 4] = 0xFFFFFFFF
    masked[:, w // 2:w // 2 + 5] = 0xFFFFFFFE
    large = base.copy()
    hit = rng.random((h, w)) < 0.02
    large[hit] = rng.choice(np.array([7280, 7281, 7282, 9361, 9362, 9363, 13107, 13108, 65532,
                                      (1 << 24) - 1, 1 << 24, 0xFFFFFFFD], np.uint32), int(hit.sum()))
    spots = base.copy()
    for _ in range(3):
        spots[rng.integers(0, h), rng.integers(0, w)] = rng.choice([9362, 40000, 3_000_000_000])
    high = rng.integers(30000, 41000, (h, w)).astype(np.uint32)
    high[rng.random((h, w)) < 0.01] = 0xFFFFFFFF
    return [base, masked, large, spots, high]


def _as16(f):
    return np.where(f >= 0xFFFFFFFE, f & 0xFFFF, np.minimum(f, 65533)).astype(np.uint16)


@pytest.mark.parametrize("algorithm", [0, 1])
@pytest.mark.parametrize("bits", [32, 16])
@pytest.mark.parametrize("kernel", [2, 3, 4])
@pytest.mark.parametrize("h,w", [(1, 1), (5, 31), (23, 360), (8, 364), (37, 361), (61, 724),
                                 (130, 1030), (257, 392)])
def test_strips_against_oracle(h, w, kernel, bits, algorithm):
    import torch
    from sfgb import api
    frames = _frames(h, w, h * 10000 + w)
    if bits == 16:
        frames = [_as16(f) for f in frames]
    for kw in (dict(), dict(gain=1.5, sigma_b=4.25, sigma_s=0.0, min_local=0),
               dict(sigma_b=1000.0, sigma_s=2.0), dict(sigma_b=2.5, gain=0.7),
               dict(gain=0.0, sigma_s=2.5, min_local=20, global_threshold=5.0)):
        p = dict(algorithm=algorithm, kernel_x=kernel, kernel_y=kernel, **kw)
        b = api.DeviceBatch(h, w, len(frames), capacity=h * w, params=api.Params(**p),
                            word_prefix=True)
        dt = np.int32 if bits == 32 else np.int16
        b([torch.from_numpy(f.view(dt)).cuda() for f in frames])
        for j, f in enumerate(frames):
            want = O.dext(f, O.Params(**p))
            assert b.result(j).tobytes() == want.tobytes(), (j, p)
            mask = np.zeros(h * w, bool)
            mask[want["index"]] = True
            assert np.array_equal(b.mask(j).ravel(), mask), (j, p)
            words = np.zeros((h, b.words_per_row * 32), bool)
            words[:, :w] = mask.reshape(h, w)
            per = words.reshape(-1, 32).sum(axis=1)
            got = b.word_prefix[j].cpu().numpy()
            assert np.array_equal(got, np.cumsum(per) - per), (j, p)


@pytest.mark.parametrize("top", [7281, 9361, 9362, 13107, (1 << 20) - 1, 1 << 20, 1 << 22])
@pytest.mark.parametrize("algorithm", [0, 1])
@pytest.mark.parametrize("kernel", [2, 3, 4])
@pytest.mark.parametrize("h,w", [(24, 84), (37, 361), (90, 412)])
def test_large_counts_against_oracle(h, w, kernel, algorithm, top):
    """Frames whose largest pixel is just below or at the counts where a strip's
    rows and a tile's check change their sums: spots and flat fields of that
    count, with and without masked pixels beside them."""
    import torch
    from sfgb import api
    rng = np.random.default_rng(h + top)
    sparse = rng.poisson(3.0, (h, w)).astype(np.uint32)
    for _ in range(max(3, h * w // 400)):
        y, x = rng.integers(0, h), rng.integers(0, w)
        sparse[max(0, y - 1):y + 2, max(0, x - 2):x + 2] = top
    dense = rng.poisson(20.0, (h, w)).astype(np.uint32)
    dense[rng.random((h, w)) < 0.02] = top
    flat = rng.integers(top - 40, top + 1, (h, w)).astype(np.uint32)
    flat[h // 2:h // 2 + 3, w // 3:w // 3 + 3] = 5
    frames = [sparse, dense, flat]
    for f in frames[:]:
        g = f.copy()
        g[rng.random((h, w)) < 0.03] = 0xFFFFFFFF
        g[:, w // 2:w // 2 + 4] = 0xFFFFFFFE
        frames.append(g)
    for kw in (dict(), dict(sigma_b=2.0, sigma_s=1.0, min_local=5), dict(sigma_b=0.0, sigma_s=0.0),
               dict(gain=1.5, sigma_b=2.5)):
        p = dict(algorithm=algorithm, kernel_x=kernel, kernel_y=kernel, **kw)
        b = api.DeviceBatch(h, w, len(frames), capacity=h * w, params=api.Params(**p))
        b([torch.from_numpy(f.view(np.int32)).cuda() for f in frames])
        for j, f in enumerate(frames):
            assert b.result(j).tobytes() == O.dext(f, O.Params(**p)).tobytes(), (j, p)

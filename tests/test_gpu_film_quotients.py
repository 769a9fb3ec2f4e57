"""The film resolve's short quotient decides every byte as the exact division
does (GPU): averages on, next to and a few to 2^20 ulps from every threshold and
bucket edge, for counts of every kind, against numpy's FP64 division and the
host's threshold table; and the tiled kernel against the one that divides.
"""

import numpy as np
import pytest
import torch

import albedo_b200 as ab

pytestmark = pytest.mark.gpu

COUNTS = [1, 2, 3, 7, 36, 49, 64, 100, 1023, 65537, (1 << 31) + 11, (1 << 32) - 1, (1 << 32) + 5, (1 << 40) + 3,
          (1 << 53) + 2]


def expected_bytes(sums, counts):
    lower, _ = ab.srgb_tables()
    with np.errstate(over="ignore", invalid="ignore", divide="ignore"):
        average = np.where(counts[:, None] > 0, sums / counts.astype(np.float64)[:, None], 0.0)
    found = np.searchsorted(lower[1:], np.nan_to_num(average, nan=-1.0, posinf=2.0, neginf=-1.0), side="right")
    return found.astype(np.uint8)


def resolved(sums, counts, offset=0):
    acc = torch.zeros(4 * len(sums) + offset, dtype=torch.float64, device="cuda")
    rows = acc[offset:].view(-1, 4)
    rows[:, :3] = torch.from_numpy(sums).cuda()
    rows.view(torch.int64)[:, 3] = torch.from_numpy(counts).cuda()
    out = torch.empty(3 * len(sums), dtype=torch.uint8, device="cuda")
    ab.resolve_srgb(acc.data_ptr() + 8 * offset, len(sums), 1, out.data_ptr())
    return out.cpu().numpy().reshape(-1, 3)


def check(sums, counts):
    got = resolved(sums, counts)
    np.testing.assert_array_equal(got, expected_bytes(sums, counts))
    # One double further on the accumulators are not 32-byte aligned: the kernel that divides.
    np.testing.assert_array_equal(got, resolved(sums, counts, offset=1))


@pytest.mark.parametrize("count", COUNTS)
def test_averages_around_every_decision(count):
    lower, _ = ab.srgb_tables()
    edges = (np.int64(ab.SRGB_BUCKET_BASE) + np.arange(ab.SRGB_BUCKETS, dtype=np.int64)) << ab.SRGB_BUCKET_SHIFT
    marks = np.concatenate([lower[1:].view(np.int64), edges])
    steps = np.array([0, 1, 2, 5, 100, 4095, 8191, 8192, 8193, 16384, 1 << 20], dtype=np.int64)
    averages = (marks[:, None] + np.concatenate([-steps[1:], steps])[None, :]).reshape(-1).view(np.float64)
    sums = averages * np.float64(count)
    sums = np.stack([sums, np.nextafter(sums, 0.0), np.nextafter(sums, np.inf)], axis=1)
    check(sums, np.full(len(sums), count, dtype=np.int64))


@pytest.mark.parametrize("pixels", [1, 31, 127, 128, 129, 1000, 300_001])
def test_seeded_films_of_ragged_sizes(pixels):
    rng = np.random.default_rng(pixels)
    counts = rng.choice(np.array([0, 1, 3, 36, 64, 225, 1 << 40], dtype=np.int64), pixels)
    sums = np.exp(rng.normal(-1.5, 2.0, (pixels, 3))) * counts[:, None]
    special = np.array([0.0, -0.0, -1.0, 1.0, 2.0, np.inf, -np.inf, np.nan, 1e308, 5e-324])
    chosen = rng.random(sums.shape) < 0.2
    sums[chosen] = rng.choice(special, int(chosen.sum()))
    check(sums, counts)

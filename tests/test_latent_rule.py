"""Which segments of a step go through keys and values per head (no GPU)."""
from __future__ import annotations

import pytest

from inference_bench_b200.parts import latent
from inference_bench_b200.parts.latent import LatentAttention
from inference_bench_b200.parts.standard import NoPositionEncoding

SMALL, LITE = dict(heads=8, dim=64, rot_dim=32, vdim=64, kv_rank=256), dict(heads=16, dim=128, rot_dim=64, vdim=128, kv_rank=512)


def _choose(z, segments, window=None):
    att = LatentAttention("a", 64, z["heads"], z["dim"], z["rot_dim"], z["vdim"], z["kv_rank"], 1.0, 1e-5, NoPositionEncoding(), window=window)
    starts = [0]
    for n, _ in segments:
        starts.append(starts[-1] + n)
    got = att._choose(starts, [p for _, p in segments])
    return got if got is None else (sorted(c[0] for c in got[0]), got[1])


DECODED = [(1, 700 + 13 * i) for i in range(8)]


@pytest.mark.parametrize("z,segments,want", [
    (SMALL, [(31, 0)], None), (SMALL, [(32, 0)], ([0], [])), (SMALL, [(32, 64 * 32 - 32)], ([0], [])), (SMALL, [(32, 64 * 32 - 31)], None),
    (SMALL, [(5, 0), (40, 900), (1, 63)], ([0, 1, 2], [])),                            # one form serves all of them
    (SMALL, [(64, 0)] + DECODED, None), (LITE, [(300, 0)] + DECODED, None),            # both forms would cost more than they save
    (SMALL, [(1000, 0), (1, 700)], None), (SMALL, [(2048, 0)] + DECODED, ([0], [(2048 + i, 2049 + i) for i in range(8)])),
    (LITE, [(1, 900), (1000, 0), (5, 700)], ([1], [(0, 1), (1001, 1006)])), (LITE, DECODED[:1] * 2 + [(200, 0)] * 4, None), (LITE, [(400, 900)] * 4 + DECODED[:1], ([0, 1, 2, 3], [(1600, 1601)])),
    (SMALL, [(0, 5), (40, 0)], ([1], [])), (SMALL, [(1, 700), (1, 5)], None)])
def test_the_choice(z, segments, want):
    assert _choose(z, segments) == want


def test_a_window_bounds_what_is_made(monkeypatch):
    """Blocks start at the first position that the segment sees, and what does not fit the limit of bytes stays with the other form."""
    assert _choose(SMALL, [(32, 5000)], window=64) == ([0], [])
    att = LatentAttention("a", 64, 16, 128, 64, 128, 512, 1.0, 1e-5, NoPositionEncoding(), window=100)
    assert att._choose([0, 40, 300], [1000, 0]) == ([(0, 0, 40, 1000, 896, 3), (1, 40, 300, 0, 0, 5)], [])
    monkeypatch.setattr(latent, "EXPAND_BESIDE_SAVED_US", -1e9)
    monkeypatch.setattr(latent, "EXPAND_MAX_BYTES", 2 * 16 * 256 * 64 * 6)
    assert att._choose([0, 40, 300], [1000, 0]) == ([(0, 0, 40, 1000, 896, 3)], [(40, 300)])


@pytest.mark.parametrize("per", [1, 2, 3, 8])
@pytest.mark.parametrize("ranges", [[(0, 1)], [(0, 7), (7, 8), (20, 36)], [(5, 5), (5, 9)], [(3, 4)] * 3])
def test_runs(per, ranges):
    assert latent._runs(ranges, per) == [v for a, b in ranges for t in range(a, b, per) for v in (t, min(per, b - t))]

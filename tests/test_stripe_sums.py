"""The tensor core cuts its running sum at every instruction: a stretch of K that one accumulator sums is off by its length times its
sum.  Products in stripes cut K into stretches no longer, all together, than the kernels whose place they take; by sizes, without a GPU."""
from __future__ import annotations

import pytest

from nncpu_b200.kernels import ops

SMS = 148
NOISE = 4          # chunks of 64 columns: shorter stretches are not nearer to 64 bits


def squared(stretches, chunks):
    return sum(c ** 3 for c in stretches) / chunks


def clusters(n, chunks):
    """Up to 64 tokens: the slices of a cluster, whose blocks all run at once (two an SM, 87 of 100 places)."""
    tiles, best = -(-n // 128), 1
    if tiles < SMS:
        for s in range(2, 9):
            if chunks // s >= 4 and tiles * s <= 2 * SMS * 87 // 100:
                best = s
    return squared([chunks * (i + 1) // best - chunks * i // best for i in range(best)], chunks)


def dealt_out(n, chunks):
    """65 to 256 tokens: all tiles' chunks (tiles of 256 rows where there are 128-row tiles for all SMs) dealt out evenly."""
    tiles = -(-n // 128)
    tiles = -(-tiles // 2) if tiles >= SMS else tiles
    units = tiles * chunks
    blocks = max(1, min(SMS, units // 4))
    cuts = sorted({c * units // blocks for c in range(blocks + 1)} | {t * chunks for t in range(tiles + 1)})
    return squared([b - a for a, b in zip(cuts, cuts[1:])], chunks) / tiles


def stripes(m, k, stretch):
    chunks = k // 64
    halves = [chunks // 8 * 4, chunks - chunks // 8 * 4] if m <= 64 and k > 5120 else [chunks]
    return squared([c for h in halves for c in [stretch] * (h // stretch) + [h % stretch]], chunks)


@pytest.mark.parametrize("m", [24, 64, 100, 200])
def test_stretches(m):
    taken = 0
    for n in (16, 256, 768, 1024, 2048, 3072, 4096, 5120, 7168, 9216, 12288, 18944, 18960, 19200, 24576, 32768, 34816, 40960, 65536, 151936):
        for k in [64 * c for c in (1, 4, 5, 6, 8, 12, 16, 24, 32, 40, 48, 56, 64, 72, 80, 81, 96, 112, 128, 160, 192, 224, 256, 272)]:
            for epilogue in ("plain", "swiglu"):
                held = ops.linear_tc_stripes(m, n, k, epilogue)
                if held is None:
                    continue
                taken += 1
                before = (clusters if m <= 64 else dealt_out)(n, k // 64)
                assert held[2] <= NOISE or stripes(m, k, held[2]) <= before, (m, n, k, epilogue, held)
    assert taken > 200


@pytest.mark.parametrize("m,n,k,epilogue", [(24, 2048, 2048, "plain"), (64, 4096, 12288, "plain"), (64, 24576, 4096, "swiglu"), (33, 20480, 2048, "swiglu"), (64, 12288, 512, "swiglu"),
                                            (100, 65536, 4096, "plain"), (128, 34816, 5120, "swiglu"), (200, 24576, 4096, "swiglu"),
                                            (200, 1024, 5184, "plain"), (256, 151936, 4096, "plain"), (256, 76000, 128, "plain")])
def test_these_run_in_stripes(m, n, k, epilogue):
    assert ops.linear_tc_stripes(m, n, k, epilogue) is not None


# few features of long rows above 64 tokens: no room for so many accumulators; gated ones whose clusters fill the SMs better
@pytest.mark.parametrize("m,n,k,epilogue", [(100, 256, 16384, "plain"), (200, 512, 12288, "plain"), (200, 4096, 17408, "plain"),
                                            (64, 512, 4096, "swiglu"), (48, 2048, 4096, "swiglu"), (40, 5120, 4096, "swiglu"),
                                            (64, 8192, 4096, "swiglu"), (33, 128, 3072, "swiglu"), (64, 24576, 4160, "swiglu"),
                                            (64, 24576, 2048, "swiglu"), (33, 65536, 512, "swiglu"), (48, 18944, 512, "swiglu"),
                                            (24, 4096, 2048, "swiglu"), (100, 2048, 2072, "plain"), (16, 4096, 4096, "plain"),
                                            (257, 4096, 4096, "plain")])
def test_these_do_not(m, n, k, epilogue):
    assert ops.linear_tc_stripes(m, n, k, epilogue) is None

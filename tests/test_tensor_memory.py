"""Blocks that cannot hold their columns of tensor memory on one SM together must not fit its shared memory together either (an
allocation waits without limit, and the block it waits for may wait for it); by the sizes that launches ask for, without a GPU."""
from __future__ import annotations

import random

from nncpu_b200.kernels import ops

COLUMNS = 512
SHARED = 228 * 1024          # of an SM
RESERVED = 1024              # of it for every block that runs there
SIZES = sorted({64 * i for i in (1, 2, 3, 5, 8, 13, 16, 17, 32, 64, 80, 81, 96, 160, 192, 256)} | {64 * 272})
FEATURES = sorted({16, 64, 80, 1024, 1210, 2048, 2368, 4096, 4097, 5120, 6144, 9480, 12288, 18944, 18945, 24576, 25008, 34816, 37888, 50000,
                   65536, 76000, 151936})
TOKENS = (17, 24, 33, 48, 64, 65, 72, 100, 128, 129, 160, 200, 256)


def least_bytes():
    """The least shared memory that any stripes of so many columns ask for."""
    rng = random.Random(1)
    sizes = [(m, n, k) for m in TOKENS for n in FEATURES for k in SIZES]
    sizes += [(rng.randint(17, 256), rng.randint(1, 40000), 64 * rng.randint(1, 256)) for _ in range(20000)]
    least = {}
    for m, n, k in sizes:
        for epilogue in ("plain", "swiglu") if n % 16 == 0 else ("plain",):
            held = ops.linear_tc_stripes(m, n, k, epilogue)
            if held is not None:
                assert held[0] in (32, 64, 128, 256, 512) and held[1] <= 227 * 1024, (m, n, k, held)
                least[held[0]] = min(least.get(held[0], SHARED), held[1])
    return least


# the other kernels that allocate tensor memory, (columns, bytes of operands): the least of each
OTHERS = [(64, 1024 + 4 * 18 * 1024), (64, 1024 + 4 * 20 * 1024), (128, 1024 + 4 * 24 * 1024),       # a tile a block
          (32, 1024 + 4 * 20 * 1024 + 40 * 512), (64, 1024 + 3 * 24 * 1024 + 72 * 512),              # a cluster a tile
          (512, 31 * 1024 + 512 * 312), (256, 31 * 1024 + 256 * 312),                                # attention over heads of 64
          (512, 1024 + 4 * 48 * 1024), (64, 1024 + 5 * 160 * 192)]                                   # larger units, float32


def test_blocks_that_cannot_allocate_together_do_not_fit_together():
    least = least_bytes()
    assert set(least) == {32, 64, 128, 256, 512}
    stripes = list(least.items())
    kinds = stripes + OTHERS

    def walk(columns, room, start):
        for i in range(start, len(kinds)):
            left = room - kinds[i][1] - RESERVED
            if left < 0:
                continue
            assert columns + kinds[i][0] <= COLUMNS, (columns, kinds[i], kinds)
            walk(columns + kinds[i][0], left, i)

    walk(0, SHARED, 0)

"""Shares of the tcgen05 kernel of two query tiles per block, on the host: the arithmetic of its plan kernel.  What the merge step
folds is every CTA counted as working on a unit, so each of them has to have a step of it (and leave a partial)."""
import ctypes as C
import random

import pytest

from inference_lib_b200 import _cabi


@pytest.fixture(scope="module")
def lib():
    return _cabi.load()


def _plan(lib, blocks, Hkv, grid):
    n = len(blocks)
    pos, parts = (C.c_int64 * (grid + 1))(), (C.c_int32 * (2 * n * Hkv))()
    rc = lib.hogatt_dense_plan((C.c_int32 * n)(*[s for s, _ in blocks]), (C.c_uint8 * n)(*[int(x) for _, x in blocks]), n, Hkv, grid, pos, parts)
    assert rc == 0
    return list(pos), list(parts)


def _check(lib, blocks, Hkv, grid):
    pos, parts = _plan(lib, blocks, Hkv, grid)
    total = Hkv * sum(s for s, _ in blocks)
    assert pos[0] == 0 and pos[grid] == total and all(a <= b for a, b in zip(pos, pos[1:]))
    at, u = 0, 0
    for steps, _ in blocks:
        for _ in range(Hkv):
            first, count = parts[2 * u:2 * u + 2]
            workers = [c for c in range(grid) if max(pos[c], at) < min(pos[c + 1], at + steps)]
            assert list(range(first, first + count)) == workers, (blocks, Hkv, grid, u)
            at += steps
            u += 1
    assert at == total


@pytest.mark.parametrize("blocks,Hkv,grid", [
    ([(8, False), (8, False), (5, True)], 8, 148),          # 160 tokens of 4 heads per kv head, fragments of 640 and 360 keys
    ([(16, True)] * 5 + [(7, True)], 1, 148),               # single tokens of a packed batch
    ([(1, True)], 1, 148), ([(1, True), (0, True), (1, False)], 2, 148), ([(3, False)], 1, 148), ([(0, False), (2, True)], 1, 2),
])
def test_every_counted_cta_has_a_step(lib, blocks, Hkv, grid):
    _check(lib, blocks, Hkv, grid)


@pytest.mark.parametrize("seed", range(4))
def test_random_block_lists(lib, seed):
    rng = random.Random(seed)
    for _ in range(2000):
        most = rng.choice([2, 6, 20, 60, 400])
        blocks = [(0 if rng.random() < 0.1 else rng.randint(1, most), rng.random() < rng.choice([0, 0.3, 1])) for _ in range(rng.randint(1, 12))]
        _check(lib, blocks, rng.choice([1, 2, 4, 8]), rng.choice([1, 3, 20, 148, 148, 148]))

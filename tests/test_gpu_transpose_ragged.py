"""Blocks <-> 128 planes whose rows start at any byte (a multiple of 8 blocks, not
of 32; outputs and inputs at any address), against the oracle's transpose:
one tile and several, last tiles of 8 to 1,024 rows, rows wider than the
columns read, and untouched bytes around the output."""
import numpy as np
import pytest

import oracle
from tests.util import to_dev, to_host

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

BLOCKS = [8, 24, 32, 40, 120, 1016, 1024, 1032, 2056, 40008]


def guarded(nbytes, offset):
    buf = torch.full((nbytes + offset + 64,), 0xA5, dtype=torch.uint8, device="cuda")
    return buf, buf[offset:offset + nbytes]


def untouched(buf, nbytes, offset):
    h = to_host(buf)
    return (h[:offset] == 0xA5).all() and (h[offset + nbytes:] == 0xA5).all()


@pytest.mark.parametrize("offset", [0, 1, 2, 3, 16])
@pytest.mark.parametrize("n", BLOCKS)
def test_blocks_to_planes(ctx, n, offset):
    x = np.random.default_rng(n).integers(0, 256, n * 16, dtype=np.uint8)
    buf, out = guarded(16 * n, offset)
    ctx.bit_transpose(to_dev(x), n, 16, 0, 128, out)
    assert np.array_equal(to_host(out), oracle.bit_transpose(x, n, 16, 0, 128).reshape(-1))
    assert untouched(buf, 16 * n, offset)


@pytest.mark.parametrize("offset,extra", [(0, 0), (1, 0), (2, 3), (3, 1), (0, 5)])
@pytest.mark.parametrize("n", BLOCKS)
def test_planes_to_blocks(ctx, n, offset, extra):
    rb = n // 8 + extra
    x = np.random.default_rng(n + 1).integers(0, 256, 128 * rb, dtype=np.uint8)
    src = torch.empty(128 * rb + offset, dtype=torch.uint8, device="cuda")[offset:]
    src.copy_(to_dev(x))
    buf, out = guarded(16 * n, 16)
    ctx.bit_transpose(src, 128, rb, 0, n, out)
    assert np.array_equal(to_host(out), oracle.bit_transpose(x, 128, rb, 0, n).reshape(-1))
    assert untouched(buf, 16 * n, 16)


# around the sizes from which tiles are used: below them, last tiles of 8, 40, 1,016 and
# 1,024 rows, and whole words at odd addresses
TILES = [18424, 18432, 18440, 73720, 73728, 73736, 73768, 74744, 74752, 131072]


@pytest.mark.parametrize("offset", [0, 1, 2, 3])
@pytest.mark.parametrize("n", TILES)
def test_tiles_to_planes(ctx, n, offset):
    test_blocks_to_planes(ctx, n, offset)


@pytest.mark.parametrize("offset,extra", [(0, 0), (1, 0), (2, 3), (3, 1), (0, 5)])
@pytest.mark.parametrize("n", TILES)
def test_tiles_to_blocks(ctx, n, offset, extra):
    test_planes_to_blocks(ctx, n, offset, extra)

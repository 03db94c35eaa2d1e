"""What a device workspace holds per block and per fastMode-1 tile: the scratch
the kernels use, and no more."""
import pytest


@pytest.fixture(scope="module")
def L():
    from szx_gb300 import build
    build.build()
    from szx_gb300._lib import lib
    return lib()


@pytest.mark.parametrize("dt,n", [(0, 1 << 27), (1, (1 << 28) + 77)])
def test_bytes_per_tile_and_block(L, dt, n):
    fixed = 110_000   # header, range partials, paddings of the regions
    tiles = (n + 4095) // 4096
    # status words 8 + 1 and 4, three decode words a tile
    assert L.SZxG_workspace_size(1, dt, n, 128) <= fixed + tiles * (8 + 1 + 4 + 24)
    blocks = (n + 127) // 128
    # payload size 2, median 4, offset 8, state bit and rank 1/8 each; a tile of eight blocks: status words of 64, 16 and
    # 32 bits, and its share of the assembler's
    per_block = 2 + 4 + 8 + 0.25 + (8 + 2 + 4 + 0.04) / 8
    assert L.SZxG_workspace_size(3, dt, n, 128) <= fixed + int(blocks * per_block) + 24 * tiles

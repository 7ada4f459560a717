"""Every tile of the CUDA-core template at its edges. The operands are whole numbers small enough that every sum is exact in
f32, so the result has to match to the bit whatever the tile; the choice of the tile is checked on the CPU."""
import os
import re

import numpy as np
import pytest

from anvil_lang_b200.backend.emit import simt_tile
from kirbuild import contraction_program, contraction_reference

# M, N, K, batch, ta, tb -> tile
CASES = [
    ((2432, 1024, 33, 1, False, False), (128, 128)),     # 19 x 8 tiles: just enough
    ((2431, 1023, 17, 1, True, True), (128, 128)),       # the same count, ragged
    ((18945, 32, 9, 1, False, True), (128, 32)),         # 149 tiles, one row in the last
    ((19000, 32, 129, 1, True, False), (128, 32)),
    ((9472, 64, 65, 1, False, False), (64, 64)),         # 148 tiles
    ((513, 257, 600, 1, True, False), (64, 64)),         # split k: parts of 160 in blocks of 32
    ((512, 128, 128, 1, False, True), (32, 32)),
    ((200, 135, 100, 1, False, False), (32, 32)),
    ((65, 63, 127, 3, True, True), (32, 32)),            # batch, every edge ragged, the last k block one short
    ((130, 70, 1000, 2, False, False), (32, 32)),        # split k: chains that end inside a block of 64
]


@pytest.mark.parametrize("case,tile", CASES, ids=lambda c: "x".join(map(str, c)))
def test_tile_choice(case, tile):
    M, N, K, batch = case[:4]
    parts = batch                                         # the emitter's split of k, from the 128 x 128 tile count
    tiles = -(-M // 128) * -(-N // 128)
    if tiles * batch < 148 and K >= 256:
        parts *= max(1, min(296 // (tiles * batch), K // 128, 32))
    assert simt_tile(M, N, parts) == tile


@pytest.mark.gpu
@pytest.mark.parametrize("case,tile", CASES, ids=lambda c: "x".join(map(str, c)))
def test_tiles_are_exact(case, tile):
    from anvil_lang_b200.program import DeviceProgram
    M, N, K, batch, ta, tb = case
    os.environ["ANVIL_B200_TC"] = "0"
    try:
        prog, kern, A, B, C, bias = contraction_program(*case, bias=True)
        dp = DeviceProgram(prog, graphs=False)
    finally:
        os.environ.pop("ANVIL_B200_TC", None)
    assert re.search(r"gemm_simt_tile<\w+, \w+, \w+, \d+, %d, %d>" % tile, dp.source)
    rng = np.random.default_rng(M)
    a, b = (rng.integers(-8, 9, batch * n * K).astype(np.float32) for n in (M, N))
    bv = rng.integers(-8, 9, N).astype(np.float32)
    dp.write(A, a)
    dp.write(B, b)
    dp.write(bias, bv)
    dp.launch(kern)
    dp.check_faults()
    got = dp.read(C).astype(np.float64)
    dp.close()
    want = contraction_reference(a, b, None, bv, M, N, K, batch, ta, tb, True, False, 1.0, False, False)
    assert np.array_equal(got.reshape(want.shape), want)

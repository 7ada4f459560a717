"""The resident tensor-core template on both sides of the chain length from which its correction terms run on bf16 operands,
and with operand values at the ends of f32's range."""
import os

import numpy as np
import pytest

from anvil_lang_b200.program import DeviceProgram
from kirbuild import contraction_program, contraction_reference

pytestmark = pytest.mark.gpu

CASES = [        # M, N, K, batch, ta, tb
    (256, 256, 508, 1, False, False),      # a chain of 512 with a ragged end: the shortest that is mixed
    (256, 256, 480, 1, True, True),        # the longest that keeps three TF32 products
    (256, 256, 512, 1, True, False),       # both operands read along their rows: 16-byte bf16 stores
    (300, 264, 516, 1, False, True),       # both read along k: 8-byte stores; ragged tiles and a ragged last k block
    (512, 128, 1000, 2, False, False),
    (256, 64, 2048, 3, True, True),        # 32 operand rows per CTA
    (2304, 1024, 544, 1, False, False),    # more than one tile per cluster: stage ring and accumulators run on
]


def run(case, a, b):
    os.environ["ANVIL_B200_TC"] = "pp"
    try:
        prog, kern, A, B, C, _ = contraction_program(*case)
        dp = DeviceProgram(prog, graphs=False)
    finally:
        os.environ.pop("ANVIL_B200_TC", None)
    assert "pp" in dp.gen.kernel_notes[0]
    dp.write(A, a)
    dp.write(B, b)
    out = []
    for _ in range(2):
        dp.launch(kern)
        dp.check_faults()
        out.append(dp.read(C).copy())
    dp.close()
    assert np.array_equal(out[0], out[1], equal_nan=True)                    # the same bits every time
    return out[0].astype(np.float64)


@pytest.mark.parametrize("case", CASES, ids=lambda c: "x".join(map(str, c[:4])) + "ta" * c[4] + "tb" * c[5])
def test_chain_lengths(case):
    """Every accumulate truncates at 2^-23 of the running sum, K / 8 + 2 K / 16 of them: 1e-5 up to K = 1024, twice that beyond."""
    M, N, K, batch, ta, tb = case
    rng = np.random.default_rng(K)
    a, b = rng.standard_normal(batch * M * K, dtype=np.float32), rng.standard_normal(batch * K * N, dtype=np.float32)
    want = contraction_reference(a, b, None, None, M, N, K, batch, ta, tb, False, False, 1.0, False, False)
    got = run(case, a, b).reshape(want.shape)
    assert np.abs(got - want).max() / np.abs(want).max() < (1e-5 if K <= 1024 else 2e-5)


def test_range_of_the_operands():
    M, N, K = 256, 256, 512
    rng = np.random.default_rng(5)
    a, b = rng.standard_normal((M, K), dtype=np.float32), rng.standard_normal((K, N), dtype=np.float32)
    a[0] *= np.float32(1e-30)
    a[1] *= np.float32(1e30)
    a[2, 7] = np.float32(3.4028235e38)                   # rounds up to an infinity in TF32 and in bf16
    a[3, 7] = np.float32(-3.4028235e38)
    b[7] *= np.float32(1e-3)
    a[4, 9] = np.inf
    a[5, 9] = np.nan
    a[6] = 0.0
    with np.errstate(all="ignore"):
        want = a.astype(np.float64) @ b.astype(np.float64)
        got = run((M, N, K, 1, False, False), a, b)[:M * N].reshape(M, N)
    rows = [i for i in range(M) if i not in (4, 5, 6)]
    scale = np.abs(want[rows]).max(axis=1, keepdims=True)
    assert np.isfinite(got[rows]).all()
    # rows 2, 3: the part of the largest f32 above the largest bf16 is a lo term of 2^-8 kept to 8 bits: 2^-17
    bound = np.where(np.isin(rows, (2, 3)), 2.0 ** -16, 1e-5)[:, None]
    assert (np.abs(got[rows] - want[rows]) <= bound * scale).all()
    assert not np.isfinite(got[4]).any() and np.isnan(got[5]).all() and not got[6].any()

"""Fused row groups of any width: the slots of a row's threads cover it exactly (CPU), and softmax and layer norm over
widths at the edges of the layouts agree with float64 (GPU)."""
import numpy as np
import pytest

from anvil_lang_b200 import kir
from anvil_lang_b200.backend import emit
from anvil_lang_b200.backend import rowgroup as rg
from kirbuild import E, F32, Affine, Kernel, KernelStmt, Reduction, Store, binop, buf, const, load, nid, var

# the shortest row, both sides of each thread count's reach, odd and even remainders of 4 and of 32, the widest row
WIDTHS = [5, 10, 16, 17, 33, 64, 65, 100, 127, 130, 462, 511, 513, 516, 1000, 2107, 4095, 4097, 4100, 8191, 8192]
ROWS = 67                                                # more than one CTA at every layout, the last one partly empty


def slots(lay, t):
    return [(i * lay.T + t if lay.cyclic else (i // 4 * lay.T + t) * 4 + i % 4) for i in range(lay.E)]


@pytest.mark.parametrize("N", WIDTHS + [128, 384, 512, 768, 1024, 2048, 4096])
def test_slots_cover_a_row_once(N):
    lay = rg.row_layout(N)
    held = sorted(j for t in range(lay.T) for j in slots(lay, t))
    assert held[:N] == list(range(N)) and (held == list(range(N))) == (not lay.masked)
    assert lay.E <= 16 and lay.T <= 512 and (lay.cyclic or lay.E % 4 == 0)


def test_rows_that_do_not_fit_are_left_alone():
    assert rg.row_layout(8193) is None and rg.row_layout(4) is None
    assert rg.row_layout(512) == rg.RowLayout(32, 16, False, False)          # what filled its threads before still does


def un(op, a):
    return E("un", F32, op=op, a=[a])


def kernel(domain, store_buf, terms, value, red=None):
    return Kernel(nid(), f"k{nid()}", "row", domain, [Store(store_buf, Affine(0, terms), value, False)], red)


def softmax_kernels(x, y, R, N):
    m, e, s = buf("m", (R,)), buf("e", (R, N)), buf("s", (R,))
    r, j = var("r", R), var("j", N)
    ks = [kernel([r], m, [(r, 1)], E("acc", F32), Reduction([j], "max", load(x, [(r, N), (j, 1)])))]
    r2, j2 = var("r", R), var("j", N)
    ks.append(kernel([r2, j2], e, [(r2, N), (j2, 1)], un("exp", binop("sub", load(x, [(r2, N), (j2, 1)]), load(m, [(r2, 1)])))))
    r3, j3 = var("r", R), var("j", N)
    ks.append(kernel([r3], s, [(r3, 1)], E("acc", F32), Reduction([j3], "sum", load(e, [(r3, N), (j3, 1)]))))
    r4, j4 = var("r", R), var("j", N)
    ks.append(kernel([r4, j4], y, [(r4, N), (j4, 1)], binop("div", load(e, [(r4, N), (j4, 1)]), load(s, [(r4, 1)]))))
    return ks, [m, e, s]


def norm_kernels(x, g, y, R, N):
    mu, v = buf("mu", (R,)), buf("v", (R,))
    r, j = var("r", R), var("j", N)
    ks = [kernel([r], mu, [(r, 1)], E("acc", F32), Reduction([j], "sum", binop("mul", const(np.float32(1 / N)), load(x, [(r, N), (j, 1)]))))]
    r2, j2 = var("r", R), var("j", N)
    d = binop("sub", load(x, [(r2, N), (j2, 1)]), load(mu, [(r2, 1)]))
    ks.append(kernel([r2], v, [(r2, 1)], E("acc", F32), Reduction([j2], "sum", binop("mul", const(np.float32(1 / N)), binop("mul", d, d)))))
    r3, j3 = var("r", R), var("j", N)
    d = binop("sub", load(x, [(r3, N), (j3, 1)]), load(mu, [(r3, 1)]))
    n = binop("div", d, un("sqrt", binop("add", load(v, [(r3, 1)]), const(1e-5))))
    ks.append(kernel([r3, j3], y, [(r3, N), (j3, 1)], binop("mul", n, load(g, [(j3, 1)]))))
    return ks, [mu, v]


def program(widths):
    kernels, bufs, io = [], [], []
    for N in widths:
        x, g = buf(f"x{N}", (ROWS, N), kind="input"), buf(f"g{N}", (N,), kind="input")
        y, z = buf(f"y{N}", (ROWS, N), kind="output"), buf(f"z{N}", (ROWS, N), kind="output")
        a, ta = softmax_kernels(x, y, ROWS, N)
        b, tb = norm_kernels(x, g, z, ROWS, N)
        kernels += a + b
        bufs += [x, g, y, z] + ta + tb
        io.append((N, x, g, y, z))
    return kir.Program(kir.Block([KernelStmt(k) for k in kernels]), bufs, "row widths"), io


def test_every_width_is_one_launch_per_run():
    prog, _ = program([10, 2107, 8192])
    src, _ = emit.generate(prog, 0)
    assert src.count("// fused row group:") == 3          # softmax and layer norm of one width join one run
    assert src.count("(masked)") == 2                  # 8192 fills its 512 x 16 slots


@pytest.mark.gpu
def test_widths_against_float64():
    """f32 sums in a fixed tree of at most 16 + 9 levels, an exp of 2 ulp and a divide: 1e-6 of a softmax value, 4e-6 of the
    unit-scale layer norm. Rows of infinities, of the type's lowest value and with a nan behave as the plain formula does."""
    from anvil_lang_b200.program import DeviceProgram
    prog, io = program(WIDTHS)
    dp = DeviceProgram(prog, seed=0, graphs=False)
    rng = np.random.default_rng(11)
    data = {}
    for N, x, g, y, z in io:
        a = (3.0 * rng.standard_normal((ROWS, N))).astype(np.float32)
        a[1, N - 1] = 40.0                                # the maximum in the last, partly masked group
        a[2, :-1] = -3.4028235e38                         # all but one element at the mask value
        a[3, 0] = -np.inf
        a[4, N // 2] = np.nan
        data[N] = (a, rng.standard_normal(N).astype(np.float32))
        dp.write(x, a)
        dp.write(g, data[N][1])
    code, _ = dp.run()
    assert code == 0, dp.error
    with np.errstate(all="ignore"):
        for N, x, g, y, z in io:
            a = data[N][0].astype(np.float64)
            e = np.exp(a - a.max(axis=1, keepdims=True))
            want = e / e.sum(axis=1, keepdims=True)
            got = dp.read(y).reshape(ROWS, N)
            assert np.array_equal(np.isnan(got), np.isnan(want)), N
            assert np.nanmax(np.abs(got - want) / np.maximum(want, 1e-30) * (want > 1e-30)) < 1e-5, N
            plain = [i for i in range(ROWS) if i not in (2, 3, 4)]
            d = a[plain] - a[plain].mean(axis=1, keepdims=True)
            want = d / np.sqrt((d * d).mean(axis=1, keepdims=True) + 1e-5) * data[N][1]
            got = dp.read(z).reshape(ROWS, N)[plain]
            assert np.abs(got - want).max() < 4e-6 * max(1.0, np.abs(want).max()), N
    dp.close()

"""GPU parity of the fp32 (FFMA) GEMM against NumPy: relative Frobenius error <= 1e-5."""
import numpy as np
import pytest

from oracle import spiral_oracle as so

pytestmark = pytest.mark.gpu
TOL_F32 = 1e-5


def _operands(seed, at, bt, m, n, k, dist="uniform"):
    g = so.rng(seed)
    draw = (lambda s: g.uniform(-1, 1, size=s)) if dist == "uniform" else (lambda s: g.normal(size=s))
    a = draw((k, m) if at else (m, k)).astype(np.float32)
    b = draw((n, k) if bt else (k, n)).astype(np.float32)
    c = draw((m, n)).astype(np.float32)
    return a, b, c


def test_config_512_nt_fp32(gpu):
    """Benchmark configuration 1: C = A @ B.T, 512^3, uniform[-1,1), seed 1, NumPy float32 oracle."""
    a, b, c = _operands(1, False, True, 512, 512, 512)
    dc = gpu.DeviceArray((512, 512), "f32")
    gpu.matmul(False, True, 1.0, gpu.DeviceArray.from_numpy(a), gpu.DeviceArray.from_numpy(b), 0.0, dc,
               in_dtype="f32")
    got = dc.numpy()
    assert so.rel_frobenius(got, a @ b.T) <= TOL_F32
    assert so.rel_frobenius(got, so.matmul(False, True, 1.0, a, b, 0.0, None)) <= TOL_F32


@pytest.mark.parametrize("at,bt", [(False, False), (False, True), (True, False), (True, True)])
@pytest.mark.parametrize("m,n,k", [(1, 1, 1), (65, 63, 17), (200, 130, 333)])
def test_layouts_and_ragged_shapes(gpu, at, bt, m, n, k):
    a, b, c = _operands(m * 7 + n + k, at, bt, m, n, k, "normal")
    dc = gpu.DeviceArray.from_numpy(c)
    gpu.matmul(at, bt, 1.5, gpu.DeviceArray.from_numpy(a), gpu.DeviceArray.from_numpy(b), -0.5, dc, in_dtype="f32")
    assert so.rel_frobenius(dc.numpy(), so.matmul(at, bt, 1.5, a, b, -0.5, c)) <= TOL_F32


@pytest.mark.parametrize("at,bt", [(False, False), (False, True), (True, False), (True, True)])
@pytest.mark.parametrize("m,n,k", [(256, 192, 320), (512, 512, 512), (1000, 520, 260), (4, 4, 4)])
def test_fp32_class_on_tensor_cores_all_layouts(gpu, at, bt, m, n, k):
    """Shapes whose contiguous dimensions are multiples of 4 take the 3 x TF32 tensor-core path (operands split
    into TF32 head and tail, one GEMM of their three products): still within 1e-5 of the float64 product."""
    a, b, c = _operands(900 + m + n + k, at, bt, m, n, k, "normal")
    dc = gpu.DeviceArray.from_numpy(c)
    l0 = gpu.launch_count()
    gpu.matmul(at, bt, 1.5, gpu.DeviceArray.from_numpy(a), gpu.DeviceArray.from_numpy(b), -0.5, dc, in_dtype="f32")
    assert gpu.launch_count() - l0 == 2                      # the split and the GEMM
    assert so.rel_frobenius(dc.numpy(), so.matmul(at, bt, 1.5, a, b, -0.5, c)) <= TOL_F32


def test_fp32_class_bias_relu_and_4096_sampled_rows(gpu):
    g = so.rng(77)
    a = g.uniform(-1, 1, size=(300, 264)).astype(np.float32)
    b = g.uniform(-1, 1, size=(128, 264)).astype(np.float32)
    bias = g.normal(size=128).astype(np.float32)
    dc = gpu.DeviceArray((300, 128), "f32")
    gpu.matmul(False, True, 1.0, gpu.DeviceArray.from_numpy(a), gpu.DeviceArray.from_numpy(b), 0.0, dc, in_dtype="f32",
               epilogue=("bias", "relu"), bias=gpu.DeviceArray.from_numpy(bias))
    assert so.rel_frobenius(dc.numpy(), so.relu(so.matmul(False, True, 1.0, a, b, 0.0, None) + bias)) <= TOL_F32
    # a large case: 4096^3, oracle on 32 sampled rows; far tighter than single-pass TF32 (about 5e-4)
    a = g.standard_normal((4096, 4096), dtype=np.float32)
    b = g.standard_normal((4096, 4096), dtype=np.float32)
    dc = gpu.DeviceArray((4096, 4096), "f32")
    gpu.matmul(False, True, 1.0, gpu.DeviceArray.from_numpy(a), gpu.DeviceArray.from_numpy(b), 0.0, dc, in_dtype="f32")
    rows = g.choice(4096, size=32, replace=False)
    err = so.rel_frobenius(dc.numpy()[rows], so.matmul(False, True, 1.0, a[rows], b, 0.0, None))
    assert err <= TOL_F32


@pytest.mark.parametrize("at,bt", [(False, True), (False, False), (True, False), (True, True)])
@pytest.mark.parametrize("m,n,k", [(132, 68, 4), (260, 300, 28), (260, 256, 32), (516, 260, 36), (128, 64, 64), (300, 192, 68),
                                   (260, 68, 100), (5120, 1024, 160), (5000, 1020, 96)])
def test_fp32_class_short_chains(gpu, at, bt, m, n, k):
    """One, two and more stages of 32 elements of K with their three products, the last one ragged; single tiles and,
    with 80 tiles for 74 pairs, half-width ones in the last wave.  A chain this short is off by 1.1e-6 (160 elements)."""
    a, b, c = _operands(40 + m + n + k, at, bt, m, n, k, "normal")
    dc = gpu.DeviceArray.from_numpy(c)
    gpu.matmul(at, bt, 1.5, gpu.DeviceArray.from_numpy(a), gpu.DeviceArray.from_numpy(b), -0.5, dc, in_dtype="f32")
    assert so.rel_frobenius(dc.numpy(), so.matmul(at, bt, 1.5, a, b, -0.5, c)) <= 3e-6


@pytest.mark.parametrize("at,bt,shift_a,shift_b", [(False, True, 1, 0), (True, False, 0, 3), (False, False, 2, 1)])
def test_fp32_class_takes_operands_off_the_16_byte_grid(gpu, at, bt, shift_a, shift_b):
    """The split kernel reads an operand that is only 4-byte aligned element by element: the same bits as the
    aligned operand gives (same arithmetic), including the sums' order when there is no split along K."""
    m, n, k = 132, 68, 36
    a, b, _ = _operands(5, at, bt, m, n, k, "normal")

    def place(x, shift):
        flat = gpu.DeviceArray.from_numpy(np.concatenate([np.zeros(shift, np.float32), x.ravel()]))
        return flat.view(x.shape, "f32", 4 * shift)

    out = []
    for sa, sb in ((0, 0), (shift_a, shift_b)):
        dc = gpu.DeviceArray((m, n), "f32")
        gpu.matmul(at, bt, 1.0, place(a, sa), place(b, sb), 0.0, dc, in_dtype="f32")
        out.append(dc.numpy())
    np.testing.assert_array_equal(out[0], out[1])
    assert so.rel_frobenius(out[0], so.matmul(at, bt, 1.0, a, b, 0.0, None)) <= TOL_F32


@pytest.mark.parametrize("at,bt,m,n,k,epilogue,beta", [
    (False, True, 129, 20, 2048, (), 0.0), (False, True, 300, 252, 2048, (), -0.5), (True, False, 128, 1020, 2048, (), 0.0),
    (False, False, 260, 36, 4096, (), 1.0), (True, True, 64, 4, 4096, (), 0.0), (False, True, 1, 36, 2048, (), -0.5),
    (False, True, 300, 128, 2048, ("bias",), 1.0), (False, False, 129, 100, 2048, ("bias",), -0.5),
    (False, True, 300, 128, 2048, ("relu",), 0.0), (True, False, 132, 252, 2048, ("bias", "relu"), 0.0),
    (False, True, 70, 256, 4096, ("bias", "relu"), -0.5), (False, True, 257, 68, 260, ("bias", "relu"), 0.0),
    (False, True, 64, 96, 256, ("bias", "relu"), 0.0), (False, True, 64, 68, 176, ("bias",), 1.0)])
@pytest.mark.parametrize("dist", ["normal", "positive"])
def test_fp32_class_holds_for_long_k_ragged_n_and_epilogues(gpu, at, bt, m, n, k, epilogue, beta, dist):
    """The chains of accumulations that the tensor core makes are cut whatever the width of C and the epilogue: a
    single chain is off by 1.1e-5 (normal) and 1.5e-5 (positive operands) at K = 1024, more in proportion beyond."""
    g = so.rng(m + n + k)
    draw = (lambda s: g.uniform(0, 1, size=s)) if dist == "positive" else (lambda s: g.normal(size=s))
    a, b = draw((k, m) if at else (m, k)).astype(np.float32), draw((n, k) if bt else (k, n)).astype(np.float32)
    c, bias = g.normal(size=(m, n)).astype(np.float32), g.normal(size=n).astype(np.float32)
    want = so.matmul(at, bt, 1.5, a, b, beta, c)
    if beta == 0:
        c[:] = np.nan                                        # not read
    if "bias" in epilogue:
        want = want + bias
    if "relu" in epilogue:
        want = so.relu(want)
    dc = gpu.DeviceArray.from_numpy(c)
    gpu.matmul(at, bt, 1.5, gpu.DeviceArray.from_numpy(a), gpu.DeviceArray.from_numpy(b), beta, dc, in_dtype="f32",
               epilogue=epilogue, bias=gpu.DeviceArray.from_numpy(bias) if "bias" in epilogue else None)
    assert so.rel_frobenius(dc.numpy(), want) <= TOL_F32


@pytest.mark.parametrize("n,epilogue", [(64, ()), (36, ("bias", "relu"))])
def test_fp32_class_holds_for_very_long_k(gpu, n, epilogue):
    """K = 200000: 782 parts."""
    m, k = 64, 200000
    g = so.rng(8)
    a, b = g.uniform(0, 1, size=(m, k)).astype(np.float32), g.uniform(0, 1, size=(n, k)).astype(np.float32)
    bias = g.normal(size=n).astype(np.float32)
    want = so.matmul(False, True, 1.0, a, b, 0.0, None)
    if epilogue:
        want = so.relu(want + bias)
    dc = gpu.DeviceArray((m, n), "f32")
    gpu.matmul(False, True, 1.0, gpu.DeviceArray.from_numpy(a), gpu.DeviceArray.from_numpy(b), 0.0, dc, in_dtype="f32",
               epilogue=epilogue, bias=gpu.DeviceArray.from_numpy(bias) if epilogue else None)
    assert so.rel_frobenius(dc.numpy(), want) <= TOL_F32


@pytest.mark.parametrize("shift", [0, 16, 200])
@pytest.mark.parametrize("m,n,k", [(4, 4, 4), (132, 68, 20), (260, 300, 1028)])
def test_fp32_class_stays_inside_the_workspace_that_it_asks_for(gpu, m, n, k, shift):
    """Two parts per operand and the slack of their alignment, wherever the workspace starts; what lies around a
    workspace of exactly that size stays as it was."""
    import ctypes
    from spiral_b200 import _lib
    need = ctypes.c_size_t()
    _lib.call("sb_matmul_f32_workspace_bytes", m, n, k, ctypes.byref(need))
    assert need.value <= 8 * (m + n) * k + 1024
    a, b, c = _operands(60 + m, False, True, m, n, k, "normal")
    da, db, dc = (gpu.DeviceArray.from_numpy(v) for v in (a, b, c))
    guard = np.full(shift + need.value + 512, 0xA5, np.uint8)
    ws = gpu.DeviceArray.from_numpy(guard)
    _lib.call("sb_matmul_f32x3", 0, 1, 1.0, da.ptr, db.ptr, 0.0, dc.ptr, m, n, k, 0, None, ws.ptr + shift, need.value, None)
    assert so.rel_frobenius(dc.numpy(), so.matmul(False, True, 1.0, a, b, 0.0, None)) <= TOL_F32
    after = ws.numpy()
    assert np.all(after[:shift] == 0xA5) and np.all(after[shift + need.value:] == 0xA5)


@pytest.mark.parametrize("at,bt", [(False, True), (False, False), (True, False)])
@pytest.mark.parametrize("m,n,k,beta", [(100, 56, 64, 1.0), (468, 56, 144, 1.0), (468, 56, 144, 0.0), (64, 1000, 300, 0.5), (300, 256, 1000, 0.0),
                                        (1000, 520, 160, -0.5)])
def test_fp32_class_on_narrow_tiles(gpu, at, bt, m, n, k, beta):
    """Few tiles in the fp32 class: narrow ones with one chain of K or several, and a C of less than 64 columns that is
    read, which keeps one tile."""
    a, b, c = _operands(80 + m + n, at, bt, m, n, k, "normal")
    dc = gpu.DeviceArray.from_numpy(c)
    gpu.matmul(at, bt, 1.0, gpu.DeviceArray.from_numpy(a), gpu.DeviceArray.from_numpy(b), beta, dc, in_dtype="f32")
    assert so.rel_frobenius(dc.numpy(), so.matmul(at, bt, 1.0, a, b, beta, c)) <= TOL_F32


@pytest.mark.parametrize("at,bt", [(False, True), (False, False), (True, False)])
@pytest.mark.parametrize("m,n,k", [(100, 252, 300), (128, 256, 64), (64, 1000, 512), (300, 256, 300)])
def test_fp32_class_beside_a_shared_memory_reserve(gpu, at, bt, m, n, k):
    """Two stages of a single CTA's 256-column tile take all of the pipeline's memory: with 64 KB reserved its tiles are
    narrower (pairs keep theirs), and the product is the same within the class."""
    from spiral_b200 import _lib
    a, b, c = _operands(70 + n, at, bt, m, n, k, "normal")
    da, db, dc = (gpu.DeviceArray.from_numpy(v) for v in (a, b, c))
    _lib.call("sb_gemm_reserve_smem", 65536)
    try:
        gpu.matmul(at, bt, 1.0, da, db, 0.5, dc, in_dtype="f32")
    finally:
        _lib.call("sb_gemm_reserve_smem", 0)
    assert so.rel_frobenius(dc.numpy(), so.matmul(at, bt, 1.0, a, b, 0.5, c)) <= TOL_F32

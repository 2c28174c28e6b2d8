"""The C-ABI library loads without a GPU and exports every symbol the header declares (CPU only)."""
import ctypes
import os
import re

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
HEADER = os.path.join(ROOT, "include", "spiral_b200.h")


def declared_symbols():
    text = open(HEADER).read()
    text = re.sub(r"/\*.*?\*/", "", text, flags=re.S)
    return sorted(set(re.findall(r"\b(sb_[a-z0-9_]+)\s*\(", text)))


def test_header_declares_entry_points():
    names = declared_symbols()
    assert "sb_matmul_tf32" in names and "sb_matmul_ex" in names
    assert len(names) >= 25


def test_library_exports_every_declared_symbol(sb):
    lib = ctypes.CDLL(sb.LIB_PATH)
    missing = [n for n in declared_symbols() if not hasattr(lib, n)]
    assert not missing, "declared in include/spiral_b200.h but not exported: %s" % missing


def test_binding_table_covers_header(sb):
    from spiral_b200 import _lib
    assert sorted(_lib.SIGNATURES) == declared_symbols()


def test_plan_needs_no_device(sb):
    plan = sb.matmul_plan(False, True, 4096, 4096, 4096, "bf16")
    assert plan["block_m"] in (128, 256) and plan["block_n"] % 16 == 0 and plan["grid"] <= 148
    assert plan["block_k"] in (64, 128) and plan["stages"] >= 2      # one or two 128-byte sub-blocks per stage
    if plan["block_m"] == 256:          # CTA pairs: an even grid, each CTA stages half of the B columns
        assert plan["grid"] % 2 == 0 and plan["block_n"] % 32 == 0
    plan = sb.matmul_plan(False, False, 4000, 3000, 1000, "tf32")
    assert plan["block_k"] in (32, 64) and plan["block_n"] % 32 == 0
    small = sb.matmul_plan(False, True, 16384, 3, 256, "tf32")
    assert small["block_n"] == 16 and small["grid"] == 128 and small["block_m"] == 128


@pytest.mark.parametrize("epilogue,m,n,k,in_dtype,want", [
    (("ln_l2", "relu"), 512, 256, 128, "tf32", (256, 256, 4)),              # the tile spans the row, however few there are
    (("ln_l2",), 300, 256, 128, "bf16", (256, 256, 4)),
    (("masked_softmax", "argmax"), 512, 64, 128, "bf16", (128, 64, 4)),     # a row head: single CTAs, whole rows
    (("regret_matching",), 512, 256, 128, "bf16", (256, 64, 16)),           # a head beyond 64 columns runs behind a plain product
    (("bias", "relu"), 512, 256, 128, "bf16", (256, 64, 16)),
    (("bias", "relu", "relu_mask_out"), 128, 96, 128, "bf16", (128, 32, 3)),
    ((), 512, 256, 128, "tf32", (256, 64, 16))])
def test_plan_is_that_of_the_launch_with_its_epilogue(sb, epilogue, m, n, k, in_dtype, want):
    plan = sb.matmul_plan(False, True, m, n, k, in_dtype, epilogue=epilogue)
    assert (plan["block_m"], plan["block_n"], plan["grid"]) == want


@pytest.mark.parametrize("in_dtype,m,n,k,block_n", [
    ("bf16", 9472, 96, 1024, 96), ("bf16", 9472, 128, 1024, 128), ("tf32", 6144, 96, 1024, 96), ("bf16", 6400, 64, 64, 64),
    ("bf16", 7424, 128, 1024, 64), ("bf16", 7680, 128, 1024, 128),        # 29 and 30 of 74 pairs
    ("bf16", 5632, 96, 1024, 64), ("bf16", 5888, 96, 1024, 96),           # 22 and 23
    ("bf16", 9472, 256, 1024, 128), ("bf16", 9472, 160, 256, 160), ("bf16", 9472, 192, 1024, 128), ("bf16", 1280, 160, 256, 64),
    ("bf16", 6144, 48, 256, 32), ("bf16", 18944, 256, 1024, 256)])
def test_tiles_that_occupy_the_chip_stay_whole(sb, in_dtype, m, n, k, block_n):
    assert sb.matmul_plan(False, True, m, n, k, in_dtype)["block_n"] == block_n


def test_padded_narrow_tiles_with_column_sums(sb):
    for epilogue, block_n in ((("relu", "relu_mask_out"), 64), (("relu_grad_mask",), 64), (("relu_grad_mask", "colsum_out"), 96)):
        assert sb.matmul_plan(False, True, 3072, 96, 256, "bf16", epilogue=epilogue)["block_n"] == block_n


@pytest.mark.parametrize("m,n,epilogue,block_n", [
    (9000, 99, (), 64), (9000, 96, (), 96),                                       # rows of C that are no whole 16-byte pieces, and that are
    (9000, 33, (), 48), (2000, 33, (), 32), (9000, 131, (), 160), (9000, 61, (), 32),
    (9000, 72, ("relu_grad",), 64), (9000, 72, (), 96), (9000, 40, ("relu_grad",), 48), (2000, 40, ("relu_grad",), 32)])
def test_tiles_whose_chunks_leave_from_registers(sb, m, n, epilogue, block_n):
    assert sb.matmul_plan(False, True, m, n, 400, "bf16", epilogue=epilogue)["block_n"] == block_n


def test_bad_arguments_are_rejected_before_any_launch(sb):
    from spiral_b200 import _lib
    with pytest.raises(sb.SpiralError) as e:
        _lib.call("sb_matmul_tf32", 0, 1, ctypes.c_float(1), None, None, ctypes.c_float(0), None, 4, 4, 4, None)
    assert e.value.code == -1
    with pytest.raises(sb.SpiralError):
        _lib.call("sb_matmul_tf32", 0, 1, ctypes.c_float(1), 16, 16, ctypes.c_float(0), 16, -1, 4, 4, None)
    # zero-sized outputs are a no-op, not an error
    _lib.call("sb_matmul_tf32", 0, 1, ctypes.c_float(1), None, None, ctypes.c_float(0), None, 0, 4, 4, None)


def test_shape_inference_follows_the_reference(sb):
    class Fake:
        def __init__(self, shape):
            self.shape, self.dtype = shape, "float32"
    from spiral_b200.matmul import _dims
    assert _dims(False, True, Fake((8, 5)), Fake((3, 5)), Fake((8, 3))) == (8, 3, 5)
    assert _dims(True, False, Fake((5, 8)), Fake((5, 3)), Fake((8, 3))) == (8, 3, 5)
    with pytest.raises(ValueError):
        _dims(False, False, Fake((8, 5)), Fake((3, 5)), Fake((8, 3)))

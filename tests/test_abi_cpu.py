"""CPU-only checks of the drop-in boundary: the C-ABI library builds, loads and
exports every symbol the header declares, and the host-side validation raises
the reference's error texts before anything touches a device."""

import ctypes
import os
import re

import pytest
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def native():
    from halops_b200 import build

    build.build()
    from halops_b200 import _native

    _native.lib()
    return _native


def _declared_functions():
    text = open(os.path.join(ROOT, "include", "halops_b200.h")).read()
    text = re.sub(r"/\*.*?\*/", "", text, flags=re.S)
    return sorted(set(re.findall(r"\b(hq_[a-z_0-9]+)\s*\(", text)))


def test_library_exports_every_declared_symbol(native):
    names = _declared_functions()
    assert "hq_group_wise_quant" in names and "hq_dense_gemm" in names
    handle = ctypes.CDLL(native.lib_path())
    for name in names:
        assert getattr(handle, name) is not None
    assert sorted(native.SIGNATURES) == names, "ctypes table and header disagree"
    assert b"sm_100a" in native.lib().hq_version()


def test_no_torch_types_in_the_header():
    text = open(os.path.join(ROOT, "include", "halops_b200.h")).read()
    assert "torch" not in text.replace("TORCH_CHECK", "") and "at::" not in text


def test_mode_helpers(native):
    lib = native.lib()
    assert lib.hq_parse_mode(b"w8a8-mxfp8") == 0
    assert lib.hq_parse_mode(b"w4a4-mxfp4") == 1
    assert lib.hq_parse_mode(b"w4a4-nvfp4") == 2
    assert lib.hq_parse_mode(b"nvfp4") == -1
    assert [lib.hq_group_size(i) for i in range(4)] == [32, 32, 16, 0]
    assert [lib.hq_sf_rows(m) for m in (0, 1, 128, 129, 1000)] == [0, 128, 128, 256, 1024]


def _gemm_rc(native, m, n, k, mode, alpha=None, epilogue=0):
    err = ctypes.create_string_buffer(512)
    rc = native.lib().hq_dense_gemm(None, None, None, None, None, None, alpha, m, n, k, 1 << 40, 1 << 40, n,
                                    mode, epilogue, -1, 0, 0, None, err, len(err))
    return rc, err.value.decode()


@pytest.mark.parametrize("mode, m, n, k, text", [
    (0, 128, 256, 96, "No dense w8a8-mxfp8 tile for M=128 (grid M=128), N=256, K=96"),
    (0, 128, 255, 128, "No dense w8a8-mxfp8 tile for M=128 (grid M=128), N=255, K=128"),
    (2, 128, 256, 48, "No dense w4a4-nvfp4 tile for M=128 (grid M=128), N=256, K=48"),
    (0, 200, 100, 128, "No dense w8a8-mxfp8 tile for M=256 (grid M=256), N=100, K=128"),
])
def test_shape_legality_messages(native, mode, m, n, k, text):
    """Texts pinned by the reference's tests/test_dense_gemm.py:398-492."""
    alpha = ctypes.cast(16, ctypes.c_void_p) if mode == 2 else None
    rc, msg = _gemm_rc(native, m, n, k, mode, alpha)
    assert rc == 1 and text in msg


def test_gemm_argument_rules(native):
    rc, msg = _gemm_rc(native, 128, 256, 512, 1, alpha=ctypes.cast(16, ctypes.c_void_p))
    assert rc == 1 and "does not take alpha" in msg
    rc, msg = _gemm_rc(native, 128, 256, 512, 2, alpha=None)
    assert rc == 1 and "requires alpha" in msg
    rc, msg = _gemm_rc(native, 128, 256, 512, 0, epilogue=4)
    assert rc == 3 and "Unsupported epilogue" in msg
    rc, msg = _gemm_rc(native, 128, 256, 512, 7)
    assert rc == 1 and "Unsupported mode" in msg
    assert _gemm_rc(native, 0, 256, 512, 0)[0] == 0  # empty problem: nothing to do


def test_quant_argument_rules(native):
    err = ctypes.create_string_buffer(512)
    f = native.lib().hq_group_wise_quant
    assert f(None, 96, 0, 128, 96, 0, 1, 0, None, None, 0, None, err, len(err)) == 1
    assert b"scale kb_dim must be divisible by 4" in err.value
    assert f(None, 100, 0, 128, 100, 0, 0, 0, None, None, 0, None, err, len(err)) == 1
    assert b"k must be divisible by the quantization group size (32)" in err.value
    assert f(None, 1024, 0, 128, 1024, 9, 1, 0, None, None, 0, None, err, len(err)) == 1
    assert b"Unsupported quantization mode" in err.value
    assert f(None, 1024, 5, 128, 1024, 0, 1, 0, None, None, 0, None, err, len(err)) == 1
    assert b"bfloat16 or float16" in err.value
    assert f(None, 1024, 0, 0, 1024, 0, 1, 0, None, None, 0, None, err, len(err)) == 0  # m = 0


def test_python_wrapper_errors_without_a_device():
    import halops_b200 as hq

    x = torch.zeros([128, 1024], dtype=torch.bfloat16)
    with pytest.raises(RuntimeError, match=re.escape("Unsupported quantization mode")):
        hq.group_wise_quant(x, mode="w4a4-fp6")
    with pytest.raises(RuntimeError, match=re.escape("scale kb_dim must be divisible by 4")):
        hq.group_wise_quant(torch.zeros([128, 96], dtype=torch.bfloat16))
    with pytest.raises(RuntimeError, match="no CPU path"):
        hq.group_wise_quant(x)

    def empties(m, n, k, mode, x_shape=None, out_shape=None):
        if mode == "w8a8-mxfp8":
            a = torch.empty(x_shape or [m, k], dtype=torch.float8_e4m3fn)
            w = torch.empty([n, k], dtype=torch.float8_e4m3fn)
            sfa, sfb = torch.empty([m, k // 32], dtype=torch.uint8), torch.empty([n, k // 32], dtype=torch.uint8)
            alpha = None
        else:
            a = torch.empty(x_shape or [m, k // 2], dtype=torch.uint8)
            w = torch.empty([n, k // 2], dtype=torch.uint8)
            g = 16 if mode == "w4a4-nvfp4" else 32
            sfa, sfb = torch.empty([m, k // g], dtype=torch.uint8), torch.empty([n, k // g], dtype=torch.uint8)
            alpha = torch.ones([1]) if mode == "w4a4-nvfp4" else None
        return a, w, sfa, sfb, torch.empty(out_shape or [m, n], dtype=torch.bfloat16), alpha

    cases = [
        ("w8a8-mxfp8", 128, 256, 96, None, None, "No dense w8a8-mxfp8 tile for M=128 (grid M=128), N=256, K=96"),
        ("w8a8-mxfp8", 128, 255, 128, None, None, "No dense w8a8-mxfp8 tile for M=128 (grid M=128), N=255, K=128"),
        ("w4a4-nvfp4", 128, 256, 48, None, None, "No dense w4a4-nvfp4 tile for M=128 (grid M=128), N=256, K=48"),
        ("w8a8-mxfp8", 128, 256, 128, [128, 1, 128], None, "input must be a 2D tensor"),
        ("w8a8-mxfp8", 128, 256, 128, None, [128, 256, 1], "output must be a 2D tensor"),
    ]
    for mode, m, n, k, xs, os_, text in cases:
        a, w, sfa, sfb, out, alpha = empties(m, n, k, mode, xs, os_)
        with pytest.raises(RuntimeError, match=re.escape(text)):
            hq.dense_gemm(a, w, sfa, sfb, out, None, alpha, -1, mode)

    a, w, sfa, sfb, out, _ = empties(128, 256, 512, "w4a4-mxfp4")
    with pytest.raises(RuntimeError, match=re.escape("does not take alpha")):
        hq.dense_gemm(a, w, sfa, sfb, out, None, torch.ones([1]), -1, "w4a4-mxfp4")
    a, w, _, _, out, _ = empties(128, 256, 512, "w4a4-mxfp4")
    bad = torch.empty([128, 32], dtype=torch.uint8), torch.empty([256, 32], dtype=torch.uint8)
    with pytest.raises(RuntimeError, match=re.escape("scale-factor shape does not match mode")):
        hq.dense_gemm(a, w, bad[0], bad[1], out, None, None, -1, "w4a4-mxfp4")
    a, w, sfa, sfb, out, _ = empties(200, 1024, 1024, "w8a8-mxfp8")
    with pytest.raises(RuntimeError, match=re.escape("multiple of 256")):
        hq.dense_gemm(a, w, torch.empty([256, 32], dtype=torch.uint8), sfb, out, torch.zeros([1024], dtype=torch.bfloat16))
    with pytest.raises(RuntimeError, match="Unsupported mode"):
        hq.dense_gemm(a, w, sfa, sfb, out, mode="nvfp4")
    with pytest.raises(RuntimeError, match="no CPU path"):
        a, w, sfa, sfb, out, _ = empties(128, 256, 512, "w8a8-mxfp8")
        hq.dense_gemm(a, w, sfa, sfb, out)


def test_batch_gemm_rules_without_a_device(native):
    """Host checks of the batch GEMM (texts of the reference's tests/test_batch_gemm.py:313-363,
    537-590) through the C entry point with null operands and through the Python wrapper."""
    import halops_b200 as hq

    def rc(batches, m, n, k, mode, alpha=None, bias=None, epilogue=0):
        err = ctypes.create_string_buffer(512)
        code = native.lib().hq_batch_gemm(None, None, None, None, None, bias, alpha, batches, m, n, k, 1 << 40,
                                          1 << 40, batches * n, mode, epilogue, -1, 0, 0, None, err, len(err))
        return code, err.value.decode()

    fake = ctypes.cast(16, ctypes.c_void_p)
    code, msg = rc(2, 128, 256, 96, 0)
    assert code == 1 and "No batch w8a8-mxfp8 tile for M=128 (grid M=256), N=256, K=96" in msg
    code, msg = rc(2, 128, 256, 256, 2)
    assert code == 1 and "requires alpha input (per-batch scaling)" in msg
    code, msg = rc(2, 128, 256, 512, 1, alpha=fake)
    assert code == 1 and "does not take alpha; the per-batch scaling factor" in msg
    code, msg = rc(2, 128, 256, 256, 2, alpha=fake, bias=fake)
    assert code == 1 and "W4A4 batch GEMM does not support bias" in msg
    code, msg = rc(2, 128, 256, 128, 0, epilogue=1)
    assert code == 3 and "Unsupported epilogue 1" in msg
    assert rc(0, 128, 256, 128, 0)[0] == 0 and rc(2, 0, 256, 128, 0)[0] == 0
    err = ctypes.create_string_buffer(512)
    assert native.lib().hq_batch_gemm(fake, fake, fake, fake, fake, None, None, 2, 100, 256, 128, 256 * 4 - 1,
                                      1 << 40, 512, 0, 0, -1, 0, 0, None, err, len(err)) == 1
    assert b"sfa must hold whole 128-row SfAtoms over the stacked rows" in err.value

    x = torch.empty([2, 128, 128], dtype=torch.float8_e4m3fn)
    w = torch.empty([2, 256, 128], dtype=torch.float8_e4m3fn)
    sfa = torch.empty([256, 4], dtype=torch.uint8)
    sfb = torch.empty([2, 256, 4], dtype=torch.uint8)
    out = torch.empty([128, 512], dtype=torch.bfloat16)
    with pytest.raises(RuntimeError, match="input must be a 3D tensor"):
        hq.batch_gemm(x[0], w, sfa, sfb, out)
    with pytest.raises(RuntimeError, match="weight batch dim must match input batch dim, got 3"):
        hq.batch_gemm(x, torch.empty([3, 256, 128], dtype=torch.float8_e4m3fn), sfa, sfb, out)
    with pytest.raises(RuntimeError, match=re.escape("output must be a 2D tensor of shape [M, B * N]")):
        hq.batch_gemm(x, w, sfa, sfb, out.view(2, 64, 512))
    with pytest.raises(RuntimeError, match=re.escape("output shape must be [M, B * N]")):
        hq.batch_gemm(x, w, sfa, sfb, out[:, :256])
    with pytest.raises(RuntimeError, match="Unsupported mode: w2a2"):
        hq.batch_gemm(x, w, sfa, sfb, out, mode="w2a2")
    with pytest.raises(RuntimeError, match="no CPU path"):
        hq.batch_gemm(x, w, sfa, sfb, out)
    assert "mode=batch" in hq.describe_group_tile("batch", 4, 200, 256, 128)


def test_group_gemm_rules_without_a_device(native):
    """Host checks of the masked / contiguous grouped GEMMs (texts of the reference's
    tests/test_group_masked_gemm.py:840-866 and tests/test_group_contiguous_gemm.py:628-652)."""
    import halops_b200 as hq

    fake = ctypes.cast(16, ctypes.c_void_p)
    err = ctypes.create_string_buffer(512)
    masked = native.lib().hq_group_masked_gemm
    contiguous = native.lib().hq_group_contiguous_gemm
    big = 1 << 40
    assert masked(None, None, None, None, None, None, None, None, 2, 129, 256, 128, big, big, 256, 0, -1, 1, 0, None,
                  err, len(err)) == 1
    assert b"No masked w8a8-mxfp8 tile for M=129 (grid M=258), N=256, K=128" in err.value
    assert masked(None, None, None, None, None, None, None, None, 2, 0, 256, 128, big, big, 256, 0, -1, 1, 0, None,
                  err, len(err)) == 1
    assert b"max_m_per_expert must be greater than 0, got 0" in err.value
    assert masked(None, None, None, None, None, None, fake, fake, 2, 128, 128, 512, big, big, 128, 2, -1, 1, 0, None,
                  err, len(err)) == 1
    assert b"W4A4 mode does not support bias yet." in err.value
    assert masked(None, None, None, None, None, None, None, None, 2, 128, 128, 512, big, big, 128, 2, -1, 1, 0, None,
                  err, len(err)) == 1
    assert b"requires alpha input (per-expert scaling factor)" in err.value
    assert contiguous(None, None, None, None, None, None, None, None, 1, 129, 256, 128, big, big, 256, 0, -1, 1, 0,
                      None, err, len(err)) == 1
    assert b"No contiguous w8a8-mxfp8 tile for M=129 (grid M=129), N=256, K=128" in err.value
    assert contiguous(None, None, None, None, None, None, None, fake, 1, 128, 256, 512, big, big, 256, 1, -1, 1, 0,
                      None, err, len(err)) == 1
    assert b"does not take alpha; the per-expert scaling factor" in err.value
    assert contiguous(None, None, None, None, None, None, None, None, 1, 0, 256, 128, big, big, 256, 0, -1, 1, 0,
                      None, err, len(err)) == 0  # no rows: nothing to do
    # mode 3: e4m3 activations x packed e2m1 weights (tests/test_group_masked_gemm.py:727-768)
    assert masked(None, None, None, None, None, None, fake, None, 2, 128, 128, 512, big, big, 128, 3, -1, 1, 0, None,
                  err, len(err)) == 1
    assert b"W4A8 mode does not support bias yet." in err.value
    assert contiguous(None, None, None, None, None, None, None, fake, 1, 128, 256, 512, big, big, 256, 3, -1, 1, 0,
                      None, err, len(err)) == 1
    assert b"W4A8 mode does not take alpha" in err.value

    x = torch.empty([256, 128], dtype=torch.float8_e4m3fn)
    w = torch.empty([2, 256, 128], dtype=torch.float8_e4m3fn)
    sfa = torch.empty([256, 4], dtype=torch.uint8)
    sfb = torch.empty([2, 256, 4], dtype=torch.uint8)
    out = torch.empty([256, 256], dtype=torch.bfloat16)
    counts = torch.full([2], 128, dtype=torch.int32)
    ids = torch.zeros([256], dtype=torch.int32)
    with pytest.raises(RuntimeError, match="masked_m must have dtype torch.int32"):
        hq.group_masked_gemm(x, w, sfa, sfb, counts.long(), out, None, None, 128)
    with pytest.raises(RuntimeError, match=re.escape("masked_m shape must be [num_experts], got 1, expected 2")):
        hq.group_masked_gemm(x, w, sfa, sfb, counts[:1], out, None, None, 128)
    with pytest.raises(RuntimeError, match="input M must equal num_experts . max_m_per_expert, got 256, expected 128"):
        hq.group_masked_gemm(x, w, sfa, sfb, counts, out, None, None, 64)
    with pytest.raises(RuntimeError, match="no CPU path"):
        hq.group_masked_gemm(x, w, sfa, sfb, counts, out, None, None, 128)
    with pytest.raises(RuntimeError, match="expert_ids must have dtype torch.int32"):
        hq.group_contiguous_gemm(x, w, sfa, sfb, ids.long(), out)
    with pytest.raises(RuntimeError, match=re.escape("output shape must be [M, N], got [256, 128], expected [256, 256]")):
        hq.group_contiguous_gemm(x, w, sfa, sfb, ids, out[:, :128])
    with pytest.raises(RuntimeError, match="no CPU path"):
        hq.group_contiguous_gemm(x, w, sfa, sfb, ids, out)
    assert "mode=masked" in hq.describe_group_tile("masked", 20, 64, 7168, 3584)
    assert "mode=contiguous" in hq.describe_group_tile("contiguous", 16, 256, 7168, 3584)
    assert "w4a8-mxfp4" in hq.describe_group_tile("masked", 8, 128, 7168, 2048, "w4a8-mxfp4", sm_count=148)
    with pytest.raises(RuntimeError):
        hq.describe_group_tile("batch", 8, 128, 7168, 2048, "w4a8-mxfp4", sm_count=148)


def test_low_latency_rules_without_a_device(native):
    """Host checks of the plain-scale M <= 16 GEMM (texts of the reference's
    tests/test_low_latency_mma_gemm.py:297-345)."""
    import halops_b200 as hq

    fake = ctypes.cast(16, ctypes.c_void_p)
    f = native.lib().hq_low_latency_gemm

    def rc(m, n, n2, k1, k2, strides=(128, 128, 128, 128), a2=None, b2=None, sfa2=None, sfb2=None, out2=None,
           sigmoid=0):
        err = ctypes.create_string_buffer(512)
        code = f(None, None, None, None, None, a2, b2, sfa2, sfb2, out2, m, n, n2, k1, k2, *strides, n, n2, sigmoid,
                 -1, 1, 0, None, err, len(err))
        return code, err.value.decode()

    assert "supports M <= 16, got M=17" in rc(17, 512, 0, 4096, 0)[1]
    assert "weight rows must be divisible by 8, got 516 and 0" in rc(8, 516, 0, 256, 0, strides=(16, 16, 0, 0))[1]
    assert "K must be divisible by 256, got K=1152" in rc(8, 512, 0, 1152, 0, strides=(48, 48, 0, 0))[1]
    assert "plain row-major" in rc(8, 512, 0, 1024, 0, strides=(36, 32, 0, 0))[1]
    assert "weight2 / sfb2 must come with" in rc(8, 512, 0, 2048, 0, b2=fake, sfb2=fake)[1]
    assert "does not support input2 or output2" in rc(8, 512, 512, 2048, 0, b2=fake, sfb2=fake, out2=fake, sigmoid=1)[1]
    assert "K1 must be a multiple of 512, got K1=1920" in rc(8, 512, 0, 1920, 2176, a2=fake, b2=fake, sfa2=fake,
                                                             sfb2=fake)[1]
    assert rc(0, 512, 0, 1024, 0, strides=(32, 32, 0, 0))[0] == 0  # no rows: nothing to do

    x = torch.empty([8, 1024], dtype=torch.float8_e4m3fn)
    w = torch.empty([512, 1024], dtype=torch.float8_e4m3fn)
    sfa, sfb = torch.empty([8, 32], dtype=torch.uint8), torch.empty([512, 32], dtype=torch.uint8)
    out = torch.empty([8, 512], dtype=torch.bfloat16)
    with pytest.raises(RuntimeError, match="plain row-major"):
        hq.low_latency_mma_gemm(x, w, torch.empty([128, 32], dtype=torch.uint8), sfb, out)
    with pytest.raises(RuntimeError, match="supports M <= 16"):
        hq.low_latency_mma_gemm(torch.empty([17, 1024], dtype=torch.float8_e4m3fn), w, sfa, sfb, out)
    with pytest.raises(RuntimeError, match="no CPU path"):
        hq.low_latency_mma_gemm(x, w, sfa, sfb, out)


def test_enum_and_interleave():
    import halops_b200 as hq

    assert [int(e) for e in hq.EpilogueOp] == [0, 1, 2, 3, 4, 5]
    assert hq.EpilogueOp.SituQuant == 4
    t = torch.arange(64).reshape(64, 1)
    r = hq.interleave_gate_up(t).reshape(-1)
    assert r[:16].tolist() == list(range(16)) and r[16:32].tolist() == list(range(32, 48))
    assert r[32:48].tolist() == list(range(16, 32))


def test_decode_unit_deal_is_consistent(native):
    """The small-M kernel's deal of (128 weight rows x 256 bytes of K) units to the CTAs: every
    unit once, contiguous runs, distinct scratch slots per tile -- checked by the library's
    host-side self-check over many shapes and SM counts, with and without the even split."""
    from halops_b200 import _native

    for n in list(range(64, 2049, 64)) + [4736, 7168, 8192, 24576, 32768, 57344]:
        for k in (128, 256, 384, 1024, 1152, 1536, 2048, 4096, 8192):
            for sm in (1, 2, 7, 74, 132, 148, 160):
                for force_split in (0, 1, 2):
                    _native.call("hq_selftest_decode_plan", n, k, sm, force_split)
    with pytest.raises(RuntimeError, match="multiple of 128"):
        _native.call("hq_selftest_decode_plan", 128, 100, 148, 0)


def test_weight_prefetch_of_the_small_m_kernel_is_bounded(native):
    """24 MB over the grid, and at most one tile's steps of 32 KB (or 8) from the one thread of a CTA that asks for them."""
    import halops_b200 as hq

    for m, n, k in ((8, 24576, 1536), (16, 7168, 2048), (33, 23552, 7808), (1, 64, 128), (64, 64, 8192)):
        for sm in (1, 4, 16, 64, 148):
            line = hq.describe_tile(m, n, k, sm_count=sm)
            steps, ctas = (int(re.search(rf"{name}=(\d+)", line).group(1)) for name in ("prefetch", "ctas"))
            assert 1 <= steps <= max(8, -(-k // 256)) and (steps == 1 or steps * ctas <= 24 * 32), line


def test_describe_tile(native):
    import halops_b200 as hq

    assert "256x256/128 pair=1" in hq.describe_tile(8192, 8192, 8192, sm_count=148)
    assert "128x256/256 pair=0" in hq.describe_tile(4096, 14336, 4096, "w4a4-nvfp4", sm_count=148)
    assert "256x256/128 pair=1" in hq.describe_tile(8192, 4096, 4096, sm_count=148)
    # 144 single-CTA tiles fit one wave, 80 pair tiles need two
    assert "128x256/128 pair=0" in hq.describe_tile(1152, 4096, 4096, sm_count=148)
    # small M: the operand-swapped kernel; whole tiles per CTA, or every tile dealt to several
    # CTAs when the weight has too few tiles to keep HBM busy
    assert "swap 128x16/256 pair=0 splitk=0 ctas=56" in hq.describe_tile(8, 7168, 2048, sm_count=148)
    assert "swap 128x64/256 pair=0 splitk=0 ctas=148" in hq.describe_tile(64, 24576, 1536, sm_count=148)
    assert "swap 128x16/256 pair=0 splitk=0 ctas=64" in hq.describe_tile(8, 8192, 1024, sm_count=148)
    assert "swap 128x64/256 pair=0 splitk=1 ctas=128" in hq.describe_tile(64, 4096, 8192, sm_count=148)
    assert "swap" not in hq.describe_tile(65, 7168, 2048, sm_count=148)
    with pytest.raises(RuntimeError, match="No dense"):
        hq.describe_tile(128, 96, 128, sm_count=148)


def test_switches_can_be_read_under_the_callers_lock(native, monkeypatch):
    """A held reading serves the calls of its thread until it is let go, whatever happens to the environment."""
    import threading

    import halops_b200 as hq

    def width():
        return int(re.search(r"128x(\d+)/", hq.describe_tile(1000, 4096, 4096, sm_count=148)).group(1))

    lib = native.lib()
    monkeypatch.setenv("HALOPS_B200_TILE", "64")
    lib.hq_hold_switches(1)
    try:
        monkeypatch.setenv("HALOPS_B200_TILE", "256")
        assert width() == 64
        seen = []
        other = threading.Thread(target=lambda: seen.append(width()))
        other.start()
        other.join()
        assert seen == [256]
        lib.hq_hold_switches(1)
        assert width() == 256
    finally:
        lib.hq_hold_switches(0)
    monkeypatch.setenv("HALOPS_B200_TILE", "128")
    assert width() == 128


def test_switches_of_the_native_front_are_read_under_the_interpreter_lock():
    """Assignments to os.environ may move the array that the C library's functions walk; only the lock keeps them apart."""
    with open(os.path.join(ROOT, "halops_b200", "csrc", "gemm.cu")) as f:
        gemm = f.read()
    assert len(re.findall(r"\benviron\b(?=[;,) ])", re.sub(r"//[^\n]*", "", gemm))) == 1  # one walk, of the held reading
    assert re.findall(r"\.walk\(\)", gemm) == [".walk()"]
    assert re.search(r"void hq_hold_switches\(int hold\) \{[^}]*\.walk\(\);\s*\}", gemm)
    with open(os.path.join(ROOT, "halops_b200", "csrc", "fast_path.cpp")) as f:
        front = re.sub(r"//[^\n]*", "", f.read())
    held = front.index("hold_switches(1)")
    assert held < front.index("return unlocked(f);", held)
    gemms = front[front.index("PyObject* dense_gemm("):]
    assert gemms.count("unlocked_gemm(") == 3 and not re.search(r"\bunlocked\(", gemms)


def test_wide_tiles_for_columns_that_do_not_fill_them(native):
    """A width need not divide N (timed: 71 us on the pair tile against 115 on the 64-wide one, 110 against 175, 67 against 75)."""
    import halops_b200 as hq

    assert "256x256/128 pair=1" in hq.describe_tile(3000, 7232, 4096, sm_count=148)
    assert "256x256/128 pair=1" in hq.describe_tile(8192, 4160, 4096, sm_count=148)
    assert "x256/256" in hq.describe_tile(8192, 4480, 4096, "w4a4-nvfp4", sm_count=148)


def test_contiguous_tile_with_experts_that_meet_inside_tiles(native):
    """Runs start on multiples of 64 rows, so more experts than that leave the choice as it is; every run is cut into tiles of its
    own (or, on fixed tiles, worked in a pass of its own), so short runs do not ask for wide tiles."""
    import halops_b200 as hq

    def tile(count, m, n, k, mode="w8a8-mxfp8"):
        return hq.describe_group_tile("contiguous", count, max(1, m // count), n, k, mode, total_m=m, sm_count=148).split("-> ")[1]

    for mode in ("w8a8-mxfp8", "w4a4-nvfp4"):
        for m, n, k in ((2048, 4096, 2048), (1024, 7168, 2048), (4096, 2048, 4096)):
            assert {tile(c, m, n, k, mode) for c in (m // 64, m // 32, m // 8)} == {tile(m // 64, m, n, k, mode)}
    # timed on every tile: 10.5 / 10.8 us on the 128- and 64-wide tile against 16.3, 12.8 against 18.3, 13.0 against 18.7,
    # 60 against 76 on the pair tile
    assert "128x256" not in tile(16, 512, 2048, 2048)
    assert "128x128" in tile(16, 512, 4096, 2048) and "128x128" in tile(64, 2048, 1024, 2048)
    assert "128x128" in tile(16, 4096, 4096, 2048)
    # one expert has no boundary: the dense choice
    assert tile(1, 4096, 4096, 2048) == hq.describe_tile(4096, 4096, 2048, sm_count=148).split("-> ")[1].split(" splitk")[0]


def test_split_k_from_the_k_that_repays_its_exchange(native):
    """Timed split and whole: 9.6 / 9.2 us at 48 k-tiles, 10.2 / 10.4 at 56 on 11 tiles; 13.9 / 13.1 at 64, 17.1 / 17.9 at 96 on 58."""
    import halops_b200 as hq

    def split(n, k_tiles):
        return re.search(r"splitk=(\d)", hq.describe_tile(100, n, 128 * k_tiles, sm_count=148)).group(1)

    assert [split(704, kt) for kt in (8, 48, 55, 56, 64, 192)] == ["0", "0", "0", "1", "1", "1"]
    assert [split(3712, kt) for kt in (56, 95, 96)] == ["0", "0", "1"]
    assert split(2368, 56) == "1" and split(2432, 56) == "0" and split(4800, 192) == "0"


def test_contiguous_experts_that_the_run_table_does_not_repay(native):
    """Timed both ways on the 128-wide tile: 6.8 us by runs and 5.0 by rows, 6.8 and 5.6, 15.9 and 14.6; 7.2 and 8.3, 46 and 56,
    30 and 35 the other way round (a second wave only by rows, several waves, runs of two quarters and more)."""
    import halops_b200 as hq

    def cut(count, m, n, k, mode="w8a8-mxfp8"):
        return re.search(r"cut=(\w+)", hq.describe_group_tile("contiguous", count, max(1, m // count), n, k, mode, total_m=m, sm_count=148)).group(1)

    assert cut(25, 1600, 1024, 512, "w4a4-nvfp4") == "rows" and cut(10, 640, 3200, 512) == "rows" and cut(64, 2048, 1024, 2048) == "rows"
    assert cut(16, 512, 2048, 2048, "w4a4-nvfp4") == "runs" and cut(15, 960, 5888, 3840) == "runs" and cut(16, 1024, 2944, 3328) == "runs"
    assert cut(10, 40960, 4096, 4096, "w4a4-nvfp4") == "runs" and cut(8, 1024, 1024, 512) == "runs"


def test_the_tile_is_chosen_among_those_that_can_run(native):
    """Slots and batches that are no multiple of 256 rows and the quantising epilogues have no (or not every) pair tile, and 64-row
    slots never straddle 128-row tiles.  Timed on every tile: 6.5 us on 128 x 128, 8.4 on 128 x 256; 19 and 21; 6.3 and 8.7;
    26 and 29; SituQuant 13.9 on 128 x 128, 14.6 on 128 x 256 and 15.3 on the pair tile; 11.3 and 12.5."""
    import halops_b200 as hq

    def tile(kind, count, m, n, k, mode):
        return hq.describe_group_tile(kind, count, m, n, k, mode, sm_count=148).split("-> ")[1]

    assert "128x128" in tile("masked", 8, 64, 2048, 2048, "w4a4-nvfp4") and "128x128" in tile("masked", 16, 64, 2688, 3072, "w4a4-nvfp4")
    assert "128x128" in tile("batch", 7, 192, 1152, 2048, "w4a4-mxfp4") and "128x128" in tile("batch", 22, 128, 3968, 2560, "w4a4-mxfp4")
    for m in (64, 128, 192, 320):
        for n in (1024, 2176, 7168):
            assert "pair=0" in tile("masked", 12, m, n, 2048, "w8a8-mxfp8") and "pair=0" in tile("batch", 12, m, n, 2048, "w8a8-mxfp8")
    # one slot fills tiles of its own: as many as the rows have, whatever the number of slots
    assert tile("masked", 64, 128, 2048, 1024, "w8a8-mxfp8") == tile("masked", 64, 64, 2048, 1024, "w8a8-mxfp8")
    assert "situ=128x128" in hq.describe_tile(458, 9984, 1664, sm_count=148)
    assert "situ=128x128" in hq.describe_tile(609, 4096, 2176, sm_count=148)
    assert "situ=256x256" in hq.describe_tile(4096, 7168, 2048, sm_count=148)
    for m in (129, 300, 916, 2048, 8192):
        for n in (2048, 5120, 9728, 14336):
            assert "situ=256x128" not in hq.describe_tile(m, n, 2048, sm_count=148)


def test_product_never_imports_the_oracle():
    """The library must not route through the CPU oracle."""
    pkg = os.path.join(ROOT, "halops_b200")
    for dirpath, _, files in os.walk(pkg):
        for f in files:
            if f.endswith((".py", ".cu", ".cuh", ".h")):
                assert "oracle" not in open(os.path.join(dirpath, f)).read(), f


def test_gemm_allgather_rules_without_a_device(native):
    import ctypes

    from halops_b200 import _native

    def call(world, rank, m, n_local, k, ldo):
        outs = (ctypes.c_void_p * 8)(*([256] * 8))
        _native.call("hq_dense_gemm_allgather", 256, 256, 256, 256, outs, world, rank, m, n_local, k, 1 << 40, 1 << 40,
                     ldo, -1, 0, 0, None)

    with pytest.raises(RuntimeError, match="world must be"):
        call(9, 0, 256, 256, 128, 256 * 9)
    with pytest.raises(RuntimeError, match="world must be"):
        call(2, 2, 256, 256, 128, 512)
    with pytest.raises(RuntimeError, match="multiple of 256"):
        call(2, 0, 256, 128, 128, 256)
    with pytest.raises(RuntimeError, match="multiple of 256"):
        call(2, 0, 128, 256, 128, 512)
    with pytest.raises(RuntimeError, match="row stride"):
        call(2, 0, 256, 256, 128, 256)

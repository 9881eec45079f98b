"""Where the native front of the entry points cannot be loaded, the wrappers make the calls."""

import warnings

import pytest
import torch

import halops_b200 as hq
from halops_b200 import _native


@pytest.fixture
def without(monkeypatch, tmp_path, request):
    from halops_b200 import build

    build.build()
    path = tmp_path / "halops_b200_fast_path.so"
    if request.param == "broken":
        path.write_bytes(b"not a shared object")
    monkeypatch.setattr(_native, "_FAST_PATH", str(path))
    monkeypatch.setattr(_native, "fast_path", None)


@pytest.mark.parametrize("without", ["missing", "broken"], indirect=True)
def test_calls_go_to_the_wrappers(without):
    x = torch.zeros([4, 256], dtype=torch.bfloat16)
    with pytest.warns(RuntimeWarning, match="native front of the Python calls is not used"):
        # (the wrapper's own check: no library has been asked)
        with pytest.raises(RuntimeError, match="CUDA tensor"):
            hq.group_wise_quant(x)
    calls = [lambda: hq.group_wise_quant(x), lambda: hq.rms_norm_quant(x, x[0].contiguous()),
             lambda: hq.dense_gemm(x, x, x, x, x, mode="none"),
             lambda: hq.group_masked_gemm(x, x, x, x, x, x, mode="none"),
             lambda: hq.group_contiguous_gemm(x, x, x, x, x, x, mode="none")]
    with warnings.catch_warnings():
        warnings.simplefilter("error")  # said once
        for call in calls:
            with pytest.raises(RuntimeError, match="CUDA tensor|Unsupported mode"):
                call()
    assert _native.fast_path is _native._NoFastPath

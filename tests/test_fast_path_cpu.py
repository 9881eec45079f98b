"""Where the native front of the entry points cannot be loaded, the wrappers make the calls.  It is rebuilt for
another torch, another Python and a changed C ABI, whose signatures it takes from the header."""

import os
import re
import warnings

import pytest
import torch

import halops_b200 as hq
from halops_b200 import _native


@pytest.fixture(autouse=True)
def built():
    from halops_b200 import build

    build.build()


@pytest.fixture
def without(monkeypatch, tmp_path, request):
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


def test_rebuilt_for_what_it_was_compiled_against(tmp_path, monkeypatch):
    from halops_b200 import _paths, build

    here = build.fast_path_file(torch.__version__)
    assert _native._FAST_PATH == here and os.path.exists(here) and not build.fast_path_is_stale(torch.__version__)
    assert build.fast_path_is_stale("0.0.1")  # another torch: another file
    monkeypatch.setattr(_paths.sysconfig, "get_config_var", lambda name: "cpython-399-x86_64-linux-gnu")
    assert build.fast_path_file(torch.__version__) != here
    monkeypatch.undo()
    newer = tmp_path / "halops_b200.h"
    newer.write_text("")
    os.utime(newer, (os.path.getmtime(here) + 10,) * 2)
    assert os.path.samefile(build.FAST_PATH_DEPS[1], os.path.join(os.path.dirname(build.PKG), "include", "halops_b200.h"))
    monkeypatch.setattr(build, "FAST_PATH_DEPS", (build.FAST_PATH_DEPS[0], str(newer)))
    assert build.fast_path_is_stale(torch.__version__)


def test_signatures_come_from_the_header():
    from halops_b200 import build

    with open(build.FAST_PATH_DEPS[0]) as f:
        text = f.read()
    assert '#include "../../include/halops_b200.h"' in text
    types = re.findall(r"using (\w+Fn) = (.*);", text)
    assert len(types) == 7 and all(re.fullmatch(r"decltype\(&hq_\w+\)", t) for _, t in types)


def test_library_alone_builds_without_torch(monkeypatch, capsys):
    import sys

    from halops_b200 import build

    monkeypatch.setitem(sys.modules, "torch", None)  # import torch raises ImportError
    build._build_fast_path(False, False)
    assert "not built" in capsys.readouterr().err

"""The C-ABI library without a GPU: it loads, exports every symbol the header declares, reports
errors through the error-string convention and refuses to work without a CUDA device."""
import ctypes as C
import os
import re

import numpy as np
import pytest

from cuml_b200.fil import _lib
from cuml_b200.fil._desc import CCreateOpts, CInfo
from tests.conftest import ROOT, has_gpu
from tests.helpers import random_forest_desc


def declared_symbols():
    text = open(os.path.join(ROOT, "include", "b2fil.h")).read()
    text = re.sub(r"/\*.*?\*/", "", text, flags=re.S)
    return sorted(set(re.findall(r"\b(b2fil_[a-z_0-9]+)\s*\(", text)))


def test_header_symbols_are_exported(lib):
    names = declared_symbols()
    assert "b2fil_predict" in names and "b2fil_forest_create" in names and len(names) >= 12
    for n in names:
        assert hasattr(lib, n), f"{n} is declared in include/b2fil.h but not exported"


def test_version_and_error_string(lib):
    assert lib.b2fil_version() >= 100
    rc = lib.b2fil_forest_create(None, None, None)
    assert rc == -1
    assert b"NULL" in lib.b2fil_last_error()
    assert lib.b2fil_forest_free(None) == 0
    info = CInfo()
    assert lib.b2fil_forest_info(None, C.byref(info)) == -1
    assert lib.b2fil_output_elems_per_row(None, 0) == 0
    assert lib.b2fil_predict(None, 0, None, 0, 0, None, 0, 0.5, None) == -1


def test_struct_sizes_match_header():
    # the header's structs, compiled by gcc, must have the sizes of the ctypes mirrors
    import subprocess
    import tempfile

    from cuml_b200.fil._desc import CForestDesc

    src = ('#include <stdio.h>\n#include "b2fil.h"\nint main(){printf("%zu %zu %zu\\n", '
           "sizeof(b2fil_forest_desc), sizeof(b2fil_create_opts), sizeof(b2fil_info));return 0;}")
    with tempfile.TemporaryDirectory() as d:
        c = os.path.join(d, "s.c")
        open(c, "w").write(src)
        exe = os.path.join(d, "s")
        subprocess.check_call(["gcc", "-I", os.path.join(ROOT, "include"), c, "-o", exe])
        sizes = [int(x) for x in subprocess.check_output([exe]).split()]
    assert sizes == [C.sizeof(CForestDesc), C.sizeof(CCreateOpts), C.sizeof(CInfo)]


@pytest.mark.skipif(has_gpu(), reason="checks the behaviour on a box without a GPU")
def test_no_gpu_means_error_not_fallback(lib):
    from cuml_b200.fil import ForestInference

    desc = random_forest_desc(0)
    with pytest.raises(_lib.B2FilError) as ei:
        ForestInference.load_from_treelite_model(desc)
    assert ei.value.code == -4


def test_python_argument_validation():
    from cuml_b200.fil import ForestInference

    with pytest.raises(ValueError):
        ForestInference(layout="zigzag")
    with pytest.raises(ValueError):
        ForestInference(precision="half")
    with pytest.raises(ValueError):
        ForestInference(default_chunk_size=3)
    with pytest.raises(ValueError):
        ForestInference(storage="ragged")


def test_product_never_imports_the_oracle():
    # the oracle is test infrastructure: nothing under cuml_b200/ may name it
    for dirpath, _, files in os.walk(os.path.join(ROOT, "cuml_b200")):
        for fn in files:
            if fn.endswith((".py", ".cu", ".cpp", ".hpp", ".h")):
                text = open(os.path.join(dirpath, fn)).read()
                assert "fil_oracle" not in text and "import oracle" not in text, fn
                assert "from oracle" not in text, fn


def test_without_the_compiled_torch_path_device_calls_go_through_ctypes(monkeypatch):
    """The module for the installed torch may be missing (another torch, no compiler): a forest then
    says so once, and the ctypes path serves its calls."""
    from cuml_b200.fil.forest_inference import _Forest

    def missing():
        raise ImportError("b2fil_torch-9.9.so is missing")

    monkeypatch.setattr(_lib, "torch_module", missing)
    f = _Forest.__new__(_Forest)
    f.handle, f.info, f._device_call = C.c_void_p(), CInfo(), None
    with pytest.warns(RuntimeWarning, match="b2fil_torch"):
        assert f.device_call() is False
    assert f.device_call() is False


def test_torch_path_that_does_not_compile_leaves_the_library_alone(monkeypatch, tmp_path, capfd):
    import sys

    from cuml_b200 import build

    if build.torch_module_path() is None:
        pytest.skip("no torch")
    monkeypatch.setattr(build, "LIB_DIR", str(tmp_path))
    assert not build._torch_module_settled()
    built = []
    monkeypatch.setattr(build, "_lib_up_to_date", lambda: True)
    monkeypatch.setattr(build, "_torch_command",
                        lambda out: built.append(out) or [sys.executable, "-c", "import sys; sys.exit(3)"])
    assert build.build() == build.LIB and len(built) == 1
    assert "ctypes" in capfd.readouterr().err
    # not tried again until its source changes or a build is forced
    assert build.up_to_date() and build.build() == build.LIB and len(built) == 1
    assert not os.path.exists(build.torch_module_path())


_ODD_TENSOR = """
import torch
from cuml_b200.fil import _lib

class Odd(torch.Tensor):  # says it is a CUDA tensor and raises when asked for its sizes
    @staticmethod
    def __new__(cls):
        return torch.Tensor._make_wrapper_subclass(
            cls, (3, 4), strides=(4, 1), dtype=torch.float32, device="cuda:0",
            dispatch_sizes_strides_policy="sizes")

    @classmethod
    def __torch_dispatch__(cls, func, types, args=(), kwargs=None):
        raise ValueError("no sizes here")

call = _lib.torch_module().DeviceCall(1, 1, 4, 3, 1, 0, False, False)
try:
    call(Odd(), None, 0, 0, 0.5)
except ValueError as e:
    print("raised:", e)
"""


def test_device_call_raises_what_a_tensor_raises(lib):
    """Errors of torch's C++ side come out as Python exceptions; they used to end the process."""
    import subprocess
    import sys

    r = subprocess.run([sys.executable, "-c", _ODD_TENSOR], cwd=ROOT, capture_output=True, text=True)
    assert r.returncode == 0 and "raised: no sizes here" in r.stdout, r.stderr[-500:]

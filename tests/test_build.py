"""The operator library fits one PyTorch: another one makes it stale, and loading it says so."""
import subprocess
import sys

from lact_b200 import build

CODE = """
import lact_b200
from lact_b200 import _lib, ops
_lib._ops_loaded, _lib.OPS_PATH = False, {path!r}
for call in (_lib.load_ops, lambda: ops._op("swiglu_ffn_fwd")):
    try:
        call()
    except ImportError as e:
        assert "another PyTorch" in str(e), e
    else:
        raise SystemExit("loaded")
"""


def test_library_of_another_torch_is_stale_and_refused(tmp_path):
    build.build()
    assert build.built_for_this_torch()
    other = tmp_path / "ops.so"
    other.write_bytes(open(build.TORCH_LIB, "rb").read().replace(build.torch_stamp().encode(), b"lact_b200 operators for PyTorch 0.1;"))
    assert not build.built_for_this_torch(str(other))
    r = subprocess.run([sys.executable, "-c", CODE.format(path=str(other))], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr


MISSING = """
import lact_b200
from lact_b200 import _fakes, _lib
_lib._ops_loaded = False
_fakes._fake("added_later")(lambda x: x)
for _ in range(2):
    try:
        _lib.load_ops()
    except ImportError as e:
        assert "older than this package" in str(e) and "added_later" in str(e), e
    else:
        raise SystemExit("loaded")
"""


def test_library_without_an_operator_is_refused():
    build.build()
    r = subprocess.run([sys.executable, "-c", MISSING], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr


def test_build_compiles_again_for_another_torch(monkeypatch):
    built = []
    monkeypatch.setattr(build, "build_torch", lambda verbose=False: built.append(1))
    build.build()
    assert not built
    monkeypatch.setattr(build, "torch_stamp", lambda: "lact_b200 operators for PyTorch 0.1;")
    build.build()
    assert built

"""What the build makes on hosts that lack something, and what the package does without the part that was not made."""
import subprocess
import sys
import textwrap
from pathlib import Path

import pytest

from turbopi_b200 import _lib

ROOT = Path(__file__).resolve().parent.parent

PREPARE = """
import sys
from pathlib import Path
{hide}
from turbopi_b200 import build
build.OBJ, build.LIB = Path({tmp!r}) / "obj", Path({tmp!r}) / "lib" / "libturbopi_b200.so"

class Done:
    returncode, stdout, stderr = 0, "", ""

class Failed(Done):
    returncode = 1

def run(cmd, **kw):                      # a compiler that succeeds at once; g++ can be made to fail
    if Path(cmd[0]).name == "g++":
        return {gxx}()
    Path(cmd[cmd.index("-o") + 1]).write_bytes(b"")
    return Done()
build.subprocess.run, build._nvcc = run, lambda: "/usr/local/cuda/bin/nvcc"
"""


def _run(tmp, body, hide="", gxx="Done"):
    code = PREPARE.format(tmp=str(tmp), hide=hide, gxx=gxx) + textwrap.dedent(body)
    r = subprocess.run([sys.executable, "-c", code], cwd=ROOT, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr


def test_the_library_needs_no_torch(tmp_path):
    _run(tmp_path, """
        assert build.build(force=True).exists() and "torch" not in {m.partition(".")[0] for m, v in sys.modules.items() if v}
    """, hide="sys.modules['torch'] = None")


def test_the_library_is_linked_also_when_the_extension_fails(tmp_path):
    _run(tmp_path, """
        try:
            build.build(force=True)
        except RuntimeError as e:
            assert "g++" in str(e) and build.LIB.exists()
        else:
            raise SystemExit("the failure was swallowed")
    """, gxx="Failed")


def test_another_torch_or_python_finds_no_module_of_this_one(monkeypatch):
    import sysconfig

    import torch
    here = _lib.calls_path()
    monkeypatch.setattr(torch, "__version__", "2.12.0")
    assert _lib.calls_path() != here
    monkeypatch.undo()
    monkeypatch.setattr(sysconfig, "get_config_var", lambda name: "cpython-313-x86_64-linux-gnu")
    assert _lib.calls_path() != here


def test_calls_without_the_module_take_their_python_form(monkeypatch, tmp_path):
    import torch

    from turbopi_b200 import ops
    monkeypatch.setattr(_lib, "_native", None)
    monkeypatch.setattr(_lib, "calls_path", lambda: tmp_path / "_calls.so")
    with pytest.warns(UserWarning, match="python -m turbopi_b200.build"), pytest.raises(_lib.TurboPiError, match="CUDA tensors"):
        ops.quantize_activation_to_fp8(torch.zeros(1, 16, dtype=torch.bfloat16))
    assert _lib.native().attention() is None

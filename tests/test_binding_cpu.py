"""What the compiled binding cannot read ends in a Python error or in the ctypes path, which raises its own: no abort, no call."""
import shutil
import subprocess
import sys
import types
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent
SCRIPT = """
import sys, torch
from torch._subclasses.fake_tensor import FakeTensorMode
from torch.fx.experimental.symbolic_shapes import DimDynamic, ShapeEnv, StatelessSymbolicContext
from breeze_tts_cpp_b200 import _native, ops

mode = FakeTensorMode(shape_env=ShapeEnv())
closed = ops.Context.__new__(ops.Context)  # a context without a device, as after close()
closed._handle, closed._address = None, 0
answers = []

def call(x):
    for attempt in (lambda: _native.row_quantize(0, x, view), lambda: closed.quantize_rows(x, view)):
        try:
            answers.append(attempt() is NotImplemented)
        except Exception:
            answers.append(True)
    return x.float().sum()

with mode:
    view = ops.RowScaledView.empty(4, 256, ops.I8)
    x = torch.empty(3, 4, 256, dtype=torch.bfloat16, device="cuda")
    if sys.argv[1] == "vmap":
        torch.vmap(call)(x)
    elif sys.argv[1] == "functionalize":
        torch.func.functionalize(call)(x[0])
    elif sys.argv[1] == "symbolic":
        real = torch.empty(5, 256, dtype=torch.bfloat16)
        sizes = StatelessSymbolicContext(dynamic_sizes=[DimDynamic.DYNAMIC, DimDynamic.STATIC])
        call(mode.from_tensor(real, symbolic_context=sizes).to("cuda"))
    else:  # a flag that int() refuses
        answers.append(_native.quantized_norm(0, x[0], None, x[0, :1], view, 1e-6, None, None) is NotImplemented)
        try:
            closed.quantized_norm(x[0], None, x[0, :1], view, 1e-6, gemma=None)
        except TypeError:
            answers.append(True)
assert answers == [True] * len(answers) and len(answers) >= 2, answers
print("declined")
"""


@pytest.mark.parametrize("kind", ["vmap", "functionalize", "symbolic", "flag"])
def test_binding_declines(kind):
    done = subprocess.run([sys.executable, "-c", SCRIPT, kind], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert done.returncode == 0 and "declined" in done.stdout, done.stderr[-2000:]


def test_import_without_a_build_names_the_command_when_called(tmp_path):
    package = tmp_path / "breeze_tts_cpp_b200"
    package.mkdir()
    for source in (ROOT / "breeze_tts_cpp_b200").glob("*.py"):
        shutil.copy(source, package)
    script = ("from breeze_tts_cpp_b200 import ops\n"
              "closed = ops.Context.__new__(ops.Context)\nclosed._handle, closed._address = None, 0\n"
              "try:\n    closed.quantize_rows(None, None)\nexcept RuntimeError as e:\n    assert 'breeze_tts_cpp_b200.build' in str(e), e\n"
              "    print('named')\n")
    done = subprocess.run([sys.executable, "-c", script], cwd=tmp_path, capture_output=True, text=True, timeout=300)
    assert done.returncode == 0 and "named" in done.stdout, done.stderr[-2000:]


def test_binding_is_rebuilt_for_another_torch_and_on_demand(tmp_path, monkeypatch):
    import torch
    from breeze_tts_cpp_b200 import build
    commands = []

    def compiler(cmd, **_):
        commands.append(cmd)
        (tmp_path / "_native.so").write_text("")
        return types.SimpleNamespace(returncode=0)

    monkeypatch.setattr(build, "BINDING", tmp_path / "_native.so")
    monkeypatch.setattr(build, "OBJ", tmp_path)
    monkeypatch.setattr(build.subprocess, "run", compiler)
    for force, version, expected in ((False, None, 1), (False, None, 1), (False, "0.0.1", 2), (False, "0.0.1", 2), (True, "0.0.1", 3)):
        if version:
            monkeypatch.setattr(torch, "__version__", version)
        build._build_binding(False, force)
        assert len(commands) == expected

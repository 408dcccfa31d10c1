"""What the build and the name-keyed call need: no PyTorch for the C library and for calls on host buffers, and an extension that is
built again when the PyTorch it was compiled against is another one."""
import os
import subprocess
import sys

import pytest

from metaltile_b200 import build

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
# a Python in which PyTorch is not installed
NO_TORCH = "import sys\nsys.modules['torch'] = None\n"


def _python(code):
    r = subprocess.run([sys.executable, "-c", NO_TORCH + code], cwd=ROOT, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
    assert r.returncode == 0, r.stdout
    return r.stdout


def test_the_name_keyed_call_does_not_need_torch():
    out = _python("from metaltile_b200 import context\n"
                  "mod = context._binding()\n"
                  "class C:\n"
                  "    _handle = None\n"
                  "    def _check(self, rc): raise RuntimeError('rc %d' % rc)\n"
                  "try:\n"
                  "    mod.dispatch(C(), 'mt_qmv', 0, {'x': b'1234'}, ('out',), (1, 1, 1), (1, 1, 1))\n"
                  "except RuntimeError as e:\n"
                  "    print(e)\n")
    assert "rc -8" in out                                 # the library refuses the null context; nothing else was missing


def test_the_c_library_is_built_without_torch(tmp_path):
    """A build from nothing (the compilers stood in for): the library, the binding of the name-keyed call, no error."""
    out = _python("import types\n"
                  "from metaltile_b200 import build\n"
                  f"build.OBJ = {str(tmp_path / 'obj')!r}\n"
                  "ran = []\n"
                  "build._compile = lambda nvcc, src, obj, *rest: obj\n"
                  "build.subprocess = types.SimpleNamespace(run=lambda cmd, **kw: ran.append(cmd) or types.SimpleNamespace(returncode=0, stdout=''),\n"
                  "                                         PIPE=None, STDOUT=None)\n"
                  "assert build.build(force=True) == build.LIB\n"
                  "made = [cmd[cmd.index('-o') + 1] for cmd in ran]\n"
                  "assert made == [build.LIB, build.DISPATCH], made\n")
    assert "PyTorch is not installed" in out


def test_another_pytorch_or_python_means_another_extension(monkeypatch, tmp_path):
    import torch
    if not os.path.exists(os.path.join(build.OBJ, "native.stamp")):
        pytest.skip("the build's stamps do not travel with the built files")
    made = []
    monkeypatch.setattr(build, "_compile_native", lambda torch, log: made.append("native"))
    monkeypatch.setattr(build, "_stamp", lambda path, digest: made.append(os.path.basename(path)))
    monkeypatch.setattr(build, "_compile", lambda *a: pytest.fail("the C library does not depend on PyTorch"))
    build.build()
    assert made == []
    monkeypatch.setattr(torch, "__version__", torch.__version__ + ".other")
    build.build()
    assert made == ["native", "native.stamp"]
    monkeypatch.undo()
    here = build.native_digest()
    monkeypatch.setattr(sys, "version", "other " + sys.version)
    assert build.native_digest() != here


def test_an_extension_of_another_pytorch_is_refused():
    r = subprocess.run([sys.executable, "-c", "import torch\ntorch.__version__ += '.other'\nimport metaltile_b200.ops"], cwd=ROOT,
                       stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
    assert r.returncode != 0 and "compiled against PyTorch" in r.stdout

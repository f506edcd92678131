"""What the native build depends on, and the declarations that its parts repeat."""

import re
import subprocess
import sys
from pathlib import Path

import pytest
import torch

from torchft_b200.ops import _lib
from torchft_b200.utils import build

ROOT = Path(build.PKG).parent


@pytest.mark.skipif(not build.autograd_module_path().exists(), reason="the native autograd nodes are not built here")
def test_autograd_module_belongs_to_the_installed_torch(monkeypatch):
    build.build_autograd()
    assert build.autograd_module_current()
    monkeypatch.setattr(torch, "__version__", "2.11.0+other")
    assert not build.autograd_module_current()


def test_build_module_works_without_torch_and_says_what_to_do():
    code = ("import sys; sys.modules['torch'] = None\n"
            "from torchft_b200.utils import build\n"
            "assert 'no-build-isolation' in build.autograd_obstacle()\n"
            "try:\n    build.build_autograd()\nexcept RuntimeError as e:\n    assert 'no-build-isolation' in str(e)\nelse:\n    raise SystemExit(1)\n")
    done = subprocess.run([sys.executable, "-c", code], cwd=ROOT, capture_output=True, text=True)
    assert done.returncode == 0, done.stderr


def _kind(declaration):
    """P, L, I or F of one C parameter, as the Python prototypes write them."""
    if "*" in declaration or "cudaStream_t" in declaration or declaration.split()[0] == "P":
        return "P"
    words = declaration.split()
    return "F" if "float" in words else "L" if "long" in words or "int64_t" in words else "I"


def _kinds(parameters):
    return [_kind(p) for p in re.sub(r"//[^\n]*", "", parameters).split(",") if p.strip() not in ("", "void")]


def test_entry_points_are_declared_alike_everywhere():
    """An entry point's parameters stand in its ``.cu`` file, in the Python prototypes and, for some, in the native nodes; only
    casts join them."""
    entries = {}
    for path in build.KERNEL_SRC.glob("*.cu"):
        for name, parameters in re.findall(r"TFT_API int (\w+)\(([^)]*)\)\s*\{", path.read_text()):
            entries[name] = _kinds(parameters)
    letters = {_lib.P: "P", _lib.I: "I", _lib.L: "L", _lib.F: "F"}
    for name, types in _lib._PROTOTYPES.items():
        assert entries[name] == [letters[t] for t in types], name

    source = (build.HOST_SRC / "autograd.cc").read_text()
    members = dict(re.findall(r"int \(\*(\w+)\)\(([^)]*)\);", source))
    taken = re.findall(r'take\(entries, "(\w+)", kernels\.(\w+)\)', source)
    assert {member for _, member in taken} == set(members)
    for entry, member in taken:
        assert _kinds(members[member]) == entries[entry], entry

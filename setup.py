"""Builds the native parts in-tree (nvcc for sm_100a, g++ for the control plane) before packaging.

``python setup.py build_ext --inplace`` and ``pip install -e .`` both end up in
``torchft_b200.utils.build``; the shared objects live inside the package directory.  The native autograd nodes are built
against the torch that is installed, so the package has to be built without isolation:
``pip install --no-build-isolation -e .``.
"""

import os
import sys

from setuptools import setup
from setuptools.command.build_ext import build_ext
from setuptools.command.build_py import build_py

sys.path.insert(0, os.path.dirname(os.path.abspath(__file__)))


def _build_native() -> None:
    from torchft_b200.utils import build

    obstacle = build.autograd_obstacle()
    if obstacle is None:
        build.build_all()
        return
    # everything but the one part that needs torch's headers; using that part later raises and says what to run
    build.build_control()
    build.build_kernels()
    print(f"native autograd nodes not built: {obstacle}", file=sys.stderr)


class BuildNative(build_ext):
    def run(self) -> None:
        _build_native()


class BuildPy(build_py):
    def run(self) -> None:
        _build_native()
        super().run()


setup(cmdclass={"build_ext": BuildNative, "build_py": BuildPy})

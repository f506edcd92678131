"""In-tree native builds.

Three artefacts are produced next to the Python sources:

* ``torchft_b200/lib/libtft_kernels.so`` -- every ``.cu`` file under ``csrc/kernels``
  compiled with nvcc for ``sm_100a`` and exported through a plain C ABI (loaded with
  ctypes, no link-time dependency on torch or libcuda).
* ``torchft_b200/_autograd.*.so`` -- native autograd nodes over the kernels (``csrc/host``), the one
  artefact compiled against torch's headers.
* ``torchft_b200/_control.*.so`` -- the C++ control plane (lighthouse, manager server and
  client) as a pybind11 extension module, plus the ``tft_lighthouse`` executable.

Objects are rebuilt only when a source or header is newer than the object.
"""

from __future__ import annotations

import os
import subprocess
import sys
import sysconfig
from concurrent.futures import ThreadPoolExecutor
from pathlib import Path
from typing import List, Optional

PKG = Path(__file__).resolve().parent.parent
KERNEL_SRC = PKG / "csrc" / "kernels"
CONTROL_SRC = PKG / "csrc" / "control"
HOST_SRC = PKG / "csrc" / "host"
LIB_DIR = PKG / "lib"
OBJ_DIR = PKG / "lib" / "obj"

NVCC_FLAGS = [
    "-gencode",
    "arch=compute_100a,code=sm_100a",
    "-lineinfo",
    "-O3",
    "-std=c++17",
    "--use_fast_math",
    "-Xcompiler",
    "-fPIC",
    "-Xcompiler",
    "-fvisibility=hidden",
]


def _nvcc() -> str:
    cuda_home = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    cand = Path(cuda_home) / "bin" / "nvcc"
    return str(cand) if cand.exists() else "nvcc"


def _newest(paths: List[Path]) -> float:
    return max((p.stat().st_mtime for p in paths if p.exists()), default=0.0)


def kernels_lib_path() -> Path:
    return LIB_DIR / "libtft_kernels.so"


def control_module_path() -> Path:
    suffix = sysconfig.get_config_var("EXT_SUFFIX") or ".so"
    return PKG / f"_control{suffix}"


def autograd_module_path() -> Path:
    suffix = sysconfig.get_config_var("EXT_SUFFIX") or ".so"
    return PKG / f"_autograd{suffix}"


def lighthouse_bin_path() -> Path:
    return LIB_DIR / "tft_lighthouse"


def build_kernels(force: bool = False, verbose: bool = False) -> Path:
    """Compiles all CUDA sources for sm_100a and links ``libtft_kernels.so``."""
    OBJ_DIR.mkdir(parents=True, exist_ok=True)
    sources = sorted(KERNEL_SRC.glob("*.cu"))
    headers = sorted(KERNEL_SRC.glob("*.cuh")) + sorted(KERNEL_SRC.glob("*.h"))
    hdr_time = _newest(headers)
    objs: List[Path] = []
    jobs = []
    for src in sources:
        obj = OBJ_DIR / (src.stem + ".o")
        objs.append(obj)
        if force or not obj.exists() or obj.stat().st_mtime < max(src.stat().st_mtime, hdr_time):
            cmd = [_nvcc(), *NVCC_FLAGS, "-I", str(KERNEL_SRC), "-c", str(src), "-o", str(obj)]
            if verbose:
                cmd.insert(1, "-Xptxas")
                cmd.insert(2, "-v")
            jobs.append(cmd)

    def run(cmd: List[str]) -> None:
        res = subprocess.run(cmd, capture_output=True, text=True)
        if res.returncode != 0:
            raise RuntimeError(f"nvcc failed: {' '.join(cmd)}\n{res.stdout}\n{res.stderr}")
        if verbose:
            sys.stderr.write(res.stderr)

    if jobs:
        with ThreadPoolExecutor(max_workers=min(8, len(jobs))) as ex:
            list(ex.map(run, jobs))
    out = kernels_lib_path()
    if force or jobs or not out.exists():
        cmd = [_nvcc(), "-shared", "-o", str(out), *map(str, objs), "-cudart", "shared"]
        run(cmd)
    return out


def _host_cxx() -> str:
    # Prefer the distribution compiler: it links libstdc++ dynamically, so a module
    # shares one C++ runtime with torch.
    return os.environ.get("TFT_CXX") or ("/usr/bin/g++" if Path("/usr/bin/g++").exists() else os.environ.get("CXX", "g++"))


def _torch_mark(version: str) -> str:
    """What the module carries inside itself about the torch that it was built against."""
    return f"built against torch {version};"


def autograd_obstacle() -> Optional[str]:
    """Why the native autograd nodes cannot be built in this environment, or ``None``."""
    try:
        import torch
    except ImportError:
        return ("torch is not installed here.  A package build in an isolated environment does not see the torch it will run with: "
                "install with `pip install --no-build-isolation`, or run `python -m torchft_b200.utils.build` afterwards")
    if torch.version.cuda is None:
        return f"torch {torch.__version__} was built without CUDA"
    return None


def autograd_module_current() -> bool:
    """Whether the module is there, newer than its source and built against the torch that is installed.  The file itself
    says against which: the times of torch's files do not, since installers keep those of the archive or of a cache."""
    import torch

    out = autograd_module_path()
    return (out.exists() and out.stat().st_mtime >= _newest([HOST_SRC / "autograd.cc"])
            and _torch_mark(torch.__version__).encode() in out.read_bytes())


def build_autograd(force: bool = False) -> Path:
    """Builds the native autograd nodes against the installed torch."""
    obstacle = autograd_obstacle()
    if obstacle is not None:
        raise RuntimeError(f"the native autograd nodes cannot be built: {obstacle}")
    import torch

    out = autograd_module_path()
    if not force and autograd_module_current():
        return out
    torch_dir = Path(torch.__file__).parent
    cuda_home = Path(os.environ.get("CUDA_HOME", "/usr/local/cuda"))
    cmd = [_host_cxx(), "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", "-DTORCH_EXTENSION_NAME=_autograd",
           f'-DTFT_TORCH_MARK="{_torch_mark(torch.__version__)}"',
           "-DTORCH_API_INCLUDE_EXTENSION_H", "-I", str(torch_dir / "include"),
           "-I", str(torch_dir / "include" / "torch" / "csrc" / "api" / "include"), "-I", str(cuda_home / "include"),
           "-I", sysconfig.get_paths()["include"], str(HOST_SRC / "autograd.cc"), "-o", str(out), "-L", str(torch_dir / "lib"),
           "-ltorch", "-ltorch_cpu", "-ltorch_python", "-lc10", "-lc10_cuda"]
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError(f"autograd build failed:\n{res.stdout}\n{res.stderr}")
    return out


def build_control(force: bool = False) -> Path:
    """Builds the pybind11 control-plane module and the standalone lighthouse binary."""
    import pybind11

    LIB_DIR.mkdir(parents=True, exist_ok=True)
    sources = sorted(p for p in CONTROL_SRC.glob("*.cc") if p.name not in ("lighthouse_main.cc", "stress_main.cc"))
    headers = sorted(CONTROL_SRC.glob("*.h"))
    out = control_module_path()
    newest = max(_newest(sources), _newest(headers))
    # -Bsymbolic keeps a statically linked runtime (other toolchains) from being
    # half-interposed by the process-wide one.
    cxx = _host_cxx()
    common = ["-O2", "-std=c++17", "-fPIC", "-pthread", "-Wall", "-Wno-unused-function", "-Wl,-Bsymbolic"]
    if force or not out.exists() or out.stat().st_mtime < newest:
        py_inc = sysconfig.get_paths()["include"]
        cmd = [cxx, *common, "-shared", "-fvisibility=hidden", "-I", pybind11.get_include(), "-I", py_inc,
               "-I", str(CONTROL_SRC), *map(str, sources), "-o", str(out)]
        res = subprocess.run(cmd, capture_output=True, text=True)
        if res.returncode != 0:
            raise RuntimeError(f"control build failed:\n{res.stdout}\n{res.stderr}")
    main_src = CONTROL_SRC / "lighthouse_main.cc"
    exe = lighthouse_bin_path()
    if main_src.exists() and (force or not exe.exists() or exe.stat().st_mtime < max(newest, main_src.stat().st_mtime)):
        lib_sources = [str(p) for p in sources if p.name != "bindings.cc"]
        cmd = [cxx, *common, "-I", str(CONTROL_SRC), str(main_src), *lib_sources, "-o", str(exe)]
        res = subprocess.run(cmd, capture_output=True, text=True)
        if res.returncode != 0:
            raise RuntimeError(f"lighthouse binary build failed:\n{res.stdout}\n{res.stderr}")
    return out


def build_all(force: bool = False, verbose: bool = False) -> None:
    build_control(force=force)
    build_kernels(force=force, verbose=verbose)
    build_autograd(force=force)


if __name__ == "__main__":
    build_all(force="--force" in sys.argv, verbose="-v" in sys.argv)
    print("built", kernels_lib_path(), control_module_path(), autograd_module_path())

"""Builds and loads the CUDA kernel libraries.

Every `<name>.cu` beside this file is one shared library with a plain C interface
(`extern "C"` functions taking device pointers, sizes and a stream), compiled by nvcc for
sm_100a only and loaded with ctypes. A library is compiled the first time something asks
for it, so a run compiles what its model needs and nothing else; `build_all()` compiles
everything. A built file is named by a hash of its source, the shared headers and the
compiler flags, so an edited source is never served by a stale binary.

Built files go to `_build/` beside the sources when that folder can be written, else to
`$QWENFORGE_B200_BUILD_DIR`, else to a per-user folder under the system's temporary
directory. Nothing here needs HOME or a network.

One source, `host.cpp`, is a Python module instead (`host_module()`): it launches the others' kernels from native code. It is built the
same way, against the headers of the torch in use, whose version is part of its name.

There is no fallback: if nvcc is missing or a compilation fails, `KernelLibraryError`
says which file and why, and nothing runs. `host.cpp` alone can be done without: it needs Python's and torch's C++ headers, which a
machine with nvcc may lack, and what it launches can be launched one by one (`ops/host.py`).
"""
from __future__ import annotations

import ctypes
import hashlib
import os
import shutil
import subprocess
import sys
import tempfile
import threading
import time
from concurrent.futures import ThreadPoolExecutor
from pathlib import Path

_SRC = Path(__file__).resolve().parent
_NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-lineinfo", "-std=c++17",
    "-Xcompiler", "-fPIC", "-shared",
]
_HOST = "host"           # the one source that is a Python module
_loaded: dict[str, ctypes.CDLL] = {}
_modules: dict = {}
_unavailable: dict = {}  # what was tried and could not be had, and why: not tried again in this process
_lock = threading.Lock()


class KernelLibraryError(RuntimeError):
    pass


def library_names() -> list[str]:
    return sorted([p.stem for p in _SRC.glob("*.cu")] + [_HOST])


def _source(name: str) -> Path:
    return _SRC / f"{name}.{'cpp' if name == _HOST else 'cu'}"


def _flags(name: str) -> list[str]:
    """What makes a build what it is; where the headers and libraries lie is `_places`' part."""
    if name != _HOST:
        return _NVCC_FLAGS
    import torch
    return ["-O2", "-std=c++17", "-Xcompiler", "-fPIC", "-shared", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
            "-ltorch_python", "-ltorch_cpu", "-lc10", "-lc10_cuda"]


def _places(name: str) -> list[str]:
    if name != _HOST:
        return ["-I", str(_SRC)]
    import sysconfig

    import torch
    root = Path(torch.__file__).resolve().parent
    return ["-I", sysconfig.get_paths()["include"], "-I", str(root / "include"), "-I", str(root / "include/torch/csrc/api/include"),
            "-L", str(root / "lib")]


def _say(message: str) -> None:
    print(f"[qwenforge_b200] {message}", file=sys.stderr, flush=True)


def _nvcc() -> str:
    candidates = [os.environ.get("QWENFORGE_B200_NVCC"), shutil.which("nvcc")]
    for home in (os.environ.get("CUDA_HOME"), os.environ.get("CUDA_PATH"), "/usr/local/cuda"):
        if home:
            candidates.append(str(Path(home) / "bin" / "nvcc"))
    for c in candidates:
        if c and Path(c).exists():
            return c
    raise KernelLibraryError("nvcc not found (looked in PATH, $CUDA_HOME and /usr/local/cuda): the CUDA kernels of "
                             "this library cannot be built, and there is no other execution path")


def _writable(folder: Path) -> bool:
    try:
        folder.mkdir(parents=True, exist_ok=True)
        probe = folder / f".probe-{os.getpid()}-{threading.get_ident()}"
        probe.write_bytes(b"")
        probe.unlink()
        return True
    except OSError:
        return False


def _build_dir() -> Path:
    choices = [_SRC / "_build"]
    if os.environ.get("QWENFORGE_B200_BUILD_DIR"):
        choices.append(Path(os.environ["QWENFORGE_B200_BUILD_DIR"]))
    choices.append(Path(tempfile.gettempdir()) / f"qwenforge_b200-build-{os.getuid()}")
    for c in choices:
        if _writable(c):
            return c
    raise KernelLibraryError(f"no writable folder for built kernels (tried {', '.join(map(str, choices))})")


def _digest(name: str) -> str:
    h = hashlib.sha256()
    if name == _HOST:
        import torch
        h.update(f"{torch.__version__} {sys.version} ".encode())
    h.update(" ".join(_flags(name)).encode())
    shared = [] if name == _HOST else sorted(_SRC.glob("*.cuh")) + sorted(_SRC.glob("*.h"))
    for path in shared + [_source(name)]:
        h.update(path.name.encode())
        h.update(path.read_bytes())
    return h.hexdigest()[:16]


def _find_built(name: str, digest: str) -> Path | None:
    file_name = f"{name}.{digest}.so"
    places = [_SRC / "_build"]
    if os.environ.get("QWENFORGE_B200_BUILD_DIR"):
        places.append(Path(os.environ["QWENFORGE_B200_BUILD_DIR"]))
    places.append(Path(tempfile.gettempdir()) / f"qwenforge_b200-build-{os.getuid()}")
    for p in places:
        if (p / file_name).exists():
            return p / file_name
    return None


def _compile(name: str) -> Path:
    source = _source(name)
    if not source.exists():
        raise KernelLibraryError(f"no kernel source {source.name}; known: {', '.join(library_names())}")
    digest = _digest(name)
    built = _find_built(name, digest)
    if built is not None:
        return built
    out_dir = _build_dir()
    target = out_dir / f"{name}.{digest}.so"
    partial = out_dir / f".{name}.{digest}.{os.getpid()}.{threading.get_ident()}.tmp.so"
    command = [_nvcc(), *_places(name), *_flags(name), "-o", str(partial), str(source)]
    _say(f"compiling {source.name} for sm_100a ...")
    started = time.time()
    env = dict(os.environ)
    env.setdefault("TMPDIR", str(out_dir))
    process = subprocess.Popen(command, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True, env=env)
    while True:
        try:
            output, _ = process.communicate(timeout=15)
            break
        except subprocess.TimeoutExpired:
            _say(f"still compiling {source.name} ({time.time() - started:.0f} s)")
    if process.returncode != 0:
        partial.unlink(missing_ok=True)
        raise KernelLibraryError(f"nvcc failed on {source.name} (exit {process.returncode}):\n{output}")
    os.replace(partial, target)
    for stale in out_dir.glob(f"{name}.*.so"):  # builds of earlier versions of this source
        if stale != target:
            stale.unlink(missing_ok=True)
    _say(f"compiled {source.name} in {time.time() - started:.1f} s")
    return target


def library(name: str) -> ctypes.CDLL:
    """The loaded library `name` (compiling it first if no current build exists)."""
    lib = _loaded.get(name)
    if lib is not None:
        return lib
    with _lock:
        lib = _loaded.get(name)
        if lib is None:
            path = _compile(name)
            try:
                lib = ctypes.CDLL(str(path))
            except OSError as exc:
                raise KernelLibraryError(f"cannot load {path}: {exc}") from exc
            _loaded[name] = lib
    return lib


def host_module():
    """The module of `host.cpp` (compiling it first if no current build exists); a kernel library's address is handed to it by whoever
    loads one (`ops/host.py`). `KernelLibraryError` where it cannot be built or loaded, at every call and tried once."""
    module = _modules.get(_HOST)
    if module is None:
        with _lock:
            module = _modules.get(_HOST)
            if module is None:
                if _HOST in _unavailable:
                    raise KernelLibraryError(_unavailable[_HOST])
                try:
                    module = _modules[_HOST] = _load_module(_compile(_HOST))
                except KernelLibraryError as exc:
                    _unavailable[_HOST] = str(exc)
                    _say(f"no native launches of prompt steps (they only save time): {exc}")
                    raise
    return module


def _load_module(path: Path):
    import importlib.machinery
    import importlib.util

    import torch  # noqa: F401  (its libraries are what the module is linked against)
    loader = importlib.machinery.ExtensionFileLoader("qf_host", str(path))
    try:
        module = importlib.util.module_from_spec(importlib.util.spec_from_file_location("qf_host", str(path), loader=loader))
        loader.exec_module(module)
    except ImportError as exc:
        raise KernelLibraryError(f"cannot load {path}: {exc}") from exc
    return module


def prepare(names) -> None:
    """Compile (in parallel) and load the named libraries; used when a model is built, so
    that all compilation happens up front with progress lines instead of inside the first step. The one that can be done without is
    left out where it cannot be had (`host_module` says so)."""
    todo = [n for n in sorted(set(names)) if n not in _loaded and n not in _modules and n not in _unavailable]
    if not todo:
        return

    def host() -> None:
        try:
            host_module()
        except KernelLibraryError:
            pass

    missing = [n for n in todo if _find_built(n, _digest(n)) is None]
    if missing:
        _say(f"{len(missing)} kernel librar{'y' if len(missing) == 1 else 'ies'} to compile: {', '.join(missing)}")
        with ThreadPoolExecutor(max_workers=min(8, len(missing))) as pool:
            list(pool.map(lambda n: host() if n == _HOST else _compile(n), missing))
    for n in todo:
        host() if n == _HOST else library(n)


def build_all() -> list[str]:
    names = library_names()
    prepare(names)
    host_module()   # (whoever builds everything hears of it)
    return names

"""Builds libsage_b200.so in-tree with nvcc for sm_100a (cross-compiles without a GPU), and
`_native.so`, the torch side of its operators in C++, with the host compiler.

    python -m sage_b200.build [--force] [--verbose]

One object per source, compiled side by side; only what changed is compiled again.

No fast-math: the dense dequantisation must round exactly like the reference
(its `_C` target is also built without fast-math, CMakeLists.txt:36-41,52-53 there).
"""

from __future__ import annotations

import argparse
import concurrent.futures
import os
import pathlib
import shutil
import subprocess
import sys
import sysconfig

PACKAGE = pathlib.Path(__file__).resolve().parent
CSRC = PACKAGE / "csrc"
LIBRARY = PACKAGE / "libsage_b200.so"
TRACE_LIBRARY = PACKAGE / "libsage_b200_trace.so"
NATIVE = PACKAGE / "_native.so"
OBJECTS = PACKAGE / "_obj"
INCLUDE = PACKAGE.parent / "include"

NVCC_FLAGS = [
    "-O3",
    "-std=c++17",
    "-gencode",
    "arch=compute_100a,code=sm_100a",
    "-lineinfo",
    "-Xcompiler",
    "-fPIC",
    "-Xptxas",
    "-v",
]


def sources() -> list[pathlib.Path]:
    return sorted(CSRC.glob("*.cu"))


def _nvcc() -> str:
    for candidate in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if candidate and pathlib.Path(candidate).exists():
            return candidate
    raise RuntimeError("nvcc not found; libsage_b200.so cannot be built")


def _inputs() -> list[pathlib.Path]:
    headers = list(CSRC.glob("*.h")) + list(CSRC.glob("*.cuh")) + list(INCLUDE.glob("*.h"))
    return headers + [pathlib.Path(__file__)]


def _older(target: pathlib.Path, inputs: list[pathlib.Path]) -> bool:
    if not target.exists():
        return True
    built = target.stat().st_mtime
    return any(path.stat().st_mtime > built for path in inputs)


def _library_stale() -> bool:
    return _older(LIBRARY, [*sources(), *_inputs()])


def _native_stale() -> bool:
    """Older than its sources, or not to be had by a fresh interpreter: torch's C++ interface has no stable ABI, so a
    module that another torch version was built against may miss symbols, or worse, find them."""
    if _older(NATIVE, [CSRC / "torch_ops.cpp", *_inputs()]):
        return True
    check = f"from {PACKAGE.name} import _lib; _lib._import_native()"
    return subprocess.run([sys.executable, "-c", check], cwd=PACKAGE.parent, capture_output=True).returncode != 0


def is_stale() -> bool:
    return _library_stale() or _native_stale()


def _run(command: list[str], what: str, verbose: bool) -> str:
    result = subprocess.run(command, capture_output=True, text=True)
    if verbose or result.returncode:
        sys.stderr.write(" ".join(command) + "\n" + result.stdout + result.stderr)
    if result.returncode:
        raise RuntimeError(f"{command[0]} failed building {what}")
    return result.stdout + result.stderr


def _build_native(verbose: bool) -> None:
    """`_native.so`: a Python extension module over torch's C++ headers.  It is not linked against
    libsage_b200.so: the ctypes binding hands it the addresses of the functions it calls."""
    import torch

    root = pathlib.Path(torch.__file__).resolve().parent
    includes = [root / "include", root / "include" / "torch" / "csrc" / "api" / "include",
                pathlib.Path(_nvcc()).resolve().parent.parent / "include", sysconfig.get_paths()["include"]]
    command = [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-shared", "-fPIC",
               f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
               f'-DSAGEB200_TORCH_VERSION="{torch.__version__}"']
    for path in includes:
        command += ["-isystem", str(path)]
    command += [str(CSRC / "torch_ops.cpp"), "-o", str(NATIVE), f"-L{root / 'lib'}",
                "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch", "-ltorch_python"]
    _run(command, NATIVE.name, verbose)


def build(force: bool = False, verbose: bool = False, trace: bool = False) -> pathlib.Path:
    """Compile every .cu under csrc/ into one shared library; returns its path.  `trace` adds
    -DSAGEB200_TRACE: the decode kernel's phase clocks (sageb200_debug_trace) and the
    SAGEB200_PATHS switch, both compiled out of the default build."""
    native_stale = not trace and (force or _native_stale())
    if not force and not trace and not native_stale and not _library_stale():
        return LIBRARY
    flags = NVCC_FLAGS + (["-DSAGEB200_TRACE"] if trace else [])
    # the profiling build goes beside the product library (select it with SAGEB200_LIBRARY)
    target = TRACE_LIBRARY if trace else LIBRARY
    objects = OBJECTS / ("trace" if trace else "product")
    objects.mkdir(parents=True, exist_ok=True)

    def compile_one(source: pathlib.Path) -> tuple[pathlib.Path, str]:
        out, log = objects / (source.stem + ".o"), objects / (source.stem + ".log")
        if force or _older(out, [source, *_inputs()]):
            command = [_nvcc(), *flags, f"-I{INCLUDE}", "-c", "-o", str(out), str(source)]
            log.write_text(_run(command, source.name, verbose))
        return out, log.read_text()

    with concurrent.futures.ThreadPoolExecutor(max_workers=os.cpu_count() or 4) as pool:
        native = pool.submit(_build_native, verbose) if native_stale else None
        done = list(pool.map(compile_one, sources()))
        if native is not None:
            native.result()
    command = [_nvcc(), "-gencode", "arch=compute_100a,code=sm_100a", "-shared", "-o", str(target),
               *(str(out) for out, _ in done)]
    log = "".join(text for _, text in done) + _run(command, target.name, verbose)
    if not trace:
        (PACKAGE / "build_log.txt").write_text(log)
    return target


if __name__ == "__main__":
    parser = argparse.ArgumentParser()
    parser.add_argument("--force", action="store_true")
    parser.add_argument("--verbose", action="store_true")
    parser.add_argument("--trace", action="store_true", help="profiling build (-DSAGEB200_TRACE)")
    args = parser.parse_args()
    print(build(force=args.force, verbose=args.verbose, trace=args.trace))

"""CPU: the build entry point from an empty tree, and what a process sees that imported the package before it."""

import pathlib
import shutil
import subprocess
import sys

import pytest

ROOT = pathlib.Path(__file__).resolve().parent.parent
SOURCES = ("__graft_entry__.py", "sage_b200", "oracle", "include")


def run(script: str, tree: pathlib.Path) -> str:
    done = subprocess.run([sys.executable, "-c", script], cwd=tree, capture_output=True, text=True)
    assert done.returncode == 0, done.stdout + done.stderr
    return done.stdout


@pytest.fixture(scope="module")
def unbuilt(tmp_path_factory):
    """The sources of the package without anything that a build writes."""
    tree = tmp_path_factory.mktemp("unbuilt")
    built = shutil.ignore_patterns("*.so", "*.o", "_obj", "_ref", "__pycache__", "build_log.txt")
    for name in SOURCES:
        source = ROOT / name
        if source.is_dir():
            shutil.copytree(source, tree / name, ignore=built)
        else:
            shutil.copy(source, tree / name)
    return tree


BEFORE = """
import torch
import sage_b200
from sage_b200 import SAGELinear, _lib, synthetic_sage

packed = synthetic_sage(128, 16, seed=0)
linear, x = SAGELinear(packed, 16), torch.zeros(1, 128, dtype=torch.float16)

def missing(call):
    try:
        call()
    except RuntimeError as error:
        assert "python -m sage_b200.build" in str(error), error
    else:
        raise AssertionError("an unbuilt tree served a call")
"""


def test_unbuilt_tree_says_how_to_build_it(unbuilt):
    run(BEFORE + """
missing(_lib.load)
missing(_lib.native_module)
missing(lambda: linear(x))
missing(lambda: sage_b200.sage(x, *packed.values(), 16))
missing(lambda: sage_b200.sage_forward(x, *packed.values(), 16))
meta = [value.to("meta") for value in packed.values()]
assert sage_b200.sage(x.to("meta"), *meta, 16).shape == (1, 16)  # (shapes need no build)
""", unbuilt)


def test_one_process_imports_builds_and_runs(unbuilt):
    """One call of the entry point in a tree that holds sources only, by a process that had already imported the
    package and met its errors; afterwards that process reaches the operators' C++ checks."""
    run(BEFORE + """
missing(lambda: linear(x))
import __graft_entry__
__graft_entry__.build()

def cuda_only(call, kind, text):
    try:
        call()
    except kind as error:
        assert text in str(error), error
    else:
        raise AssertionError("a CPU call was served")

native = "SAGE requires contiguous CUDA FP16 input"
cuda_only(lambda: sage_b200.sage_forward(x, *packed.values(), 16), RuntimeError, native)
cuda_only(lambda: linear(x), NotImplementedError, "CUDA")
cuda_only(lambda: sage_b200.sage(x, *packed.values(), 16), NotImplementedError, "CUDA")
assert torch._C._dispatch_has_kernel_for_dispatch_key(sage_b200.sage.name(), "CUDA")
assert torch._C._dispatch_has_kernel_for_dispatch_key(sage_b200.sage.name(), "AutogradCUDA")
assert torch._C._dispatch_has_kernel_for_dispatch_key(sage_b200.sphquant.name(), "CUDA")
""", unbuilt)
    # an interpreter that imports the package, and one that loads it
    maps = "print(sum('sage_b200' in line and '.so' in line for line in open('/proc/self/maps')))"
    assert run(f"import sage_b200\n{maps}", unbuilt).strip() == "0"
    assert int(run(f"from sage_b200 import _lib\n_lib.load()\n{maps}", unbuilt)) > 0


@pytest.fixture
def built(tmp_path):
    """The package with its built files, newer than every source."""
    from sage_b200 import build

    build.build()
    shutil.copytree(ROOT / "sage_b200", tmp_path / "sage_b200", ignore=shutil.ignore_patterns("_obj", "__pycache__"))
    shutil.copytree(ROOT / "include", tmp_path / "include")
    for name in ("libsage_b200.so", "_native.so"):
        (tmp_path / "sage_b200" / name).touch()
    return tmp_path


STALE = "from sage_b200 import build; print(build._native_stale())"


def test_a_module_that_does_not_import_says_why_and_is_built_again(built):
    assert run(STALE, built).strip() == "False"
    (built / "sage_b200" / "_native.so").write_bytes(b"not a shared object")
    run("""
from sage_b200 import _lib
try:
    _lib.load()
except ImportError as error:  # the loader's own words, not "missing"
    assert "missing" not in str(error) and "_native.so" in str(error), error
else:
    raise AssertionError("loaded")
""", built)
    assert run(STALE, built).strip() == "True"


def test_a_module_of_another_torch_version_is_refused(built):
    run("""
import torch
torch.__version__ = "0.0"  # as if torch had been exchanged after the build
from sage_b200 import _lib
try:
    _lib._import_native()  # (what the build's check of an existing module calls as well)
except RuntimeError as error:
    assert "torch 0.0" in str(error) and "python -m sage_b200.build" in str(error), error
else:
    raise AssertionError("loaded")
""", built)

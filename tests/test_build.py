"""The build from nothing: a checkout without ``lib/`` can import the package and run its build.  The compilers are stand-ins that
only write their output files, so that the test is about the Python around them."""
import os
import shutil
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _compilers(folder):
    """nvcc and g++ that write a line to the file behind -o and say so; returns the environment that finds them."""
    folder.mkdir()
    for name in ("nvcc", "g++"):
        tool = folder / name
        tool.write_text('#!/bin/sh\nwhile [ "$1" != "-o" ]; do shift; done\necho built > "$2"\n')
        tool.chmod(0o755)
    return {**os.environ, "NVCC": str(folder / "nvcc"), "PATH": f"{folder}{os.pathsep}{os.environ['PATH']}", "PYTHONDONTWRITEBYTECODE": "1"}


@pytest.fixture
def checkout(tmp_path):
    """The sources of the package as a fresh clone has them."""
    root = tmp_path / "checkout"
    skip = shutil.ignore_patterns("lib", "build", "__pycache__", "*.so")
    for name in ("lisa_b200", "include", "oracle"):
        shutil.copytree(os.path.join(ROOT, name), root / name, ignore=skip)
    shutil.copy(os.path.join(ROOT, "__graft_entry__.py"), root)
    return root


def _python(root, *args, env=None):
    return subprocess.run([sys.executable, *args], cwd=root, env={**(env or os.environ), "PYTHONPATH": str(root)}, capture_output=True, text=True, timeout=300)


def test_build_from_a_clean_checkout(checkout, tmp_path):
    res = _python(checkout, "-m", "lisa_b200.build", env=_compilers(tmp_path / "bin"))
    assert res.returncode == 0, res.stderr
    assert (checkout / "lisa_b200" / "lib" / "liblisa_cuda.so").exists() and (checkout / "lisa_b200" / "lib" / "_lisa_torch.so").exists()


def test_import_without_a_library_and_a_call_says_what_is_missing(checkout):
    res = _python(checkout, "-c", "import lisa_b200, torch\n"
                                  "try:\n    lisa_b200.ops.quantized_matmul(torch.zeros(1), None, None, None)\n"
                                  "except RuntimeError as e:\n    print('said:', e)")
    assert res.returncode == 0, res.stderr
    assert "said:" in res.stdout and "python -m lisa_b200.build" in res.stdout

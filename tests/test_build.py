"""The build from nothing: a checkout without ``lib/`` can import the package and run its build.  The compilers are stand-ins that
only write their output files, so that the test is about the Python around them."""
import os
import shutil
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _compilers(folder):
    """nvcc and g++ that write a line to the file behind -o; returns the environment that finds them.  What links a library copies
    `$REAL_LIB` instead where that is given, as a new file with a mark at its end."""
    folder.mkdir()
    for name in ("nvcc", "g++"):
        tool = folder / name
        tool.write_text('#!/bin/sh\nwhile [ "$1" != "-o" ]; do shift; done\n'
                        'case "$2" in *.so) if [ -n "$REAL_LIB" ]; then cp "$REAL_LIB/$(basename "$2")" "$2.new"; mv "$2.new" "$2"; fi;; esac\n'
                        'echo built >> "$2"\n')
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


@pytest.fixture
def older(checkout, tmp_path):
    """A checkout with a built library, one of whose sources has changed since; and its environment."""
    lib = os.path.join(ROOT, "lisa_b200", "lib")
    if not os.path.exists(os.path.join(lib, "_lisa_torch.so")):
        pytest.skip("the library is not built")
    env = {**_compilers(tmp_path / "bin"), "REAL_LIB": lib}
    res = _python(checkout, "-m", "lisa_b200.build", env=env)
    assert res.returncode == 0, res.stderr
    with open(checkout / "lisa_b200" / "csrc" / "api.cu", "a") as f:
        f.write("// a change\n")
    return checkout, env


def test_entry_point_loads_the_library_that_it_built(older):
    root, env = older
    before = os.stat(root / "lisa_b200" / "lib" / "liblisa_cuda.so").st_ino
    res = _python(root, "-c", "import __graft_entry__ as entry, lisa_b200\nentry.build()\nlisa_b200.native.ext.moe_block\n"
                              "print(*{line.split()[4] + ' ' + line.split(maxsplit=5)[5].strip() for line in open('/proc/self/maps') if 'lisa_b200/lib' in line}, sep='\\n')", env=env)
    assert res.returncode == 0, res.stderr
    mapped = dict(reversed(line.split(maxsplit=1)) for line in res.stdout.splitlines() if "lisa_b200/lib" in line)
    assert len(mapped) == 2 and not any("deleted" in name for name in mapped), mapped
    for name, inode in mapped.items():
        assert os.stat(name).st_ino == int(inode) and (int(inode) != before or "liblisa_cuda" not in name)


def test_build_refuses_to_replace_a_loaded_library(older):
    root, env = older
    res = _python(root, "-c", "from lisa_b200 import _cabi, build\n_cabi.lib()\nbuild.build()", env=env)
    assert res.returncode != 0 and "already loaded" in res.stderr, res.stderr


def test_a_copy_of_a_built_tree_is_built(older, tmp_path):
    root, env = older
    assert _python(root, "-m", "lisa_b200.build", env=env).returncode == 0
    shutil.copytree(root, tmp_path / "copy")
    res = _python(tmp_path / "copy", "-c", "import lisa_b200.build as b\nb._compile = None\nb.build()", env=env)
    assert res.returncode == 0, res.stderr


def test_another_torch_or_compiler_line_builds_anew(older):
    root, env = older
    code = ("import torch, lisa_b200.build as b\nb._compile = lambda *a: built.append(a) or '/dev/null'\nbuilt = []\n{}\nb.build()\n"
            "assert not built, 'built without a change'\n{}\nb.build()\nassert built, 'not built'")
    for change in ("torch.__version__ += 'x'", "line = b._torch_command()\nb._torch_command = lambda: [*line, '-O1']", "b.NVCC_FLAGS.append('-O2')"):
        res = _python(root, "-c", code.format("b.build()\nbuilt.clear()", change), env=env)
        assert res.returncode == 0, res.stderr

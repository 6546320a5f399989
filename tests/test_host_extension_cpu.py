"""A host extension that is missing or does not load is reported; a tree in which nothing is built still constructs quantizers."""
import os
import shutil
import subprocess
import sys

import pytest

PACKAGE = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "var-q_b200", "VAR_Q")


def run_in_copy(tmp_path, files, code):
    """`code` in a process that sees a copy of the package's Python files and, as its binaries, `files` (name -> bytes)"""
    target = tmp_path / "VAR_Q"
    target.mkdir()
    for name in os.listdir(PACKAGE):
        if name.endswith(".py"):
            shutil.copy(os.path.join(PACKAGE, name), target)
    for name, content in files.items():
        (target / name).write_bytes(content)
    return subprocess.run([sys.executable, "-c", code], cwd=tmp_path, capture_output=True, text=True, env={**os.environ, "PYTHONPATH": str(tmp_path)})


@pytest.mark.parametrize("files", [{"libvarq_b200.so": b"", "_host.so": b"built against another torch"}, {"libvarq_b200.so": b""}])
def test_a_library_without_a_host_extension_that_loads_is_an_error(tmp_path, files):
    res = run_in_copy(tmp_path, files, "import VAR_Q.quant")
    assert res.returncode != 0 and "ImportError" in res.stderr and "_host.so" in res.stderr and "build.py" in res.stderr, res.stderr


def test_without_any_binary_quantizers_are_built_and_device_calls_say_what_is_missing(tmp_path):
    res = run_in_copy(tmp_path, {}, "from VAR_Q.quant import VAR_Q\nfrom VAR_Q import _cabi\nassert VAR_Q(quant_bits=4).bound_max == 7\n_cabi.lib()")
    assert res.returncode != 0 and "libvarq_b200.so is missing" in res.stderr, res.stderr

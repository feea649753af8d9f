"""The operators' native call path is found for the interpreter and the torch it was built for, and the package works without it."""
import os
import shutil
import subprocess
import sys
import sysconfig

import pytest
import torch

import wuda_b200
from wuda_b200 import native_calls


def test_name_says_what_it_was_built_for(monkeypatch):
    name = native_calls.file_name()
    assert torch.__version__ in name and sysconfig.get_config_var("SOABI") in name
    assert os.path.exists(os.path.join(native_calls.HERE, name)) and wuda_b200._fast.__file__.endswith(name)
    monkeypatch.setattr(torch, "__version__", "2.0.0")
    assert native_calls.file_name() != name


@pytest.mark.parametrize("there", ["nothing", "another torch's", "one that does not load", "one of an earlier build"])
def test_package_without_it(tmp_path, there):
    package = tmp_path / "wuda_b200"
    shutil.copytree(native_calls.HERE, package, ignore=lambda d, names: [n for n in names if n.endswith(".so") or n in ("build", "csrc")])
    os.symlink(os.path.join(native_calls.HERE, "libwuda_b200.so"), package / "libwuda_b200.so")
    name = {"another torch's": "_fast.cpython-310-torch2.0.0-abi1.so", "one that does not load": native_calls.file_name(),
            "one of an earlier build": "_fast.so"}.get(there)
    if name:
        (package / name).write_bytes(b"\x7fELF, but no more of it")
    said = subprocess.run([sys.executable, "-W", "always", "-c", """
import torch, wuda_b200 as w
assert w.ops._fast.topk(1, 2, 3, 4, 5, 6, 7) is None
try:
    w.rmsnorm_quant(torch.zeros(2, 256), None)
except w.WudaError as e:
    print("refused:", e)
"""], cwd=tmp_path, capture_output=True, text=True, env=dict(os.environ, PYTHONPATH=str(tmp_path)))
    assert said.returncode == 0, said.stderr
    assert "refused: " in said.stdout and "native call path is not there" in said.stderr and "wuda_b200.build" in said.stderr

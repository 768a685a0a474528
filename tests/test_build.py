"""CPU: what the compiler makes of the kernels."""
import os
import re
import shutil
import subprocess
import warnings
from importlib import import_module
from types import SimpleNamespace

import pytest
import torch

from .conftest import PKG_NAME, ROOT, load_pkg


@pytest.mark.skipif(shutil.which("nvcc") is None, reason="no nvcc")
def test_few_rows_kernels_do_not_spill(tmp_path):
    """Their epilogues hold whole accumulators in registers: an instantiation that spills them is slower than one that reads
    and writes a group at a time (gate/up of 9000 rows 164 against 146 us)."""
    src = os.path.join(ROOT, PKG_NAME, "csrc", "gemm_few.cu")
    res = subprocess.run(["nvcc", "-O3", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-Xcompiler", "-fPIC", "-Xptxas", "-v",
                          "-c", src, "-o", str(tmp_path / "few.o")], capture_output=True, text=True)
    assert res.returncode == 0, res.stderr[-2000:]
    spills = re.findall(r"Function properties for (\S+)\n\s*(\d+) bytes stack frame, (\d+) bytes spill stores, (\d+) bytes spill loads", res.stderr)
    few = [s for s in spills if "few_rows_kernel" in s[0]]
    assert len(few) >= 7 and all(s[1:] == ("0", "0", "0") for s in spills), spills


def _script(path, text):
    path.write_text(text)
    path.chmod(0o755)
    return str(path)


def test_make_targets(tmp_path):
    """An interpreter without torch builds the library and no more; one with torch builds the module too, once, and again for another
    torch.  Compilers are scripts that note what they write."""
    csrc = tmp_path / "pkg" / "csrc"
    shutil.copytree(os.path.join(ROOT, PKG_NAME, "csrc"), csrc, ignore=shutil.ignore_patterns("build"))
    shutil.copytree(os.path.join(ROOT, "include"), tmp_path / "include")
    log, torch_dir = tmp_path / "log", tmp_path / "torch"
    torch_dir.mkdir()
    (torch_dir / "version.py").write_text("__version__ = '1'")
    tool = _script(tmp_path / "cc", f'#!/bin/sh\nwhile [ "$1" != -o ]; do shift; done\necho "$2" >> {log}\ntouch "$2"\n')
    with_torch = _script(tmp_path / "py", f'#!/bin/sh\ncase "$1" in -c) echo {torch_dir};; -VV) echo Python;; *) echo;; esac\n')
    without = _script(tmp_path / "py0", '#!/bin/sh\nexit 1\n')

    def make(python, *targets):
        log.write_text("")
        res = subprocess.run(["make", "-s", "-C", str(csrc), f"NVCC={tool}", f"CXX={tool}", f"PYTHON={python}", *targets], capture_output=True, text=True)
        assert res.returncode == 0, res.stderr
        return [os.path.basename(f) for f in log.read_text().split()]

    made = make(without)
    assert "libb200moe.so" in made and "_fast.so" not in made
    assert make(with_torch, "lib") == []
    assert make(with_torch) == ["_fast.so"] and make(with_torch) == []
    (torch_dir / "version.py").write_text("__version__ = '2'")
    assert make(with_torch) == ["_fast.so"] and make(with_torch) == []


@pytest.mark.parametrize("why", ["is missing", "was built for torch 0.0", "cannot be loaded"])
def test_a_missing_or_foreign_fast_module_leaves_the_python_functions(tmp_path, monkeypatch, why):
    load_pkg()
    L = import_module(PKG_NAME + "._lib")
    path = tmp_path / "_fast.so"

    def load(*_):
        if "loaded" in why:
            raise ImportError("undefined symbol")
        return SimpleNamespace(torch_version="0.0")

    if "missing" not in why:
        path.touch()
    monkeypatch.setattr(L, "_fast", None)
    monkeypatch.setattr(L, "FAST_PATH", str(path))
    monkeypatch.setattr(L.importlib, "import_module", load)
    with pytest.warns(RuntimeWarning, match=why):
        assert L.fast() is None
    with warnings.catch_warnings():
        warnings.simplefilter("error")
        assert L.fast() is None      # said once


def test_the_fast_module_that_was_built_fits():
    pkg = load_pkg()
    L = import_module(PKG_NAME + "._lib")
    pkg.build()
    assert L.fast().torch_version == torch.__version__.split("+")[0]

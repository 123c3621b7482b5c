"""The build script: what each kind of host gets from it."""
from __future__ import annotations

import os
import shutil
import subprocess
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _copy(tmp_path):
    """The package and the header as they are, time stamps and all: what is built is not built again."""
    for d in ("comfyui-backend-but-rust_b200", "include"):
        shutil.copytree(os.path.join(ROOT, d), tmp_path / d, ignore=shutil.ignore_patterns("__pycache__"))
    return os.path.join(tmp_path, "comfyui-backend-but-rust_b200")


def _run(args, cwd, **env):
    return subprocess.run([sys.executable] + args, cwd=cwd, env={**os.environ, **env}, capture_output=True, text=True, timeout=900)


def test_the_c_library_builds_without_torch(tmp_path):
    """A Rust or C host runs the same script; without torch it gets the shared and the static library and a note."""
    there = _copy(tmp_path)
    (tmp_path / "stub").mkdir()
    (tmp_path / "stub" / "torch.py").write_text("raise ImportError('not on this host')\n")
    r = _run([os.path.join(there, "build.py")], tmp_path, PYTHONPATH=str(tmp_path / "stub"))
    assert r.returncode == 0, r.stderr
    assert r.stdout.strip().endswith("libb200_qlinear.so") and "left out" in r.stderr
    assert os.path.exists(os.path.join(there, "libb200_qlinear.a"))
    r = _run([os.path.join(there, "build.py"), "--c-only"], tmp_path)
    assert r.returncode == 0 and r.stdout.strip().endswith("libb200_qlinear.so"), r.stderr


def test_an_extension_of_another_interpreter_or_torch_is_built_again(tmp_path):
    """Two pythons or two torches of one version may share a checkout: the extension is bound to one of them."""
    from types import SimpleNamespace

    import torch

    from __graft_entry__ import _load_file
    b = _load_file("build_under_test", os.path.join(ROOT, "comfyui-backend-but-rust_b200", "build.py"))
    here = b._host_ops_stamp(torch)
    assert here == b._host_ops_stamp(torch) and sys.implementation.cache_tag in here
    other = SimpleNamespace(__version__=torch.__version__, __file__=str(tmp_path / "torch" / "__init__.py"),
                            compiled_with_cxx11_abi=torch.compiled_with_cxx11_abi)
    assert b._host_ops_stamp(other) != here


def test_a_missing_extension_says_how_to_build_it(tmp_path):
    there = _copy(tmp_path)
    ext = os.path.join(there, "_host_ops.so")
    for broken in (b"not an extension", None):
        os.remove(ext)
        if broken:
            with open(ext, "wb") as f:
                f.write(broken)
        r = _run(["-c", "import importlib; importlib.import_module('comfyui-backend-but-rust_b200')"], tmp_path, PYTHONPATH=str(tmp_path))
        assert r.returncode != 0 and "build.py" in r.stderr.strip().splitlines()[-1], r.stderr

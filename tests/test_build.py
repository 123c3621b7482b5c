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


def _run(args, **env):
    return subprocess.run([sys.executable] + args, env={**os.environ, **env}, capture_output=True, text=True, timeout=900)


def test_the_c_library_builds_without_torch(tmp_path):
    """A Rust or C host runs the same script; without torch it gets the shared and the static library and a note."""
    there = _copy(tmp_path)
    (tmp_path / "stub").mkdir()
    (tmp_path / "stub" / "torch.py").write_text("raise ImportError('not on this host')\n")
    r = _run([os.path.join(there, "build.py")], PYTHONPATH=str(tmp_path / "stub"))
    assert r.returncode == 0, r.stderr
    assert r.stdout.strip().endswith("libb200_qlinear.so") and "left out" in r.stderr
    assert os.path.exists(os.path.join(there, "libb200_qlinear.a"))
    r = _run([os.path.join(there, "build.py"), "--c-only"])
    assert r.returncode == 0 and r.stdout.strip().endswith("libb200_qlinear.so"), r.stderr

"""CACHALOT_B200_LIB: both ways of an operator's call - ctypes and the native call path - end in the library it names."""
import os
import shutil
import subprocess
import sys
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]

CHECK = """
import cachalot_b200.ops as ops
maps = open("/proc/self/maps").read()
loaded = {l.split()[-1] for l in maps.splitlines() if l.endswith(".so") and ("cachalot_b200" in l or "libdev" in l)}
print(sorted(p.rsplit("/", 1)[-1] for p in loaded))
"""


def _run(env, code=CHECK):
    return subprocess.run([sys.executable, "-c", code], cwd=ROOT, env={**os.environ, **env}, capture_output=True, text=True)


def test_one_library_is_loaded(tmp_path):
    from cachalot_b200 import build

    dev = tmp_path / "libdev.so"
    shutil.copy(build.build(), dev)
    res = _run({"CACHALOT_B200_LIB": str(dev)})
    assert res.returncode == 0, res.stderr
    assert eval(res.stdout.splitlines()[-1]) == ["_host.so", "libdev.so"]


def test_host_module_names_no_library_of_the_package():
    """Built with or without the override it is the same file: nothing of it depends on where the library is."""
    from cachalot_b200 import build

    text = subprocess.run(["readelf", "-d", str(build.build_host())], capture_output=True, text=True, check=True).stdout
    assert "NEEDED" in text and "cachalot" not in text and "ORIGIN" not in text


def test_missing_host_module_says_how_to_build_it(tmp_path):
    shutil.copytree(ROOT / "cachalot_b200", tmp_path / "cachalot_b200", ignore=shutil.ignore_patterns("build", "_host.so", "csrc"))
    res = subprocess.run([sys.executable, "-c", "import cachalot_b200.ops"], cwd=tmp_path, capture_output=True, text=True)
    assert res.returncode != 0 and "_host.so is missing" in res.stderr and "python -m cachalot_b200.build" in res.stderr


def test_host_module_is_built_again_for_another_torch(monkeypatch):
    from cachalot_b200 import build

    build.build_host()
    ran = []
    monkeypatch.setattr(build.metadata, "version", lambda name: "0.0")
    monkeypatch.setattr(build.subprocess, "run", lambda *a, **k: ran.append(a) or subprocess.CompletedProcess(a, 1, "", "stop"))
    try:
        build.build_host()
    except RuntimeError:
        pass
    assert len(ran) == 1

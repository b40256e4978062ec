"""The build recipe (biofvm-b_b200/build.py): a change to any file that the
library includes rebuilds it, and the plain C++ headers compile on their own."""
from __future__ import annotations

import importlib.util
import re
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
CSRC = ROOT / "biofvm-b_b200" / "csrc"


@pytest.fixture(scope="module")
def recipe():
    spec = importlib.util.spec_from_file_location("bfb_build_recipe", ROOT / "biofvm-b_b200" / "build.py")
    mod = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(mod)
    return mod


def test_every_included_file_is_a_dependency(recipe):
    deps = {p.resolve() for p in recipe.dependencies()}
    assert {CSRC / s for s in recipe.SOURCES} <= deps
    for src in list(CSRC.iterdir()):
        if src.is_file():
            for name in re.findall(r'^\s*#\s*include\s+"([^"]+)"', src.read_text(), re.M):
                found = [d / name for d in (CSRC, ROOT / "include") if (d / name).exists()]
                assert found and found[0].resolve() in deps, f"{src.name} includes {name}"


@pytest.mark.parametrize("header", sorted(p.name for p in CSRC.glob("*.h")))
def test_host_headers_compile_alone(tmp_path, header):
    src = tmp_path / "alone.cpp"
    src.write_text(f'#include "{header}"\n#include "{header}"\nint main() {{ return 0; }}\n')
    r = subprocess.run(["/usr/bin/g++", "-std=c++17", "-Wall", "-Werror", "-fsyntax-only", "-I/usr/local/cuda/include",
                        f"-I{CSRC}", str(src)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr

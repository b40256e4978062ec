"""Host-to-device copies (csrc/bfb_upload.h): their sources outlive them also
where the runtime reads them as late as it may, and no other code in the
library copies from a table of its own."""
from __future__ import annotations

import re
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]
CSRC = ROOT / "biofvm-b_b200" / "csrc"


def test_sources_live_until_the_wait(tmp_path):
    exe = tmp_path / "upload_check"
    subprocess.run(["/usr/bin/g++", "-std=c++17", "-O1", "-g", "-fsanitize=address", "-Wall", "-I/usr/local/cuda/include",
                    f"-I{CSRC}", "-o", str(exe), str(ROOT / "tests" / "upload_check.cpp")], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr


def test_only_caller_buffers_are_copied_elsewhere():
    """Outside Uploads, a host-to-device copy reads the array that the caller gave (`host`)."""
    for src in CSRC.iterdir():
        if src.name == "bfb_upload.h":
            continue
        for call in re.findall(r"\w+\([^;]*?cudaMemcpyHostToDevice[^;]*;", src.read_text()):
            assert re.search(r"\bhost\b", call) and ".data()" not in call, f"{src.name}: {call}"

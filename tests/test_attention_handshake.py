"""The barriers between the warps of the attention kernels, on the CPU: the kernels' own sources
run under stand-ins for the hardware's barriers (tests/host_kernels), with schedules that hold
back each warp, the tensor pipe or the TMA unit for as long as any other can go on.  A wait that
is right only because one side is fast enough in practice misses its phase in one of them."""
import re
import shutil
import subprocess
from pathlib import Path

import pytest

HOST = Path(__file__).resolve().parent / "host_kernels"
KERNELS = Path(__file__).resolve().parent.parent / "monarch_b200" / "csrc" / "kernels"
CUDA = Path("/usr/local/cuda/include")

needs = pytest.mark.skipif(shutil.which("g++") is None or not (CUDA / "cuda.h").exists(),
                           reason="needs g++ and the CUDA headers")


def _build(tmp, source: str, text: str = None) -> Path:
    text = (KERNELS / source).read_text() if text is None else text
    # single instructions without a meaning here (register split, three-input maximum)
    text = re.sub(r"\basm(\s+volatile)?\s*\([^;]*;[^;]*\);|\basm(\s+volatile)?\s*\([^;]*\);", ";", text)
    (tmp / source).write_text(text)
    for f in ("ptx.cuh", "launch.cuh", "attention.cpp"):
        shutil.copy(HOST / f, tmp / f)
    shutil.copy(KERNELS / "mb200.h", tmp / "mb200.h")
    exe = tmp / "run"
    cmd = ["g++", "-std=c++17", "-O1", "-w", f"-I{CUDA}", "-x", "c++",
           f'-DKERNEL_SOURCE="{source}"', *(["-DBACKWARD"] if "bwd" in source else []),
           "attention.cpp", "-o", str(exe)]
    p = subprocess.run(cmd, cwd=tmp, capture_output=True, text=True)
    assert p.returncode == 0, p.stderr[-3000:]
    return exe


@needs
@pytest.mark.parametrize("source,warps", [("attn_fwd.cu", 12), ("attn_bwd.cu", 18)])
@pytest.mark.parametrize("hd", [64, 128])
def test_no_schedule_misses_a_phase(tmp_path, source, warps, hd):
    p = subprocess.run([str(_build(tmp_path, source)), str(hd), str(warps), "4"],
                       capture_output=True, text=True, timeout=240)
    assert p.returncode == 0, p.stdout

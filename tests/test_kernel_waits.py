"""The waits inside pipelined kernels, on the CPU: the kernels' own sources run under stand-ins for
the hardware's barriers (tests/host_kernels), with schedules that hold back each warp, the tensor
pipe or the TMA unit for as long as any other can go on.  A wait that is right only because one
side is fast enough in practice misses its phase in one of them.  The launches alternate between
two devices, whose kernels need their shared memory allowed one by one."""
import re
import shutil
import subprocess
from pathlib import Path

import pytest

HOST = Path(__file__).resolve().parent / "host_kernels"
KERNELS = Path(__file__).resolve().parent.parent / "monarch_b200" / "csrc" / "kernels"
CUDA = Path("/usr/local/cuda/include")

pytestmark = pytest.mark.skipif(shutil.which("g++") is None or not (CUDA / "cuda.h").exists(),
                                reason="needs g++ and the CUDA headers")


def _build(tmp, source, text, driver):
    # single instructions without a meaning here (register split, three-input maximum)
    text = re.sub(r"\basm(\s+volatile)?\s*\([^;]*;[^;]*\);", ";", text)
    text = text.replace("extern __shared__", "extern").replace("__shared__", "static")
    (tmp / source).write_text(text)
    for f in ("ptx.cuh", "launch.cuh", driver):
        shutil.copy(HOST / f, tmp / f)
    shutil.copy(KERNELS / "mb200.h", tmp / "mb200.h")
    cmd = ["g++", "-std=c++17", "-O1", "-w", f"-I{CUDA}", "-x", "c++",
           f'-DPER_DEVICE_HEADER="{KERNELS / "per_device.cuh"}"', f'-DKERNEL_SOURCE="{source}"', *(["-DBACKWARD"] if "bwd" in source else []),
           driver, "-o", "run"]
    p = subprocess.run(cmd, cwd=tmp, capture_output=True, text=True)
    assert p.returncode == 0, p.stderr[-3000:]
    return tmp / "run"


def _run(exe, *args):
    p = subprocess.run([str(exe), *map(str, args)], capture_output=True, text=True, timeout=240)
    assert p.returncode == 0, (args, p.stdout)


@pytest.mark.parametrize("source,warps", [("attn_fwd.cu", 12), ("attn_bwd.cu", 18)])
def test_no_schedule_of_the_attention_kernels_misses_a_phase(tmp_path, source, warps):
    exe = _build(tmp_path, source, (KERNELS / source).read_text(), "attention.cpp")
    for hd in (64, 128):
        _run(exe, hd, warps, 4)


def test_rmsnorm_backward_reports_a_copy_that_never_lands(tmp_path):
    """The status word is set, no row of the gradient keeps what its memory held, and the block
    ends as a whole, with no copy in flight."""
    text = (KERNELS / "elementwise.cu").read_text()
    text = text[: text.index("// ---", text.index("static int launch_rmsnorm_bwd("))] + "}\n"
    exe = _build(tmp_path, "elementwise.cu", text, "rmsnorm_bwd.cpp")
    # all rows of a block staged at once and a ring that is filled again; one chunk and two per
    # thread; every copy lands, one of the first rows' does not, one of a refilled stage does not
    for d in (264, 2048, 4096, 8192):
        for lost in (-1, 0, 4, 17):
            _run(exe, d, lost, 2)

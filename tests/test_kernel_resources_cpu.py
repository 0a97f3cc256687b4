"""What the compiler gives the kernels: registers that cost no block which shared memory has room for, and few spills."""
import os
import re
import shutil
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "chunk-attention_b200"))
import build  # noqa: E402


def resources(source, kernel):
    """(template arguments, registers, bytes of spill stores) of every instance of a kernel."""
    out = subprocess.run(["nvcc"] + build.NVCC_FLAGS + ["-Xptxas", "-v", "-cubin", os.path.join(build.CSRC, source), "-o", os.devnull],
                         capture_output=True, text=True, check=True)
    text = out.stdout + out.stderr
    found = re.findall(r"Compiling entry function '\S*?%sI((?:L[ib]\d+E)+)E\S*'.*?(\d+) bytes spill stores.*?Used (\d+) registers" % kernel, text, re.S)
    return [([int(x) for x in re.findall(r"L[ib](\d+)E", args)], int(regs), int(spills)) for args, spills, regs in found]


@pytest.mark.skipif(shutil.which("nvcc") is None, reason="needs the CUDA compiler")
def test_grouped_attention_keeps_the_blocks_that_its_stages_leave_room_for():
    instances = resources("ca_attn_rows.cu", "rows_mma_kernel")
    assert len(instances) == 27
    for (dk, dv, stages, span, bulk, few), regs, spills in instances:
        ring = stages * 64 * (dk + dv) * 2 + stages * 8
        blocks = 228 * 1024 // (ring + 1024)
        if span and dk < dv:
            blocks = 2  # a third one costs more in spills than it brings
        what = "%s: %d registers, %d bytes spilled" % ((dk, dv, stages, span, bulk, few), regs, spills)
        assert blocks * 128 * (-(-regs // 8) * 8) <= 65536, what
        assert spills <= 76, what  # the widest heads with 16-row tiles

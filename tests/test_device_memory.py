"""What the library keeps of the device's memory between calls and handles.

Each test runs in a process of its own, so that no other handle is alive, and
reads the free memory of the device.
"""
import subprocess
import sys
import textwrap
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

ROOT = Path(__file__).resolve().parent.parent
SETUP = """
import torch
from implexity_b200 import LbmSolver, workloads

MB = 1 << 20
w = workloads.objective_weights()


def free():
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def open_channel(shape, steps):
    s = LbmSolver(workloads.channel_problem(shape=shape, steps=steps, box_half_width=0))
    s.set_design(workloads.uniform_design(shape, 1))
    return s


torch.cuda.init()
"""


def _run(body):
    r = subprocess.run([sys.executable, "-c", SETUP + textwrap.dedent(body)], cwd=ROOT, capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr


def test_last_handle_gives_the_memory_back(gpu_lib):
    """The records of 300 steps at 64^3 are 1.2 GB.  The first cycle loads the
    kernels; 256 MB is left for what the driver itself keeps."""
    _run("""
        def cycle():
            with open_channel((64, 64, 64), 300) as s:
                s.gradient(w)
                return free()

        with open_channel((64, 64, 64), 20) as s:
            s.forward()
            s.gradient(w)
        start = free()
        for _ in range(2):
            assert cycle() < start - 1024 * MB  # kept while the handle lives
            assert free() > start - 256 * MB, (start - free()) / MB
    """)


def test_freed_records_stay_beside_live_handles(gpu_lib):
    """Up to 16 GiB of freed memory stays for the next gradient, whatever the
    live handles hold (two of 21M cells, 3.2 GB of populations each); what is
    freed beyond that goes back."""
    _run("""
        with open_channel((64, 64, 64), 20) as s:
            s.forward()
            s.gradient(w)
        base = free()
        big = [open_channel((320, 256, 256), 2) for _ in range(2)]
        s = open_channel((128, 128, 128), 300)
        s.forward()
        start = free()
        for _ in range(2):
            s.gradient(w)
            assert start - free() > 301 * 128**3 * 16, (start - free()) / MB  # the records of 301 states
        for b in big:
            b.close()
        assert base - free() < s.device_bytes() + (16 << 30) + 256 * MB, (base - free()) / MB
    """)

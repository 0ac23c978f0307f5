"""A grid made in a forked process whose parent has used torch's threads."""

import os
import subprocess
import sys

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SCRIPT = """
import os, signal, sys
import numpy as np
import torch
from pyftle_b200.interpolate import GridSpec

torch.set_num_threads(4)
torch.rand(4_000_000).sum()  # starts torch's threads
axis = 0.1 * np.arange(512)
points = np.stack([m.ravel() for m in np.meshgrid(axis, axis)])
want = GridSpec.from_points(points, (512, 512))
torch.aminmax(torch.from_numpy(points))
pid = os.fork()
if pid == 0:
    signal.alarm(30)  # ends a child that waits for threads it does not have
    os._exit(0 if GridSpec.from_points(points, (512, 512)) == want else 1)
sys.exit(os.waitstatus_to_exitcode(os.waitpid(pid, 0)[1]))
"""


def test_grid_from_points_in_a_forked_process():
    run = subprocess.run([sys.executable, "-W", "ignore", "-c", SCRIPT], cwd=REPO, timeout=240)
    assert run.returncode == 0

"""A device holds the driver's block for small allocations, so that a small scene's buffers neither make nor free it."""
import subprocess
import sys
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]

SCRIPT = """
import torch
import selas_gb300 as sel
from selas_gb300 import scenes
dev = sel.Device(0)
data = scenes.displaced_icospheres(count=1, level=0)
free = [torch.cuda.mem_get_info()[0]]
for _ in range(2):
    sc = sel.Scene(dev, sel.SEL_BVH_WIDE8_Q8, sel.SEL_BUILD_HOST)
    data.attach_to(sc)
    sc.commit()
    free.append(torch.cuda.mem_get_info()[0])
    sc.release()
    free.append(torch.cuda.mem_get_info()[0])
dev.release()
assert len(set(free)) == 1, free
"""


@pytest.mark.gpu
def test_a_small_scene_leaves_the_free_memory_as_it_was(device):  # in a process without other scenes
    done = subprocess.run([sys.executable, "-c", SCRIPT], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert done.returncode == 0, done.stderr[-2000:]

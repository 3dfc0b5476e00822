"""What the kernels' stacks take of the device. The driver reserves the deepest
stack of the kernels run so far for every thread the chip can hold, so one
kernel with a deep frame costs every process gigabytes. In a fresh process all
stages together take less than 3,072 bytes a thread (0.93 GB on 148
multiprocessors), beside their buffers."""
import os
import subprocess
import sys

import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = """
import sys
sys.path.insert(0, {repo!r})
import numpy as np, torch
from trinity_b200.meshgen import field_multi, grid_mesh
from tests.oracle_lib import tags_of
from trinity_b200.api import Coarse, GradientSmooth, Mesh, Metrics, Partit, Refine, Smooth, Swap
torch.zeros(1, device="cuda")
p = torch.cuda.get_device_properties(0)
before = torch.cuda.mem_get_info()[0]
m = grid_mesh(80, 0.2, 1)
for precision in ("fp64", "mixed"):
    g = Mesh((m.nb_nodes, m.nb_elems), 64, 1, 0, 1, capa_scale=4)
    g.set_precision(precision)
    g.load_arrays(m.points, m.tris, tags_of(m), field_multi(m.points))
    h = Partit(g, 8)
    for k in (Metrics(g, 0.5, 2), Refine(g, 1), Coarse(g, h), Swap(g), Smooth(g, h, 1), GradientSmooth(g, h, 1)):
        k.run()
    g.quality_adjoint()
    g.round_graph(1)
    g.close()
torch.cuda.synchronize()
print(before - torch.cuda.mem_get_info()[0], p.multi_processor_count * p.max_threads_per_multi_processor)
"""


@pytest.mark.gpu
def test_stacks_of_all_stages():
    out = subprocess.run([sys.executable, "-c", PROGRAM.format(repo=REPO)], check=True, capture_output=True, text=True,
                         cwd=REPO)
    taken, threads = map(int, out.stdout.split()[-2:])
    print(f"{taken / 2**20:.0f} MB, {taken / threads:.0f} bytes a thread")
    assert taken < 3072 * threads

"""The second call of a program replays the graph that its first call captured.  A process of its
own: the first call also makes the library's buffers, and what it leaves on the stack must not tell
two equal calls apart."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
CHILD = """
import torch
from torch.profiler import ProfilerActivity, profile
from snowsimulation_b200 import scene
from snowsimulation_b200.world import Simulation
torch.zeros(1, device="cuda")
sim = Simulation(scene.tiny(seed=4, water=(6, 6, 6), snow=(8, 5, 8), init_links=True)).setup()
for call in range(4):
    with profile(activities=[ProfilerActivity.CPU, ProfilerActivity.CUDA], acc_events=True) as p:
        sim.step(use_graph=True)
        torch.cuda.synchronize()
    print(sum(e.name.startswith("cudaGraphInstantiate") for e in p.events()))
"""


def test_second_call_replays(cuda):
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", CHILD], cwd=root, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    assert r.stdout.split() == ["1", "0", "0", "0"]

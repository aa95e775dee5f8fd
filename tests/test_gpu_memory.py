"""Solver memory: where the GPU has little left, and what is kept and given back."""
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

SCRIPT = """
import dataclasses, sys
import torch
from dacti_b200 import cases
from dacti_b200.solver import Solver

def make():
    c = cases.lax_liu3(5, 2)
    return Solver(dataclasses.replace(c, params=dataclasses.replace(c.params, pool_capacity=500000)))

def run(s):
    for _ in range(4):
        assert not s.integrate()[1]
    a = s.active_cells()
    s.close()
    return [getattr(a, f).tobytes() for f in ("tree_level", "acti_level", "center", "t", "u", "p", "error")]

first = Solver(cases.lax_liu3(3, 1))  # the kernels' own memory is reserved at their first launch
first.integrate()
first.close()
s = make()
hold = torch.empty(torch.cuda.mem_get_info()[0] - (150 << 20), dtype=torch.uint8, device="cuda")
tight = run(s)
del hold
torch.cuda.empty_cache()
assert tight == run(make())
"""


def test_resort_without_room_for_a_second_pool():
    """A pool of half a million slots (about 200 MB) on a GPU with 150 MB left, in a fresh process so that nothing freed
    before helps: the re-sort's one-field buffer serves, with the same cells in the same order."""
    r = subprocess.run([sys.executable, "-c", SCRIPT], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-2000:]


KEPT = """
import dataclasses
import torch
from dacti_b200 import cases
from dacti_b200.solver import Solver

def make(slots):
    c = cases.lax_liu3(5, 2)
    return Solver(dataclasses.replace(c, params=dataclasses.replace(c.params, pool_capacity=slots)))

def free():
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0] / 2 ** 30

first = make(1)  # contexts, modules, the kernels' own memory
first.integrate()
first.close()
start = free()
small = [make(140000) for _ in range(40)]            # 85 MB each, in blocks below 64 MiB
held = free()
assert start - held > 2.5, (start, held)
for s in small[:5]:
    s.close()
assert abs(free() - held) < 0.1, (held, free())      # what they had stays mapped for the next
small[:5] = [make(140000) for _ in range(5)]
assert abs(free() - held) < 0.1, (held, free())
large = make(14000000)                               # 8 GiB in large blocks
large.integrate()
assert held - free() > 6.0, (held, free())
large.close()
assert held - free() < 0.1, (held, free())           # which all go back
for s in small:
    s.close()
assert start - free() < 0.6, start - free()          # 512 MiB when no solver lives
"""


def test_memory_is_kept_while_in_use_and_given_back():
    """With more in use than is kept unused (2 GiB) a synchronisation unmaps nothing that was just freed; a large solver's
    blocks go back as it closes; half a GiB stays when the last solver is gone."""
    r = subprocess.run([sys.executable, "-c", KEPT], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-2000:]

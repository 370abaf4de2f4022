"""Uploads on a device that is nearly full: what only makes a pass faster is
left out, and the pass gives the same lump.  A process of its own fills the
device, so that no other test's cached blocks count."""
from __future__ import annotations

import os
import pathlib
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = pathlib.Path(__file__).resolve().parent.parent

FILL = """
import dataclasses
import sys
import numpy as np, torch
from hl2sdk_tools_sharp_b200 import lighting as L, roomgrid as rg

hold = []

def fill(room):
    while torch.cuda.mem_get_info()[0] > room + (2 << 20):
        size = torch.cuda.mem_get_info()[0] - room
        try:
            hold.append(torch.empty(min(size, 8 << 30), dtype=torch.uint8, device="cuda"))
        except torch.OutOfMemoryError:
            break
    assert torch.cuda.mem_get_info()[0] < room + (12 << 20)

def give_back():
    hold.clear()
    torch.cuda.empty_cache()
"""

WORLD = FILL + """
few = rg.config_3x3(seed=2)
few = dataclasses.replace(few, side=1, lights=2, sky_ambient=True)
# 850 sun samples a point: the split launches' buffer takes over 60 MB.
inp = L.prepare(rg.generate(dataclasses.replace(few, sun_spread=2.0, sun_samples=850)))
w = rg.generate(few)
with L.LightingStage(w, L.prepare(w)) as st:
    st.direct()    # the kernels' code is on the device
    fill(48 << 20)
    st.upload_world(inp)
    got, _ = st.direct()
    give_back()
    st.upload_world(inp)
    want, _ = st.direct()
    assert want.view(np.uint8).any() and np.array_equal(got.view(np.uint8), want.view(np.uint8))
print("ok")
"""

# What the bounce upload of a map takes, or the same with `short` MB less room;
# and the lump.
BOUNCE = FILL + """
out, taken, short = sys.argv[1], int(sys.argv[2]), int(sys.argv[3]) << 20
w = rg.generate(dataclasses.replace(rg.config_8x8(seed=1), side=7, lights=49))
off, lst = L.pvs_lists(w)
refl = L.face_reflectivity(w)
small = rg.generate(rg.config_3x3(seed=2))
with L.LightingStage(small, L.prepare(small)) as st:   # the kernels' code is on the device
    so, sl = L.pvs_lists(small)
    st.upload_bounce(L.face_reflectivity(small), so, sl)
    st.light_pass()
    with L.LightingStage(w, L.prepare(w)) as st:
        before = torch.cuda.mem_get_info()[0]
        if taken:
            fill(taken - short)
        st.upload_bounce(refl, off, lst, threshold=1.0)
        if not taken:
            print(before - torch.cuda.mem_get_info()[0])
        give_back()
        lump, _, _ = st.light_pass()
        np.save(out, lump)
"""


def python(code, *args):
    # Each tensor an allocation of its own size, so that the room left is exact.
    env = dict(os.environ, PYTORCH_NO_CUDA_MEMORY_CACHING="1")
    run = subprocess.run([sys.executable, "-c", code, *map(str, args)], cwd=ROOT, capture_output=True, text=True,
                         timeout=300, env=env)
    assert run.returncode == 0, run.stdout + run.stderr
    return run.stdout.split()


def test_world_upload_without_room_for_the_split_launches():
    assert python(WORLD) == ["ok"]


def test_bounce_upload_without_room_for_the_windows(tmp_path):
    """The slices of windows take some 100 MB more of this map than one window
    for all receivers; with 60 MB less than the upload would take it is done
    all the same, and the lump is the same."""
    taken, = python(BOUNCE, tmp_path / "a.npy", 0, 0)
    python(BOUNCE, tmp_path / "b.npy", taken, 60)
    a, b = np.load(tmp_path / "a.npy"), np.load(tmp_path / "b.npy")
    assert a.any() and np.array_equal(a, b)

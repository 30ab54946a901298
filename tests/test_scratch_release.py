"""What the scratch pool holds and when it lets go of it, each case in a process of its own."""
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

HEAD = """
import sys
import numpy as np, torch
from luz_b200 import native, scenes
sys.path.insert(0, 'tests')
from test_scratch import buffers
torch.cuda.init(); torch.zeros(1, device='cuda')
free = lambda: torch.cuda.mem_get_info()[0]
"""


def run(code: str):
    r = subprocess.run([sys.executable, "-c", HEAD + code], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr


def test_a_denoise_without_handles_keeps_nothing():
    """No scene or cache is ever opened: after a denoise the device holds what it held after a
    denoise of 8 x 8 pixels, which loads the same kernels (to 32 MiB; the 960 x 540 buffers are
    more than ten times that)."""
    run("""
native.nfor_denoise(buffers(8, 8, 1))
free0 = free()
for k in range(3):
    native.nfor_denoise(buffers(960, 540, k))
left = free0 - free()
assert left <= 32 << 20, left
""")


def test_allocations_take_back_what_the_pool_holds_idle():
    """With more than 1 GiB idle in the pool and all but 64 MiB of the device taken by others, a
    scene of 131 MB and its first render (one wave of 2^19 paths, 145 MB of state) find room."""
    run("""
w = scenes.mesh_glossy(256, 256, 8, 3, level=8)
b = w.scene.build()
small = scenes.mesh_glossy(64, 64, 1, 3, level=3)
p, ps = (native.params(x.width, x.height, x.spp, 3, 5) for x in (w, small))
g = native.GpuScene(b); want, _ = g.render(p); g.close()
keep = native.GpuScene(small.scene.build())
keep.render(ps); native.batch_render([keep], [ps])
f0 = free()
native.nfor_denoise(buffers(1920, 1080, 1))
idle = f0 - free()
assert idle > 1 << 30, idle
hog = torch.empty(max(0, free() - (64 << 20)), dtype=torch.uint8, device='cuda')
g = native.GpuScene(b)
film, st = g.render(p)
assert np.array_equal(film, want) and st.waves == 1
""")


def test_the_denoiser_holds_133_doubles_a_pixel():
    """At most, were all of a call's arrays alive at once: inputs and output 43, suppressed colours
    9, prefiltered features 22, regressions 12, patch distances 25, maps 6, blended colours,
    features and variance 15, list 1. The pool keeps what a call took, below its bound of 3 GiB.
    Allowed beside that: 128 MiB of granularity."""
    run("""
w = scenes.mesh_glossy(8, 8, 1, 1, level=2)
g = native.GpuScene(w.scene.build())
native.nfor_denoise(buffers(8, 8, 1))
f0 = free()
n = 1600 * 900
native.nfor_denoise(buffers(1600, 900, 2))
held = f0 - free()
assert held <= 133 * 8 * n + (128 << 20), (held, 133 * 8 * n)
""")

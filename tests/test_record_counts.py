"""The record counts of LUZ_RENDER_COUNT."""
import pytest

from luz_b200 import native, scenes
from luz_b200.desc import RENDER_COUNT


@pytest.mark.gpu
def test_record_counts_do_not_depend_on_the_launch():
    """LUZ_RENDER_COUNT counts the records a ray's walk reads: a property of the ray, whichever
    lanes share its warp."""
    w = scenes.mesh_glossy(128, 96, 8, 4, level=5)
    g = native.GpuScene(w.scene.build())
    try:
        p = native.params(128, 96, 8, 4, 7)
        p.flags = RENDER_COUNT
        counts = []
        for blocks, paths in ((1, 4096), (2, 16384), (1, 0), (0, 0)):
            g.set_tuning(extend_blocks_per_sm=blocks, shadow_blocks_per_sm=blocks, wave_paths=paths)
            _, st = g.render(p)
            counts.append((st.ext_nodes, st.ext_tris, st.ext_top, st.sh_nodes, st.sh_tris, st.sh_top))
        assert all(c == counts[0] for c in counts), counts
    finally:
        g.close()

"""The tile schedule's scratch is optional: where the device has no memory left
for it, the slab schedule runs and gives the same field."""
import numpy as np
import pytest

from test_gpu_solver2d_memory import fill  # noqa: F401  (fixture)
from test_gpu_tiles import H, SLABS, TILES, _cells, _src

pytestmark = pytest.mark.gpu


def test_slabs_run_without_memory_for_the_tiles(fk, fill):  # noqa: F811
    n = (90, 128, 128)                    # 56 MB of edge words in FP64
    s = fk.fteik3d()
    s.initialize(n[1], n[2], n[0], H[1], H[2], H[0], nsweep=1, eps=5.0, precision=8)
    s.setCellSlownessNatural(_cells(n, 2))
    src = _src(n, "inside")
    s.setSources(src[1], src[2], src[0])
    old = fk.set_slab_config(*SLABS)
    try:
        s.solveSourceLSM(1)
        want = s.getTravelTimeField()
        fill(24 << 20)
        fk.set_slab_config(*TILES)
        for _ in range(2):
            s.solveSourceLSM(1)
            assert np.array_equal(s.getTravelTimeField(), want)
    finally:
        fk.set_slab_config(*old)
        s.free()

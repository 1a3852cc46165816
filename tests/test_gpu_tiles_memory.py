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


def test_a_batch_on_slabs_keeps_no_tile_memory(fk):
    """The search times the tiles; where it takes the slabs (28 sources need ten
    launches of tiles) their scratch, 48 MB, is given back."""
    import torch
    grid = (60, 97, 83, 50.0, 50.0, 50.0)

    def used(cfg, src):
        old = fk.set_slab_config(*cfg)
        try:
            b = fk.Batch3D([grid], nsweep=2, eps=5.0, precision=4)
            b.setVelocityModel(1, np.full((82, 96, 59), 3000.0))
            b.setSources(1, *[np.linspace(100.0, (m - 3) * 50.0, src) for m in grid[:3]])
            before = torch.cuda.mem_get_info()[0]
            b.solve()
            after = torch.cuda.mem_get_info()[0]
            c = b.slabConfig()
            b.finalize()
        finally:
            fk.set_slab_config(*old)
        return before - after, c

    for cfg in (SLABS, TILES):            # kernels loaded, the stream's pools grown
        used(cfg, 2)
    want, _ = used(SLABS, 28)
    got, c = used(TILES, 28)
    assert c["tune_runs"] > 0 and c["init_ms"] > 0.0
    assert got - want < 16 << 20, (got, want)

"""A large model's slowness upload keeps no second copy on the device: after a
solve on 3501 x 3501 nodes there is the field and the slowness (98 MB each).  And an
allocation that fails is that call's error only, not the next one's."""
import numpy as np
import pytest

from test_gpu_solver2d_memory import fill  # noqa: F401  (fixture)

pytestmark = pytest.mark.gpu


def _used(fk, n):
    import torch
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    s = fk.fteik2d()
    s.initialize(n, n, 5.0, 5.0, nsweep=0, eps=5.0)
    s.setCellVelocityNatural(np.full((n - 1) * (n - 1), 3000.0))
    s.setSources([5.0 * (n // 2)], [5.0 * (n // 3)])
    s.solveSourceLSM(1)
    after = torch.cuda.mem_get_info()[0]
    s.free()
    return before - after


def test_no_staging_copy_stays(fk):
    _used(fk, 600)                        # kernels loaded
    n = 3501
    assert _used(fk, n) < 2.5 * 8 * n * n


def test_a_failed_allocation_stays_with_its_call(fk, fill):  # noqa: F811
    _used(fk, 600)
    fill(64 << 20)
    with pytest.raises(fk.FteikError):
        _used(fk, 3501)                   # two arrays of 98 MB
    _used(fk, 600)

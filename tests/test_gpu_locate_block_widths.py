"""The block-bounded grid search at the table counts around which two or three
thread blocks share an SM."""
import pytest

import test_gpu_locate_blocks as B

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ntf,nev", [(31, 192), (32, 200), (33, 200), (40, 192)])
@pytest.mark.parametrize("kind", ["times", "random"])
def test_widths(fk, ntf, nev, kind):
    B.test_blocks_match_points_and_oracle_bitwise(fk, ntf, (1 << 18) + ntf, nev, kind)

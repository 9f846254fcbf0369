"""The grid build of long lists on either side of the number of cells a point (16) where
the tile sums change from a kernel over the counts to the key pass's atomics; order and
offsets must equal the oracle's."""
import pytest

from test_gpu_grid_sizes import test_build_sizes as check_build

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built():
    from twoscalesplit_gb300 import build
    build.build()


@pytest.mark.parametrize("n,dims", [(150000, (1600, 1500)), (150000, (2400015, 1)), (150000, (1, 2400016)),
                                    (150001, (3001, 801)), (200003, (2049, 1562)), (623617, (4096, 4099))])
def test_sparse_builds(n, dims):
    check_build(n, dims)

"""Points of a shot at the counts where the resident kernel's instances change: 256 are linked
per tile, 64 more looked up in its list, beyond that the tile's points go over all its
threads. Against the streaming kernels as in the kernel's other tests."""
import pytest

from test_resident_dense_gpu import test_points_at_the_linked_count as _check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nsrc,nrec", [(1, 319), (1, 320), (1, 321), (320, 20), (321, 20), (700, 900)])
@pytest.mark.parametrize("order,update", [(2, "leapfrog"), (4, "auto"), (8, "auto")])
def test_points_at_the_walk_count(cuda, order, update, nsrc, nrec):
    _check(cuda, order, update, nsrc, nrec)

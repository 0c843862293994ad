"""Each block of the resident CG kernel updates its own copy of the direction
entries that it reads of other blocks.  The copies have to be the owners' bits,
or the product and p.q are not of one vector."""
import pytest

from femorph_b200 import api, mesh

pytestmark = pytest.mark.gpu


# 10 blocks of 133 rows; one of 201 an SM; of more than 1,024 (1,024 threads);
# and 912,673 rows (q and r alone beside the direction in shared memory)
@pytest.mark.parametrize("n,elem_type", [(10, mesh.HEXA8), (30, mesh.TET4), (56, mesh.HEXA8), (96, mesh.HEXA8)])
def test_halo_copies_have_the_owners_bits(n, elem_type):
    s = api.GpuPoisson(mesh.poisson_box(n, elem_type, seed=n))
    for iterations in (1, 2, 3, 40):
        copies, differing = s.check_direction(iterations)
        assert copies > 0 and differing == 0, (iterations, copies, differing)
    s.close()


def test_one_block_has_no_copies():
    s = api.GpuPoisson(mesh.poisson_box(8, mesh.HEXA8, seed=8))
    assert s.check_direction(3) == (0, 0)
    s.close()

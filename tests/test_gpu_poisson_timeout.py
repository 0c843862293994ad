"""A resident Poisson solve whose blocks give up waiting for one another.  The
bound is a launch parameter: with a limit of 0 polls every block gives up in
its first exchange, so nothing has to hang or fault for the path to run."""
import numpy as np
import pytest

from femorph_b200 import api, mesh

pytestmark = pytest.mark.gpu

LIMIT = 1 << 22  # the default


@pytest.mark.parametrize("n", [10, 30])
def test_timed_out_solve_leaves_nothing_to_read(n, tmp_path):
    """1,331 and 29,791 rows (10 blocks and one an SM): a solve that timed out
    reports it, writes no outputs and hides the earlier solution; the next one
    has the first one's bits."""
    p = mesh.poisson_box(n, mesh.HEXA8, seed=n)
    s = api.GpuPoisson(p)
    it, rr, _ = s.solve(1e-12)
    x, _ = s.solution()
    s.set_wait_limit(0)
    out = [api.C.c_int32(-7), api.C.c_double(-7.0), api.C.c_double(-7.0)]
    r = api.lib().fm_poisson_solve(s.h, 1e-12, 20000, *[api.C.byref(o) for o in out])
    assert r == api.FM_ERR_TIMEOUT
    assert [o.value for o in out] == [-7, -7.0, -7.0]
    with pytest.raises(api.FmError) as ei:
        s.solution()
    assert ei.value.code == api.FM_ERR_INVALID
    with pytest.raises(api.FmError):
        s.write_vtk(str(tmp_path / "x.vtk"))
    s.set_wait_limit(LIMIT)
    it2, rr2, _ = s.solve(1e-12)
    x2, _ = s.solution()
    assert it2 == it and rr2 == rr and np.array_equal(x2, x)
    s.close()


def test_one_block_has_no_wait():
    """729 rows are one block's: the limit does not matter."""
    p = mesh.poisson_box(8, mesh.TET4, seed=8)
    s = api.GpuPoisson(p)
    s.set_wait_limit(0)
    _, rr, _ = s.solve(1e-12)
    assert rr <= 1e-12
    s.close()

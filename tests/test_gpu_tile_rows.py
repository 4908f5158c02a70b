"""The threads that share a row in the one-pass tile build: which form a
rebuild takes, and what sends it back to one thread a row."""
import numpy as np
import pytest

from test_gpu_md import fcc, mb_velocities

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def M():
    import mrmd_gb300 as m

    return m


# Two tiles per SM (304 on 152 SMs, 77,824 rows) take four threads; rows whose
# quarter of the columns holds more than 64 entries (r_list 4.0) do not fit.
@pytest.mark.parametrize("cells,atoms,rc,threads", [(8, 2031, 2.5, 4), (27, 77824, 2.5, 4), (27, 77825, 2.5, 1),
                                                    (10, 4000, 3.7, 1)])
def test_row_threads(M, cells, atoms, rc, threads):
    pos, L = fcc(cells)
    keep = np.sort(np.random.default_rng(atoms).permutation(len(pos))[:atoms])
    s = M.LJSystem(pos[keep], mb_velocities(len(pos), 0.728, 9)[keep], [0, 0, 0], [L] * 3, rc=rc,
                   precision=M.PREC_MIXED)
    s.run(25)
    st = s.tile_stats()
    assert st["row_threads"] == threads and st["two_pass_builds"] == 0


def test_unsorted_atoms_leave_the_row_threads(M):
    """A rebuild over atoms without spatial order does not fit the tile tables
    and makes int32 rows; the next sorted one has four threads a row again."""
    pos, L = fcc(12)
    vel = mb_velocities(len(pos), 0.728, 5)
    s = M.LJSystem(pos, vel, [0, 0, 0], [L] * 3, precision=M.PREC_MIXED, sort_atoms=4)
    s.run(15)  # three rebuilds, the first sorted
    assert s.tile_stats()["row_threads"] == 4
    s.set_state(pos[np.random.default_rng(1).permutation(len(pos))], vel)
    s.eval_forces()
    st = s.tile_stats()
    assert st["unfit_tiles"] > 0 and st["two_pass_builds"] == 1 and st["row_threads"] == 0
    s.run(5)  # the fifth rebuild sorts
    st = s.tile_stats()
    assert st["row_threads"] == 4 and st["two_pass_builds"] == 1

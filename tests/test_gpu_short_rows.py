"""Pair kernels over lists with rows of a few entries (a gas), at the sizes
where one lane a row takes over, against the oracle."""
import numpy as np
import pytest

from test_gpu_pair_kernels import both

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def M():
    import mrmd_gb300 as m

    return m


# One lane a row from 97,280 rows (640 per SM on 152) of fewer than four
# entries up; 0.9 entries a row at density 0.02, 4.6 at 0.1.
@pytest.mark.parametrize("n,rho,pred", [(97279, 0.02, None), (97281, 0.02, None), (97281, 0.02, "both"), (97281, 0.1, None)])
def test_mixed_half_short_rows(M, orc, n, rho, pred):
    """Forces within the mixed form's bar of the oracle's (1e-6 of the rms
    force), the energy within 1e-7.  One atom in 400 sits in a dense
    droplet, whose rows are long."""
    rng = np.random.default_rng(n)
    L = (n / rho) ** (1 / 3)
    pos = rng.uniform(0, L, (n, 3))
    drop = rng.permutation(n)[: n // 400]
    pos[drop] = L / 2 + rng.uniform(-3.0, 3.0, (len(drop), 3))
    lo = [-1.0, 0.0, 7.0]
    (Fo, Eo, Wo), gpu = both(M, orc, pos + np.asarray(lo), lo, L, 2.5, orc.lj_table(0.8, 2.5, 1.0, 1.0, 1, True), pred)
    F, E, W = gpu(M.LennardJones(2.5, 1.0, 1.0, 0.8, is_shifted=True), M.PREC_MIXED)
    rms = np.sqrt((Fo ** 2).sum(1).mean())
    assert np.linalg.norm(F - Fo, axis=1).max() <= 1e-6 * rms
    assert abs(E - Eo) <= 1e-7 * abs(Eo)

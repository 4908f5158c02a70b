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


# One lane a molecule from 60,800 of them (400 per SM on 152) with less than
# one pair of sites each up: 0.9 entries a row, and 8 pairs of sites with three.
@pytest.mark.parametrize("prec", ["fp64", "mixed"])
@pytest.mark.parametrize("n,sites", [(60799, 1), (60801, 1), (60801, 3)])
def test_lj_ideal_gas_short_rows(M, orc, n, sites, prec):
    """Forces before the fold-back and the energy against the oracle, by the
    bars of the FP64 and the mixed form."""
    from conftest import assert_fp64_forces
    from test_gpu_adress import adress_system, upload_molecules

    mo, ao, corr, sd, slab, (rc, skin, _) = adress_system(orc, n, (310.0, 100.0, 100.0), 17, sites)
    co, no = orc.build_half_list(mo.pos, mo.numLocal + mo.numGhost, 0, mo.numLocal, rc + skin, sd.minGhostCorner,
                                 sd.maxGhostCorner, 1.0, 64)
    assert 0.5 * n < co.sum() < n
    ao.force[:] = 0
    mo.force[:] = 0
    Eo = orc.LJIdealGas(0.8, rc, 1.0, 1.0, True).run(mo, co, no, ao)
    na, nm = ao.n, mo.numLocal + mo.numGhost
    a = M.Atoms.from_arrays(ao.pos[:na], relative_mass=ao.relativeMass[:na], capacity=ao.capacity)
    a.numLocalAtoms, a.numGhostAtoms = ao.numLocal, ao.numGhost
    m = upload_molecules(M, mo, mo.numLocal, mo.numGhost)
    m.setForce(0.0)
    a.setForce(0.0)
    vl = M.HalfVerletList()
    vl.build(m, 0, mo.numLocal, rc + skin, 1.0, sd.minGhostCorner[:], sd.maxGhostCorner[:], 60)
    ig = M.LJ_IdealGas(0.8, rc, 1.0, 1.0, True)
    E = ig.run(m, vl, a, M.PREC_FP64 if prec == "fp64" else M.PREC_MIXED)
    F, Fm = a.getForce(), m.download()["force"]
    Fo, Fmo = ao.force[:na], mo.force[:nm]
    if prec == "fp64":
        assert_fp64_forces(F, Fo)
        assert_fp64_forces(Fm, Fmo)
        assert abs(E - Eo) <= 1e-10 * abs(Eo)
    else:
        rms = np.sqrt((Fo ** 2).sum(1).mean())
        assert np.linalg.norm(F - Fo, axis=1).max() <= 1e-6 * rms
        assert abs(E - Eo) <= 1e-7 * abs(Eo)

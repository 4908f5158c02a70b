"""Calls at the limits of indices and buffers: refused with an error, or
reported by the bounds-checked build, and the objects stay usable."""
import os
import subprocess
import sys
import textwrap

import numpy as np
import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def M():
    import mrmd_gb300 as m

    return m


def test_molecule_images_beyond_31_bits_are_refused(M):
    """A molecule in a corner has seven images; 7 x 2^29 atoms have no 32-bit
    index.  Refused before anything is reserved or written."""
    box = M.Subdomain([0, 0, 0], [10.0] * 3, 2.8)
    a = M.Atoms.from_arrays([[0.5, 0.5, 0.5]], capacity=64)
    m = M.Molecules(16)
    up = dict(pos=np.array([[0.5, 0.5, 0.5]]), force=np.zeros((1, 3)), lambda_=np.zeros(1),
              modulated_lambda=np.zeros(1), grad_lambda=np.zeros((1, 3)), atoms_offset=[0])
    m.upload(1, 0, num_atoms=[1 << 29], **up)
    gl = M.MultiResGhostLayer()
    with pytest.raises(M.MrmdError) as e:
        gl.createGhostAtoms(m, a, box)
    assert e.value.code == -8  # MRMD_ERR_CAPACITY
    assert (m.numGhostMolecules, a.numGhostAtoms) == (0, 0)
    m.upload(1, 0, num_atoms=[1], **up)
    gl.createGhostAtoms(m, a, box)
    assert (m.numGhostMolecules, a.numGhostAtoms) == (7, 7)


# Runs with the bounds-checked library alone, where an index outside its array
# is recorded and the access is skipped.
CHILD = textwrap.dedent(r"""
    import ctypes, sys
    import numpy as np
    sys.path.insert(0, ROOT)
    sys.path.insert(0, ROOT + "/tests")
    import mrmd_gb300 as M
    from test_gpu_md import fcc, mb_velocities
    ctx = M.default_context()
    if ctx.lib.mrmd_bounds_checked() != 1:
        print("not the bounds-checked library")
        sys.exit(3)
    cudart = None
    for name in ("libcudart.so.13", "libcudart.so.12", "libcudart.so"):
        try:
            cudart = ctypes.CDLL(name)
            break
        except OSError:
            pass
    clean = M.Atoms.from_arrays(np.ones((4, 3)), capacity=64)

    def reported(f, source, value):
        try:
            f()
            clean.setForce(0.0)  # the next synchronisation
        except M.MrmdError as e:
            assert e.code == -9 and source in str(e) and str(value) in str(e), e
            print("reported:", e)
        else:
            print("no violation reported for", source)
            sys.exit(4)

    # the FP64 stepper's real atoms of its ghosts, from the host
    pos, L = fcc(6)
    s = M.LJSystem(pos, mb_velocities(len(pos), 0.728, 3), [0, 0, 0], [L] * 3, precision=M.PREC_FP64)
    s.run(5)
    g = ctx.lib.mrmd_md_ghosts(s.h).contents
    real = ctypes.c_void_p(ctypes.cast(g.correspondingRealAtom, ctypes.c_void_p).value + 4 * g.numLocal)
    for bad in (1 << 30, -1):
        entries = np.full(g.numGhost, bad, dtype=np.int32)
        assert cudart.cudaMemcpy(real, entries.ctypes.data_as(ctypes.c_void_p), ctypes.c_size_t(4 * g.numGhost), 1) == 0
        reported(s.launch_pair_kernel, "lj.cu", bad)
    s.close()
    # a molecule whose atoms are not there
    a = M.Atoms.from_arrays([[0.5, 5.0, 5.0], [5.0, 5.0, 5.0]], capacity=64)
    m = M.Molecules(16)
    up = dict(pos=np.array([[0.5, 5.0, 5.0], [5.0, 5.0, 5.0]]), force=np.zeros((2, 3)), lambda_=np.zeros(2),
              modulated_lambda=np.zeros(2), grad_lambda=np.zeros((2, 3)), num_atoms=[1, 1])
    box, gl = M.Subdomain([0, 0, 0], [10.0] * 3, 2.8), M.MultiResGhostLayer()
    m.upload(2, 0, atoms_offset=[1 << 30, 1], **up)
    reported(lambda: gl.createGhostAtoms(m, a, box), "ghost.cu", 1 << 30)
    m.upload(2, 0, atoms_offset=[0, 1], **up)
    gl.createGhostAtoms(m, a, box)
    print("ok")
""")


def test_bounds_build_reports_bad_real_atoms_and_molecules():
    from mrmd_gb300 import build as B

    B.build(bounds_check=True)
    env = dict(os.environ, MRMD_GB300_BOUNDS_CHECK="1")
    r = subprocess.run([sys.executable, "-c", f"ROOT = {ROOT!r}\n" + CHILD], env=env, capture_output=True,
                       text=True, timeout=600)
    assert r.returncode == 0, r.stdout + r.stderr
    assert r.stdout.count("reported: MRMD_ERR_BOUNDS") == 3 and r.stdout.strip().endswith("ok"), r.stdout


def test_a_list_that_could_not_grow_is_empty(M):
    """A build with room for 2^40 neighbours a row fails; the list has no rows
    then, and the next build allocates anew."""
    pos = np.random.default_rng(3).uniform(0, 6.0, (500, 3))
    a = M.Atoms.from_arrays(pos)
    vl, lj = M.HalfVerletList(), M.LennardJones(1.0, 1.0, 1.0, 0.7)
    args = (a, 0, 500, 1.3, 1.0, [0.0] * 3, [6.0] * 3)
    vl.build(*args, 60)
    pairs = vl.total_pairs
    a.setForce(0.0)
    lj.apply(a, vl)
    energy = lj.getEnergy()
    with pytest.raises(M.MrmdError) as e:
        vl.build(*args, 1 << 40)
    assert e.value.code == -2  # MRMD_ERR_OOM
    assert vl.total_pairs == 0 and len(vl.download()[0]) == 0
    lj.apply(a, vl)
    assert lj.getEnergy() == 0.0
    vl.build(*args, 60)
    a.setForce(0.0)
    lj.apply(a, vl)
    assert vl.total_pairs == pairs and abs(lj.getEnergy() - energy) <= 1e-12 * abs(energy)


@pytest.mark.parametrize("kind", ["md", "adress"])
def test_a_run_too_long_to_record_leaves_the_system(M, kind):
    """2^45 steps have no room for their energies; a run after that is the one
    of a fresh system."""
    from test_gpu_md import fcc, mb_velocities

    pos, L = fcc(6)
    vel = mb_velocities(len(pos), 0.728, 3)

    def system():
        if kind == "md":
            return M.LJSystem(pos, vel, [0, 0, 0], [L] * 3, precision=M.PREC_MIXED)
        return M.AdResSSystem(pos, vel, [0, 0, 0], [L] * 3, [L / 2] * 3, 3.0, 2.0, capping_distance=0.7842,
                              precision=M.PREC_MIXED, composed=True)

    a, b = system(), system()
    with pytest.raises(M.MrmdError) as e:
        a.run(1 << 45, energies=False)
    assert e.value.code == -2  # MRMD_ERR_OOM
    ea, eb = a.run(12), b.run(12)
    np.testing.assert_allclose(ea, eb, rtol=1e-9)
    np.testing.assert_allclose(a.state()[0], b.state()[0], rtol=0, atol=1e-9)


@pytest.mark.parametrize("interface", [0, 1])
@pytest.mark.parametrize("at,hy", [(np.nan, 10.0), (-np.nan, 10.0), (np.nan, np.inf), (-np.inf, np.inf), (np.inf, 10.0),
                                   (30.0, np.inf), (-5.0, 10.0)])
def test_slab_diameters_out_of_the_ordinary(M, orc, at, hy, interface):
    """Weights of slabs with NaN, infinite and negative diameters (a hybrid width
    that is not positive is refused) are the reference's: NaN compares with
    nothing, so that a smooth slab has NaN weights (not ones) and an abrupt one
    weights of one."""
    apos = np.random.default_rng(2).uniform(0, 120, (500, 3))
    mo = orc.Molecules(500)
    mo.atomsOffset[:], mo.numAtoms[:], mo.numLocal = np.arange(500), 1, 500
    ao = orc.Atoms.from_positions(apos)
    ao.relativeMass[:500] = 1.0
    with np.errstate(all="ignore"):
        orc.update_molecules(mo, ao, orc.slab([60, 12, 12], at, hy, 1, interface))
    m, a = M.Molecules(500), M.Atoms.from_arrays(apos)
    m.upload(500, 0, pos=apos, force=np.zeros((500, 3)), lambda_=np.zeros(500), modulated_lambda=np.zeros(500),
             grad_lambda=np.zeros((500, 3)), atoms_offset=np.arange(500), num_atoms=np.ones(500))
    M.UpdateMolecules.update(m, a, M.Slab([60, 12, 12], at, hy, 1, interface))
    d = m.download(500)
    np.testing.assert_allclose(d["lambda_"], mo.lambda_[:500], rtol=1e-13, atol=1e-15, equal_nan=True)
    np.testing.assert_allclose(d["modulatedLambda"], mo.modulatedLambda[:500], rtol=1e-13, atol=1e-15, equal_nan=True)
    np.testing.assert_allclose(d["gradLambda"][:, 0], mo.gradLambda[:500, 0], rtol=1e-12, atol=1e-15, equal_nan=True)

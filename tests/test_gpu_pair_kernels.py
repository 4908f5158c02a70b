"""The half-list pair kernels at the sizes where their split of the work
changes (rows per warp, list chunks, ragged last groups), against the oracle."""
import numpy as np
import pytest

from conftest import assert_fp64_forces

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def M():
    import mrmd_gb300 as m

    return m


def fluid(cells, drop, rho, seed, lo):
    """Lattice sites with displacements of 0.08 sigma, `drop` of them vacant,
    in a box with its lower corner at lo."""
    rng = np.random.default_rng(seed)
    a = (4.0 / rho) ** (1.0 / 3.0)
    base = np.array([[0, 0, 0], [0.5, 0.5, 0], [0.5, 0, 0.5], [0, 0.5, 0.5]])
    g = np.stack(np.meshgrid(*[np.arange(cells)] * 3, indexing="ij"), -1).reshape(-1, 3)
    pos = ((g[:, None, :] + base[None, :, :]).reshape(-1, 3) + 0.25) * a
    pos = np.delete(pos, rng.choice(len(pos), drop, replace=False), axis=0)
    L = cells * a
    return np.mod(pos + rng.normal(0, 0.08, pos.shape), L) + np.asarray(lo), L


def both(M, orc, pos, lo, L, rc, table, pred=None, types=None):
    """(forces, energy, virial) of the oracle and a function giving those of a
    precision on the GPU, before the ghosts' forces are folded back."""
    hi = [x + L for x in lo]
    rl = rc + 0.3
    sd_o, sd_g = orc.subdomain(lo, hi, rl), M.Subdomain(lo, hi, rl)
    cap = int(len(pos) * (1 + 2.1 * rl / L) ** 3) + 256
    ao = orc.Atoms.from_positions(pos, capacity=cap)
    if types is not None:
        ao.type[: len(pos)] = types
    orc.create_ghosts(ao, sd_o)
    most = int(4.5 * rl ** 3) + 32
    co, no = orc.build_half_list(ao.pos, ao.n, 0, ao.numLocal, rl, sd_o.minGhostCorner, sd_o.maxGhostCorner, 1.0, most)
    ao.force[:] = 0
    kinds = {None: None, "either": (orc.PRED_EITHER_IN_SLAB, M.PRED_EITHER_IN_SLAB),
             "both": (orc.PRED_BOTH_IN_SLAB, M.PRED_BOTH_IN_SLAB)}[pred]
    args = (0, lo[0] + L / 2, 0.0, L / 4)
    Eo, Wo = orc.lj_apply(table, rc * rc, ao, co, no, None if kinds is None else orc.pred(kinds[0], *args),
                          1 if types is None else 2)
    ag = M.Atoms.from_arrays(pos, type=types, capacity=cap)
    M.GhostLayer().createGhostAtoms(ag, sd_g)
    vl = M.HalfVerletList()
    vl.build(ag, 0, ag.numLocalAtoms, rl, 1.0, sd_g.minGhostCorner, sd_g.maxGhostCorner, 60)
    assert vl.total_pairs == int(co.sum())

    def gpu(lj, precision):
        ag.setForce(0.0)
        lj.apply_if(ag, vl, None if kinds is None else M.pred(kinds[1], *args), precision)
        return ag.getForce(), lj.getEnergy(), lj.getVirial()

    return (ao.force[: ao.n], Eo, Wo), gpu


# Rows per warp change at 3,040, 19,456 and 233,472 atoms on 152 SMs; rc 4
# gives rows of more than 64 entries (several chunks).
@pytest.mark.parametrize("cells,drop,rc,cap,pred,lo,types", [
    (4, 255, 2.5, 0.0, None, [0.0, 0.0, 0.0], False),              # a single atom
    (5, 3, 2.5, 0.95, None, [-3.0, 2.5, 0.0], False),
    (9, 1, 4.0, 0.0, "either", [0.0, 0.0, 0.0], False),
    (10, 961, 2.5, 0.0, None, [0.0, 0.0, 0.0], False),             # 3,039
    (10, 959, 2.5, 0.95, "both", [5000.0, -70000.0, 0.1], False),  # 3,041, far from the origin
    (10, 5, 4.0, 0.9, None, [0.0, 0.0, 0.0], True),
    (17, 197, 2.5, 0.95, None, [0.0, 0.0, 0.0], False),            # 19,455
    (17, 195, 4.0, 0.0, "either", [-10.0, -10.0, -10.0], True),    # 19,457
    (39, 3800, 2.5, 0.0, None, [0.0, 0.0, 1000.0], False),         # 233,476
    (39, 3790, 3.2, 0.95, "both", [0.0, 0.0, 0.0], False),
])
def test_fp64_rows_per_warp(M, orc, cells, drop, rc, cap, pred, lo, types):
    pos, L = fluid(cells, drop, 0.8 if cells > 4 else 0.4, cells + drop, lo)
    t = np.random.default_rng(cells).integers(0, 2, len(pos)) if types else None
    sig, eps = (np.array([1.0, 0.95, 0.95, 0.9]), np.array([1.0, 0.8, 0.8, 1.3])) if types else (1.0, 1.0)
    k = 2 if types else 1
    caps, rcs = (np.full(4, cap), np.full(4, rc)) if types else (cap, rc)
    (Fo, Eo, Wo), gpu = both(M, orc, pos, lo, L, rc, orc.lj_table(caps, rcs, sig, eps, k, True), pred, t)
    F, E, W = gpu(M.LennardJones(rcs, sig, eps, caps, num_types=k, is_shifted=True, num_types_index=k), M.PREC_FP64)
    if not np.any(Fo):
        assert not np.any(F) and E == Eo == 0.0 and W == Wo == 0.0
        return
    assert_fp64_forces(F, Fo)
    assert abs(E - Eo) <= 1e-10 * max(abs(Eo), 1.0)
    assert abs(W - Wo) <= 1e-10 * max(abs(Wo), 1.0)


# The AdResS stepper takes 8, 4, 2 or 1 lanes per row by size and form; the
# batched engine with one lane per row is the same system.
LANES = [((36, 6, 6), 20.0), ((31, 13, 13), 20.0), ((60, 21, 21), 30.0), ((61, 31, 31), 60.0)]


def gas(M, cells, at, precision):
    """(AdResS stepper, one-lane batch) of one density-0.5 system."""
    rng = np.random.default_rng(cells[0])
    base = np.array([[0, 0, 0], [0.5, 0.5, 0], [0.5, 0, 0.5], [0, 0.5, 0.5]])
    g = np.stack(np.meshgrid(*[np.arange(c) for c in cells], indexing="ij"), -1).reshape(-1, 3)
    L = 2.0 * np.array(cells)
    pos = np.mod(((g[:, None, :] + base).reshape(-1, 3) + 0.25) * 2.0 + rng.normal(0, 0.1, (4 * len(g), 3)), L)[:-3]
    vel = rng.normal(0, 1, pos.shape)
    kw = dict(rc=2.5, skin=0.3, capping_distance=0.7842, precision=precision, dt=0.005)
    return (M.AdResSSystem(pos, vel, [0, 0, 0], list(L), list(L / 2), at, 10.0, seed=7, **kw),
            M.BatchSystem([M.Replica(len(pos), [0, 0, 0], list(L), list(L / 2), at, 7)], pos, vel, 10.0, **kw))


@pytest.mark.parametrize("cells,at", LANES)
def test_adress_lanes_per_row_fp64(M, cells, at):
    """Sums of some hundred doubles in another order: 1e-12 of the rms force."""
    a, b = gas(M, cells, at, M.PREC_FP64)
    ea, eb = a.run(1)[0], b.run(1)[0, 0]
    (pa, va, fa), (pb, vb, fb) = a.state(), b.state()
    assert np.array_equal(pa, pb)
    assert np.abs(fa - fb).max() <= 1e-12 * np.sqrt((fb ** 2).sum(1).mean())
    assert abs(ea - eb) <= 1e-12 * abs(eb)
    ea, eb = a.run(49), b.run(49)[:, 0]
    np.testing.assert_allclose(a.state()[0], b.state()[0], rtol=0, atol=1e-9)
    np.testing.assert_allclose(ea, eb, rtol=1e-9)


@pytest.mark.parametrize("cells,at", LANES)
def test_adress_lanes_per_row_mixed(M, cells, at):
    """The FP32 energies are summed in the order of one lane per row: equal
    but for the FP64 additions across rows.  Forces within the mixed form's
    bar of the FP64 ones (1e-6 of the rms force)."""
    a, b = gas(M, cells, at, M.PREC_MIXED)
    f64 = gas(M, cells, at, M.PREC_FP64)[1]
    ea, eb = a.run(1)[0], b.run(1)[0, 0]
    f64.run(1)
    fa, f = a.state()[2], f64.state()[2]
    assert np.abs(fa - f).max() <= 1e-6 * np.sqrt((f ** 2).sum(1).mean())
    assert abs(ea - eb) <= 1e-12 * abs(eb)


def test_list_order_does_not_depend_on_lanes(M):
    """Small batches build their rows with eight lanes each, large ones with
    one: the entries come in the same order, so that a replica run in a
    large batch (near/far rows, FP32 far sums) is bitwise the one run alone."""
    rng = np.random.default_rng(5)
    reps, pos, vel = [], [], []
    for k, (c, at) in enumerate([((120, 30, 30), 60.0), ((30, 6, 7), 14.0)]):
        base = np.array([[0, 0, 0], [0.5, 0.5, 0], [0.5, 0, 0.5], [0, 0.5, 0.5]])
        g = np.stack(np.meshgrid(*[np.arange(m) for m in c], indexing="ij"), -1).reshape(-1, 3)
        L = 2.0 * np.array(c)
        x = np.mod(((g[:, None, :] + base).reshape(-1, 3) + 0.25) * 2.0 + rng.normal(0, 0.1, (4 * len(g), 3)), L)
        reps.append(M.Replica(len(x), [0, 0, 0], list(L), list(L / 2), at, 50 + k))
        pos.append(x)
        vel.append(rng.normal(0, 1, x.shape))
    kw = dict(hybrid_diameter=8.0, capping_distance=0.7842, precision=M.PREC_MIXED, rebuild_interval=5,
              sort_every=1, graph_steps=10, list_layout=1)
    b = M.BatchSystem(reps, np.concatenate(pos), np.concatenate(vel), **kw)
    b.run(20)
    sl = b.replica_slice(1)
    alone = M.BatchSystem(reps[1:], pos[1], vel[1], **kw)
    alone.run(20)
    for x, y in zip(b.state(), alone.state()):
        assert np.array_equal(x[sl], y)


@pytest.mark.parametrize("cells,drop", [(13, 0), (14, 1), (29, 0), (30, 3)])
def test_half_list_lanes_are_the_oracle_rows(M, orc, cells, drop):
    """Eight lanes per row below 9,728 rows on 152 SMs, four below 97,280, one
    above: each row holds exactly the oracle's neighbours."""
    lo = [-1.0, 0.0, 7.0]
    pos, L = fluid(cells, drop, 0.8442, 3 * cells, lo)
    hi = [x + L for x in lo]
    sd_o, sd_g = orc.subdomain(lo, hi, 2.8), M.Subdomain(lo, hi, 2.8)
    ao = orc.Atoms.from_positions(pos, capacity=int(len(pos) * (1 + 6 / L) ** 3) + 256)
    orc.create_ghosts(ao, sd_o)
    co, no = orc.build_half_list(ao.pos, ao.n, 0, ao.numLocal, 2.8, sd_o.minGhostCorner, sd_o.maxGhostCorner, 1.0, 96)
    ag = M.Atoms.from_arrays(pos, capacity=len(ao.pos))
    M.GhostLayer().createGhostAtoms(ag, sd_g)
    vl = M.HalfVerletList()
    vl.build(ag, 0, ag.numLocalAtoms, 2.8, 1.0, sd_g.minGhostCorner, sd_g.maxGhostCorner, 20)
    cg, ng = vl.download(96)
    np.testing.assert_array_equal(cg, co)
    k = np.arange(96)[None, :] < co[:, None]
    np.testing.assert_array_equal(np.sort(np.where(k, ng, -1), 1), np.sort(np.where(k, no, -1), 1))


def test_sparse_box_keeps_full_radius_cells(M):
    """A box with far more half-radius cells than particles (4.4e9 of them,
    beyond 2^31) still builds its list."""
    L = 2300.0
    pos = np.array([[1.0, 1.0, 1.0], [2.0, 1.0, 1.0], [L / 2] * 3, [L / 2, L / 2, L / 2 + 2.7]])
    a = M.Atoms.from_arrays(pos, capacity=64)
    vl = M.HalfVerletList()
    vl.build(a, 0, 4, 2.8, 1.0, [0.0] * 3, [L] * 3, 8)
    assert vl.total_pairs == 2


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
@pytest.mark.parametrize("n,box,apm", [(2200, (40.0, 9.0, 9.0), 3), (19759, (110.0, 19.0, 19.0), 1),
                                       (19761, (110.0, 19.0, 19.0), 1), (20001, (110.0, 19.0, 19.0), 2)])
def test_lj_ideal_gas_lanes(M, orc, n, box, apm, prec):
    """LJ_IdealGas with four lanes per molecule (below 19,760 molecules on 152
    SMs) and two, single- and multi-site, rows of more than one chunk (random
    placement, density 0.2 to 0.5): forces before the fold-back and the energy
    against the oracle, by the bars of the FP64 and the mixed form."""
    from test_gpu_adress import adress_system, upload_molecules

    mo, ao, corr, sd, slab, (rc, skin, _) = adress_system(orc, n, box, 17, apm)
    co, no = orc.build_half_list(mo.pos, mo.numLocal + mo.numGhost, 0, mo.numLocal, rc + skin, sd.minGhostCorner,
                                 sd.maxGhostCorner, 1.0, 256)
    assert co.max() > 40
    ig_o = orc.LJIdealGas(0.8, rc, 1.0, 1.0, True)
    ao.force[:] = 0
    mo.force[:] = 0
    Eo = ig_o.run(mo, co, no, ao)
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


# Eight lanes per row below 6,080 atoms on 152 SMs, four below 97,280, two
# above; rows of more than 40 entries (several chunks) with rc 4.
@pytest.mark.parametrize("cells,drop,rc,cap,pred,lo", [
    (4, 255, 2.5, 0.0, None, [0.0, 0.0, 0.0]),
    (5, 3, 2.5, 0.95, None, [-3.0, 2.5, 0.0]),
    (12, 833, 2.5, 0.0, "either", [0.0, 0.0, 0.0]),      # 6,079
    (12, 831, 4.0, 0.95, None, [0.0, 0.0, 0.0]),         # 6,081
    (29, 277, 2.5, 0.95, "both", [0.0, 0.0, 0.0]),       # 97,279
    (29, 275, 3.2, 0.0, None, [100.0, -100.0, 0.1]),     # 97,281
])
def test_mixed_half_lanes(M, orc, cells, drop, rc, cap, pred, lo):
    """Forces within the mixed form's bar of the oracle's (1e-6 of the rms
    force), the energy within 1e-7."""
    pos, L = fluid(cells, drop, 0.8 if cells > 4 else 0.4, cells + drop, lo)
    (Fo, Eo, Wo), gpu = both(M, orc, pos, lo, L, rc, orc.lj_table(cap, rc, 1.0, 1.0, 1, True), pred)
    F, E, W = gpu(M.LennardJones(rc, 1.0, 1.0, cap, is_shifted=True), M.PREC_MIXED)
    rms = np.sqrt((Fo ** 2).sum(1).mean())
    assert np.linalg.norm(F - Fo, axis=1).max() <= 1e-6 * rms
    assert abs(E - Eo) <= 1e-7 * abs(Eo)


# Blocks of 1,024 atoms, the scan of 256 blocks at a time; boxes thinner than
# two ghost layers (an atom with images on both sides of an axis).
@pytest.mark.parametrize("n,box,thickness", [
    (1, (6.0, 6.0, 6.0), 2.8), (1023, (14.0, 11.0, 9.0), 2.8), (1024, (5.0, 9.0, 4.0), 2.8),
    (1025, (4.0, 4.0, 4.0), 3.5), (5000, (40.0, 3.0, 12.0), 2.8), (263200, (90.0, 60.0, 50.0), 2.8), (320001, (90.0, 60.0, 50.0), 2.8),
    (700, (20.0, 20.0, 20.0), 0.0),
])
def test_ghost_images_bit_exact(M, orc, n, box, thickness):
    """Ghost positions, order, real atoms and the folded-back forces are the
    oracle's, bit for bit."""
    rng = np.random.default_rng(n)
    pos = rng.uniform(0, 1, (n, 3)) * np.asarray(box)
    pos[:3] = np.array([[0.0, 0.0, 0.0], [thickness] * 3, np.asarray(box) - thickness])[: min(n, 3)] % np.asarray(box)
    sd_o, sd_g = orc.subdomain([0, 0, 0], list(box), thickness), M.Subdomain([0, 0, 0], list(box), thickness)
    ao = orc.Atoms.from_positions(pos, capacity=28 * n + 64 if n < 10000 else 2 * n)
    corr = orc.create_ghosts(ao, sd_o)
    ag = M.Atoms.from_arrays(pos, vel=pos * 2, type=np.arange(n) % 7, mass=1.0 + np.arange(n) % 3)  # room for n ghosts
    gl = M.GhostLayer()
    gl.createGhostAtoms(ag, sd_g)
    assert ag.numGhostAtoms == ao.n - n
    d = ag.download()
    np.testing.assert_array_equal(d["pos"], ao.pos[: ao.n])
    real = gl.correspondingRealAtom(ao.n)
    np.testing.assert_array_equal(real[n:], corr[n: ao.n])
    assert np.all(real[:n] == -1)
    np.testing.assert_array_equal(d["vel"][n:], d["vel"][real[n:]])
    np.testing.assert_array_equal(d["type"][n:], d["type"][real[n:]])
    np.testing.assert_array_equal(d["mass"][n:], d["mass"][real[n:]])
    f = rng.normal(0, 1, (ao.n, 3))
    ao.force[: ao.n] = f
    orc.ghost_to_real(ao, corr)
    ag.upload(n, ao.n - n, force=f)
    gl.contributeBackGhostToReal(ag)
    np.testing.assert_array_equal(ag.getForce(), ao.force[: ao.n])


# Half-radius cells of the list grid: one scan tile (1,024 cells) and one more
# cell than that, many tiles, and more than 2,048 tiles (2,097,152 cells),
# where the tile totals are scanned in a launch of their own.
@pytest.mark.parametrize("n,box", [(900, (8.0, 8.0, 8.0)), (900, (20.5, 5.0, 2.5)), (5000, (30.0, 30.0, 30.0)),
                                   (200000, (66.0, 66.0, 66.0))])
def test_list_counts_over_scan_sizes(M, n, box):
    """The half list's pairs are those within the radius, and its totals are
    the sums of its counts."""
    spatial = pytest.importorskip("scipy.spatial")
    pos = np.random.default_rng(n).uniform(0, 1, (n, 3)) * np.asarray(box)
    a = M.Atoms.from_arrays(pos)
    vl = M.HalfVerletList()
    vl.build(a, 0, n, 1.0, 1.0, [0.0] * 3, list(box), 30)
    counts, nbrs = vl.download()
    tree = spatial.cKDTree(pos)
    assert vl.total_pairs == counts.sum() == (tree.count_neighbors(tree, 1.0) - n) // 2
    got = np.concatenate([np.stack([np.full(c, i), nbrs[i, :c]], 1) for i, c in enumerate(counts) if c])
    got = np.unique(np.sort(got, 1), axis=0)
    np.testing.assert_array_equal(got, np.unique(np.sort(tree.query_pairs(1.0, output_type="ndarray"), 1), axis=0))


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
@pytest.mark.parametrize("n", [2, 9, 128, 129, 130, 300])
def test_adjoint_rows_over_chunk_edges(M, n, prec):
    """The adjoint of one force evaluation with rows of n - 1 entries (chunks
    of 128; n = 130, 300: more than one), all pairs in range and atomistic,
    against the sum over pairs in FP64.  FP64: 1e-12 of the summed magnitudes
    (under 100 roundings a pair and 300 adds, each 2^-53, is 5e-14).  Mixed:
    pairs beyond r_split in FP32, about 20 roundings a term and 75 adds a lane,
    each 2^-24: 6e-6 of the magnitudes."""
    rng = np.random.default_rng(n)
    box, rc, cap = [40.0, 10.0, 10.0], 2.5, 0.7842
    pos = np.array([19.3, 4.3, 4.3]) + rng.uniform(0, 1.4, (n, 3))
    rep = M.Replica(n, [0, 0, 0], box, [20.0, 5.0, 5.0], 10.0, 31)
    d = M.DiffSystem(rep, pos, np.zeros((n, 3)), hybrid_diameter=5.0, steps=5, window=5, checkpoint_interval=5,
                     loss_bins=32, loss_sigma=1.0, capping_distance=cap, rebuild_interval=5,
                     precision=M.PREC_FP64 if prec == "fp64" else M.PREC_MIXED)
    a = rng.normal(size=(n, 3))
    _, xbar, _, ge, gs = d.force_vjp(np.zeros(d.num_bins), 1.0, 1.0, a)
    r = pos[:, None] - pos[None]
    da = a[:, None] - a[None]
    s = (r * r).sum(2) + np.eye(n)
    q = (da * r).sum(2)
    far = s >= cap * cap
    C = 48 * cap ** -13 - 24 * cap ** -7  # force at the cap, d/dsigma below
    Cs = 12 * 48 * cap ** -13 - 6 * 24 * cap ** -7
    f = np.where(far, 48 * s ** -7 - 24 * s ** -4, C / np.sqrt(s))
    fp = np.where(far, -7 * 48 * s ** -8 + 4 * 24 * s ** -5, -0.5 * C * s ** -1.5)
    fs = np.where(far, 12 * 48 * s ** -7 - 6 * 24 * s ** -4, Cs / np.sqrt(s))
    off = 1.0 - np.eye(n)
    t1, t2 = 2 * (fp * q * off)[:, :, None] * r, (f * off)[:, :, None] * da
    tol = 1e-12 if prec == "fp64" else 6e-6
    assert np.all(np.abs(xbar - (t1 + t2).sum(1)) <= tol * (np.abs(t1) + np.abs(t2)).sum(1))
    assert abs(ge - 0.5 * (q * f * off).sum()) <= tol * np.abs(q * f * off).sum()
    assert abs(gs - 0.5 * (q * fs * off).sum()) <= tol * np.abs(q * fs * off).sum()


# Bins wider than the kernel's reach allows for one visit each (4, 5), the
# first count that takes the direct form (6), the Gaussian by factors (16: bins of
# 2.5 sigma, to 100: 16 bins on a side), 32 columns a bin and one (4,097)
@pytest.mark.parametrize("bins", [4, 5, 6, 15, 16, 17, 33, 100, 107, 4096, 4097])
def test_density_loss_over_bin_counts(M, bins):
    """The loss of one step's smoothed density against NumPy in FP64 (a sum of
    n terms rounds to under 1e-13 of itself)."""
    n, L, area = 500, 40.0, 100.0
    rng = np.random.default_rng(5)
    pos = rng.uniform(0, 1, (n, 3)) * [L, 10.0, 10.0]
    rep = M.Replica(n, [0, 0, 0], [L, 10.0, 10.0], [20.0, 5.0, 5.0], 10.0, 31)
    d = M.DiffSystem(rep, pos, rng.normal(size=(n, 3)), hybrid_diameter=5.0, steps=1, window=1, checkpoint_interval=5,
                     loss_bins=bins, loss_sigma=1.0, capping_distance=0.7842, rebuild_interval=5,
                     precision=M.PREC_FP64)
    tab = rng.normal(0, 0.3, d.num_bins)
    L0 = d.forward(tab, 1.0, 1.0)
    x = d.state()[0][:, 0]
    dd = x[:, None] - (np.arange(bins) + 0.5) * (L / bins)
    dd -= L * np.rint(dd / L)
    k = np.where(np.abs(dd) > 6.0, 0.0, np.exp(-0.5 * dd * dd) / np.sqrt(2 * np.pi))
    rho = k.sum(0) / area
    assert abs(L0 - ((rho - n / (L * area)) ** 2).sum()) <= 1e-11 * (rho ** 2).sum()


# Blocks of 256 and of 1,024 molecules (above 152 * 2,048), one to three atoms
# in a molecule, boxes thinner than two ghost layers
@pytest.mark.parametrize("n,box,thickness", [
    (1, (6.0, 6.0, 6.0), 2.8), (255, (4.0, 9.0, 5.0), 2.8), (257, (14.0, 3.5, 9.0), 2.8), (5000, (40.0, 12.0, 12.0), 2.8),
    (320000, (90.0, 60.0, 50.0), 2.8), (300, (20.0, 20.0, 20.0), 0.0),
])
def test_molecule_images_bit_exact(M, orc, n, box, thickness):
    """Ghost molecules and their atoms, in the oracle's order, bit for bit."""
    rng = np.random.default_rng(n)
    size = rng.integers(1, 4, n)
    first = np.concatenate([[0], np.cumsum(size)[:-1]])
    na = int(size.sum())
    mpos = rng.uniform(0, 1, (n, 3)) * np.asarray(box)
    apos = np.repeat(mpos, size, axis=0) + rng.normal(0, 0.15, (na, 3))
    room = 27 if n < 10000 else 3
    mo = orc.Molecules(n * room + 64)
    mo.pos[:n], mo.atomsOffset[:n], mo.numAtoms[:n], mo.numLocal = mpos, first, size, n
    mo.lambda_[:n] = rng.uniform(0, 1, n)
    ao = orc.Atoms.from_positions(apos, capacity=na * room + 64)
    corr = orc.multires_create_ghosts(mo, ao, orc.subdomain([0, 0, 0], list(box), thickness))
    m = M.Molecules(n)  # room for no ghost
    m.upload(n, 0, pos=mpos, force=np.zeros((n, 3)), lambda_=mo.lambda_[:n], modulated_lambda=np.zeros(n),
             grad_lambda=np.zeros((n, 3)), atoms_offset=first, num_atoms=size)
    a = M.Atoms.from_arrays(apos, type=np.arange(na) % 7)
    gl = M.MultiResGhostLayer()
    gl.createGhostAtoms(m, a, M.Subdomain([0, 0, 0], list(box), thickness))
    nm, nt = mo.numLocal + mo.numGhost, ao.numLocal + ao.numGhost
    assert (m.numGhostMolecules, a.numGhostAtoms) == (mo.numGhost, ao.numGhost)
    d, da = m.download(), a.download()
    np.testing.assert_array_equal(d["pos"], mo.pos[:nm])
    np.testing.assert_array_equal(d["atomsOffset"], mo.atomsOffset[:nm])
    np.testing.assert_array_equal(d["numAtoms"], mo.numAtoms[:nm])
    np.testing.assert_array_equal(d["lambda_"], mo.lambda_[:nm])
    np.testing.assert_array_equal(da["pos"], ao.pos[:nt])
    real = gl.correspondingRealAtom(nt)
    np.testing.assert_array_equal(real[na:], corr[na:nt])
    np.testing.assert_array_equal(da["type"][na:], da["type"][real[na:]])


# Rows of one lane and of several (97,280 and 9,728 rows on 152 SMs); particles
# up to 3 beyond the grid (they sit in its outermost cells), a grid far from
# the origin (FP32 coordinates good to 1e-4 there), one cell on an axis.
@pytest.mark.parametrize("n,box,origin,out", [(3000, (9.0, 7.0, 6.0), 0.0, 3.0), (3000, (9.0, 7.0, 1.0), 1000.0, 0.0),
                                              (12000, (22.0, 14.0, 17.0), -37.3, 0.4), (100000, (50.0, 50.0, 50.0), 0.0, 2.0)])
def test_list_keeps_every_pair_when_cells_are_cut(M, n, box, origin, out):
    """Cells out of reach of a row are skipped; the list is still every pair
    within the radius."""
    spatial = pytest.importorskip("scipy.spatial")
    box = np.asarray(box)
    pos = origin + np.random.default_rng(n).uniform(0, 1, (n, 3)) * (box + 2 * out) - out
    a = M.Atoms.from_arrays(pos)
    vl = M.HalfVerletList()
    vl.build(a, 0, n, 1.3, 1.0, [origin] * 3, list(origin + box), 60)
    counts, nbrs = vl.download()
    got = np.concatenate([np.stack([np.full(c, i), nbrs[i, :c]], 1) for i, c in enumerate(counts) if c])
    got = np.unique(np.sort(got, 1), axis=0)
    assert len(got) == counts.sum()
    tree = spatial.cKDTree(pos)
    np.testing.assert_array_equal(got, np.unique(np.sort(tree.query_pairs(1.3, output_type="ndarray"), 1), axis=0))


# Tiles of 256 rows with four threads a row up to two tiles per SM (304 on 152
# SMs, 77,824 rows), one above; a row more than a tile, less than a warp; rows
# whose quarter of the columns holds more than 64 entries (r_list 4.0: one
# thread a row from then on).
@pytest.mark.parametrize("cells,atoms,rc", [(8, 2048, 2.5), (8, 2031, 2.5), (10, 3841, 2.5), (27, 77824, 2.5),
                                            (27, 77825, 2.5), (10, 4000, 3.7)])
def test_tile_list_threads_per_row(M, cells, atoms, rc):
    """The one-pass tile list has the rows, and in them the order, of the one
    made from the int32 rows: bitwise equal forces after a few rebuilds."""
    from test_gpu_md import fcc, mb_velocities

    pos, L = fcc(cells)
    keep = np.sort(np.random.default_rng(atoms).permutation(len(pos))[:atoms])
    pos, vel = pos[keep], mb_velocities(len(pos), 0.728, 9)[keep]
    a, b = (M.LJSystem(pos, vel, [0, 0, 0], [L] * 3, rc=rc, precision=M.PREC_MIXED, tile_build=t)
            for t in ("one_pass", "two_kernel"))
    a.run(25)
    b.run(25)
    assert a.tile_stats()["tiled"] and b.tile_stats()["tiled"]
    for x, y in zip(a.state(), b.state()):
        np.testing.assert_array_equal(x, y)
    np.testing.assert_array_equal(a.pair_keys(), b.pair_keys())

"""The kernels' dispatch rules at the sizes where they change: list sort, pair work, plane
transform, stencil orders, virial, kinetic energy, state copies, against the CPU oracle (or numpy).

Tolerances as tests/test_gpu_parity.py: FP64 1e-9 and mixed 1e-5 of the norm of the forces; virials
ten times that of their largest component."""
import numpy as np
import pytest

from oracle import oracle as O
from protomol3_b200 import forces as F
from protomol3_b200 import waterbox as W

pytestmark = pytest.mark.gpu
TOL = {"fp64": 1e-9, "mixed": 1e-5}


def rel(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


def shaken(n, seed):
    """A water box with stretched bonds and bent angles."""
    b = W.water_box(n, seed=seed)
    b["pos"] = b["pos"] + np.random.default_rng(seed).normal(0.0, 0.02, b["pos"].shape)
    return b


def evaluate(boxes, fl, precision, virial=False):
    topo = F.Topology(boxes, precision)
    f, e = np.zeros((topo.n_atoms, 3)), F.ScalarStructure(topo.n_boxes, virial=virial)
    F.evaluate_all(topo, fl, topo.positions(), f, e)
    return f, e, topo


# 1024 waters are the last box that one CTA sorts (3,072 atoms); 2 waters are less than a block
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("waters", [2, 3, 341, 1024, 1025])
def test_list_sort_and_units(precision, waters):
    b = shaken(waters, 31)
    cut = min(8.0, 0.45 * b["box"][0])
    f, e, topo = evaluate(b, [F.NonbondedCutoffSystemForce(lj=("C2", 0.8 * cut, cut), coulomb=("C1", 0.0, cut)),
                              F.BondedSystemForce()], precision, virial=True)
    fo, _, vo, _ = O.evaluate(O.System(b), b["pos"], cutoff=O.cutoff_params(lj=("C2", 0.8 * cut, cut), coul=("C1", 0.0, cut)),
                              bonded=True, virial=True)
    assert rel(f, fo) < TOL[precision]
    np.testing.assert_allclose(e.virial().ravel(), vo, rtol=0, atol=10 * TOL[precision] * np.abs(vo).max() + 1e-7)
    assert topo.list_tiles() >= -(-topo.n_atoms // 8)


def test_large_boxes_of_one_system_sort_alike():
    """Boxes above and below the one-CTA size in one system (a launch per phase) give each box's
    own forces bit for bit."""
    boxes = [shaken(n, 40 + n) for n in (1500, 40, 1025)]
    fl = lambda: [F.NonbondedCutoffSystemForce(lj=("C2", 6.0, 7.0))]  # noqa: E731
    f, _, _ = evaluate(boxes, fl(), "mixed")
    at = 0
    for b in boxes:
        n = len(b["charge"])
        alone, _, _ = evaluate(b, fl(), "mixed")
        np.testing.assert_array_equal(f[at:at + n], alone)
        at += n


# every radix of the plane transform, one to three stages, odd rows, a virial; 128 x 125 FP64 does not
# fit shared memory and takes the line kernels
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("grid", [(8, 9, 10), (12, 15, 16), (25, 27, 20), (10, 81, 24), (50, 6, 45), (125, 24, 8),
                                  (128, 125, 9), (4, 5, 6), (72, 54, 12)])
def test_plane_transform(precision, grid):
    b = shaken(60, 7)
    pme = F.NonbondedPMEwaldSystemForce(grid, 6.0, real=False, correction=False)
    f, e, _ = evaluate(b, [pme], precision, virial=True)
    fo, _, vo, _ = O.evaluate(O.System(b), b["pos"], pme=O.pme_params(grid, 6.0, real=0, recip=1, corr=0), virial=True)
    assert rel(f, fo) < TOL[precision]
    np.testing.assert_allclose(e.virial().ravel(), vo, rtol=0, atol=10 * TOL[precision] * np.abs(vo).max())


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("order", [2, 4, 6, 8])
def test_stencil_orders(precision, order):
    b = shaken(77, 5)
    f, _, _ = evaluate(b, [F.NonbondedPMEwaldSystemForce((16, 18, 20), 6.0, order=order)], precision)
    fo, _, _, _ = O.evaluate(O.System(b), b["pos"], pme=O.pme_params((16, 18, 20), 6.0, order=order))
    assert rel(f, fo) < TOL[precision]


# edges just above and below what lets a tile skip the image per pair (2 (cutoff + cluster extent + skin))
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("waters", [130, 260, 420, 700])
def test_virial_with_and_without_wrapped_tiles(precision, waters):
    b = shaken(waters, 19)
    g = W.pme_grid_for(b["box"][0])
    f, e, _ = evaluate(b, [F.NonbondedCutoffSystemForce(lj=("C2", 6.0, 7.5)), F.NonbondedPMEwaldSystemForce((g, g, g), 7.5)],
                       precision, virial=True)
    fo, _, vo, _ = O.evaluate(O.System(b), b["pos"], cutoff=O.cutoff_params(lj=("C2", 6.0, 7.5)),
                              pme=O.pme_params((g, g, g), 7.5), virial=True)
    assert rel(f, fo) < TOL[precision]
    np.testing.assert_allclose(e.virial().ravel(), vo, rtol=0, atol=10 * TOL[precision] * np.abs(vo).max())


# one part, exactly one, one atom more, several; summation order only: n ulp at most
@pytest.mark.parametrize("waters", [1, 682, 683, 7300])
def test_kinetic_energy_and_state(waters):
    """The kinetic energy of boxes of one and several parts; 7,300 waters (65,700 doubles) also take
    the staged state copy."""
    b = W.water_box(waters, seed=2)
    topo = F.Topology(b, "mixed")
    md = F.Integrator(topo, [F.BondedSystemForce()])
    md.set_state(b["pos"], b["vel"])
    _, kin = md.energies()
    want = 0.5 * (b["mass"][:, None] * b["vel"] ** 2).sum()
    assert abs(kin[0] - want) <= 3 * waters * 2.3e-16 * want
    for _ in range(2):  # the second copy reuses the staging
        pos, vel = md.state()
        np.testing.assert_array_equal(pos, b["pos"])
        np.testing.assert_array_equal(vel, b["vel"])


@pytest.mark.parametrize("kind", ["leapfrog", "langevin"])
def test_forces_outlive_the_list(kind):
    """A run whose list storage is replaced between two calls goes on with the same forces: equal to
    an uninterrupted one but for the order of the sums (other clusters), 1e-12 relative per step in
    FP64, which ten steps amplify by less than 1e2."""
    b = shaken(300, 3)
    out = []
    for change in (False, True):
        topo = F.Topology(b, "fp64")
        md = F.Integrator(topo, [F.NonbondedCutoffSystemForce(lj=("C2", 6.0, 7.0)), F.BondedSystemForce()], kind=kind, seed=5)
        md.set_state(b["pos"], b["vel"])
        md.run(5)
        if change:
            topo.set_tuning(skin=0.5, sort_cell=1.9)
        md.run(5)
        out.append(np.concatenate(md.state()))
    assert rel(out[1], out[0]) < 1e-10


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("extra", ["", "bonded"])
def test_slots_rebuilt_without_pair_lists(precision, extra):
    """Sets without a pair term sort their atoms but build no lists.  1,100 waters take the launch per
    phase: two unrelated configurations, then a pair set and the first set again on the same system,
    so every build starts from the bins that a build of either kind left."""
    b, other = shaken(1100, 61), shaken(1100, 62)
    grid = (20, 24, 18)
    topo = F.Topology(b, precision)
    slow = [F.NonbondedPMEwaldSystemForce(grid, 7.0, real=False, correction=False)]
    if extra:
        slow.append(F.BondedSystemForce())
    fast = [F.NonbondedCutoffSystemForce(lj=("C2", 6.0, 7.0), coulomb=("C1", 0.0, 7.0))]
    pme = O.pme_params(grid, 7.0, real=0, recip=1, corr=0)
    cut = O.cutoff_params(lj=("C2", 6.0, 7.0), coul=("C1", 0.0, 7.0))
    for pos, fl in [(b["pos"], slow), (other["pos"], slow), (b["pos"], fast), (other["pos"], slow), (b["pos"], slow),
                    (other["pos"], fast)]:
        pos = np.ascontiguousarray(pos)
        f = np.zeros((topo.n_atoms, 3))
        F.evaluate_all(topo, fl, pos, f, F.ScalarStructure(1))
        kw = dict(cutoff=cut) if fl is fast else dict(pme=pme, bonded=bool(extra))
        fo, _, _, _ = O.evaluate(O.System(b), pos, **kw)
        assert rel(f, fo) < TOL[precision]


@pytest.mark.parametrize("rc", [5.0, 10.0])
@pytest.mark.parametrize("edge", [200.0, 2000.0, 4000.0])
def test_list_of_a_dilute_box(edge, rc):
    """Chains of three charges in a wide box, neighbours 1e-6 to 1e-4 A inside the cutoff, and no skin:
    blocks of eight atoms spread over up to half the box (the list's test in FP32 has 1e-3 A to
    spare).  A charge pair that the list leaves out changes two forces by 332 / rc^2."""
    rng = np.random.default_rng(17)
    n = 300
    step = rng.normal(size=(n, 2, 3))
    step *= ((rc - 10.0 ** rng.uniform(-6, -4, (n, 2))) / np.linalg.norm(step, axis=2))[:, :, None]
    first = rng.uniform(0.0, edge, (n, 3))
    pos = np.stack([first, first + step[:, 0], first + step.sum(1)], 1).reshape(-1, 3)
    b = W.water_box(n, seed=1, edge=edge)
    none = np.zeros((0, 2), np.int32)
    b.update(pos=pos, charge=np.tile([18.2, -18.2, 18.2], n), molecule=np.arange(3 * n, dtype=np.int32),
             excl_pairs=none, excl_kind=np.zeros(0, np.int32))
    topo = F.Topology(b, "fp64")
    topo.set_tuning(skin=0.0, sort_cell=50.0)
    f = np.zeros_like(pos)
    F.evaluate_all(topo, [F.NonbondedCutoffSystemForce(coulomb=("cutoff", 0.0, rc))], pos, f, F.ScalarStructure(1))
    fo, _, _, _ = O.evaluate(O.System(b), pos, cutoff=O.cutoff_params(coul=("cutoff", 0.0, rc)))
    assert rel(f, fo) < TOL["fp64"]


def test_kinetic_energy_of_many_boxes():
    """More boxes than a grid's second dimension holds (65,535)."""
    n = 65600
    one = dict(box=np.full(3, 10.0), charge=[0.0], type=[0], molecule=[0], lj=np.zeros(4), mass=[2.0])
    topo = F.Topology([one] * n, "mixed")
    md = F.Integrator(topo, [F.BondedSystemForce()])
    vel = np.zeros((n, 3))
    vel[:, 0] = np.arange(n)
    md.set_state(np.ones((n, 3)), vel)
    _, kin = md.energies()
    np.testing.assert_array_equal(kin, vel[:, 0] ** 2)


# a slab of 2.1 million sort cells, a cluster alone in such a box (fewer atoms than one CTA sorts), and
# the latter beside an ordinary box
@pytest.mark.parametrize("boxes", [["slab"], ["cluster"], ["cluster", "liquid"]])
def test_sort_of_a_wide_box(boxes):
    """Sort cells follow the longest edge: many are scanned by the whole chip, and cleared for the next
    build.  Several unrelated configurations, each against the oracle."""
    rng = np.random.default_rng(23)
    rc = 8.0
    fill = {"slab": ([40.0, 40.0, 400.0], [40.0, 40.0, 400.0], 5000), "cluster": ([400.0] * 3, [20.0] * 3, 300),
            "liquid": ([30.0] * 3, [30.0] * 3, 2000)}
    systems = []
    for name in boxes:
        edges, _, n = fill[name]
        systems.append(dict(box=np.array(edges), charge=np.where(np.arange(n) % 2, 18.2, -18.2), type=np.zeros(n, np.int32),
                            molecule=np.arange(n, dtype=np.int32), lj=np.zeros(4), mass=np.ones(n)))
    topo = F.Topology(systems, "fp64")
    force = F.NonbondedCutoffSystemForce(coulomb=("C1", 0.0, rc))
    for _ in range(3):
        pos = [rng.uniform(0.0, 1.0, (fill[n][2], 3)) * fill[n][1] for n in boxes]
        f = np.zeros((topo.n_atoms, 3))
        F.evaluate_all(topo, [force], np.concatenate(pos), f, F.ScalarStructure(len(boxes)))
        at = 0
        for b, p in zip(systems, pos):
            fo, _, _, _ = O.evaluate(O.System(dict(b, pos=p)), p, cutoff=O.cutoff_params(coul=("C1", 0.0, rc)))
            assert rel(f[at:at + len(p)], fo) < TOL["fp64"]
            at += len(p)


# 80 boxes at both sides of the largest that one CTA each sorts (8,192 atoms), and small ones beside one
# that all would wait for
@pytest.mark.parametrize("sizes", [[8192, 8185], [8200, 8185], [24, 5000]])
def test_sort_of_many_boxes(sizes):
    """Each box of a system of many gets the forces it gets alone, bit for bit, at the first build and
    at the next one."""
    rng = np.random.default_rng(29)
    edge = lambda n: (10.0 * n) ** (1.0 / 3.0)  # noqa: E731
    box = lambda n: dict(box=np.full(3, max(edge(n), 15.0)), charge=np.where(np.arange(n) % 2, 18.2, -18.2),  # noqa: E731
                         type=np.zeros(n, np.int32), molecule=np.arange(n, dtype=np.int32), lj=np.zeros(4), mass=np.ones(n))
    boxes = [box(sizes[0])] * 40 + [box(sizes[1])] + [box(sizes[0])] * 39
    at = np.concatenate([[0], np.cumsum([len(b["charge"]) for b in boxes])])
    force = lambda: [F.NonbondedCutoffSystemForce(coulomb=("C1", 0.0, 6.0))]  # noqa: E731
    topo = F.Topology(boxes, "mixed")
    fl = force()
    alone = {k: (F.Topology(boxes[k], "mixed"), force()) for k in (0, 40, 79)}
    for _ in range(2):
        pos = np.concatenate([rng.uniform(0.0, b["box"][0], (len(b["charge"]), 3)) for b in boxes])
        f = np.zeros_like(pos)
        F.evaluate_all(topo, fl, pos, f, F.ScalarStructure(len(boxes)))
        for k, (t, one) in alone.items():
            p = np.ascontiguousarray(pos[at[k]:at[k + 1]])
            g = np.zeros_like(p)
            F.evaluate_all(t, one, p, g, F.ScalarStructure(1))
            np.testing.assert_array_equal(f[at[k]:at[k + 1]], g)


# planes above 227 KB: lines of both forms in either direction, the shortest and longest of each
@pytest.mark.parametrize("precision,grid", [
    ("mixed", (160, 192, 8)), ("mixed", (240, 128, 9)), ("mixed", (192, 160, 8)), ("mixed", (128, 240, 10)),
    ("mixed", (250, 200, 8)), ("mixed", (256, 256, 8)), ("fp64", (64, 240, 8)), ("fp64", (240, 64, 9)),
    ("fp64", (250, 96, 8)), ("fp64", (96, 250, 10)), ("fp64", (128, 128, 8)), ("fp64", (160, 160, 8)), ("fp64", (150, 125, 8))])
def test_planes_too_large_for_shared_memory(precision, grid):
    b = shaken(60, 7)
    pme = F.NonbondedPMEwaldSystemForce(grid, 6.0, real=False, correction=False)
    f, e, _ = evaluate(b, [pme], precision, virial=True)
    fo, eo, vo, _ = O.evaluate(O.System(b), b["pos"], pme=O.pme_params(grid, 6.0, real=0, recip=1, corr=0), virial=True)
    assert rel(f, fo) < TOL[precision]
    np.testing.assert_allclose(e.virial().ravel(), vo, rtol=0, atol=10 * TOL[precision] * np.abs(vo).max())


# the largest box of each block size of the one-CTA sort (64 to 1,024 threads), and one atom more
@pytest.mark.parametrize("atoms", [63, 64, 65, 128, 129, 256, 257, 512, 513, 1023, 1025])
def test_one_cta_sort_of_each_size(atoms):
    rng = np.random.default_rng(atoms)
    edge = max(10.0, (10.0 * atoms) ** (1.0 / 3.0))
    b = dict(box=np.full(3, edge), charge=np.where(np.arange(atoms) % 2, 18.2, -18.2), type=np.zeros(atoms, np.int32),
             molecule=np.arange(atoms, dtype=np.int32), lj=np.zeros(4), mass=np.ones(atoms))
    topo = F.Topology(b, "fp64")
    for _ in range(2):
        pos = rng.uniform(0.0, edge, (atoms, 3))
        f = np.zeros_like(pos)
        F.evaluate_all(topo, [F.NonbondedCutoffSystemForce(coulomb=("C1", 0.0, 4.5))], pos, f, F.ScalarStructure(1))
        fo, _, _, _ = O.evaluate(O.System(dict(b, pos=pos)), pos, cutoff=O.cutoff_params(coul=("C1", 0.0, 4.5)))
        assert rel(f, fo) < TOL["fp64"]

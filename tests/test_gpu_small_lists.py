"""Edges of the size rules: purification sizes, atoms per warp of the one-electron kernels, lanes of short
quartet lists, the line between short and long lists, and work lists of more bras than one pass of the prefix
sums.

Tolerances: integrals, Fock matrices and gradients as in test_gpu_hf.py (1e-10, 1e-8); the purified density
stops where tr(P - P^2) < 1e-12 before a last squaring step, so that in an orthonormal basis the idempotency error
is rounding of m-term sums of elements of order one over some 40 steps, below m^2 eps; the tests' limits
around P S P allow for the condition of S on top.
"""
import numpy as np
import pytest

import oracle
from conftest import ANGSTROM_TO_BOHR
from pdynamo3_b200 import geometry
from pdynamo3_b200.basis import ShellTable

pytestmark = pytest.mark.gpu


def _context(basis, z, xyz):
    from pdynamo3_b200.lib import Context
    ctx = Context(0)
    ctx.set_basis(ShellTable(basis, z))
    ctx.set_geometry(xyz)
    return ctx


def _full(packed):
    n = int((np.sqrt(8 * len(packed) + 1) - 1) / 2)
    M = np.zeros((n, n))
    M[np.tril_indices(n)] = packed
    return M + np.tril(M, -1).T


# functions: 4 (one tile), 57 and 72 (either side of one row tile per warp), 126 (below the
# largest of the one-launch form, 128), 133, 144 and 152 (GEMMs)
@pytest.mark.parametrize("basis,waters", [("6-31g_st_cart", 0), ("6-31g_st_cart", 3), ("6-31g_st", 4), ("6-31g_st", 7),
                                          ("6-31g_st_cart", 7), ("6-31g_st", 8), ("6-31g_st_cart", 8)])
def test_purified_density_is_a_projector(cuda_device, basis, waters):
    if waters:
        z, xyz = geometry.water_cluster(waters, max(3.0, 3.2 * waters ** (1.0 / 3.0)), 7)
    else:
        z, xyz = np.array([1, 1]), np.array([[0.0, 0.0, 0.0], [0.0, 0.0, 0.74]])
    ctx = _context(basis, z, xyz * ANGSTROM_TO_BOHR)
    P, res = ctx.scf(density_tolerance=1e-9, energy_tolerance=1e-8)
    S = _full(ctx.one_electron()[0])
    P = _full(P)
    assert res.converged
    assert abs((P * S).sum() - z.sum()) < 1e-9
    assert np.abs(P @ S @ P - 2.0 * P).max() < 1e-10


def test_one_launch_form_has_its_cluster(cuda_device):
    from pdynamo3_b200.lib import load
    assert [load().pdg_purify_clusters(m) > 0 for m in (1, 64, 65, 128, 129)] == [True, True, True, True, False]


def _stretched_ethene():
    """C2H4 with bonds 1.6 times the ordinary: a gap of some 0.05 hartree in PBE, 1/400 of the spectrum's width."""
    c, h = 0.67, 1.09
    x = [[-c, 0, 0], [c, 0, 0]] + [[s * (c + h * 0.5), t * h * 0.866, 0] for s in (-1, 1) for t in (-1, 1)]
    return np.array([6, 6, 1, 1, 1, 1]), 1.6 * np.array(x)


# iterations of many steps, where rounding errors that a step amplifies would show: molecules of small gaps
# on either side of the tile counts of the one-launch form
@pytest.mark.parametrize("basis,molecule", [("6-31g_st_cart", "ethene"), ("6-31g_st", "ethene"), ("6-31g_st_cart", 5),
                                            ("6-31g_st", 5), ("6-31g_st_cart", 7)])
def test_purified_density_of_small_gaps(cuda_device, basis, molecule):
    z, xyz = _stretched_ethene() if molecule == "ethene" else geometry.organic_molecule(molecule, {5: 5, 7: 1}[molecule])
    ctx = _context(basis, z, xyz * ANGSTROM_TO_BOHR)
    ctx.set_functional("pbe")
    ctx.grid_build(3)
    P, res = ctx.scf(density_tolerance=1e-8, energy_tolerance=1e-7)
    s, U = np.linalg.eigh(_full(ctx.one_electron()[0]))
    root = (U * np.sqrt(s)) @ U.T
    Q = 0.5 * root @ _full(P) @ root  # the lower triangle mirrored: an antisymmetric part shows to first order
    assert res.converged
    assert np.abs(Q @ Q - Q).max() < ctx.n ** 2 * np.finfo(float).eps


@pytest.mark.parametrize("natom", [1, 2, 4, 5, 16, 17, 32, 33])
def test_hydrogen_chains_against_oracle(cuda_device, natom):
    z = np.ones(natom, dtype=int)
    rng = np.random.default_rng(natom)
    xyz = np.stack([1.7 * np.arange(natom), rng.normal(scale=0.3, size=natom), rng.normal(scale=0.3, size=natom)], 1)
    shells = ShellTable("6-31g_st_cart", z)
    ctx = _context("6-31g_st_cart", z, xyz)
    o = oracle.Oracle(shells, xyz)
    S, H, _ = ctx.one_electron()
    So, Ho, _ = o.one_electron()
    assert np.abs(S - So).max() < 1e-10
    assert np.abs(H - Ho).max() < 1e-9
    n = len(So)
    P = 0.2 * rng.normal(size=n)
    W = 0.2 * rng.normal(size=n)
    # one-electron and nuclear terms alone (the oracle's quartets of a long chain take a minute)
    g = np.zeros(3 * natom)
    oracle.lib().orc_one_electron_gradient(P, -0.5 * W, g)
    assert np.abs(ctx.gradients(P, W, 0.0, False) - g.reshape(-1, 3)).max() < 1e-8
    if natom <= 5:
        F, _ = ctx.fock_two_electron(P, 1.0)
        assert np.abs(F - o.fock(P, 1.0)[0]).max() < 1e-10
        assert np.abs(ctx.gradients(P, W, 1.0) - o.gradients(P, W)).max() < 1e-8


def test_work_list_totals(cuda_device):
    """12 waters have more than 1024 (ps) pairs: the device's totals against the host's count of the rule."""
    z, xyz = geometry.water_cluster(12, 7.5, 3)
    ctx = _context("6-31g_st_cart", z, xyz * ANGSTROM_TO_BOHR)
    _, res = ctx.scf(maximum_iterations=50)
    assert res.quartets == ctx.work_estimate("eri_jk")[2]


def test_builds_launch_what_the_autotuner_reports(cuda_device):
    """4 waters have short lists only; 8 waters long ones too, which have no lanes to tune."""
    for waters, long_lists in ((4, False), (8, True)):
        z, xyz = geometry.water_cluster(waters, max(3.0, 3.2 * waters ** (1.0 / 3.0)), 3)
        ctx = _context("6-31g_st_cart", z, xyz * ANGSTROM_TO_BOHR)
        ctx.fock_two_electron(np.full(ctx.npacked(), 0.01), 1.0)
        tuned = ctx.autotune_eri()
        forms = {(b, k): ctx.L.pdg_jk_form_of(ctx.h, b, k) for b in range(6) for k in range(b + 1)}
        assert tuned and all(forms[p] == v for p, v in tuned.items())
        assert ((0, 0) not in tuned) == long_lists == (forms[0, 0] == 8)
        ctx.close()


@pytest.fixture(scope="module")
def four_atoms():
    """s, p and d shells on four atoms: geometry, densities and the oracle's Fock matrices and gradients."""
    from test_gpu_limits import RawShells
    xyz = np.array([[0.0, 0.1, 0.0], [1.9, 0.2, 0.1], [-0.3, 1.7, 0.4], [0.4, -0.2, 2.1]])
    o = oracle.Oracle(RawShells([3, 1, 2, 1], _spd_shells(4)), xyz)
    rng = np.random.default_rng(17)
    npk = o.n * (o.n + 1) // 2
    P, W = 0.3 * rng.normal(size=npk), 0.1 * rng.normal(size=npk)
    kinds = ((1.0, True), (0.0, True), (1.0, False))  # J and K, J, K
    return xyz, P, W, {k: (o.fock(P, *k)[0], o.gradients(P, W, *k)) for k in kinds}


def _spd_shells(n):
    return [s for a in range(n) for s in ((a, 0, 0, [9.0, 1.9, 0.5], [0.1, 0.4, 0.6]), (a, 0, 0, [0.17], [1.0]),
                                          (a, 1, 1, [2.1, 0.4], [0.4, 0.7]), (a, 2, 2, [0.8], [1.0]))]


# The quartets of the four atoms alone (short lists, lanes split over primitives) and among 36 centres without
# charge, density or weight (long lists of every class, one quartet per lane): their Fock block and
# gradient are the same.  In the mixed mode with every quartet in FP32 an element is a sum of some 44^2
# products of 0.3 and an integral of order one, each with a few roundings of 6e-8: 1e-4.
@pytest.mark.parametrize("ghosts,mixed_cut,ftol,gtol", [(0, 0.0, 1e-10, 1e-8), (36, 0.0, 1e-10, 1e-8),
                                                        (0, 1e9, 1e-4, 1e-4), (36, 1e9, 1e-4, 1e-4)])
def test_short_and_long_lists_against_oracle(cuda_device, four_atoms, ghosts, mixed_cut, ftol, gtol):
    from test_gpu_limits import RawShells
    from pdynamo3_b200.lib import Context
    xyz, P, W, expected = four_atoms
    ctx = Context(0)
    ctx.set_basis(RawShells([3, 1, 2, 1] + [0] * ghosts, _spd_shells(4 + ghosts)))
    ctx.set_geometry(np.concatenate([xyz, np.random.default_rng(5).uniform(-4.0, 4.0, size=(ghosts, 3))]))
    ctx.set_eri_options(precision_mode=1 if mixed_cut else 0, mixed_cut=mixed_cut or 1e-6)
    pad = lambda v: np.concatenate([v, np.zeros(ctx.npacked() - len(v))])  # noqa: E731
    for (cx, coulomb), (Fo, go) in expected.items():
        F, _ = ctx.fock_two_electron(pad(P), cx, coulomb)
        assert np.abs(F[:len(P)] - Fo).max() < ftol
        g = ctx.gradients(pad(P), pad(W), cx, coulomb)
        assert np.abs(g[:4] - go).max() < gtol
        assert np.abs(g[4:]).max(initial=0.0) < 1e-12
    forms = {ctx.L.pdg_jk_form_of(ctx.h, b, k) for b in range(6) for k in range(b + 1)} - {-1}
    assert forms == {8} if ghosts else 8 not in forms

"""Partition weights against full products of all cell functions, at the edges of their atom tiles: 1 to 3
atoms in the last tile, 64 full tiles, and warps whose points belong to two or more atoms (few points per
atom).  Wide Gaussians on every atom keep all functions at all points, so that the electron count is the sum
of weight x density over the points and shows every weight.
"""
import os
import re

import numpy as np
import pytest
import torch

from conftest import ANGSTROM_TO_BOHR, ROOT
from test_gpu_limits import RawShells

pytestmark = pytest.mark.gpu

EXPONENT = 0.02
BRAGG = {1: 0.35, 6: 0.70, 8: 0.60}
XPASC = [1.0, -10 / 3, 9.0, -120 / 7, 70 / 3, -252 / 11, 210 / 13, -8.0, 45 / 17, -10 / 19, 1 / 21]  # C(10,t) (-1)^t / (2t+1)


def lebedev(order):
    text = open(os.path.join(ROOT, "pdynamo3_b200", "csrc", "lebedev_table.inc")).read()
    row = lambda n: [int(v) for v in re.search(n + r"\[LEB_NORDERS\] = \{([^}]*)\}", text).group(1).split(",")]  # noqa: E731
    k = row("leb_order").index(order)
    body = re.search(r"leb_data\[[^\]]*\] = \{(.*?)\};", text, re.S).group(1)
    data = np.array([float(v) for v in body.split(",") if v.strip()]).reshape(-1, 4)
    return data[row("leb_offset")[k]:][:row("leb_count")[k]]


def quadrature(z, xyz, n_radial, order):
    """Points and weights, all cell functions formed in full."""
    ang = lebedev(order)
    bragg = np.array([BRAGG[int(k)] for k in z]) * ANGSTROM_TO_BOHR
    x = (np.arange(n_radial) + 1) / (1.0 + n_radial)
    R = np.linalg.norm(xyz[:, None] - xyz[None], axis=2)
    t = (bragg[:, None] / bragg[None] - 1) / (bragg[:, None] / bragg[None] + 1)
    a = np.clip(t / (t * t - 1), -0.5, 0.5)
    c = (XPASC / np.sum(XPASC) / 2).tolist()
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    X, R, a = (torch.as_tensor(v, device=dev) for v in (xyz, R, a))
    pts, wts = [], []
    for g in range(len(z)):
        r, wr = bragg[g] * (x / (1 - x)) ** 2, 2 * bragg[g] ** 3 * x ** 5 / (1 - x) ** 7 / (1 + n_radial)
        q = (xyz[g] + r[:, None, None] * ang[None, :, :3]).reshape(-1, 3)
        d = (torch.as_tensor(q, device=dev)[:, None] - X[None]).norm(dim=2)
        mu = (d[:, :, None] - d[:, None, :]) / R
        nu = mu + a * (1 - mu * mu)
        n2, s = nu * nu, torch.full_like(nu, c[-1])
        for v in c[-2::-1]:
            s = s * n2 + v
        s = 0.5 - s * nu
        s.diagonal(dim1=1, dim2=2).fill_(1.0)
        A = s.prod(dim=2)
        pts.append(q)
        wts.append((4 * np.pi * wr[:, None] * ang[None, :, 3]).reshape(-1) * (A[:, g] / A.sum(dim=1)).cpu().numpy())
    return np.concatenate(pts), np.concatenate(wts)


def cluster(natom):
    """Atoms at least 1.6 bohr apart in a cube of 27 bohr^3 per atom."""
    rng = np.random.default_rng(natom)
    xyz = []
    while len(xyz) < natom:
        p = rng.uniform(0.0, 3.0 * natom ** (1 / 3), 3)
        if all(np.linalg.norm(p - q) > 1.6 for q in xyz):
            xyz.append(p)
    return rng.choice([1, 6, 8], size=natom), np.array(xyz)


@pytest.mark.parametrize("natom", [1, 2, 3, 4, 5, 6, 7, 8, 9, 61, 62, 63, 64, 200, 201, 253, 254, 255, 256])
def test_weights_against_full_products(cuda_device, natom):
    from pdynamo3_b200.lib import Context
    z, xyz = cluster(natom)
    ctx = Context(0)
    ctx.set_basis(RawShells(z, [(i, 0, 0, [EXPONENT], [1.0]) for i in range(natom)]))
    ctx.set_geometry(xyz)
    ctx.set_functional("pbe")
    n_radial, order = 3, 9  # 114 points per atom: most warps hold points of one atom, the last of two
    npts = ctx.grid_build(5, n_radial, order)
    P = np.zeros((natom, natom))
    np.fill_diagonal(P, np.random.default_rng(1).uniform(0.5, 1.5, size=natom))
    _, _, electrons = ctx.fock_quadrature(P[np.tril_indices(natom)])
    pts, w = quadrature(z, xyz, n_radial, order)
    norm = (2 * EXPONENT / np.pi) ** 1.5
    rho = (np.diag(P) * norm * np.exp(-2 * EXPONENT * ((pts[:, None] - xyz[None]) ** 2).sum(2))).sum(1)
    # factors below the rounding of 1/2 are noise, and so is which points of such weights are kept
    assert abs(npts - (np.abs(w) > 1e-30).sum()) <= 2e-4 * len(w) + 2
    assert abs(electrons - (w * rho).sum()) < 1e-12 * (np.abs(w) * rho).sum()


@pytest.mark.parametrize("natom", [5, 62, 200, 201, 255])
def test_weight_gradient_along_a_displacement(cuda_device, natom):
    """d E_xc / d lambda by central differences of fourth order (steps of 2e-3, error of 1e-8 and less)."""
    from pdynamo3_b200.lib import Context
    z, xyz = cluster(natom)
    rng = np.random.default_rng(2)
    d = rng.normal(size=xyz.shape)
    d /= np.abs(d).max()
    P = np.zeros((natom, natom))
    np.fill_diagonal(P, rng.uniform(0.5, 1.5, size=natom))
    P = P[np.tril_indices(natom)]
    ctx = Context(0)
    ctx.set_basis(RawShells(z, [(i, 0, 0, [0.3], [1.0]) for i in range(natom)]))
    ctx.set_functional("pbe")

    def energy(x):
        ctx.set_geometry(x)
        ctx.grid_build(5, 6, 9)
        return ctx.fock_quadrature(P)[1]

    h = 2e-3
    e = [energy(xyz + k * h * d) for k in (-2, -1, 1, 2)]
    energy(xyz)
    slope = (ctx.gradients_quadrature(P) * d).sum()
    assert abs((e[0] - 8 * e[1] + 8 * e[2] - e[3]) / (12 * h) - slope) < 1e-7 * natom

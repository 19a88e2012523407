"""Measured workloads of the Fock-build engine: what a program that uses it asks for.

A user's program asks for energies and gradients of molecules (System.Energy through GPUQCEngine), or
drives the integral and quadrature entry points of ``lib.Context`` from its own SCF.  The cases are the
calls of both: whole energy + gradient calls, one two-electron Fock build, one gradient, one quadrature
Fock build, one quadrature gradient, and the work of a new geometry, in FP64 and in the mixed mode, from
one water to the largest molecules of the organic batch and 32 waters, in Cartesian and spherical 6-31G*.

Inputs: the molecule is fixed by the case (``system``, ``size``, ``tree``) and every atom is displaced by
a seeded 0.02 A Gaussian, as an MD or optimisation step does.  Densities are the occupied projectors
of an extended-Hueckel matrix (Wolfsberg-Helmholz), so that they decay and are idempotent as converged
ones are; they are made here from the overlap integrals of the molecule, without the library.
``exact`` gives overlap, core, Fock and gradient values from McMurchie-Davidson integrals in 64 bits.
"""
import math

import numpy as np
import torch

from pdynamo3_b200 import geometry
from pdynamo3_b200.basis import ShellTable
from pdynamo3_b200.lib import Context
from pdynamo3_b200.qcmodel import ANGSTROM_TO_BOHR, GPUQCEngine

CART, SPH = "6-31g_st_cart", "6-31g_st"
EXCHANGE = {"hf": 1.0, "pbe": 0.0, "blyp": 0.0, "b3lyp": 0.2}


def _case(name, kind, system, size, tree, functional, mixed=False, basis=CART):
    return {"name": name, "kind": kind, "system": system, "size": size, "tree": tree, "functional": functional,
            "mixed": mixed, "basis": basis}


def listed():
    return [
        # the smallest whole call: one molecule of a force-field fit or a test, latency and launches count
        _case("energy_hf_water1", "energy", "water", 1, 11, "hf"),
        # a small molecule of the organic batch as the server runs it: mixed precision, from a cold start
        _case("energy_b3lyp_organic5_mixed", "energy", "organic", 5, 5, "b3lyp", mixed=True),
        # one Fock build in a caller's own SCF: small (4 waters), the batch's median, its largest, pure functional
        _case("fock_hf_water4", "fock", "water", 4, 0, "hf"),
        _case("fock_b3lyp_organic14", "fock", "organic", 14, 3, "b3lyp"),
        _case("fock_b3lyp_organic23_mixed", "fock", "organic", 23, 2, "b3lyp", mixed=True),
        _case("fock_pbe_water16", "fock", "water", 16, 1000, "pbe", basis=SPH),
        # gradients of optimisation and MD steps
        _case("gradient_hf_water2", "gradient", "water", 2, 1, "hf"),
        _case("gradient_b3lyp_organic14", "gradient", "organic", 14, 3, "b3lyp"),
        _case("gradient_b3lyp_organic20_mixed", "gradient", "organic", 20, 7, "b3lyp", mixed=True),
        # the quadrature: V_xc of one SCF cycle, the XC gradient with grid-weight terms
        _case("xc_b3lyp_organic14", "xc", "organic", 14, 3, "b3lyp"),
        _case("xc_gradient_pbe_water16", "xc_gradient", "water", 16, 1000, "pbe"),
        # what each new geometry costs: pair lists, one-electron matrices, the grid and its first V_xc
        _case("geometry_pbe_water32", "geometry", "water", 32, 32, "pbe"),
    ]


# kind -> (systems, smallest and largest size of each, functionals, may be mixed, may be spherical)
_RANGES = {
    "energy": ({"water": (1, 3), "organic": (1, 5)}, ("hf", "pbe", "b3lyp"), True, True),
    "fock": ({"water": (1, 24), "organic": (1, 22)}, ("hf", "pbe", "b3lyp"), True, True),
    "gradient": ({"water": (1, 20), "organic": (1, 16)}, ("hf", "pbe", "b3lyp"), True, True),
    "xc": ({"water": (1, 24), "organic": (1, 20)}, ("pbe", "blyp", "b3lyp"), False, True),
    "xc_gradient": ({"water": (1, 16), "organic": (1, 16)}, ("pbe", "blyp", "b3lyp"), False, True),
    "geometry": ({"water": (1, 32), "organic": (1, 22)}, ("pbe", "blyp", "b3lyp"), False, True),
}


def draw(rng):
    kind = rng.choice(sorted(_RANGES))
    systems, functionals, mixed, spherical = _RANGES[kind]
    system = rng.choice(sorted(systems))
    lo, hi = systems[system]
    size = min(hi, int(math.exp(rng.uniform(math.log(lo), math.log(hi + 1)))))
    c = _case("", kind, system, size, rng.randrange(1, 10000), rng.choice(functionals),
              mixed=mixed and rng.random() < 0.4, basis=SPH if spherical and rng.random() < 0.3 else CART)
    del c["name"]
    return c


# ---- inputs -------------------------------------------------------------------------------------


def _molecule(case):
    if case["system"] == "water":
        return geometry.water_cluster(case["size"], max(3.0, 3.2 * case["size"] ** (1.0 / 3.0)), case["tree"])
    tree = case["tree"]
    while True:
        try:
            return geometry.organic_molecule(case["size"], tree)
        except RuntimeError:  # a tree that cannot be grown without clashes: the next one
            tree += 1


def _inputs(case, seed):
    """Atomic numbers and displaced coordinates (bohr)."""
    z, xyz = _molecule(case)
    return z, (xyz + np.random.default_rng(seed).normal(scale=0.02, size=xyz.shape)) * ANGSTROM_TO_BOHR


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


# valence-state energies (hartree) of the extended-Hueckel matrix: 1s, valence s, p, d of each element
_HUECKEL = {1: (-0.50, -0.50, 0.2, 0.4), 6: (-11.3, -0.79, -0.42, 0.4), 7: (-15.6, -0.96, -0.49, 0.4),
            8: (-20.7, -1.19, -0.54, 0.4)}


def _hueckel(mol, xyz):
    """Density and energy-weighted density (the library's convention, -2 sum n e C C^T) of the
    extended-Hueckel ground state, full matrices in the output basis."""
    S = mol.to_output(mol.one_electron(xyz)[0])
    h = torch.as_tensor(mol.site_energies, dtype=torch.float64, device=S.device)
    H = 0.875 * S * (h[:, None] + h[None, :])
    H.diagonal().copy_(h * S.diagonal())
    s, U = torch.linalg.eigh(S)
    X = U / s.sqrt()
    e, C = torch.linalg.eigh(X.T @ H @ X)
    nocc = int(mol.z.sum()) // 2
    C = (X @ C)[:, :nocc]
    return 2.0 * C @ C.T, -4.0 * (C * e[:nocc]) @ C.T


def _pack(M):
    i, j = torch.tril_indices(len(M), len(M))
    return M.cpu()[i, j].numpy().copy()


def prepare(case, seed):
    z, xyz = _inputs(case, seed)
    state = {"case": case, "xyz": xyz}
    if case["kind"] == "energy":
        eng = GPUQCEngine(z, orbital_basis=case["basis"], functional=case["functional"])
        if case["mixed"]:
            eng.ctx.set_eri_options(precision_mode=1)
        state["engine"] = eng
        return state
    mol = _Molecule(case["basis"], z)
    ctx = Context(0)
    ctx.set_basis(mol.table)
    ctx.set_functional(case["functional"])
    ctx.set_eri_options(precision_mode=1 if case["mixed"] else 0)
    ctx.set_geometry(xyz)
    if case["kind"] in ("xc", "xc_gradient"):
        ctx.grid_build(3)
    state["context"] = ctx
    P, W = _hueckel(mol, torch.as_tensor(xyz, device=_device()))
    state["density"], state["weighted"] = _pack(P), _pack(W)
    return state


def run(state):
    case = state["case"]
    kind, cx = case["kind"], EXCHANGE[case["functional"]]
    if kind == "energy":
        eng = state["engine"]
        eng.forget_density()
        r = eng.energy(state["xyz"])
        return {"energy": r.energy, "gradients": r.gradients, "density": r.density}
    ctx = state["context"]
    if kind == "fock":
        F, e2 = ctx.fock_two_electron(state["density"], cx)
        return {"fock": F, "e2": e2}
    if kind == "gradient":
        return {"gradients": ctx.gradients(state["density"], state["weighted"], cx)}
    if kind == "xc":
        F, exc, rho = ctx.fock_quadrature(state["density"])
        return {"fock": F, "exc": exc, "electrons": rho}
    if kind == "xc_gradient":
        return {"gradients": ctx.gradients_quadrature(state["density"])}
    ctx.set_geometry(state["xyz"])
    ctx.grid_build(3)
    S, H, e = ctx.one_electron()
    F, exc, rho = ctx.fock_quadrature(state["density"])
    return {"overlap": S, "core": H, "nuclear": e, "fock": F, "exc": exc, "electrons": rho}


def tolerance(case):
    """Relative 2-norm limits, about four times what was measured against ``exact`` or against the same
    call with every screening threshold tightened (in brackets the largest measured)."""
    kind = case["kind"]
    if kind == "energy":
        # an SCF stops where the RMS density change is 1e-8: other sums stop elsewhere [2e-8], and one
        # cycle more or less changes the density by 1e-8 n over its norm [1e-7 in the largest]
        return {"rel": 3e-7}
    if kind == "fock":
        return {"rel": 1e-10 if case["mixed"] else 3e-11}  # [6.7e-12 in both]
    if kind == "gradient":
        # quartets below Schwarz x density bounds of 1e-13, in the mixed mode 1e-10, are left out
        return {"rel": 6e-7 if case["mixed"] else 6e-10}  # [1.4e-7 and 1.5e-10]
    return {"rel": 1e-10}  # quadrature: weights and basis values to 1e-12, sums of 1e5 to 1e6 points


def work(case):
    z, xyz = _molecule(case)
    mol = _Molecule(case["basis"], z)
    packed = 8.0 * mol.n * (mol.n + 1) / 2
    kind = case["kind"]
    if kind == "fock":
        return {"bytes": 2 * packed, "flops": mol.quartet_flops(xyz * ANGSTROM_TO_BOHR, 0)}
    if kind == "gradient":
        return {"bytes": 2 * packed + 48.0 * len(z), "flops": mol.quartet_flops(xyz * ANGSTROM_TO_BOHR, 1)}
    points, xc = mol.quadrature_flops(xyz * ANGSTROM_TO_BOHR)
    if kind == "xc":
        return {"bytes": 2 * packed, "flops": xc}
    if kind == "xc_gradient":
        return {"bytes": packed + 48.0 * len(z), "flops": 2.0 * xc + 40.0 * points * len(z)}
    if kind == "geometry":
        return {"bytes": 4 * packed, "flops": xc + 40.0 * points * len(z)}
    cycles = 12.0  # Fock builds of a cold SCF
    flops = cycles * mol.quartet_flops(xyz * ANGSTROM_TO_BOHR, 0) + mol.quartet_flops(xyz * ANGSTROM_TO_BOHR, 1)
    if case["functional"] != "hf":
        flops += (cycles + 2.0) * xc
    return {"bytes": 24.0 * len(z) + packed, "flops": flops}


# ---- exact values: McMurchie-Davidson integrals in 64 bits ---------------------------------------


class _Boys(torch.autograd.Function):
    """F_0 .. F_m of the Boys function; dF_n/dx = -F_(n+1)."""

    @staticmethod
    def forward(ctx, x, m):
        a = m + 1.5
        big = x.clamp(min=0.1)
        top = torch.special.gammainc(torch.full_like(big, a), big) * (0.5 * math.gamma(a)) / big ** a
        small, term = torch.zeros_like(x), torch.ones_like(x)
        for k in range(14):
            small += term / (2 * m + 3 + 2 * k)
            term = -term * x / (k + 1)
        F = [torch.where(x < 0.1, small, top)]
        ex = torch.exp(-x)
        for n in range(m, -1, -1):
            F.append((2.0 * x * F[-1] + ex) / (2 * n + 1))
        F.reverse()
        ctx.save_for_backward(*F)
        return tuple(F[:-1])

    @staticmethod
    def backward(ctx, *g):
        F = ctx.saved_tensors
        return -sum(gn * F[n + 1] for n, gn in enumerate(g)), None


def _cartesian(l):
    """Powers of the components: for z, for y, x = l - y - z."""
    return [(l - y - z, y, z) for z in range(l + 1) for y in range(l - z + 1)]


def _hermite(L):
    return [(t, u, v) for t in range(L + 1) for u in range(L + 1 - t) for v in range(L + 1 - t - u)]


def _R(L, alpha, d):
    """Hermite Coulomb integrals R_tuv, t + u + v <= L, of exponent alpha at the differences d[..., 3]."""
    F = _Boys.apply(alpha * (d * d).sum(-1), L)
    known = {}

    def r(n, t, u, v):
        if (n, t, u, v) not in known:
            if t + u + v == 0:
                val = (-2.0 * alpha) ** n * F[n]
            else:
                k = 0 if t else 1 if u else 2
                low = [t, u, v]
                low[k] -= 1
                val = d[..., k] * r(n + 1, *low)
                if low[k]:
                    lower = list(low)
                    lower[k] -= 1
                    val = val + low[k] * r(n + 1, *lower)
            known[n, t, u, v] = val
        return known[n, t, u, v]

    return {h: r(0, *h) for h in _hermite(L)}


class _Molecule:
    """Split shells of a molecule's basis, primitive by primitive, with the integrals over them."""

    CUT = 18.0 * math.log(10.0)  # primitive pairs below 1e-18 are dropped, as the method defines

    def __init__(self, basis, z):
        self.z = np.asarray(z)
        t = self.table = ShellTable(basis, z)
        self.spherical = t.spherical
        prims = {l: [] for l in range(3)}  # (shell, atom, first function, exponent, coefficient)
        self.shells, norm, sites, blocks, s_seen = [], [], [], [], set()
        e0 = c0 = f = 0
        for s in range(t.n_shells):
            at, n = int(t.shell_atom[s]), int(t.shell_nprim[s])
            ex = t.exponents[e0:e0 + n]
            for l in range(int(t.shell_l_low[s]), int(t.shell_l_high[s]) + 1):
                fac = (math.pi / (2 * ex)) ** 1.5
                for i in range(1, l + 1):
                    fac = fac * (2 * i - 1) / (4 * ex)
                co = t.coefficients[c0:c0 + n] / (np.sqrt(fac) if t.normalized_primitives else 1.0)
                c0 += n
                prims[l] += [(len(self.shells), at, f, e, c) for e, c in zip(ex, co)]
                self.shells.append((l, at, ex, co))
                nc = (l + 1) * (l + 2) // 2
                norm += [math.sqrt(3.0) if l == 2 and max(p) == 1 else 1.0 for p in _cartesian(l)]
                core = l == 0 and at not in s_seen and int(z[at]) > 1
                if l == 0:
                    s_seen.add(at)
                sites += [_HUECKEL[int(z[at])][0 if core else 1 + l]] * (2 * l + 1 if self.spherical else nc)
                blocks.append(_solid(l))
                f += nc
            e0 += n
        self.ncart, self.norm, self.site_energies, self.n = f, np.array(norm), sites, len(sites)
        self.prims = {l: [np.array(c) for c in zip(*p)] for l, p in prims.items() if p}
        self.c2s = torch.block_diag(*blocks) if self.spherical else None

    def to_output(self, M):
        if not self.spherical:
            return M
        C = self.c2s.to(M.device)
        return C @ M @ C.T

    def to_cartesian(self, M):
        if not self.spherical:
            return M
        C = self.c2s.to(M.device)
        return C.T @ M @ C

    def pairs(self, xyz, extra=0):
        """Primitive pairs by (la, lb): exponents, centre, 1D Hermite coefficients (b up to lb + extra),
        function indices and the weight of the unordered shell pair."""
        out = {}
        host = xyz.detach().cpu().numpy()
        for la in self.prims:
            for lb in range(la + 1):
                if lb not in self.prims:
                    continue
                (sa, aa, fa, ea, ca), (sb, ab, fb, eb, cb) = self.prims[la], self.prims[lb]
                r2 = ((host[aa][:, None] - host[ab][None]) ** 2).sum(-1)
                keep = ea[:, None] * eb[None] / (ea[:, None] + eb[None]) * r2 <= self.CUT
                if la == lb:
                    keep &= sa[:, None] >= sb[None]
                i, j = np.nonzero(keep)
                T = lambda v: torch.as_tensor(v, dtype=torch.float64, device=xyz.device)  # noqa: E731
                a, b = T(ea[i]), T(eb[j])
                A, B = xyz[torch.as_tensor(aa[i], device=xyz.device)], xyz[torch.as_tensor(ab[j], device=xyz.device)]
                p = a + b
                P = (a[:, None] * A + b[:, None] * B) / p[:, None]
                K = torch.exp(-(a * b / p)[:, None] * (A - B) ** 2)
                E = [self._hermite_1d(la, lb + extra, p, P[:, k] - A[:, k], P[:, k] - B[:, k], K[:, k]) for k in range(3)]
                comps = lambda f, l: torch.as_tensor(f[:, None] + np.arange(len(_cartesian(l))), device=xyz.device)  # noqa: E731
                out[la, lb] = {"p": p, "b": b, "P": P, "E": E, "c": T(ca[i] * cb[j]), "fa": comps(fa[i], la),
                               "fb": comps(fb[j], lb), "w": T(np.where(sa[i] == sb[j], 1.0, 2.0))}
        return out

    @staticmethod
    def _hermite_1d(la, lb, p, PA, PB, K):
        E = {(0, 0, 0): K}

        def get(i, j, t):
            if t < 0 or t > i + j or i < 0 or j < 0:
                return None
            if (i, j, t) not in E:
                x = PA if i else PB
                i1, j1 = (i - 1, j) if i else (i, j - 1)
                val = 0.0
                for c, e in ((0.5 / p, get(i1, j1, t - 1)), (x, get(i1, j1, t)), (t + 1.0, get(i1, j1, t + 1))):
                    if e is not None:
                        val = val + c * e
                E[i, j, t] = val
            return E[i, j, t]

        for i in range(la + 1):
            for j in range(lb + 1):
                for t in range(i + j + 1):
                    get(i, j, t)
        return E

    def _expansion(self, la, lb, pr):
        """Hermite expansion [pair, component of a, component of b, tuv] with contraction and norms."""
        zero = torch.zeros_like(pr["p"])
        rows = []
        for ax in _cartesian(la):
            for bx in _cartesian(lb):
                for h in _hermite(la + lb):
                    v = pr["c"]
                    for k in range(3):
                        e = pr["E"][k].get((ax[k], bx[k], h[k]))
                        v = zero if e is None or v is zero else v * e
                    rows.append(v)
        na, nb = len(_cartesian(la)), len(_cartesian(lb))
        E = torch.stack(rows, -1).reshape(len(zero), na, nb, -1)
        norm = torch.as_tensor(self.norm, device=E.device)
        return E * norm[pr["fa"]][:, :, None, None] * norm[pr["fb"]][:, None, :, None]

    def one_electron(self, xyz, charges=None):
        """Overlap, and with ``charges`` the core Hamiltonian (nuclei as the method's narrow Gaussians),
        normalised Cartesian full matrices."""
        n, dev = self.ncart, xyz.device
        S, H = (torch.zeros(n * n, dtype=torch.float64, device=dev) for _ in range(2))
        norm = torch.as_tensor(self.norm, device=dev)
        zeta = 4.0 / (1.0e-8 * math.pi)
        for (la, lb), pr in self.pairs(xyz, 2 if charges is not None else 0).items():
            root = (math.pi / pr["p"]) ** 1.5 * pr["c"]
            ov = lambda k, i, j: pr["E"][k][i, j, 0]  # noqa: E731

            def kin(k, i, j):
                v = -2.0 * pr["b"] ** 2 * ov(k, i, j + 2) + pr["b"] * (2 * j + 1) * ov(k, i, j)
                return v - 0.5 * j * (j - 1) * ov(k, i, j - 2) if j > 1 else v

            s, h = [], []
            for a in _cartesian(la):
                for b in _cartesian(lb):
                    o = [ov(k, a[k], b[k]) for k in range(3)]
                    s.append(o[0] * o[1] * o[2] * root)
                    if charges is not None:
                        t = [kin(k, a[k], b[k]) for k in range(3)]
                        h.append((t[0] * o[1] * o[2] + o[0] * t[1] * o[2] + o[0] * o[1] * t[2]) * root)
            shape = (-1, pr["fa"].shape[1], pr["fb"].shape[1])
            # a shell with itself is there in both orders, the other pairs once: half of the former, then M + M^T
            nn = 0.5 * pr["w"][:, None, None] * norm[pr["fa"]][:, :, None] * norm[pr["fb"]][:, None, :]
            at = (pr["fa"][:, :, None] * n + pr["fb"][:, None, :]).reshape(-1)
            S = S.index_add(0, at, (torch.stack(s, -1).reshape(shape) * nn).reshape(-1))
            if charges is None:
                continue
            H = H.index_add(0, at, (torch.stack(h, -1).reshape(shape) * nn).reshape(-1))
            E = self._expansion(la, lb, pr)
            p = pr["p"][:, None]
            R = _R(la + lb, p * zeta / (p + zeta), pr["P"][:, None] - xyz[None])
            pref = -2.0 * math.pi ** 2.5 * (zeta / math.pi) ** 1.5 / (p * zeta * torch.sqrt(p + zeta)) * charges[None]
            R = torch.stack([(pref * R[t]).sum(1) for t in _hermite(la + lb)], -1)
            H = H.index_add(0, at, torch.einsum("i,iabt,it->iab", 0.5 * pr["w"], E, R).reshape(-1))
        S, H = S.reshape(n, n), H.reshape(n, n)
        return S + S.T, H + H.T

    def two_electron_energy(self, xyz, D, cx):
        """1/2 sum [D_ab D_cd - cx/4 (D_ac D_bd + D_ad D_bc)] (ab|cd) and its derivatives with respect
        to the coordinates and to D; normalised Cartesian full D."""
        xyz = xyz.detach().requires_grad_(True)
        D = D.detach().requires_grad_(True)
        total = 0.0
        sizes = {k: len(v["p"]) for k, v in self.pairs(xyz).items()}
        for bra in sizes:
            for ket in sizes:
                L, nh = sum(bra) + sum(ket), len(_hermite(sum(ket)))
                per = sizes[ket] * (3 * len(_hermite(L)) + 2 * len(_hermite(sum(bra))) * nh + (200 if cx else 0) + 20)
                step = max(1, int(3e8 / per))
                for i0 in range(0, sizes[bra], step):
                    e = self._block(xyz, D, cx, bra, ket, slice(i0, i0 + step))
                    e.backward()
                    total += float(e.detach())
        return total, xyz.grad, D.grad

    def _block(self, xyz, D, cx, bra, ket, rows):
        pairs = self.pairs(xyz)
        cut = lambda v: {k: v[k][rows] for k in ("p", "P", "fa", "fb", "w")}  # noqa: E731
        I, J = pairs[bra], pairs[ket]
        Ei, Ej = self._expansion(*bra, I)[rows], self._expansion(*ket, J)
        I = cut(I)
        hb, hk = _hermite(sum(bra)), _hermite(sum(ket))
        sign = torch.as_tensor([(-1.0) ** sum(h) for h in hk], dtype=torch.float64, device=xyz.device)
        Ej = Ej * sign
        p, q = I["p"][:, None], J["p"][None]
        R = _R(sum(bra) + sum(ket), p * q / (p + q), I["P"][:, None] - J["P"][None])
        pref = 2.0 * math.pi ** 2.5 / (p * q * torch.sqrt(p + q)) * (0.5 * I["w"][:, None] * J["w"][None])
        add = lambda x, y: tuple(m + n for m, n in zip(x, y))  # noqa: E731
        at = lambda a, b: D[a, b]  # noqa: E731
        Dab = at(I["fa"][:, :, None], I["fb"][:, None, :])
        Dcd = at(J["fa"][:, :, None], J["fb"][:, None, :])
        if not cx:
            hi, hj = torch.einsum("iab,iabt->it", Dab, Ei), torch.einsum("jcd,jcdt->jt", Dcd, Ej)
            e = 0.0
            for s, x in enumerate(hb):
                v = sum(hj[:, t][None] * R[add(x, y)] for t, y in enumerate(hk))
                e = e + (hi[:, s] * (pref * v).sum(1)).sum()
            return e
        RR = torch.stack([torch.stack([pref * R[add(x, y)] for y in hk], -1) for x in hb], -2)
        V = torch.einsum("iabs,ijst,jcdt->ijabcd", Ei, RR, Ej)
        g = lambda a, b: at(a[:, None, :, None], b[None, :, None, :])  # noqa: E731
        ac, bd = g(I["fa"], J["fa"]), g(I["fb"], J["fb"])
        ad, bc = g(I["fa"], J["fb"]), g(I["fb"], J["fa"])
        return torch.einsum("ijabcd,iab,jcd->", V, Dab, Dcd) - 0.25 * cx * (
            torch.einsum("ijabcd,ijac,ijbd->", V, ac, bd) + torch.einsum("ijabcd,ijad,ijbc->", V, ad, bc))

    # ---- what the paths cannot do without ----

    def quartet_flops(self, xyz, derivative):
        """FLOPs of the Rys quadrature over the primitive quartets whose shell-pair bounds (estimated
        with s functions) reach 1e-13: per quartet n_R [4 n_c + 12 (L_ab+1)(L_cd+1) + 6 (la+1)(lb+1)(L_cd+1)
        + 6 n_c], gradients with each of three centres raised by one."""
        bound, count, cls = [], [], []
        for i, (la, ai, ea, ca) in enumerate(self.shells):
            for lb, aj, eb, cb in self.shells[:i + 1]:
                r2 = ((xyz[ai] - xyz[aj]) ** 2).sum()
                p = ea[:, None] + eb[None]
                arg = ea[:, None] * eb[None] / p * r2
                ok = arg <= self.CUT
                if ok.any():
                    k = np.abs(ca[:, None] * cb[None]) * np.exp(-arg) / p ** 1.25
                    bound.append(4.2 * k.sum())
                    count.append(ok.sum())
                    cls.append((max(la, lb), min(la, lb)))
        bound, count = np.array(bound), np.array(count, dtype=np.float64)
        kinds = sorted(set(cls))
        group = {}
        for c in kinds:
            at = np.array([x == c for x in cls])
            order = np.argsort(-bound[at])
            group[c] = (bound[at][order], count[at][order])
        nc = lambda l: (l + 1) * (l + 2) // 2  # noqa: E731
        total = 0.0
        for m, x in enumerate(kinds):
            for y in kinds[:m + 1]:
                (bx, cx), (by, cy) = group[x], group[y]
                run = np.concatenate([[0.0], np.cumsum(cy)])
                quartets = (cx * run[np.searchsorted(-by, -1e-13 / np.maximum(bx, 1e-300), side="right")]).sum()
                la, lb, lc, ld = x[0] + derivative, x[1] + derivative, y[0] + derivative, y[1]
                lab, lcd, comp = la + lb - derivative, lc + ld, nc(x[0]) * nc(x[1]) * nc(y[0]) * nc(y[1])
                w = ((lab + lcd) // 2 + 1) * (4 * comp + 12 * (lab + 1) * (lcd + 1) + 6 * (la + 1) * (lb + 1) * (lcd + 1)
                                              + (18 if derivative else 6) * comp)
                total += quartets * w * (0.5 if x == y else 1.0)
        return float(total)

    def quadrature_flops(self, xyz):
        """Points of the medium grid and FLOPs of rho and V_xc over the functions within 7 bohr."""
        per_atom = 15000.0
        funcs = np.zeros(len(self.z))
        for l, at, _, _ in self.shells:
            funcs[at] += (l + 1) * (l + 2) // 2
        near = ((xyz[:, None] - xyz[None]) ** 2).sum(-1) < 49.0
        nb = near.astype(np.float64) @ funcs
        return per_atom * len(self.z), float((4.0 * nb * nb + 8.0 * nb).sum() * per_atom)


def _solid(l):
    """Real solid harmonics (m = 0, 1c, 1s, 2c, 2s) over normalised Cartesian components."""
    if l == 0:
        return torch.ones(1, 1, dtype=torch.float64)
    if l == 1:
        return torch.tensor([[0, 0, 1], [1, 0, 0], [0, 1, 0]], dtype=torch.float64)
    s = 0.5 * math.sqrt(3.0)
    return torch.tensor([[-0.5, 0, -0.5, 0, 0, 1], [0, 0, 0, 1, 0, 0], [0, 0, 0, 0, 1, 0], [s, 0, -s, 0, 0, 0],
                         [0, 1, 0, 0, 0, 0]], dtype=torch.float64)


def exact(case, seed):
    kind = case["kind"]
    z, xyz = _inputs(case, seed)
    mol = _Molecule(case["basis"], z)
    dev = _device()
    r = torch.as_tensor(xyz, device=dev)
    charges = torch.as_tensor(z, dtype=torch.float64, device=dev)

    def nuclear(x):
        i, j = torch.tril_indices(len(z), len(z), -1)
        return (charges[i] * charges[j] / (x[i] - x[j]).norm(dim=1)).sum()

    if kind == "geometry" and len(z) <= 48:
        S, H = mol.one_electron(r, charges)
        return {"overlap": _pack(mol.to_output(S)), "core": _pack(mol.to_output(H)), "nuclear": float(nuclear(r)),
                "fock": None, "exc": None, "electrons": None}
    cx = EXCHANGE[case["functional"]]
    if kind not in ("fock", "gradient") or len(z) > (12 if cx else 48 if kind == "fock" else 24):
        return None
    P, W = _hueckel(mol, r)
    D = mol.to_cartesian(P)
    e2, gradient, F = mol.two_electron_energy(r, D, cx)
    if kind == "fock":
        return {"fock": _pack(mol.to_output(0.5 * (F + F.T))), "e2": e2}
    x = r.clone().requires_grad_(True)
    S, H = mol.one_electron(x, charges)
    (nuclear(x) + (D * H).sum() + 0.5 * (mol.to_cartesian(W) * S).sum()).backward()
    return {"gradients": (gradient + x.grad).cpu().numpy()}

"""Performance cases of the SOAP framework: what users of ``cusoap_b200.SOAP`` run, over its whole range.

The calls are the public ones (``create``, ``create_flat``, ``derivatives``, ``batch``, and autograd
through them).  Structures are water clusters and boxes (0.1 atoms/A^3) and periodic cells of mixed
species at the same density; bases are those of the repository's workloads and tests.

``exact`` restates each call in float64 torch: images and pairs by a plain distance test, GTO or
polynomial radial functions, solid harmonics by recurrence, and derivatives by forward- or
reverse-mode differentiation of that expression.
"""
import math

import numpy as np
import torch

DENSITY = 0.1  # atoms / A^3

# Basis parameters of the repository's workloads, and of its large-basis test.
BASES = {
    "small": dict(r_cut=5.0, n_max=4, l_max=3, sigma=0.5),     # 192-atom cluster
    "sharp": dict(r_cut=10.0, n_max=7, l_max=3, sigma=0.5),    # 3000-atom cluster
    "cells": dict(r_cut=6.0, n_max=8, l_max=6, sigma=0.4),     # 512-cell batch
    "box": dict(r_cut=6.0, n_max=8, l_max=6, sigma=1.0),       # 2001-atom water box
    "scale": dict(r_cut=6.0, n_max=8, l_max=4, sigma=1.0),     # 1M-atom cluster
    "large": dict(r_cut=5.0, n_max=10, l_max=9, sigma=0.6),    # beyond the one-lane-per-n range
}
WEIGHTINGS = {
    "none": None,
    "poly": {"function": "poly", "r0": 5.0, "c": 1.0, "m": 2.0},
    "pow": {"function": "pow", "r0": 2.0, "c": 1.0, "d": 1.0, "m": 2.0, "w0": 0.5},
}


def _case(name, op, structure, n, basis, **more):
    c = {"name": name, "op": op, "structure": structure, "n": n, "cells": 1, "host": True, "centres": 0,
         "average": "off", "rbf": "gto", "weighting": "none", "crossover": True}
    c.update(BASES[basis])
    c.update(more)
    return c


def listed():
    return [
        # one small molecule cluster from host arrays: the smallest call, all latency
        _case("create_24", "create", "cluster", 8, "small"),
        # the 192-atom cluster, descriptor and Jacobian of every centre
        _case("deriv_192", "deriv", "cluster", 64, "small"),
        # descriptors of a mid-size cluster at a long cutoff (700 neighbours a centre inside)
        _case("create_3000", "create", "cluster", 1000, "sharp"),
        # a driver loop's step over the same cluster: create and derivatives of 50 centres
        _case("deriv_50_of_3000", "create_deriv", "cluster", 1000, "sharp", centres=50),
        # the full dense Jacobian, bound by writing 12 GB
        _case("deriv_1536", "deriv", "cluster", 512, "sharp"),
        # a triclinic cell with a high-resolution basis, an odd number of atoms
        _case("create_501_n10_l9", "create", "triclinic", 167, "large"),
        # cc derivatives with weighting and centres moving with their atoms, in a triclinic cell
        _case("deriv_cc_attach_192", "deriv", "triclinic", 64, "small", average="cc", weighting="pow"),
        # a data set of small cells, descriptors only, as one list
        _case("create_48_cells", "create", "cells", 0, "cells", cells=48, average="inner"),
        # a training batch of 512 cells: descriptors, energy and forces
        _case("forces_512_cells", "forces", "cells", 0, "cells", cells=512, average="inner", host=False),
        # one molecular-dynamics step of a water box, eager
        _case("forces_2001", "forces", "box", 667, "box", host=False),
        # the same step through the captured plan
        _case("plan_2001", "plan", "box", 667, "box", host=False),
        # a million atoms, descriptors only, positions on the device
        _case("create_1M", "create", "cluster", 333334, "scale", host=False),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["create", "create", "cells", "deriv", "create_deriv", "forces", "forces", "plan"])
    b = dict(r_cut=round(rng.uniform(4.0, 8.0), 2), n_max=rng.randint(3, 10), l_max=rng.randint(2, 8),
             sigma=round(rng.uniform(0.4, 1.0), 2)) if rng.random() < 0.5 else \
        dict(BASES[rng.choice(["small", "sharp", "cells", "box", "scale"])])
    more = {"average": rng.choice(["off", "off", "off", "cc"]), "crossover": rng.random() < 0.8,
            "weighting": rng.choice(["none", "none", "none", "poly", "pow"]), "host": rng.random() < 0.5}
    if op == "cells":
        op, structure, n = rng.choice(["create", "forces"]), "cells", 0
        more["cells"] = _log(rng, 2, 60)
    elif op == "create":
        structure, n = rng.choice(["cluster", "cluster", "box", "triclinic"]), _log(rng, 5, 30000)
        if structure == "triclinic":
            n = _log(rng, 5, 1000)
        if rng.random() < 0.2 and n < 300:  # the polynomial radial basis
            b = dict(b, n_max=min(b["n_max"], 4), l_max=min(b["l_max"], 6))
            more["rbf"] = "polynomial"
    elif op == "deriv":
        structure, n = rng.choice(["cluster", "box", "triclinic"]), _log(rng, 5, 200)
    elif op == "create_deriv":
        structure, n = rng.choice(["cluster", "box"]), _log(rng, 100, 1000)
        more["centres"] = rng.randint(1, 60)
    else:
        structure, n = rng.choice(["cluster", "box", "triclinic"]), _log(rng, 5, 3000)
        more["host"] = False
    c = {"op": op, "structure": structure, "n": n, "cells": 1, "centres": 0, "rbf": "gto"}
    c.update(b)
    c.update(more)
    if op in ("forces", "plan"):
        c["host"] = False
    return c


# ---- structures -------------------------------------------------------------------------------

def _species(case):
    return (1, 6, 7, 8) if case["structure"] == "cells" else (1, 8)


def _water(rng, n_mol, grid, spacing, jitter):
    """n_mol water molecules on the first sites of a jittered lattice: (3 n_mol, 3), atoms O, H, H."""
    site = np.arange(n_mol)
    O = np.stack([site // (grid[1] * grid[2]), site // grid[2] % grid[1], site % grid[2]], 1) * spacing
    O = O + rng.uniform(-jitter, jitter, O.shape)
    u = rng.standard_normal((n_mol, 3))
    u /= np.linalg.norm(u, axis=1, keepdims=True)
    v = rng.standard_normal((n_mol, 3))
    v -= (u * v).sum(1, keepdims=True) * u
    v /= np.linalg.norm(v, axis=1, keepdims=True)
    half = math.radians(104.5) / 2
    pos = np.empty((n_mol, 3, 3))
    pos[:, 0] = O
    pos[:, 1] = O + 0.96 * (math.cos(half) * u + math.sin(half) * v)
    pos[:, 2] = O + 0.96 * (math.cos(half) * u - math.sin(half) * v)
    return pos.reshape(-1, 3), np.tile(np.array([8, 1, 1], np.int64), n_mol)


def _structures(case, seed):
    """The structures of a case as dicts of host arrays."""
    rng = np.random.default_rng(seed)
    n = case["n"]
    if case["structure"] == "cells":
        out = []
        for i in range(case["cells"]):  # 8 to 400 atoms, the same sizes for every seed
            A = 8 + int(393 * ((i * 0.6180339887498949 + 0.37) % 1.0))
            side = (A / DENSITY) ** (1.0 / 3.0)
            k = math.ceil(A ** (1.0 / 3.0) - 1e-9)
            site = rng.permutation(k ** 3)[:A]
            jit = max(0.0, (side / k - 0.9) / 2)
            pos = np.stack([site // (k * k), site // k % k, site % k], 1) * (side / k) + rng.uniform(-jit, jit, (A, 3))
            out.append({"positions": np.mod(pos, side), "atomic_numbers": rng.choice(np.array([1, 6, 7, 8]), A),
                        "cell": np.eye(3) * side, "pbc": np.array([True, True, True])})
        return out
    k = math.ceil(n ** (1.0 / 3.0) - 1e-9)
    if case["structure"] == "cluster":
        pos, Z = _water(rng, n, (k, k, k), 3.1, 0.3)
        return [{"positions": pos, "atomic_numbers": Z}]
    spacing = (3.0 / DENSITY * n / k ** 3) ** (1.0 / 3.0)  # a box of n molecules at the density
    spacing, jitter = max(spacing, 2.6), min(0.3, max(0.0, (spacing - 2.6) / 2))
    pos, Z = _water(rng, n, (k, k, k), spacing, jitter)
    cell = np.eye(3)
    if case["structure"] == "triclinic":
        cell = np.array([[1.0, 0.0, 0.0], [0.2, 0.97, 0.0], [0.1, -0.15, 0.95]])
    frac = pos / (k * spacing)
    return [{"positions": np.mod(frac, 1.0) @ cell * (k * spacing), "atomic_numbers": Z, "cell": cell * (k * spacing),
             "pbc": np.array([True, True, True])}]


def _periodic(case):
    return case["structure"] != "cluster"


def _energy_weights(F, seed):
    return np.random.default_rng(seed + 77).standard_normal(F).astype(np.float32)


# ---- the framework's side ---------------------------------------------------------------------

def prepare(case, seed):
    from cusoap_b200 import SOAP
    soap = SOAP(species=list(_species(case)), r_cut=case["r_cut"], n_max=case["n_max"], l_max=case["l_max"],
                sigma=case["sigma"], rbf=case["rbf"], weighting=WEIGHTINGS[case["weighting"]],
                average=case["average"], crossover=case["crossover"], periodic=_periodic(case))
    systems = _structures(case, seed)
    state = {"case": case, "soap": soap, "systems": systems}
    if case["op"] in ("forces", "plan"):
        counts = [len(s["atomic_numbers"]) for s in systems]
        state["counts"] = counts
        state["positions"] = torch.as_tensor(np.concatenate([s["positions"] for s in systems]), device=soap.device)
        state["w"] = torch.as_tensor(_energy_weights(soap.get_number_of_features(), seed), device=soap.device)
        if case["op"] == "plan":
            state["plan"] = soap.batch(systems)
    elif not case["host"]:
        for s in systems:
            s["positions"] = torch.as_tensor(s["positions"], device=soap.device)
    return state


def run(state):
    case, soap, systems = state["case"], state["soap"], state["systems"]
    op = case["op"]
    if op == "create":
        return soap.create(systems if case["structure"] == "cells" else systems[0])
    if op == "deriv":
        J, D = soap.derivatives(systems[0], attach=case["average"] == "cc")
        return {"jacobian": J, "descriptor": D}
    if op == "create_deriv":
        n = len(systems[0]["atomic_numbers"])
        first = (n - case["centres"]) // 2
        centres = list(range(first, first + case["centres"]))
        D = soap.create(systems[0], centers=centres)
        J = soap.derivatives(systems[0], centers=centres, return_descriptor=False)
        return {"descriptor": D, "jacobian": J}
    pos = state["positions"].clone().requires_grad_(True)
    if op == "plan":
        D = state["plan"].create(pos)
    elif case["structure"] == "cells":
        parts = torch.split(pos, state["counts"])
        D, _ = soap.create_flat([dict(s, positions=p) for s, p in zip(systems, parts)])
    else:
        D = soap.create(dict(systems[0], positions=pos))
    (D @ state["w"]).sum().backward()
    return {"descriptor": D.detach(), "gradient": pos.grad}


# ---- work -------------------------------------------------------------------------------------

def _features(case):
    S, N, L1 = len(_species(case)), case["n_max"], case["l_max"] + 1
    cc = S * N * L1 * L1
    if case["average"] == "cc":
        return cc, cc
    same, cross = N * (N + 1) // 2 * L1, N * N * L1
    return S * same + (S * (S - 1) // 2 * cross if case["crossover"] else 0), cc


def _cutoff(case):
    return case["r_cut"] + case["sigma"] * math.sqrt(-2.0 * math.log(1e-3))


def _counts(case):
    """(atoms, centres, pairs) of a case; pairs at the structures' mean density."""
    rc = _cutoff(case)
    if case["structure"] == "cells":
        A = sum(8 + int(393 * ((i * 0.6180339887498949 + 0.37) % 1.0)) for i in range(case["cells"]))
    else:
        A = 3 * case["n"]
    C = case["centres"] or A
    rho = DENSITY
    r = (np.arange(200) + 0.5) / 200 * rc
    inside = np.ones_like(r)
    if case["structure"] == "cluster":  # share of a cube of side a that stays inside it at distance r
        rho = 3.0 / 3.1 ** 3
        a = 3.1 * case["n"] ** (1.0 / 3.0)
        x = r / a
        inside = np.where(x < 1, 1 - 1.5 * x + 2 / math.pi * x ** 2 - x ** 3 / (4 * math.pi), 0.0).clip(0.0)
    return A, C, C * (1.0 + float((4 * math.pi * r * r * rho * inside).sum() * rc / 200))


def work(case):
    A, C, P = _counts(case)
    F, cc = _features(case)
    N, L1 = case["n_max"], case["l_max"] + 1
    K, S = L1 * L1, len(_species(case))
    ps = case["average"] != "cc"
    forward = P * (2 * N * K + 14 * N * L1 + 4 * K) + (C * 2.0 * F * K / L1 if ps else 0.0)
    data, flops = 28.0 * A + 4.0 * C * F, forward
    if case["op"] in ("deriv", "create_deriv"):
        data += 12.0 * C * A * F
        flops += P * (28 * N * L1 + 16 * K + 3 * (8.0 * F if ps else 4.0 * N * K))
        if case["op"] == "create_deriv":
            flops += forward  # two calls, each with its own coefficients
    elif case["op"] in ("forces", "plan"):
        data += 24.0 * A
        flops += P * (28 * N * L1 + 4 * N * K + 12 * K) + (C * 2.0 * (S * N) ** 2 * K if ps else 0.0) + 2.0 * C * F
    return {"bytes": data, "flops": flops}


# ---- float64 ----------------------------------------------------------------------------------

class _Radial:
    """w(r) B_nl(r) = w(r) I_nl(r) / r^l in float64, as a function of r^2 > 0; .at0[l] = w0 B_nl(0)."""

    def __init__(self, case, dev):
        N, L1, rc = case["n_max"], case["l_max"] + 1, case["r_cut"]
        self.eta, self.N, self.L1, self.rbf = 1.0 / (2.0 * case["sigma"] ** 2), N, L1, case["rbf"]
        self.weighting = WEIGHTINGS[case["weighting"]]
        put = lambda x: torch.as_tensor(np.ascontiguousarray(x), dtype=torch.float64, device=dev)  # noqa: E731
        if self.rbf == "gto":
            a = np.linspace(1.0, rc, N)
            self.gamma, self.q = [], []
            for l in range(L1):
                alpha = -np.log(1e-3 / a ** l) / a ** 2
                ev, V = np.linalg.eigh(0.5 * math.gamma(l + 1.5) * (alpha[:, None] + alpha[None, :]) ** -(l + 1.5))
                beta = (V / np.sqrt(np.clip(ev, 1e-12, None))) @ V.T
                p = alpha + self.eta
                self.gamma.append(put(alpha * self.eta / p))
                self.q.append(put((math.pi ** 1.5 * (self.eta / p) ** l * p ** -1.5)[:, None] * beta.T))
            at0 = [q.sum(0) for q in self.q[:2]]
        else:
            i = np.arange(1, N + 1)
            t = i[:, None] + i[None, :]
            ev, V = np.linalg.eigh(2 * rc ** (7.0 + t) / ((5 + t) * (6 + t) * (7 + t)))
            beta = (V / np.sqrt(ev)) @ V.T
            k = np.arange(1, 100, dtype=np.float64)
            b = k / np.sqrt(4 * k * k - 1)
            x, U = np.linalg.eigh(np.diag(b, 1) + np.diag(b, -1))
            rx, wr = rc * 0.5 * (x + 1), rc * U[0] ** 2
            self.rx, self.top = put(rx), case["l_max"] + 60 + int(2 * self.eta * rc * _cutoff(case))
            self.g = put(4 * math.pi * rx ** 2 * wr * (beta @ np.stack([(rc - rx) ** (j + 2) for j in i])))
            f = torch.exp(-self.eta * self.rx ** 2)
            at0 = [self.g @ f, self.g @ (f * 2 * self.eta * self.rx / 3)]
        w0 = 1.0 if self.weighting is None else self.weighting.get("w0", 1.0)
        self.at0 = [w0 * v for v in at0]

    def __call__(self, r2):
        r = torch.sqrt(r2)
        if self.rbf == "gto":
            B = torch.stack([torch.exp(-r2[:, None] * self.gamma[l]) @ self.q[l] for l in range(self.L1)], 2)
        else:  # ratios i_{l+1}/i_l of the modified spherical Bessel functions by downward recurrence
            t = 2 * self.eta * self.rx * r[:, None]
            ratio, keep = torch.zeros_like(t), []
            for l in range(self.top, -1, -1):
                ratio = 1.0 / ((2 * l + 3) / t + ratio)
                if l < self.L1 - 1:
                    keep.append(ratio)
            f = torch.exp(-self.eta * (self.rx - r[:, None]) ** 2) * (-torch.expm1(-2 * t)) / (2 * t)
            cols = [f @ self.g.T]
            for l, ratio in enumerate(reversed(keep)):
                f = f * ratio
                cols.append((f @ self.g.T) / r[:, None] ** (l + 1))
            B = torch.stack(cols, 2)
        w = self.weighting
        if w is not None and w["function"] == "poly":
            x = r / w["r0"]
            base = torch.where(x < 1, 1 + 2 * x ** 3 - 3 * x ** 2, torch.zeros_like(x)).clamp(min=0)
            B = B * (w["c"] * base ** w["m"])[:, None, None]
        elif w is not None:
            B = B * (w["c"] / (w["d"] + (r / w["r0"]) ** w["m"]))[:, None, None]
        return B


def _solid_harmonics(x, y, z, L1):
    r2 = x * x + y * y + z * z
    Q, C, S = {}, [torch.ones_like(x)], [torch.zeros_like(x)]
    for m in range(L1):
        if m:
            C, S = C + [x * C[-1] - y * S[-1]], S + [x * S[-1] + y * C[-1]]
        Q[m, m] = torch.full_like(x, math.prod(range(2 * m - 1, 0, -2)))
        if m + 1 < L1:
            Q[m + 1, m] = (2 * m + 1) * z * Q[m, m]
        for l in range(m + 2, L1):
            Q[l, m] = ((2 * l - 1) * z * Q[l - 1, m] - (l + m - 1) * r2 * Q[l - 2, m]) / (l - m)
    out = []
    for l in range(L1):
        for m in range(-l, l + 1):
            a = abs(m)
            c = math.sqrt((2 * l + 1) / (4 * math.pi) * (2 if a else 1) * math.factorial(l - a) / math.factorial(l + a))
            out.append(c * Q[l, a] * (S[a] if m < 0 else C[a]))
    return torch.stack(out, 1)


def _edge_coefficients(radial, rvec):
    """(E, N, K) coefficients of unit neighbours at rvec."""
    x, y, z = rvec.unbind(1)
    B, R = radial(x * x + y * y + z * z), _solid_harmonics(x, y, z, radial.L1)
    l_of = torch.tensor([l for l in range(radial.L1) for _ in range(2 * l + 1)], device=rvec.device)
    return B[:, :, l_of] * R[:, None, :]


class _Exact:
    def __init__(self, case, s, dev):
        self.case, self.dev, self.rc = case, dev, _cutoff(case)
        self.pos = torch.as_tensor(s["positions"], dtype=torch.float64, device=dev)
        self.Z = torch.as_tensor(np.searchsorted(np.array(_species(case)), s["atomic_numbers"]), device=dev)
        shifts = np.zeros((1, 3))
        if _periodic(case):
            cell = np.asarray(s["cell"])
            perp = 1.0 / np.linalg.norm(np.linalg.inv(cell), axis=0)
            n = [int(math.ceil(self.rc / p)) for p in perp]
            shifts = np.stack(np.meshgrid(*[np.arange(-k, k + 1) for k in n], indexing="ij"), -1).reshape(-1, 3) @ cell
        # images that can be within the cutoff of an atom of the cell
        shifts = torch.as_tensor(shifts, dtype=torch.float64, device=dev)
        A = self.pos.shape[0]
        img = (self.pos[None] + shifts[:, None]).reshape(-1, 3)
        lo, hi = self.pos.min(0).values - self.rc, self.pos.max(0).values + self.rc
        keep = ((img >= lo) & (img <= hi)).all(1).nonzero()[:, 0]
        self.img, self.img_atom, self.img_shift = img[keep], keep % A, shifts[keep // A]
        self.radial = _Radial(case, dev)
        S, N, L1 = len(_species(case)), case["n_max"], case["l_max"] + 1
        self.S, self.N, self.L1, self.K = S, N, L1, L1 * L1
        # power-spectrum features: per species block and l, the (row, row) pairs of the coefficient matrix
        self.blocks = []
        for j in range(S):
            for jd in range(j, S if case["crossover"] else j + 1):
                pairs = [(j * N + n, jd * N + m) for n in range(N) for m in range(n if jd == j else 0, N)]
                self.blocks.append(tuple(torch.tensor(v, device=dev) for v in zip(*pairs)))

    def pairs(self, centres):
        """(centre slot, atom, shift) of every pair of the centres except their own r = 0 ones."""
        p = self.pos[centres]
        near = ((self.img >= p.min(0).values - self.rc) & (self.img <= p.max(0).values + self.rc)).all(1).nonzero()[:, 0]
        q = self.img[near]
        ci, ji = [], []
        step = max(1, (1 << 26) // max(1, q.shape[0]))
        for a in range(0, p.shape[0], step):
            d2 = sum((p[a:a + step, k, None] - q[None, :, k]) ** 2 for k in range(3))
            i, j = ((d2 <= self.rc ** 2) & (d2 > 1e-24)).nonzero(as_tuple=True)
            ci.append(i + a)
            ji.append(near[j])
        ci, ji = torch.cat(ci), torch.cat(ji)
        return ci, self.img_atom[ji], self.img_shift[ji]

    def coefficients(self, centres, ci, atom, rvec):
        c = torch.zeros(len(centres) * self.S, self.N, self.K, dtype=torch.float64, device=self.dev)
        c = c.index_add(0, ci * self.S + self.Z[atom], _edge_coefficients(self.radial, rvec))
        own = torch.zeros_like(c)
        own[torch.arange(len(centres), device=self.dev) * self.S + self.Z[centres], :, 0] = \
            self.radial.at0[0] / math.sqrt(4 * math.pi)
        return (c + own).reshape(len(centres), self.S * self.N, self.K)

    def cc(self, c):
        """The cc layout of (..., K): l = 1 as (z, x, y), l > 1 scaled by pi^-3/2."""
        order = torch.arange(self.K, device=self.dev)
        if self.K > 1:
            order[1:4] = torch.tensor([2, 3, 1], device=self.dev)
        scale = torch.ones(self.K, dtype=torch.float64, device=self.dev)
        scale[4:] = math.pi ** -1.5
        return c[..., order] * scale

    def select(self, gram):
        """Features from gram[l]: (..., S N, S N)."""
        return torch.cat([math.sqrt(8 * math.pi ** 2 / (2 * l + 1)) * gram[l][..., a, b]
                          for a, b in self.blocks for l in range(self.L1)], -1)

    def descriptor(self, c):
        if self.case["average"] == "cc":
            return self.cc(c).flatten(1)
        blocks = [c[:, :, l * l:(l + 1) ** 2] for l in range(self.L1)]
        return self.select([b @ b.transpose(1, 2) for b in blocks])

    def chunks(self, centres, edges):
        """Slices of the centres with about that many pairs in each."""
        per = 1 + 4.2 * self.rc ** 3 * DENSITY * 1.1
        step = max(1, min(4096, int(edges / per)))
        return [centres[a:a + step] for a in range(0, len(centres), step)]

    def create(self, centres):
        out = []
        for cen in self.chunks(centres, 1.5e8 / (self.N * self.K)):
            ci, atom, shift = self.pairs(cen)
            out.append(self.descriptor(self.coefficients(cen, ci, atom, self.pos[atom] + shift - self.pos[cen][ci])))
        return torch.cat(out)

    def jacobian(self, centres, attach):
        A, SN = self.pos.shape[0], self.S * self.N
        F = _features(self.case)[0]
        J = torch.zeros(len(centres), A, 3, F, dtype=torch.float64, device=self.dev)
        ps = self.case["average"] != "cc"
        done = 0
        for cen in self.chunks(centres, 3e8 / (3 * (SN * SN * self.L1 if ps else SN * self.K))):
            ci, atom, shift = self.pairs(cen)
            rvec = self.pos[atom] + shift - self.pos[cen][ci]
            c = self.coefficients(cen, ci, atom, rvec)
            E = ci.shape[0]
            own = torch.zeros(len(cen), 3, self.N, self.K, dtype=torch.float64, device=self.dev)
            if self.L1 > 1 and not attach:  # the centre's own atom leaving a fixed centre: R_1 = sqrt(3/4pi) (y, z, x)
                for d, m in enumerate((3, 1, 2)):
                    own[:, d, :, m] = math.sqrt(3 / (4 * math.pi)) * self.radial.at0[1]
            dc = torch.stack([torch.func.jvp(lambda v: _edge_coefficients(self.radial, v), (rvec,),
                                             (torch.eye(3, dtype=torch.float64, device=self.dev)[d].expand(E, 3),))[1]
                              for d in range(3)], 1)  # (E, 3, N, K)
            dc, E = torch.cat([dc, own]), E + len(cen)
            ci = torch.cat([ci, torch.arange(len(cen), device=self.dev)])
            atom = torch.cat([atom, cen])
            full = torch.zeros(E, self.S, 3, self.N, self.K, dtype=torch.float64, device=self.dev)
            full[torch.arange(E, device=self.dev), self.Z[atom]] = dc
            full = full.transpose(1, 2).reshape(E, 3, SN, self.K)
            if ps:
                gram = []
                for l in range(self.L1):
                    g = full[..., l * l:(l + 1) ** 2] @ c[ci][:, None, :, l * l:(l + 1) ** 2].transpose(2, 3)
                    gram.append(g + g.transpose(2, 3))
                d = self.select(gram)
            else:
                d = self.cc(full).flatten(2)
            row = J.view(-1, 3, F)
            if attach:
                moving = atom != cen[ci]
                d = d * moving[:, None, None]
                row.index_add_(0, (done + ci) * A + cen[ci], -d)
            row.index_add_(0, (done + ci) * A + atom, d)
            done += len(cen)
        return J

    def forces(self, w):
        """(descriptors, dE/dx) of E = sum of descriptor @ w."""
        pos0 = self.pos
        grad, out = torch.zeros_like(pos0), []
        for cen in self.chunks(torch.arange(pos0.shape[0], device=self.dev), 0.6e8 / (self.N * self.K)):
            ci, atom, shift = self.pairs(cen)
            rvec = (pos0[atom] + shift - pos0[cen][ci]).requires_grad_(True)
            D = self.descriptor(self.coefficients(cen, ci, atom, rvec))
            g, = torch.autograd.grad((D @ w).sum(), rvec)
            grad.index_add_(0, atom, g)
            grad.index_add_(0, cen[ci], -g)
            out.append(D.detach())
        return torch.cat(out), grad


def exact(case, seed):
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    systems = _structures(case, seed)
    op = case["op"]
    if op in ("forces", "plan"):
        w = torch.as_tensor(_energy_weights(_features(case)[0], seed), dtype=torch.float64, device=dev)
        got = [_Exact(case, s, dev).forces(w) for s in systems]
        return {"descriptor": torch.cat([g[0] for g in got]), "gradient": torch.cat([g[1] for g in got])}
    if op == "create":
        got = [(e := _Exact(case, s, dev)).create(torch.arange(e.pos.shape[0], device=dev)) for s in systems]
        return got if case["structure"] == "cells" else got[0]
    e = _Exact(case, systems[0], dev)
    A = e.pos.shape[0]
    first, n = (A - case["centres"]) // 2, case["centres"] or A
    centres = torch.arange(first if case["centres"] else 0, (first if case["centres"] else 0) + n, device=dev)
    return {"descriptor": e.create(centres), "jacobian": e.jacobian(centres, op == "deriv" and case["average"] == "cc")}

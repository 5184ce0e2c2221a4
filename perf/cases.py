"""Performance cases: the work that users of easyfea_gb300 have it do, through its public entry points.

Families (``case["what"]``):

* ``solve``   Simulations.Elastic: assembly and solve of a clamped bar under an end traction, with the reaction at the clamp
              where ``reaction`` is set (host arrays, as a script that replaces EasyFEA's class uses them).
* ``matrix``  Simulations.Elastic: the stiffness assembly alone (K on the device, in CSR order).
* ``fields``  Simulations.Elastic.Result: nodal von Mises stress, element stresses and strain energy of a known displacement.
* ``crack``   Simulations.PhaseField: one load step of a notched plate (staggered loop) from a saved, committed iteration.
* ``batch``   batching.RandomMaterialBatch: random-material cantilevers of uneven sizes, assembled and solved by one graph launch.
* ``serve``   serving.Server: a burst of elastic requests of mixed elements and sizes, every solution read back.

Meshes are the organised generators' with their interior nodes moved by a tenth of the spacing, as an unstructured mesh has
no two equal elements.
"""

import math

import numpy as np
import torch

from easyfea_gb300 import Models, Simulations
from easyfea_gb300 import mesh as gmesh
from easyfea_gb300.batching import RandomMaterialBatch, fourier_field
from easyfea_gb300.serving import ElasticRequest, Server, box_spec, cantilever_spec


def listed():
    return [
        # a first try of a model, or one of many in a parameter study: a few hundred unknowns, all latency
        {"name": "solve_quad4_25x3_fp64", "what": "solve", "elem": "QUAD4", "nx": 25, "ny": 3, "nz": 0,
         "precision": "fp64", "hetero": False, "reaction": True},
        # the plane-stress cantilever of the examples (240 x 26 QUAD4), solved as the drop-in does by default
        {"name": "solve_quad4_240x26_fp64", "what": "solve", "elem": "QUAD4", "nx": 240, "ny": 26, "nz": 0,
         "precision": "fp64", "hetero": False, "reaction": True},
        # a 3D part of ordinary size, odd counts in every direction, FP64
        {"name": "solve_hexa8_77x13x11_fp64", "what": "solve", "elem": "HEXA8", "nx": 77, "ny": 13, "nz": 11,
         "precision": "fp64", "hetero": False, "reaction": False},
        # quadratic elements with a random material per element, mixed precision
        {"name": "solve_quad9_461x50_mixed", "what": "solve", "elem": "QUAD9", "nx": 461, "ny": 50, "nz": 0,
         "precision": "mixed", "hetero": True, "reaction": False},
        # the large 3D box (400 x 40 x 40 HEXA8, 2.02 million unknowns), mixed precision
        {"name": "solve_hexa8_400x40x40_mixed", "what": "solve", "elem": "HEXA8", "nx": 400, "ny": 40, "nz": 40,
         "precision": "mixed", "hetero": False, "reaction": False},
        # stiffness of a quadratic tetrahedral mesh, the usual output of a 3D mesher
        {"name": "matrix_tetra10_31x12x11", "what": "matrix", "elem": "TETRA10", "nx": 31, "ny": 12, "nz": 11,
         "hetero": False},
        # stiffness with a modulus per element on a million-element plane mesh
        {"name": "matrix_quad4_1501x701_hetero", "what": "matrix", "elem": "QUAD4", "nx": 1501, "ny": 701, "nz": 0,
         "hetero": True},
        # stresses of a 3D solution for plotting
        {"name": "fields_hexa8_161x33x29", "what": "fields", "elem": "HEXA8", "nx": 161, "ny": 33, "nz": 29},
        # one load step of the single-edge-notched plate (80,000 TRI3, Miehe split), mixed precision
        {"name": "crack_tri3_200_miehe_mixed", "what": "crack", "elem": "TRI3", "n": 200, "nz": 0, "split": "Miehe",
         "precision": "mixed"},
        # the same plate as a thin 3D body of HEXA8 with the volumetric-deviatoric split, FP64
        {"name": "crack_hexa8_36_amor_fp64", "what": "crack", "elem": "HEXA8", "n": 36, "nz": 5, "split": "Amor",
         "precision": "fp64"},
        # a material-uncertainty study: 32 cantilevers of 2,000 to 50,000 unknowns
        {"name": "batch_32_cantilevers", "what": "batch", "count": 32, "dof_min": 2000, "dof_max": 50000, "sizes": 1},
        # a burst of requests at the service: plates and boxes of 1,000 to 150,000 unknowns
        {"name": "serve_24_requests", "what": "serve", "count": 24, "dof_min": 1000, "dof_max": 150000, "sizes": 2},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _bar(rng, elem, dof):
    """(nx, ny, nz) of a bar of about ``dof`` unknowns."""
    if elem in ("QUAD4", "QUAD9"):
        per = 2 if elem == "QUAD4" else 8
        ratio = rng.uniform(5.0, 10.0)
        ny = max(2, round(math.sqrt(dof / per / ratio)))
        return max(2, round(dof / per / ny)), ny, 0
    per = 3 if elem == "HEXA8" else 24
    ratio = rng.uniform(3.0, 10.0)
    ny = max(2, round((dof / per / ratio) ** (1 / 3)))
    nz = max(2, ny + rng.randint(-1, 1))
    return max(2, round(dof / per / ny / nz)), ny, nz


def draw(rng):
    what = rng.choice(["solve", "solve", "solve", "solve", "matrix", "fields", "crack", "crack", "batch", "serve"])
    if what == "solve":
        elem = rng.choice(["QUAD4", "QUAD9", "HEXA8", "TETRA10"])
        top = {"QUAD4": 300e3, "QUAD9": 300e3, "HEXA8": 1e6, "TETRA10": 200e3}[elem]
        nx, ny, nz = _bar(rng, elem, _log(rng, 200, top))
        return {"what": "solve", "elem": elem, "nx": nx, "ny": ny, "nz": nz,
                "precision": rng.choice(["fp64", "mixed"]), "hetero": rng.random() < 0.4, "reaction": rng.random() < 0.4}
    if what == "matrix":
        elem = rng.choice(["QUAD4", "QUAD9", "HEXA8", "TETRA10"])
        nx, ny, nz = _bar(rng, elem, _log(rng, 2e3, 1e6 if elem != "TETRA10" else 3e5))
        return {"what": "matrix", "elem": elem, "nx": nx, "ny": ny, "nz": nz, "hetero": rng.random() < 0.5}
    if what == "fields":
        elem = rng.choice(["QUAD4", "QUAD9", "HEXA8"])
        nx, ny, nz = _bar(rng, elem, _log(rng, 2e3, 1e6))
        return {"what": "fields", "elem": elem, "nx": nx, "ny": ny, "nz": nz}
    if what == "crack":
        elem = rng.choice(["TRI3", "TRI3", "HEXA8"])
        n = 2 * rng.randint(20, 110) if elem == "TRI3" else 2 * rng.randint(8, 20)
        return {"what": "crack", "elem": elem, "n": n, "nz": 0 if elem == "TRI3" else rng.randint(3, 6),
                "split": rng.choice(["Miehe", "Amor", "Bourdin"]), "precision": rng.choice(["fp64", "mixed"])}
    if what == "batch":
        return {"what": "batch", "count": rng.randint(6, 40), "dof_min": 2000, "dof_max": round(_log(rng, 8e3, 6e4)),
                "sizes": rng.randint(3, 1000)}
    return {"what": "serve", "count": rng.randint(6, 30), "dof_min": 1000, "dof_max": round(_log(rng, 8e3, 2e5)),
            "sizes": rng.randint(3, 1000)}


# ---------------------------------------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------------------------------------

SIZE = {2: (120.0, 13.0, 0.0), 3: (1000.0, 100.0, 100.0)}


def _mesh(elem, nx, ny, nz, rng, size=None, keep=None):
    """An organised mesh whose interior nodes (but those ``keep(x, y, z)`` names) are moved by up to a tenth of the spacing."""
    if nz:
        L = size or SIZE[3]
        m = gmesh.Mesh_Box(gmesh.ElemType(elem), *L, nx, ny, nz)
        n = (nx, ny, nz)
    else:
        L = (size or SIZE[2])[:2]
        m = gmesh.Mesh_Rect(gmesh.ElemType(elem), *L, nx, ny)
        n = (nx, ny)
    order = 2 if elem in ("QUAD9", "TETRA10") else 1
    x = m.coord
    inside = np.ones(len(x), dtype=bool)
    for k, (l, c) in enumerate(zip(L, n)):
        eps = 1e-9 * l
        inside &= (x[:, k] > eps) & (x[:, k] < l - eps)
    if keep is not None:
        inside &= ~keep(x[:, 0], x[:, 1], x[:, 2])
    for k, (l, c) in enumerate(zip(L, n)):
        x[inside, k] += rng.uniform(-0.1, 0.1, int(inside.sum())) * (l / (c * order))
    return m


def _moduli(m, rng):
    """A Young's modulus per element: lognormal around 210000, correlated over a tenth of the bar."""
    x = m.coord
    cent = np.zeros((m.Ne, m.dim))
    for c in np.asarray(m.connect).T:
        cent += x[c, :m.dim]
    cent /= m.connect.shape[1]
    modes = 64 if m.Ne < 300000 else 16
    return 210000.0 * np.exp(0.3 * fourier_field(cent, rng, 0.1 * float(x[:, 0].max()), modes))


def _elastic(case, seed):
    """(mesh, law arguments, traction, law) of a bar's case."""
    rng = np.random.default_rng(seed)
    m = _mesh(case["elem"], case["nx"], case["ny"], case["nz"], rng)
    E = _moduli(m, rng) if case.get("hetero") else 210000.0 * float(rng.uniform(0.9, 1.1))
    load = float(rng.uniform(0.5, 1.5)) * (-800 / 13**2 if m.dim == 2 else -1.0)
    return m, E, load, rng


def _law(dim, E):
    if dim == 2:
        return Models.Elastic.Isotropic(2, E=E, v=0.3, planeStress=True, thickness=13.0)
    return Models.Elastic.Isotropic(3, E=E, v=0.3, planeStress=False)


def _ends(m):
    x = m.coord[:, 0]
    return np.nonzero(x == 0)[0], np.nonzero(np.abs(x - x.max()) < 1e-9 * x.max())[0]


def _known_displacement(m, rng):
    """A smooth displacement of the bar: bending, stretch and a few waves."""
    x = m.coord[:, :m.dim] / m.coord[:, 0].max()
    a, k, p = rng.uniform(0.5, 1.5, m.dim), rng.uniform(2, 9, (m.dim, m.dim)), rng.uniform(0, 6, m.dim)
    u = 1e-3 * a * np.sin(x @ k + p)
    u[:, -1] += 0.1 * x[:, 0] ** 2
    u[:, 0] -= 0.2 * x[:, 0] * x[:, -1]
    return u.ravel()


def _specs(case):
    """The meshes of a service's requests: sizes spread over the range, the elements in turn."""
    rng = np.random.default_rng(case["sizes"])
    dof = np.exp(rng.uniform(math.log(case["dof_min"]), math.log(case["dof_max"]), case["count"]))
    kinds = ("quad4", "quad9", "hexa8")
    return [box_spec(max(n, 2000.0)) if kinds[i % 3] == "hexa8" else cantilever_spec(kinds[i % 3], n)
            for i, n in enumerate(dof)]


_servers = {}  # a service outlives its requests: one for each mix of meshes


def prepare(case, seed):
    what = case["what"]
    if what in ("solve", "matrix"):
        m, E, load, _ = _elastic(case, seed)
        simu = Simulations.Elastic(m, _law(m.dim, E))
        left, right = _ends(m)
        if what == "solve":
            simu.precision = case["precision"]
            simu.rtol = 1e-12 if case["precision"] == "fp64" else 1e-10
            names = ["x", "y", "z"][:m.dim]
            simu.add_dirichlet(left, [0.0] * m.dim, names)
            simu.add_surfLoad(right, [load], [names[-1]])
        simu.dmesh
        return {"case": case, "simu": simu, "clamp": simu.Bc_dofs_nodes(left, ["x", "y", "z"][:m.dim])}
    if what == "fields":
        m, E, _, rng = _elastic(case, seed)
        simu = Simulations.Elastic(m, _law(m.dim, E))
        simu._Set_solutions("elastic", _known_displacement(m, rng))
        simu.dmesh.incidence()
        return {"case": case, "simu": simu}
    if what == "crack":
        return _prepare_crack(case, seed)
    if what == "batch":
        rng = np.random.default_rng(case["sizes"])
        made = []
        for i in range(case["count"]):
            n = math.exp(rng.uniform(math.log(case["dof_min"]), math.log(case["dof_max"])))
            ny = max(2, round(math.sqrt(n / 2 * 13.0 / 120.0)))
            nx = max(2, round(n / 2 / ny))
            r = np.random.default_rng([seed, i])
            m = _mesh("QUAD4", nx, ny, 0, r)
            made.append((m, _moduli(m, r)))
        return {"case": case, "batch": RandomMaterialBatch(made)}
    key = (case["count"], case["dof_min"], case["dof_max"], case["sizes"])
    if key not in _servers:
        _servers[key] = [Server(workers=8, batch_max_dof=15000), 0]
        _servers[key][0].cache.prebuild(_specs(case))
    rng = np.random.default_rng(seed)
    specs = _specs(case)
    made = [210000.0 * np.exp(0.2 * rng.standard_normal(s.n_elems)) if i % 2 else np.full(s.n_elems, 210000.0 * rng.uniform(0.9, 1.1))
            for i, s in enumerate(specs)]
    return {"case": case, "server": _servers[key], "specs": specs, "E": made}


def _prepare_crack(case, seed):
    rng = np.random.default_rng(seed)
    n, nz = case["n"], case["nz"]
    at_notch = lambda x, y, z: (np.abs(y - 0.5) < 1e-12) & (x <= 0.5 + 1e-12)  # noqa: E731
    m = _mesh(case["elem"], n, n, nz, rng, size=(1.0, 1.0, nz / n), keep=at_notch)
    law = Models.Elastic.Isotropic(m.dim, E=210e3, v=0.3, planeStress=False)
    simu = Simulations.PhaseField(m, Models.PhaseField(law, case["split"], "AT2", 2.7, max(0.01, 2.0 / n)))
    simu.precision = case["precision"]
    simu.rtol = 1e-10
    x = m.coord
    s = {"case": case, "simu": simu, "notch": np.nonzero(at_notch(x[:, 0], x[:, 1], x[:, 2]))[0],
         "bottom": np.nonzero(x[:, 1] == 0)[0], "top": np.nonzero(x[:, 1] == 1.0)[0],
         "pull": float(rng.uniform(1.6e-3, 2.0e-3))}
    _load_step(s, s["pull"])  # the loading so far, committed
    simu.Save_Iter()
    return s


def _load_step(s, pull):
    simu, names = s["simu"], ["x", "y", "z"][:s["simu"].dim]
    simu.Bc_Init()
    simu.add_dirichlet(s["notch"], [1.0], ["d"], problemType="damage")
    simu.add_dirichlet(s["bottom"], [0.0] * len(names), names)
    simu.add_dirichlet(s["top"], [0.0, pull, 0.0][:len(names)], names)
    return simu.Solve(1e-3, 500, convOption=0)


# ---------------------------------------------------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------------------------------------------------


def run(state):
    what = state["case"]["what"]
    if what == "solve":
        simu = state["simu"]
        simu.Need_Update()
        if not state["case"]["reaction"]:
            return {"u": simu.Solve_device()}
        return {"u": simu.Solve(), "reaction": simu.Calc_Reaction(state["clamp"])}
    if what == "matrix":
        state["simu"].Need_Update()
        return {"K": state["simu"].K_device.vals64}
    if what == "fields":
        simu = state["simu"]
        return {"Svm": simu.Result_device("Svm"), "Stress": simu.Result_device("Stress", nodeValues=False),
                "Wdef": simu.Result_device("Wdef")}
    if what == "crack":
        state["simu"].Set_Iter(0)
        u, d, converged = _load_step(state, state["pull"] + 4e-5)
        return {"u": u, "d": d, "converged": bool(converged)}
    if what == "batch":
        state["batch"].replay()
        return [s.x for s in state["batch"].systems]
    server, first = state["server"]
    state["server"][1] += len(state["specs"])
    for i, (spec, E) in enumerate(zip(state["specs"], state["E"])):
        server.submit(ElasticRequest(spec, E=E, rid=first + i))
    server.drain()
    return [server.results.pop(first + i).u for i in range(len(state["specs"]))]


# ---------------------------------------------------------------------------------------------------------------------
# what a pass cannot do without: the mesh, material and loads read once, the results written once, and the arithmetic of the
# element matrices and of one product with the assembled operator (a lower limit for any solver)
# ---------------------------------------------------------------------------------------------------------------------

PER = {"QUAD4": (4, 4, 9, 1), "QUAD9": (9, 9, 16, 4), "HEXA8": (8, 8, 27, 1), "TETRA10": (10, 4, 28, 8), "TRI3": (3, 1, 7, 1)}


def _counts(elem, nx, ny, nz):
    """(nodes, elements, nodes an element, points an element, stored blocks)."""
    npe, npg, nbr, _ = PER[elem]
    q = 2 if elem in ("QUAD9", "TETRA10") else 1
    nn = (q * nx + 1) * (q * ny + 1) * (q * nz + 1)
    ne = nx * ny * max(nz, 1) * {"TRI3": 2, "TETRA10": 6}.get(elem, 1)
    return nn, ne, npe, npg, nn * nbr


def _solve_work(elem, nx, ny, nz):
    nn, ne, npe, npg, blocks = _counts(elem, nx, ny, nz)
    d = 3 if nz else 2
    return 24 * nn + 4 * npe * ne + 24 * d * nn, 2 * ne * npg * npe * npe * d * d + 2 * d * d * blocks


def work(case):
    what = case["what"]
    if what in ("solve", "matrix", "fields"):
        nn, ne, npe, npg, blocks = _counts(case["elem"], case["nx"], case["ny"], case["nz"])
        d = 3 if case["nz"] else 2
        by, fl = _solve_work(case["elem"], case["nx"], case["ny"], case["nz"])
        if what == "matrix":
            return {"bytes": 24 * nn + 4 * npe * ne + 8 * d * d * blocks + (8 * ne if case["hetero"] else 0),
                    "flops": 2 * ne * npg * npe * npe * d * d}
        if what == "fields":
            k = 3 if d == 2 else 6
            return {"bytes": 24 * nn + 4 * npe * ne + 8 * d * nn + 8 * nn + 8 * k * ne, "flops": 2 * ne * npg * npe * d * (d + d * d + k)}
        return {"bytes": by + (8 * ne if case["hetero"] else 0), "flops": fl}
    if what == "crack":
        nn, ne, npe, npg, blocks = _counts(case["elem"], case["n"], case["n"], case["nz"])
        by, fl = _solve_work(case["elem"], case["n"], case["n"], case["nz"])
        return {"bytes": by + 32 * nn + 16 * ne * 3, "flops": 2 * fl}
    if what == "batch":
        rng = np.random.default_rng(case["sizes"])
        dof = np.exp(rng.uniform(math.log(case["dof_min"]), math.log(case["dof_max"]), case["count"]))
        return {"bytes": float(np.sum(52 * dof)), "flops": float(np.sum(110 * dof))}
    each = [_solve_work({"quad4": "QUAD4", "quad9": "QUAD9", "hexa8": "HEXA8"}[s.kind], s.nx, s.ny, s.nz) for s in _specs(case)]
    return {"bytes": float(sum(b for b, _ in each)), "flops": float(sum(f for _, f in each))}


# ---------------------------------------------------------------------------------------------------------------------
# the same results in 64 bits by plain torch
# ---------------------------------------------------------------------------------------------------------------------

LOCAL = {
    "QUAD4": [(-1, -1), (1, -1), (1, 1), (-1, 1)],
    "QUAD9": [(-1, -1), (1, -1), (1, 1), (-1, 1), (0, -1), (1, 0), (0, 1), (-1, 0), (0, 0)],
    "HEXA8": [(-1, -1, -1), (1, -1, -1), (1, 1, -1), (-1, 1, -1), (-1, -1, 1), (1, -1, 1), (1, 1, 1), (-1, 1, 1)],
    "TETRA10": [(0, 0, 0), (1, 0, 0), (0, 1, 0), (0, 0, 1), (.5, 0, 0), (.5, .5, 0), (0, .5, 0), (0, 0, .5), (0, .5, .5),
                (.5, 0, .5)],
}


def _element(elem):
    """Derivatives (points, dim, nodes) of the shape functions at the Gauss points, and the weights."""
    nodes = np.array(LOCAL[elem], dtype=np.float64)
    dim = nodes.shape[1]
    if elem == "TETRA10":
        powers = [p for p in np.ndindex(3, 3, 3) if sum(p) <= 2]
        a, b = (5 - math.sqrt(5)) / 20, (5 + 3 * math.sqrt(5)) / 20
        pts, w = np.array([(a, a, a), (a, a, b), (a, b, a), (b, a, a)]), np.full(4, 1 / 24)
    else:
        q = 3 if elem == "QUAD9" else 2
        powers = list(np.ndindex(*[q] * dim))
        x1, w1 = np.polynomial.legendre.leggauss(q)
        pts = np.stack(np.meshgrid(*[x1] * dim, indexing="ij"), -1).reshape(-1, dim)
        w = np.stack(np.meshgrid(*[w1] * dim, indexing="ij"), -1).reshape(-1, dim).prod(1)
    powers = np.array(powers, dtype=np.float64)
    coef = np.linalg.inv(np.prod(nodes[:, None, :] ** powers[None], axis=2))  # monomials -> shape functions
    d = np.zeros((len(pts), dim, len(nodes)))
    for k in range(dim):
        lower = powers.copy()
        lower[:, k] = np.maximum(lower[:, k] - 1, 0)
        d[:, k] = (powers[:, k] * np.prod(pts[:, None, :] ** lower[None], axis=2)) @ coef
    return torch.from_numpy(d), torch.from_numpy(w)


def _law_matrix(dim, E):
    """(elements or 1, dim, dim, dim, dim) tensor of the isotropic law."""
    E = np.atleast_1d(np.asarray(E, dtype=np.float64))
    lam, mu = E * 0.3 / ((1 + 0.3) * (1 - 2 * 0.3)), E / (2 * (1 + 0.3))
    if dim == 2:
        lam = E * 0.3 / (1 - 0.3**2)
    i = np.eye(dim)
    C = lam[:, None, None, None, None] * np.einsum("ij,kl->ijkl", i, i)
    return torch.from_numpy(C + mu[:, None, None, None, None] * (np.einsum("ik,jl->ijkl", i, i) + np.einsum("il,jk->ijkl", i, i)))


def _gradients(elem, X):
    """Gradients (elements, points, dim, nodes) of the shape functions and the weighted measures (elements, points)."""
    d, w = _element(elem)
    d, w = d.to(X.device), w.to(X.device)
    F = torch.einsum("gdn,enk->egdk", d, X)
    return torch.linalg.solve(F, d.expand(len(X), *d.shape)), torch.linalg.det(F).abs() * w


def _stiffness(elem, X, E, thickness):
    """(elements, nodes * dim, nodes * dim)."""
    g, w = _gradients(elem, X)
    C = _law_matrix(X.shape[2], E).to(X.device)
    Ke = torch.zeros(len(X), X.shape[1], X.shape[2], X.shape[1], X.shape[2], dtype=X.dtype, device=X.device)
    for q in range(g.shape[1]):
        s = torch.einsum("eijkl,elm->eijkm", C.expand(len(X), *C.shape[1:]), g[:, q])
        Ke += torch.einsum("e,ejn,eijkm->enimk", w[:, q], g[:, q], s)
    return thickness * Ke.reshape(len(X), X.shape[1] * X.shape[2], -1)


def _bar_exact(elem, m, E, load, device="cuda"):
    """The clamped bar's displacement and the forces K u, by a dense factorisation."""
    dim, con = m.dim, torch.from_numpy(np.array(m.connect)).to(device)
    X = torch.from_numpy(m.coord[:, :dim].copy()).to(device)[con]
    thickness = 13.0 if dim == 2 else 1.0
    Ke = _stiffness(elem, X, E, thickness)
    dofs = (con[:, :, None] * dim + torch.arange(dim, device=device)).reshape(len(con), -1)
    n = m.Nn * dim
    K = torch.zeros(n * n, dtype=torch.float64, device=device)
    K.index_add_(0, (dofs[:, :, None] * n + dofs[:, None, :]).reshape(-1), Ke.reshape(-1))
    K = K.view(n, n)
    b = np.zeros(n)
    left, right = _ends(m)
    ends = m.coord[right]
    if dim == 2:  # half of each piece of the edge on its two ends
        order = right[np.argsort(ends[:, 1])]
        piece = np.diff(m.coord[order, 1]) * load * thickness / 2
        np.add.at(b, order[:-1] * 2 + 1, piece)
        np.add.at(b, order[1:] * 2 + 1, piece)
    else:  # a quarter of each rectangle of the end face on its corners
        ys, zs = np.unique(np.round(ends[:, 1], 9)), np.unique(np.round(ends[:, 2], 9))
        at = np.empty((len(zs), len(ys)), dtype=np.int64)
        at[np.searchsorted(zs, np.round(ends[:, 2], 9)), np.searchsorted(ys, np.round(ends[:, 1], 9))] = right
        area = np.diff(zs)[:, None] * np.diff(ys)[None] * load / 4
        for c in (at[:-1, :-1], at[1:, :-1], at[:-1, 1:], at[1:, 1:]):
            np.add.at(b, c.ravel() * 3 + 2, area.ravel())
    free = np.ones(n, dtype=bool)
    free[(left[:, None] * dim + np.arange(dim)).ravel()] = False
    at = torch.from_numpy(np.nonzero(free)[0]).to(device)
    A = K[at][:, at]
    f = torch.from_numpy(b).to(device)[at][:, None]
    L = torch.linalg.cholesky(A)
    u = torch.cholesky_solve(f, L)
    for _ in range(2):  # refined
        u += torch.cholesky_solve(f - A @ u, L)
    whole = torch.zeros(n, dtype=torch.float64, device=device)
    whole[at] = u[:, 0]
    return whole, K @ whole


def exact(case, seed):
    what = case["what"]
    if what == "solve":
        nodes = _counts(case["elem"], case["nx"], case["ny"], case["nz"])[0]
        if case["elem"] == "TETRA10" or nodes * (3 if case["nz"] else 2) > 14000:
            return None  # a dense factorisation of more would take too long
        m, E, load, _ = _elastic(case, seed)
        u, f = _bar_exact(case["elem"], m, E, load)
        if not case["reaction"]:
            return {"u": u}
        clamp = (_ends(m)[0][:, None] * m.dim + np.arange(m.dim)).ravel()
        return {"u": u, "reaction": f[torch.from_numpy(clamp).to(f.device)]}
    if what == "matrix":
        m, E, _, _ = _elastic(case, seed)
        con = torch.from_numpy(np.array(m.connect)).cuda()
        X = torch.from_numpy(m.coord[:, :m.dim].copy()).cuda()[con]
        n = m.Nn * m.dim
        dofs = (con[:, :, None] * m.dim + torch.arange(m.dim, device=con.device)).reshape(len(con), -1)
        at = (dofs[:, :, None] * n + dofs[:, None, :]).reshape(-1)
        places, where = torch.unique(at, return_inverse=True)
        K = torch.zeros(len(places), dtype=torch.float64, device=con.device)
        return {"K": K.index_add_(0, where, _stiffness(case["elem"], X, E, 13.0 if m.dim == 2 else 1.0).reshape(-1))}
    if what == "fields":
        m, E, _, rng = _elastic(case, seed)
        dim, con = m.dim, torch.from_numpy(np.array(m.connect)).cuda()
        X = torch.from_numpy(m.coord[:, :dim].copy()).cuda()[con]
        u = torch.from_numpy(_known_displacement(m, rng)).cuda().view(-1, dim)[con]
        g, w = _gradients(case["elem"], X)
        H = torch.einsum("egin,enk->egki", g, u)
        e = (H + H.transpose(2, 3)) / 2
        s = torch.einsum("ijkl,egkl->egij", _law_matrix(dim, E).cuda()[0], e)
        pairs = [(0, 0), (1, 1), (0, 1)] if dim == 2 else [(0, 0), (1, 1), (2, 2), (1, 2), (0, 2), (0, 1)]
        t = torch.stack([s[..., i, j] for i, j in pairs], -1)
        if dim == 2:
            vm = (t[..., 0]**2 + t[..., 1]**2 - t[..., 0] * t[..., 1] + 3 * t[..., 2]**2).sqrt()
        else:
            vm = (0.5 * ((t[..., 0] - t[..., 1])**2 + (t[..., 1] - t[..., 2])**2 + (t[..., 2] - t[..., 0])**2)
                  + 3 * (t[..., 3:]**2).sum(-1)).sqrt()
        total = torch.zeros(m.Nn, dtype=torch.float64, device=con.device)
        number = torch.zeros_like(total)
        per = vm.mean(1)[:, None].expand(con.shape)
        total.index_add_(0, con.reshape(-1), per.reshape(-1))
        number.index_add_(0, con.reshape(-1), torch.ones_like(per).reshape(-1))
        W = 0.5 * (13.0 if dim == 2 else 1.0) * torch.einsum("egij,egij,eg->", s, e, w)
        return {"Svm": total / number, "Stress": t.mean(1), "Wdef": float(W)}
    return None

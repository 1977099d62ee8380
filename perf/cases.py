"""The work a user of this library has it do, as measurable cases.

A pass of a "resident" case is one time step of a program that keeps alpha on
the GPU: load alpha, ``reconstruct_resident()``, ``advect_resident()``.  A
pass of a "host" case is one step through the host-array entry points, and of
a "facade" case one step through the solveVofEqu mirror.  A "train" pass is
one gradient evaluation of the learned-normal network's training.  Meshes,
flow, Courant number and controls are those of the repository's benchmark and
tests: the unit cube, the 3-D deformation field at Courant 0.5, nAlphaBounds 3.

``evolve`` is the number of plain steps the volume fraction has made before
the pass: a few (the first steps, most of the mesh exactly empty), or enough
that every cell holds the small remainders that a run lives with from its
first tenth on.  The meshes and the library's handles are made once and kept,
as a program keeps them; alpha, phi and U come from the seed.
"""

import math

import numpy as np
import torch

from geometricvofext_gb300 import capi, meshgen, mlp, solve_vof_equ

FORMS = {"plain": capi.PRECISION_PLAIN_FP64, "mixed": capi.PRECISION_MIXED, "learned": capi.PRECISION_LEARNED}
DEV = "cuda"


def listed():
    return [
        # the drop-in facade on a small host mesh: all latency (copies, launches, synchronisations)
        case("facade-plain-hex-24", "facade", "plain", "hex", 24, 8),
        # the smallest resident run: the launches and the serial chains of one cell
        case("plain-hex-33", "resident", "plain", "hex", 33, 8),
        # the 128^3 deformation run in its middle, plain FP64 (the drop-in's arithmetic)
        case("plain-hex-128", "resident", "plain", "hex", 128, 600),
        # the benchmark's size and its window at the start of the run, plain FP64
        case("plain-hex-256-start", "resident", "plain", "hex", 256, 4),
        # the headline form at the benchmark's size once alpha has spread over the mesh
        case("learned-hex-256", "resident", "learned", "hex", 256, 300),
        # the mixed form in a coupled solver: the mass flux is read after every step
        case("mixed-hex-128-coupled", "resident", "mixed", "hex", 128, 600, coupled=True),
        # many drops and a pool (the scale configuration's shape): a long interface in the mesh
        case("mixed-drops-150", "resident", "mixed", "hex", 150, 20, shape="drops"),
        # warped hexahedra (unstructured configuration)
        case("plain-jitter-96", "resident", "plain", "jitter", 96, 150),
        # tetrahedra (unstructured configuration), an odd size
        case("mixed-tet-45", "resident", "mixed", "tet", 45, 100),
        # 2:1 refined polyhedra with isoRDF normals, clipping and sources, coupled
        case("rdf-checker-24", "resident", "plain", "checker", 24, 40, rdf=True, clip=True, sources=True, coupled=True),
        # a CPU solver that hands its pinned arrays over every step
        case("host-learned-hex-128", "host", "learned", "hex", 128, 100),
        # one gradient evaluation of the network's training at its batch size
        {"name": "train-8192", "use": "train", "rows": 8192},
    ]


def case(name, use, form, mesh, n, evolve, shape="sphere", rdf=False, clip=False, sources=False, coupled=False):
    c = {"use": use, "form": form, "mesh": mesh, "n": n, "evolve": evolve, "shape": shape, "rdf": rdf, "clip": clip,
         "sources": sources, "coupled": coupled}
    return {"name": name, **c} if name else c


def draw(rng):
    if rng.random() < 0.1:
        return {"use": "train", "rows": 128 * rng.randint(1, 160)}
    use = rng.choice(("resident", "resident", "resident", "resident", "host", "facade"))
    mesh = rng.choice(("hex", "hex", "hex", "jitter", "tet", "checker", "refined"))
    top = {"hex": 180, "jitter": 96, "tet": 45, "checker": 36, "refined": 36}[mesh]
    if use == "facade":
        top = min(top, 64)
    n = int(round(math.exp(rng.uniform(math.log(14), math.log(top)))))
    form = rng.choice(("plain", "mixed", "learned"))
    rdf = form == "plain" and rng.random() < 0.2
    shape = "drops" if mesh == "hex" and n >= 64 and rng.random() < 0.25 else "sphere"
    evolve = rng.choice((4, 12, 40, min(400, 4 * n)))
    return case(None, use, form, mesh, n, evolve, shape, rdf, rng.random() < 0.25, rng.random() < 0.15,
                use == "resident" and rng.random() < 0.3)


# ---------------------------------------------------------------------------
# meshes and handles, made once
# ---------------------------------------------------------------------------
_MESHES = {}
_HANDLES = {}


def _hex_block(n):
    """meshgen.hex_mesh's numbering with closed-form metrics, built on the
    GPU (the numpy generator takes minutes at 256^3)."""
    n1, h = n + 1, 1.0 / n
    i64 = dict(dtype=torch.int64, device=DEV)
    c = torch.arange(n ** 3, **i64)
    ci, cj, ck = c % n, (c // n) % n, c // (n * n)

    def pid(i, j, k):
        return i + n1 * (j + n1 * k)

    corners = {  # the four corners (offsets from the cell's lowest corner) of a face, in order
        "+x": ((1, 0, 0), (1, 1, 0), (1, 1, 1), (1, 0, 1)),
        "+y": ((0, 1, 0), (0, 1, 1), (1, 1, 1), (1, 1, 0)),
        "+z": ((0, 0, 1), (1, 0, 1), (1, 1, 1), (0, 1, 1)),
        "-x": ((0, 0, 0), (0, 0, 1), (0, 1, 1), (0, 1, 0)),
        "-y": ((0, 0, 0), (1, 0, 0), (1, 0, 1), (0, 0, 1)),
        "-z": ((0, 0, 0), (0, 1, 0), (1, 1, 0), (1, 0, 0)),
    }

    def part(side, sel):
        a, b, e = ci[sel], cj[sel], ck[sel]
        q = torch.stack([pid(a + x, b + y, e + z) for x, y, z in corners[side]], 1).to(torch.int32)
        axis, sgn = "xyz".index(side[1]), 1.0 if side[0] == "+" else -1.0
        cf = torch.stack([(v.double() + 0.5) * h for v in (a, b, e)], 1)
        cf[:, axis] = ((a, b, e)[axis] + (1 if sgn > 0 else 0)).double() * h
        sf = torch.zeros_like(cf)
        sf[:, axis] = sgn * h * h
        return sel.to(torch.int32), q, cf, sf

    axes = (ci, cj, ck)
    valid = torch.stack([v < n - 1 for v in axes], 1)
    first = torch.cumsum(valid.sum(1), 0) - valid.sum(1)
    rank = torch.cumsum(valid.long(), 1) - valid.long()
    ni = int(valid.sum())
    own = torch.empty(ni, dtype=torch.int32, device=DEV)
    nei = torch.empty_like(own)
    pts4 = torch.empty((ni, 4), dtype=torch.int32, device=DEV)
    Cf = torch.empty((ni, 3), dtype=torch.float64, device=DEV)
    Sf = torch.empty_like(Cf)
    for a, step in enumerate((1, n, n * n)):
        sel = torch.nonzero(valid[:, a]).flatten()
        at = (first + rank[:, a])[sel]
        o, q, cf, sf = part("+" + "xyz"[a], sel)
        own[at], nei[at], pts4[at], Cf[at], Sf[at] = o, o + step, q, cf, sf
    own, pts4, Cf, Sf = [own], [pts4], [Cf], [Sf]
    patches, start = [], ni
    for name, side, sel in (("top", "+z", ck == n - 1), ("left", "-y", cj == 0), ("back", "-x", ci == 0),
                            ("right", "+y", cj == n - 1), ("bottom", "-z", ck == 0), ("front", "+x", ci == n - 1)):
        o, q, cf, sf = part(side, torch.nonzero(sel).flatten())
        own.append(o), pts4.append(q), Cf.append(cf), Sf.append(sf)
        patches.append((name, start, n * n))
        start += n * n
    x = torch.arange(n1, dtype=torch.float64, device=DEV) / n
    pts = torch.stack([v.expand(n1, n1, n1).reshape(-1) for v in (x[None, None, :], x[None, :, None], x[:, None, None])], 1)
    C = torch.stack([(v.double() + 0.5) * h for v in axes], 1)
    host = lambda t: t.cpu().numpy()  # noqa: E731
    Sf = torch.cat(Sf)
    m = meshgen.PolyMesh(points=host(pts), face_offsets=np.arange(start + 1, dtype=np.int32) * 4,
                         face_points=host(torch.cat(pts4)).ravel(), owner=host(torch.cat(own)), neighbour=host(nei),
                         n_cells=n ** 3, patches=patches, kind="hex")
    m.C, m.V, m.Cf, m.Sf = host(C), np.full(n ** 3, h ** 3), host(torch.cat(Cf)), host(Sf)
    m.magSf, m.h = host(Sf.abs().sum(1)), h
    return m


def _mesh(kind, n):
    """The mesh with its flow (phi and U at full speed) and Courant-0.5 step."""
    if (kind, n) not in _MESHES:
        m = _hex_block(n) if kind == "hex" else meshgen.make_mesh(kind, n)
        d = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(DEV)  # noqa: E731
        C, Cf, Sf, V = d(m.C), d(m.Cf), d(m.Sf), d(m.V)
        phi = (_velocity(Cf) * Sf).sum(1)
        speed = torch.zeros_like(V)
        own, nei = d(m.owner).long(), d(m.neighbour).long()
        speed.index_add_(0, own, phi.abs()).index_add_(0, nei, phi[: nei.numel()].abs())
        dt = 1.0 / float((speed / V).max())
        _MESHES[kind, n] = {"mesh": m, "C": C, "h": V ** (1.0 / 3.0), "phi": phi, "U": _velocity(C), "dt": dt,
                            "Ub": torch.zeros((m.n_boundary_faces, 3), dtype=torch.float64, device=DEV)}
    return _MESHES[kind, n]


def _velocity(x):
    """The 3-D deformation field of the benchmark (harness.deformation_velocity), on the GPU."""
    s, s2 = torch.sin(math.pi * x), torch.sin(2 * math.pi * x)
    return torch.stack((2 * s[:, 0] ** 2 * s2[:, 1] * s2[:, 2], -s2[:, 0] * s[:, 1] ** 2 * s2[:, 2],
                        -s2[:, 0] * s2[:, 1] * s[:, 2] ** 2), 1)


def _handle(kind, n, form, rdf=False, clip=False):
    key = (kind, n, form, rdf, clip)
    if key not in _HANDLES:
        g = capi.Simplic(_mesh(kind, n)["mesh"], precision=FORMS[form], n_alpha_bounds=3, clip=int(clip),
                         orientation_method=capi.ORIENTATION_ISO_RDF if rdf else capi.ORIENTATION_ISO_ALPHA_GRAD)
        if form == "learned":
            g.set_network(*mlp.load_weights())
        _HANDLES[key] = g
    return _HANDLES[key]


class _Buffer:
    """The library's alpha buffer as an array interface (no copy)."""

    def __init__(self, ptr, n):
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": "<f8", "data": (ptr, False), "version": 3}


_VIEWS = {}


def _alpha_view(g):
    ptr = g.alpha_device_ptr()
    if (id(g), ptr) not in _VIEWS:
        _VIEWS[id(g), ptr] = torch.as_tensor(_Buffer(ptr, g.nc), device=DEV)
    return _VIEWS[id(g), ptr]


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _alpha(case, M, seed):
    """Liquid bodies with a one-cell ramp, then ``evolve`` plain steps."""
    rng = np.random.default_rng(seed)
    C, h = M["C"], M["h"]
    if case["shape"] == "drops":
        gap = 1.0 - C[:, 2] / float(rng.uniform(0.18, 0.22))
        a = torch.clamp(0.5 + gap * 0.2 / h, 0.0, 1.0)
        for _ in range(60):
            r = float(rng.uniform(0.02, 0.05))
            c = torch.tensor(rng.uniform((0.06, 0.06, 0.3), 0.94, 3), device=DEV)
            a = torch.maximum(a, torch.clamp(0.5 - ((C - c).norm(dim=1) - r) / h, 0.0, 1.0))
    else:
        c = torch.tensor(0.35 + rng.uniform(-0.03, 0.03, 3), device=DEV)
        r = float(rng.uniform(0.13, 0.17))
        a = torch.clamp(0.5 - ((C - c).norm(dim=1) - r) / h, 0.0, 1.0)
    g = _handle(case["mesh"], case["n"], "plain")
    torch.cuda.synchronize()
    g.set_alpha(a, device=True)
    for _ in range(case["evolve"]):
        g.reconstruct_resident()
        g.advect_resident(M["phi"], M["U"], M["dt"], U_boundary=M["Ub"])
    g.synchronize()
    return _alpha_view(g).clone(), rng


def prepare(case, seed):
    if case["use"] == "train":
        return _prepare_train(case, seed)
    M = _mesh(case["mesh"], case["n"])
    a, rng = _alpha(case, M, seed)
    f = float(rng.uniform(0.6, 1.0))  # the period's time factor
    s = {"case": case, "dt": M["dt"], "pass": 0, "Sp": None, "Su": None}
    if case["sources"]:
        t = torch.Generator(device=DEV).manual_seed(seed)
        s["Sp"] = -0.01 * torch.rand(a.shape, generator=t, dtype=torch.float64, device=DEV)
        s["Su"] = 0.001 * torch.rand(a.shape, generator=t, dtype=torch.float64, device=DEV) * (a > 0.5)
    s.update(alpha=a, phi=M["phi"] * f, U=M["U"] * f, Ub=M["Ub"])
    if case["use"] == "resident":
        s["g"] = _handle(case["mesh"], case["n"], case["form"], case["rdf"], case["clip"])
        if case["coupled"]:
            s["rhoPhi"] = torch.empty_like(s["phi"])
        torch.cuda.synchronize()
        return s
    # host arrays: the flow of even passes and, reversed, of odd ones, so that
    # any number of passes keeps the liquid where it is
    pin = case["use"] == "host"

    def host(t):
        t = t.cpu()
        return (t.pin_memory() if pin else t).numpy()

    s.update(alpha=host(a), phi=(host(s["phi"]), host(-s["phi"])), U=(host(s["U"]), host(-s["U"])), Ub=host(s["Ub"]),
             Sp=None if s["Sp"] is None else host(s["Sp"]), Su=None if s["Su"] is None else host(s["Su"]))
    if pin:
        s["g"] = _handle(case["mesh"], case["n"], case["form"], case["rdf"], case["clip"])
    else:
        s["solver"] = solve_vof_equ.SolveVofEqu(
            M["mesh"], s["alpha"], s["phi"][0], s["U"][0],
            {"solvers": {"alpha.water": {"nAlphaBounds": 3, "clip": case["clip"], "precision": case["form"],
                                         "orientationMethod": "isoRDF" if case["rdf"] else "isoAlphaGrad"}}},
            U_boundary=s["Ub"])
        s["solver"].delta_t = s["dt"]
    return s


def _prepare_train(case, seed):
    """The training's initial network and inputs from its own sampler."""
    n = case["rows"]
    X = torch.empty((n, mlp.WIDTH), dtype=torch.bfloat16, device=DEV)
    T = torch.empty((n, 4), dtype=torch.float32, device=DEV)
    g = _handle("jitter", 24, "plain")
    g.samples(seed, X, T)
    g.synchronize()
    key = ("train", n)
    if key not in _HANDLES:
        _HANDLES[key] = mlp.Trainer(*mlp.init_params(1), n)
    return {"case": case, "X": X, "T": T, "trainer": _HANDLES[key]}


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def run(s):
    use = s["case"]["use"]
    if use == "train":
        t = s["trainer"]
        Y = t.forward(s["X"])
        loss, dY = mlp.loss_and_grad(Y, s["T"], s["X"])
        gW, gb = t.backward(s["X"], dY)
        return {"Y": Y, "loss": loss, "gW": gW, "gb": gb}
    if use == "resident":
        g = s["g"]
        g.set_alpha(s["alpha"], device=True)
        g.reconstruct_resident()
        g.advect_resident(s["phi"], s["U"], s["dt"], U_boundary=s["Ub"], Sp=s["Sp"], Su=s["Su"])
        out = {"alpha": _alpha_view(g)}
        if s["case"]["coupled"]:
            r = capi.load().simplic_get_rho_phi(g._h, 1000.0, 1.2, s["phi"].data_ptr(), s["rhoPhi"].data_ptr(),
                                                capi.MEM_DEVICE)
            if r != capi.OK:
                raise RuntimeError(f"simplic_get_rho_phi: {r}")
            out["rhoPhi"] = s["rhoPhi"]
        return out
    k = s["pass"] & 1
    s["pass"] += 1
    if use == "host":
        g = s["g"]
        g.reconstruct_ptr(s["alpha"])
        if s["Sp"] is None:
            g.advect_inplace(s["alpha"], s["phi"][k], s["U"][k], s["dt"], U_boundary=s["Ub"])
        else:
            s["alpha"][:] = g.advect(s["alpha"], s["phi"][k], s["U"][k], s["dt"], U_boundary=s["Ub"], Sp=s["Sp"],
                                     Su=s["Su"], unchanged=True)
        return {"alpha": s["alpha"]}
    v = s["solver"]
    v.phi, v.U = s["phi"][k], s["U"][k]
    v.reconstruct()
    v.advect(s["Sp"], s["Su"])
    return {"alpha": v.alpha()}


def work(case):
    """Bytes: alpha in and out, the cell volume (and sources) once, phi once
    and alphaPhi once, the owner and neighbour of each face unless the mesh is
    a lattice, and the velocity around the interface; host arrays also cross
    the link.  Flops: about 60 per cell for the update, and per interface cell
    the least-squares fit, the plane solve (six cuts of about 1,000) and the
    Simpson fluxes (with the network's 4 x 128 x 128 in the learned form)."""
    if case["use"] == "train":
        n = case["rows"]
        gemms = 2.0 * n * mlp.WIDTH * mlp.WIDTH * (4 + 4 + 3)
        return {"bytes": n * (256 + 16 + 512 + 3 * 512 * 2) + 4 * mlp.WIDTH * mlp.WIDTH * 6, "flops": gemms}
    n = case["n"]
    cells = {"hex": n ** 3, "jitter": n ** 3, "tet": 6 * n ** 3, "checker": 1.7 * n ** 3, "refined": 1.9 * n ** 3}[case["mesh"]]
    faces = (2 if case["mesh"] == "tet" else 3) * cells
    around = (6 if case["mesh"] == "tet" else 1) * n * n * (2.0 if case["shape"] == "drops" else 0.45)
    if case["evolve"] >= 2 * n:
        around *= 2
    b = 24 * cells + 16 * faces + (0 if case["mesh"] == "hex" else 8 * faces) + 700 * around
    if case["sources"]:
        b += 16 * cells
    per = 9000 if case["form"] == "plain" else 5000
    if case["form"] == "learned":
        per += 2 * 4 * 128 * 128
    return {"bytes": b, "flops": 60.0 * cells + per * around * (5 if case["rdf"] else 1)}


# ---------------------------------------------------------------------------
# 64-bit values
# ---------------------------------------------------------------------------
def exact(case, seed):
    """The network's gradient pass in 64 bits.  None for the steps: their
    bounding walks the cells one after the other, which plain numpy takes
    minutes over."""
    if case["use"] != "train":
        return None
    s = _prepare_train(case, seed)
    W0, b0 = mlp.init_params(1)
    W = torch.tensor(W0, dtype=torch.float64, device=DEV, requires_grad=True)
    b = torch.tensor(b0, dtype=torch.float64, device=DEV, requires_grad=True)
    x, T = s["X"].double(), s["T"].double()
    a = x
    for l in range(3):
        a = torch.nn.functional.gelu(a @ W[l].T + b[l], approximate="tanh")
    Y = a @ W[3].T + b[3]
    v = x[:, 124:127] + Y[:, :3]
    v = v / v.norm(dim=1, keepdim=True).clamp(min=1e-6)
    loss = (1.0 - (v * T[:, :3]).sum(1)).mean() + 0.1 * ((Y[:, 3] - T[:, 3]) ** 2).mean()
    loss.backward()
    return {"Y": Y.detach(), "loss": float(loss), "gW": W.grad, "gb": b.grad}

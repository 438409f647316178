"""The timed work of the implicit tet-FEM timestep, through its public entry points.

A case is one of:
  material  an energy's PK1 and clampedHessian of an array of deformation gradients
  elements  TET_MESH.computeElements: per-tet F, Sigma, force and 12x12 Hessian of a mesh
  solve     one solve() of a drop-in timestepper (host state up, one step, host state down)
  batch     one step of a BATCH of scenes: upload of every scene's state, the step, download
  serve     a server that takes a few jobs, steps them to their ends and hands back their states
Meshes are the Kuhn cubes of hobakv1_gb300.scenes; states are smooth deformations with
noise (a cube in motion) or the squashed-and-twisted start, drawn from the seed.
"""
import math

import numpy as np
import torch

from hobakv1_gb300 import hobak, scenes, serving

RAYLEIGH = (0.01, 0.01)           # Rayleigh alpha, beta of the position integrator (its defaults)
STEPPERS = {"velocity": hobak.BACKWARD_EULER_VELOCITY, "position": hobak.BACKWARD_EULER_POSITION,
            "newmark": hobak.NEWMARK}
INTEGRATORS = {"velocity": 0, "position": 1, "newmark": 2}


def listed():
    return [
        # a host that evaluates an energy itself (integration points of its own mesh, plots, tests)
        dict(name="material_snh_4096", path="material", material="snh", n=4096),
        # inspection of a mesh's element terms, as the parity tests and a debugging host do
        dict(name="elements_cube10_arap", path="elements", N=10, material="arap"),
        # the smallest real steps: one small body in an interactive host, where latency counts
        dict(name="solve_cube6_arap_position", path="solve", N=6, material="arap", integrator="position"),
        # the CPU-sized standard cube under gravity, one drop-in solve
        dict(name="solve_cube10_snh_velocity", path="solve", N=10, material="snh", integrator="velocity"),
        # a Newton loop per step, odd size
        dict(name="solve_cube13_stvk_newmark", path="solve", N=13, material="stvk", integrator="newmark"),
        # the large body, plain FP64, both energies of the standard workloads
        dict(name="cube40_snh_fp64", path="batch", scene="twist", N=40, count=1, material="snh", mixed=False,
             integrator="velocity", cluster=0),
        dict(name="cube40_arap_fp64", path="batch", scene="twist", N=40, count=1, material="arap", mixed=False,
             integrator="velocity", cluster=0),
        # the same body in mixed precision
        dict(name="cube40_snh_mixed", path="batch", scene="twist", N=40, count=1, material="snh", mixed=True,
             integrator="velocity", cluster=0),
        # many uneven scenes in one batch (N 6..24, SNH and ARAP), with the clusters the autotuner picks
        dict(name="mix96_mixed", path="batch", scene="mix", N=24, count=96, material="mix", mixed=True,
             integrator="velocity", cluster=8),
        dict(name="mix48_fp64", path="batch", scene="mix", N=24, count=48, material="mix", mixed=False,
             integrator="velocity", cluster=4),
        # self contact of two cubes, vertex-face and edge-edge, in the position integrator
        dict(name="contact_cubes24_fp64", path="batch", scene="contact", N=24, count=1, material="snh", mixed=False,
             integrator="position", cluster=0),
        # a burst of short jobs to the server, half of them in vertex-face contact, mixed precision
        dict(name="serve_6jobs", path="serve", N=12, count=6, steps=6),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    path = rng.choice(["material", "elements", "solve", "solve", "batch", "batch", "batch", "mix", "contact", "serve"])
    energy = rng.choice(["snh", "arap", "stvk", "neo_hookean_bw"])
    integrator = rng.choice(["velocity", "position", "newmark"])
    if path == "material":
        return dict(path="material", material=energy, n=_log_int(rng, 1, 20000))
    if path == "elements":
        return dict(path="elements", N=rng.randint(3, 18), material=energy)
    if path == "solve":
        return dict(path="solve", N=rng.randint(4, 15), material=energy, integrator=integrator)
    if path == "batch":
        return dict(path="batch", scene="twist", N=rng.randint(12, 40), count=1, material=rng.choice(["snh", "arap"]),
                    mixed=rng.random() < 0.4, integrator=rng.choice(["velocity", "position"]), cluster=0)
    if path == "mix":
        mixed = rng.random() < 0.5
        return dict(path="batch", scene="mix", N=rng.randint(9, 24), count=_log_int(rng, 4, 64 if mixed else 32),
                    material="mix", mixed=mixed, integrator=rng.choice(["velocity", "position"]),
                    cluster=rng.choice([0, 4, 8]))
    if path == "contact":
        return dict(path="batch", scene="contact", N=rng.randint(6, 24), count=1, material="snh",
                    mixed=rng.random() < 0.4, integrator=rng.choice(["velocity", "position"]), cluster=0)
    return dict(path="serve", N=rng.randint(8, 12), count=rng.randint(2, 6), steps=rng.randint(2, 6))


# ---- inputs ------------------------------------------------------------------------------

CONTACT = dict(eps=1e-2, stiffness=1e3, damping_beta=1e-3)  # the contact workload's distance and spring


def _smooth(rest, rng, amplitude, noise):
    """A smooth random vector field (three waves of at most one period) plus noise."""
    out = np.zeros_like(rest)
    for _ in range(3):
        k = rng.uniform(-2.0 * np.pi, 2.0 * np.pi, 3)
        out += np.sin(rest @ k + rng.uniform(0, 2 * np.pi))[:, None] * rng.normal(size=3) * amplitude / 3.0
    return out + rng.normal(size=rest.shape) * noise


def _in_motion(s, rng, strain=0.05, speed=0.3):
    """The scene with a deformed, moving state; pinned vertices stay at rest."""
    h = 1.0 / s.N
    s.x0 = _smooth(s.rest, rng, strain, 0.005 * h)
    s.v0 = _smooth(s.rest, rng, speed, 0.01 * speed)
    s.x0[s.pinned] = 0.0
    s.v0[s.pinned] = 0.0
    return s


def _body(N, material, seed, E=1e3, nu=0.45):
    """One top-pinned cube of the CPU-sized workload, in motion."""
    rng = np.random.default_rng([seed, N])
    rest, tets = scenes.kuhn_cube(N, seed=seed % (1 << 31))
    mu, lam = scenes.lame(E, nu)
    s = scenes.Scene(f"cube{N}", rest, tets, material, mu, lam, scenes.top_layer(N), None, None, N=N)
    return _in_motion(s, rng)


def _scenes(case, seed):
    rng = np.random.default_rng([seed, 7])
    kind, N = case["scene"], case["N"]
    if kind == "twist":  # squashed to 0.6 and each layer turned by up to 15 degrees
        s = _body(N, case["material"], seed, E=1e4)
        x = scenes.compress_and_twist(s.rest, N, seed=int(rng.integers(1 << 31)))
        s.x0 = x - s.rest + rng.normal(size=x.shape) * 0.005 / N
        s.v0[s.pinned] = 0.0
        return [s]
    if kind == "mix":
        sizes = np.random.default_rng([case["count"], N]).integers(6, N + 1, size=case["count"])  # the case's own
        return [_in_motion(scenes.config4_scenes(1, int(n), int(n), seed=int(rng.integers(1 << 31)))[0], rng)
                for n in sizes]
    s = scenes.two_cubes_scene(N, seed=int(rng.integers(1 << 31)))
    upper = np.arange(s.nv) >= s.nv // 2
    s.x0 = _smooth(s.rest, rng, 2e-3, 1e-4 / N)
    s.v0 = _smooth(s.rest, rng, 0.05, 1e-4)
    s.v0[upper, 1] -= 0.1
    s.x0[s.pinned] = 0.0
    s.v0[s.pinned] = 0.0
    return [s]


def _jobs(case, seed):
    """Every other job is two cubes in contact, the rest single cubes of the mix."""
    rng, shape = np.random.default_rng([seed, 11]), np.random.default_rng([case["count"], case["N"], case["steps"]])
    out = []
    for j in range(case["count"]):
        N, steps = int(shape.integers(6, case["N"] + 1)), int(shape.integers(2, case["steps"] + 1))
        s = int(rng.integers(1 << 31))
        if j % 2 == 0:
            out.append((scenes.two_cubes_scene(N, seed=s), steps, scenes.SERVE_CONTACT))
        else:
            out.append((scenes.config4_scenes(1, N, N, seed=s)[0], steps, None))
    return out


def _gradients(n, seed):
    """Deformation gradients I + strains of a few tenths, some strongly compressed; all det > 0."""
    rng = np.random.default_rng([seed, 3])
    F = np.eye(3) + rng.normal(size=(n, 3, 3)) * 0.15
    F[rng.random(n) < 0.2] *= 0.6
    bad = np.linalg.det(F) < 0.05
    F[bad] = np.eye(3) * 0.7
    return F


def _pinned(n):
    return torch.empty(n, dtype=torch.float64, pin_memory=torch.cuda.is_available()).numpy()


def prepare(case, seed):
    path = case["path"]
    if path == "material":
        mu, lam = scenes.lame(1e4, 0.45)
        return dict(path=path, material=hobak.make_material(case["material"], mu, lam), F=_gradients(case["n"], seed))
    if path == "elements":
        s = _body(case["N"], case["material"], seed)
        mesh = hobak.TET_MESH(s.rest, s.tets)
        mesh.setDisplacement(s.x0)
        return dict(path=path, mesh=mesh, material=hobak.make_material(s.material, s.mu, s.lam))
    if path == "solve":
        s = _body(case["N"], case["material"], seed)
        mesh = hobak.TET_MESH(s.rest, s.tets)
        step = STEPPERS[case["integrator"]](mesh, hobak.make_material(s.material, s.mu, s.lam))
        step.scaleMass(s.density)
        step.addGravity([s.density * g for g in s.gravity])
        step.attachKinematicConstraints(s.pinned)
        return dict(path=path, step=step, newmark=case["integrator"] == "newmark", x=s.x0.reshape(-1),
                    v=s.v0.reshape(-1))
    if path == "serve":
        return dict(path=path, jobs=_jobs(case, seed))
    group = _scenes(case, seed)
    b = hobak.BATCH(group, hobak.solver_opts(precision=int(case["mixed"]), integrator=INTEGRATORS[case["integrator"]],
                                             rayleigh=RAYLEIGH))
    if case["cluster"]:
        b.set_tuning(tile_vertices=64, element_threads=64, assembly_threads=64, cluster_pcg=1,
                     cluster_max=case["cluster"])
    if case["scene"] == "contact":
        b.set_collisions(0, True, **CONTACT)
        b.set_edge_collisions(0, True)
    n = 3 * b.total_vertices
    bufs = [_pinned(n) for _ in range(4)]
    bufs[0][:] = np.concatenate([s.x0.reshape(-1) for s in group])
    bufs[1][:] = np.concatenate([s.v0.reshape(-1) for s in group])
    return dict(path=path, batch=b, bufs=bufs)


# ---- one pass ----------------------------------------------------------------------------

def run(state):
    path = state["path"]
    if path == "material":
        return {"P": state["material"].PK1(state["F"]), "H": state["material"].clampedHessian(state["F"])}
    if path == "elements":
        return state["mesh"].computeElements(state["material"])
    if path == "solve":
        step = state["step"]
        step.position()[:] = state["x"]
        step.velocity()[:] = state["v"]
        if state["newmark"]:
            step.acceleration()[:] = 0.0
        step.solve()
        out = {"x": step.position(), "v": step.velocity()}
        if state["newmark"]:
            out["a"] = step.acceleration()
        return out
    if path == "serve":
        srv = serving.NativeServer(budget_bytes=1 << 33, precision=hobak.PRECISION_MIXED)
        jobs = [serving.Job(i, s, n, collisions=c) for i, (s, n, c) in enumerate(state["jobs"])]
        for j in jobs:
            srv.submit(j)
        while not srv.idle():
            srv.pump()
        srv.close()
        return [{"x": j.result_x, "v": j.result_v} for j in jobs]
    b, (x, v, xn, vn) = state["batch"], state["bufs"]
    b.set_state_all(x, v)
    b.step(1)
    b.get_state_all(xn, vn)
    return {"x": xn, "v": vn}


# ---- what a pass cannot do without --------------------------------------------------------

# arithmetic of one element (SVD, eigen-clamped Hessian, force) and of one 3x3 block of a product
FLOPS_TET, FLOPS_BLOCK = 1200, 18
ITERATIONS = {"twist": 100, "mix": 40, "contact": 80, "body": 40}  # of an ordinary step


def _step_work(nv, nt, word, iters):
    """Inputs (mesh, state) and outputs once each; per iteration the matrix's 14.5 blocks a row and
    the vectors are needed once more, from wherever they are kept."""
    nb = 14.5 * nv
    return {"bytes": nt * (16 + 72 + 8) + nv * (5 * 24 + 2 * 24) + iters * word * (9 * nb + 30 * nv),
            "flops": nt * FLOPS_TET + iters * (nb * FLOPS_BLOCK + 60 * nv)}


def work(case):
    path, N = case["path"], case.get("N", 0)
    if path == "material":
        return {"bytes": case["n"] * 8 * (9 + 9 + 81), "flops": case["n"] * 2000}
    if path == "elements":
        return {"bytes": 6 * N ** 3 * (16 + 8 * (9 + 3 + 12 + 144)) + 48 * (N + 1) ** 3, "flops": 6 * N ** 3 * 3000}
    if path == "solve":
        newton = 3 if case["integrator"] == "newmark" else 1
        w = _step_work((N + 1) ** 3, 6 * N ** 3, 8, ITERATIONS["body"])
        return {k: v * newton for k, v in w.items()}
    if path == "serve":
        sizes = range(6, N + 1)
        nv = sum((n + 1) ** 3 for n in sizes) / len(sizes) * 1.5
        w = _step_work(nv, 5 * nv, 4, ITERATIONS["mix"])
        return {k: v * case["count"] * (2 + case["steps"]) / 2 for k, v in w.items()}
    sizes = range(6, N + 1) if case["scene"] == "mix" else [N]
    nv = case["count"] * sum((n + 1) ** 3 for n in sizes) / len(sizes) * (2 if case["scene"] == "contact" else 1)
    nt = case["count"] * sum(6 * n ** 3 for n in sizes) / len(sizes) * (2 if case["scene"] == "contact" else 1)
    return _step_work(nv, nt, 4 if case["mixed"] else 8, ITERATIONS[case["scene"]])


# ---- the same in 64 bits by plain torch ---------------------------------------------------

def _dev():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _t(a, dtype=torch.float64):
    return torch.as_tensor(np.ascontiguousarray(a), dtype=dtype, device=_dev())


def _flat(M):
    """[n, 3, 3] -> [n, 9], columns first."""
    return M.transpose(1, 2).reshape(-1, 9)


def _cof(F):
    f0, f1, f2 = F[:, :, 0], F[:, :, 1], F[:, :, 2]
    c = torch.linalg.cross
    return torch.stack([c(f1, f2), c(f2, f0), c(f0, f1)], dim=2)


def _det_hessian(F):
    """d2 det(F) / dF2, [n, 9, 9], columns first."""
    def hat(a):
        z = torch.zeros_like(a[:, 0])
        return torch.stack([torch.stack([z, -a[:, 2], a[:, 1]], 1), torch.stack([a[:, 2], z, -a[:, 0]], 1),
                            torch.stack([-a[:, 1], a[:, 0], z], 1)], 1)
    f0, f1, f2 = (hat(F[:, :, k]) for k in range(3))
    z = torch.zeros_like(f0)
    rows = [torch.cat([z, -f2, f1], 2), torch.cat([f2, z, -f0], 2), torch.cat([-f1, f0, z], 2)]
    return torch.cat(rows, 1)


def _clamp(H):
    out = torch.empty_like(H)
    for k in range(0, len(H), 8192):
        w, Q = torch.linalg.eigh(H[k:k + 8192])
        out[k:k + 8192] = (Q * w.clamp(min=0)[:, None, :]) @ Q.transpose(1, 2)
    return out


def _svd(F):
    """F = U diag(S) V^T with U, V rotations and the sign of det F on the last value."""
    Us, Ss, Vs = [], [], []
    for k in range(0, len(F), 8192):
        U, S, Vh = torch.linalg.svd(F[k:k + 8192])
        V = Vh.transpose(1, 2).clone()
        U, S = U.clone(), S.clone()
        for M in (U, V):
            neg = torch.linalg.det(M) < 0
            M[neg, :, 2] = -M[neg, :, 2]
            S[neg, 2] = -S[neg, 2]
        Us.append(U), Ss.append(S), Vs.append(V)
    return torch.cat(Us), torch.cat(Ss), torch.cat(Vs)


def _energy(material, mu, lam, F):
    """PK1 [n, 3, 3] and the clamped 9x9 Hessian, columns first."""
    n, I9 = len(F), torch.eye(9, dtype=F.dtype, device=F.device)
    if material == "arap":
        U, S, V = _svd(F)
        P = 2 * mu * (F - U @ V.transpose(1, 2))
        H = 2 * mu * I9.expand(n, 9, 9).clone()
        for i, j in ((1, 2), (0, 2), (0, 1)):
            q = _flat(U[:, :, j:j + 1] * V[:, None, :, i] - U[:, :, i:i + 1] * V[:, None, :, j]) / math.sqrt(2)
            H -= (4 * mu / (S[:, i] + S[:, j]))[:, None, None] * q[:, :, None] * q[:, None, :]
        return P, _clamp(H)
    if material == "stvk":
        C = F.transpose(1, 2) @ F
        E = 0.5 * (C - torch.eye(3, dtype=F.dtype, device=F.device))
        tr = E.diagonal(dim1=1, dim2=2).sum(1)
        Sg = 2 * mu * E + lam * tr[:, None, None] * torch.eye(3, dtype=F.dtype, device=F.device)
        P = F @ Sg
        # column c of the Hessian: dP for dF = the c-th unit matrix
        cols = []
        for c in range(9):
            D = torch.zeros(3, 3, dtype=F.dtype, device=F.device)
            D[c % 3, c // 3] = 1
            dE = 0.5 * (D.T @ F + F.transpose(1, 2) @ D)
            dtr = dE.diagonal(dim1=1, dim2=2).sum(1)
            cols.append(_flat(D @ Sg + F @ (2 * mu * dE + lam * dtr[:, None, None]
                                            * torch.eye(3, dtype=F.dtype, device=F.device))))
        return P, _clamp(torch.stack(cols, 2))
    G, J = _cof(F), torch.linalg.det(F)
    g = _flat(G)
    if material == "snh":
        la = lam + mu
        a = la * (J - 1 - mu / la)
        b = torch.full_like(J, la)
    else:  # neo_hookean_bw
        a = (lam * torch.log(J) - mu) / J
        b = (lam * (1 - torch.log(J)) + mu) / J ** 2
    P = mu * F + a[:, None, None] * G
    H = mu * I9 + b[:, None, None] * g[:, :, None] * g[:, None, :] + a[:, None, None] * _det_hessian(F)
    return P, _clamp(H)


class _Mesh:
    def __init__(self, rest, tets, density):
        self.rest, self.tets = _t(rest), _t(tets, torch.int64)
        X = self.rest[self.tets]
        Dm = (X[:, 1:] - X[:, :1]).transpose(1, 2)
        self.inv, self.vol = torch.linalg.inv(Dm), torch.linalg.det(Dm) / 6
        self.ring = torch.zeros(len(rest), dtype=torch.float64, device=_dev())
        self.ring.index_add_(0, self.tets.reshape(-1), (self.vol / 4).repeat_interleave(4))
        self.mass = density * self.ring
        # dF/dx: F = sum_a x_a w_a^T with w_0 = -(w_1 + w_2 + w_3), rows of the inverse
        self.w = torch.cat([-self.inv.sum(1, keepdim=True), self.inv], 1)

    def terms(self, material, mu, lam, x):
        """F, element forces [n, 4, 3] and element Hessians [n, 12, 12] of -K (positive semidefinite)."""
        F = torch.einsum("nai,naj->nij", (self.rest + x)[self.tets], self.w)
        P, H = _energy(material, mu, lam, F)
        f = -self.vol[:, None, None] * torch.einsum("nij,naj->nai", P, self.w)
        B = torch.einsum("naj,ik->njiak", self.w, torch.eye(3, dtype=F.dtype, device=F.device))
        B = B.reshape(len(F), 9, 12)  # row 3 j + i, column 3 a + k
        return F, f, self.vol[:, None, None] * (B.transpose(1, 2) @ H @ B)

    def sum(self, e):
        out = torch.zeros_like(self.rest)
        return out.index_add_(0, self.tets.reshape(-1), e.reshape(-1, 3))

    def mul(self, He, y):
        return self.sum(torch.bmm(He, y[self.tets].reshape(-1, 12, 1)))


def _cg(A, diag, b, free):
    """Block-Jacobi PCG on the free vertices, to the limit of 64 bits."""
    f = free[:, None]
    inv = torch.linalg.inv(diag)
    y, r = torch.zeros_like(b), b * f
    z = torch.einsum("nij,nj->ni", inv, r) * f
    p, rz, stop = z.clone(), (r * z).sum(), 1e-28 * (r * r).sum()
    for k in range(4000):
        if k % 16 == 0 and float((r * r).sum()) <= float(stop):
            break
        q = A(p) * f
        alpha = rz / (p * q).sum()
        y, r = y + alpha * p, r - alpha * q
        z = torch.einsum("nij,nj->ni", inv, r) * f
        new = (r * z).sum()
        p, rz = z + (new / rz) * p, new
    return y


def _surface(tets):
    faces = torch.cat([tets[:, None, k] for k in ([0, 1, 3], [0, 2, 1], [0, 3, 2], [1, 2, 3])], 1).reshape(-1, 3)
    key = faces.sort(1)[0]
    _, where, count = torch.unique(key, dim=0, return_inverse=True, return_counts=True)
    return faces[count[where] == 1]


def _unit(a):
    return a / a.norm(dim=-1, keepdim=True)


def _cross(a, b):
    return torch.linalg.cross(a, b)


def _dot(a, b):
    return (a * b).sum(-1)


def _barycentric(a, b, c, p):
    n = _cross(b - a, c - a)
    nn = _dot(n, n)
    return torch.stack([_dot(n, _cross(c - b, p - b)) / nn, _dot(n, _cross(a - c, p - c)) / nn,
                        _dot(n, _cross(b - a, p - a)) / nn], -1)


def _near(lo_a, hi_a, lo_b, hi_b, eps):
    """Pairs of boxes within eps of each other."""
    out = []
    for k in range(0, len(lo_a), 2048):
        near = torch.ones(len(lo_a[k:k + 2048]), len(lo_b), dtype=torch.bool, device=lo_a.device)
        for i in range(3):
            near &= (lo_b[None, :, i] - eps <= hi_a[k:k + 2048, None, i]) & (hi_b[None, :, i] + eps >= lo_a[k:k + 2048, None, i])
        out.append(near.nonzero() + torch.tensor([k, 0], device=lo_a.device))
    return torch.cat(out).T


def _point_segment(p, a, b, ends):
    """Distance of p to segment a b where it projects inside, else `ends`."""
    l = (b - a).norm(dim=-1)
    d = _dot((b - a) / l[:, None], p - a)
    return torch.where((d > 0) & (d < l), (p - a - (d / l)[:, None] * (b - a)).norm(dim=-1), ends)


def _face_pairs(pos, tri, ring, area, eps):
    """Vertex-face pairs: ids [n, 4] (vertex, then the face backwards), weights."""
    P, v = pos[tri], tri.unique()
    vi, fi = _near(pos[v], pos[v], P.min(1)[0], P.max(1)[0], eps)
    vid = v[vi]
    ok = (tri[fi] != vid[:, None]).all(1)
    vid, fi = vid[ok], fi[ok]
    a, b, c, p = P[fi, 0], P[fi, 1], P[fi, 2], pos[vid]
    n = _unit(_cross(b - a, c - a))
    inside = _barycentric(a, b, c, p).abs().sum(-1) - 1 < 1e-8
    far = torch.full_like(p[:, 0], math.inf)
    edges = torch.stack([_point_segment(p, q, r, far) for q, r in ((a, b), (a, c), (b, c))]).min(0)[0]
    ends = torch.stack([(p - q).norm(dim=-1) for q in (a, b, c)]).min(0)[0]
    dist = torch.where(inside, _dot(n, p - a).abs(), torch.minimum(edges, ends))
    # the cell of a face: bounded through each edge by the plane of the two faces' mean normal
    key = torch.stack([torch.minimum(tri, tri.roll(-1, 1)), torch.maximum(tri, tri.roll(-1, 1))], -1)
    code = (key[..., 0] * (len(pos) + 1) + key[..., 1]).reshape(-1)
    order = code.argsort()  # a closed surface: every edge has two faces, neighbours in this order
    other = torch.empty_like(order)
    other[order[0::2]], other[order[1::2]] = order[1::2], order[0::2]
    nbr = (other // 3).reshape(-1, 3)
    cell, normal = torch.ones_like(inside), _unit(_cross(P[:, 1] - P[:, 0], P[:, 2] - P[:, 0]))
    for k in range(3):
        q, r = P[fi, k], P[fi, (k + 1) % 3]
        side = _unit(_cross(_unit(normal[nbr[fi, k]] + n), r - q))
        cell &= ~(_dot(side, p - q) < 0)
    ok = (dist < eps) & (inside | cell)
    vid, fi = vid[ok], fi[ok]
    return torch.stack([vid, tri[fi, 2], tri[fi, 1], tri[fi, 0]], 1), area[fi] + ring[vid]


def _face_spring(x, eps):
    """c [n, 4], unit direction [n, 3], signed spring length and distance of vertex-face pairs."""
    p, q = x[:, 0], x[:, 1:]
    nh = _unit(_cross(q[:, 1] - q[:, 0], q[:, 2] - q[:, 0]))
    on = p - _dot(nh, p - q[:, 0])[:, None] * nh
    bary = _barycentric(q[:, 0], q[:, 1], q[:, 2], on)
    best = torch.full_like(p[:, 0], math.inf)
    edge = torch.zeros_like(bary)
    for i, j in ((0, 1), (1, 2), (2, 0)):
        e = q[:, j] - q[:, i]
        r = (_dot(p - q[:, i], e) / _dot(e, e)).clamp(0, 1)
        d = (p - q[:, i] - r[:, None] * e).norm(dim=-1)
        b = torch.zeros_like(bary)
        b[:, i], b[:, j] = 1 - r, r
        edge = torch.where((d < best)[:, None], b, edge)
        best = torch.minimum(best, d)
    bary = torch.where((bary >= 0).all(1, keepdim=True), bary, edge)
    t = p - (bary[..., None] * q).sum(1)
    tm = t.norm(dim=-1)
    behind = _dot(_cross(q[:, 0] - q[:, 1], q[:, 2] - q[:, 1]), p - q[:, 1]) < 0
    c = torch.cat([torch.ones_like(tm)[:, None], -bary], 1)
    return c, t, torch.where(behind, tm + eps, tm - eps), tm, tm * tm >= 1e-8


def _edge_pairs(pos, tri, area, eps):
    """Edge-edge pairs: ids [n, 4], c [n, 4], weights, crossing flags."""
    e = torch.stack([tri, tri.roll(-1, 1)], -1).reshape(-1, 2).sort(1)[0]
    edges, where = torch.unique(e, dim=0, return_inverse=True)
    weight = torch.zeros(len(edges), dtype=pos.dtype, device=pos.device)
    weight.index_add_(0, where, area.repeat_interleave(3) / 3)
    order = torch.argsort(where, stable=True)  # two faces per edge, in face order
    faces = (order // 3).reshape(-1, 2)
    P = pos[edges]
    lo, hi = P.min(1)[0], P.max(1)[0]
    i, j = _near(lo, hi, lo, hi, eps)
    ok = (j >= i) & (edges[i][:, :, None] != edges[j][:, None, :]).all(2).all(1)
    i, j = i[ok], j[ok]
    a1, b1 = P[i, 0], P[j, 0]
    La, Lb = P[i, 1] - a1, P[j, 1] - b1
    L11, L22, L12 = _dot(La, La), _dot(Lb, Lb), -_dot(La, Lb)
    det, ra, rb = L11 * L22 - L12 * L12, _dot(La, b1 - a1), -_dot(Lb, b1 - a1)
    t = (L11 * rb - ra * L12) / det
    s = (ra - L12 * t) / L11
    # nearly parallel edges: the middle of their overlap
    s0, s1 = _dot(La, b1 - a1) / L11, _dot(La, P[j, 1] - a1) / L11
    mid = 0.5 * (s0.clamp(0, 1) + s1.clamp(0, 1))
    mid = torch.where((s0 < 0) & (s1 < 0) | (s0 > 1) & (s1 > 1), torch.full_like(mid, -1.0), mid)
    flat = det.abs() < 1e-8
    s = torch.where(flat, mid, s)
    t = torch.where(flat, _dot(Lb, a1 + s[:, None] * La - b1) / L22, t)
    inner = (s >= 1e-4) & (s <= 1 - 1e-4) & (t.abs() >= 1e-4) & (t.abs() <= 1 - 1e-4)
    inner &= flat | (t > 0)
    d = (b1 + t[:, None] * Lb - a1 - s[:, None] * La).norm(dim=-1)
    i, j, s, t, d = (z[inner] for z in (i, j, s, t, d))
    # the nearest partner of each edge, the later one of equals
    order = torch.argsort(-j, stable=True)
    order = order[torch.argsort(d[order], stable=True)]
    order = order[torch.argsort(i[order], stable=True)]
    i, j, s, t, d = (z[order] for z in (i, j, s, t, d))
    first = torch.ones_like(i, dtype=torch.bool)
    first[1:] = i[1:] != i[:-1]
    i, j, s, t, d = (z[first] for z in (i, j, s, t, d))
    code = (edges[:, 0] * len(pos) + edges[:, 1]).sort()[0]
    ring = torch.zeros_like(first[first])
    for a in (0, 1):
        for b in (0, 1):
            u, w = edges[i, a], edges[j, b]
            k = torch.minimum(u, w) * len(pos) + torch.maximum(u, w)
            ring |= code[torch.searchsorted(code, k).clamp(max=len(code) - 1)] == k
    ok = (d < eps) & ~ring
    i, j, s, t = i[ok], j[ok], s[ok], t.abs()[ok]
    crossing = torch.zeros_like(s, dtype=torch.bool)
    o, L = P[i, 0], P[i, 1] - P[i, 0]
    for k in (0, 1):  # the outer edge through a face next to the inner one
        A, B, C = (pos[tri[faces[j, k], m]] for m in range(3))
        n = _cross(B - A, C - A)
        r = _dot(A - o, n) / _dot(L, n)
        h = o + r[:, None] * L
        hit = (r >= 0) & (r < 1)
        for q, w in ((A, B), (B, C), (C, A)):
            hit &= ~(_dot(n, _cross(w - q, h - q)) < 0)
        crossing |= hit
    return (torch.cat([edges[i], edges[j]], 1), torch.stack([s - 1, -s, 1 - t, t], 1), weight[i] + weight[j], crossing)


class _Contact:
    """Contact forces and (positive semidefinite) Hessians w (c c^T) (x) G of a state."""

    def __init__(self, mesh, x, eps, mu, edges):
        tri = _surface(mesh.tets)
        R = mesh.rest[tri]
        area = 0.5 * _cross(R[:, 1] - R[:, 0], R[:, 2] - R[:, 0]).norm(dim=-1)
        ring = torch.zeros_like(mesh.ring).index_add_(0, tri.reshape(-1), area.repeat_interleave(3) / 3)
        pos = mesh.rest + x
        ids, w = _face_pairs(pos, tri, ring, area, eps)
        c, t, spring, r, on = _face_spring(pos[ids], eps)
        if edges:
            ids2, c2, w2, crossing = _edge_pairs(pos, tri, area, eps)
            t2 = (c2[..., None] * pos[ids2]).sum(1)
            r2 = t2.norm(dim=-1)
            ids, c, t, w, r = (torch.cat(z) for z in ((ids, ids2), (c, c2), (t, t2), (w, w2), (r, r2)))
            spring = torch.cat([spring, torch.where(crossing, r2 + eps, r2 - eps)])
            on = torch.cat([on, r2 >= 1e-7])
        self.ids, self.c = ids, c
        n, k = t / r[:, None], (spring / r).clamp(min=0)[:, None, None]
        w = torch.where(on, 2 * mu * w, torch.zeros_like(w))
        nn = n[:, :, None] * n[:, None, :]
        self.G = w[:, None, None] * (nn + k * (torch.eye(3, dtype=n.dtype, device=n.device) - nn))
        self.force = self._sum(mesh, -(w * spring)[:, None, None] * c[..., None] * n[:, None, :])
        self.diag = torch.zeros(len(x), 3, 3, dtype=x.dtype, device=x.device).index_add_(
            0, ids.reshape(-1), (c[..., None, None] ** 2 * self.G[:, None]).reshape(-1, 3, 3))

    def _sum(self, mesh, e):
        return torch.zeros_like(mesh.rest).index_add_(0, self.ids.reshape(-1), e.reshape(-1, 3))

    def mul(self, mesh, y):
        z = torch.einsum("nij,nj->ni", self.G, (self.c[..., None] * y[self.ids]).sum(1))
        return self._sum(mesh, self.c[..., None] * z[:, None, :])


def _exact_step(mesh, s, integrator, x, v, force, contact=None):
    """One step from (x, v) and zero acceleration; contact = (eps, stiffness, beta, edge pairs too)."""
    free = torch.ones(len(x), dtype=torch.bool, device=x.device)
    free[_t(s.pinned, torch.int64)] = False
    dt, m = s.dt, mesh.mass[:, None]
    eye = torch.eye(3, dtype=x.dtype, device=x.device)
    old = x.clone()

    def system(x, scale, mcoef, He, extra=None, hit=None, cscale=0.0):
        diag = mesh.diag(He) * scale + (mcoef * m)[..., None] * eye
        if extra is not None:
            diag = diag + extra[1]
        if hit is not None:
            diag = diag + cscale * hit.diag
        diag[~free] = eye

        def A(y):
            out = mcoef * m * y + scale * mesh.mul(He, y)
            if extra is not None:
                out = out + extra[0](y)
            return out + cscale * hit.mul(mesh, y) if hit is not None else out
        return A, diag

    hit = _Contact(mesh, x, contact[0], contact[1], contact[3]) if contact else None
    if integrator != "newmark":
        _, f, He = mesh.terms(s.material, s.mu, s.lam, x)
        R = mesh.sum(f) + (hit.force if hit else 0)
    if integrator == "velocity":
        b = dt * (R - dt * mesh.mul(He, v) - (dt * hit.mul(mesh, v) if hit else 0) + force)
        A, diag = system(x, dt * dt, 1.0, He, hit=hit, cscale=dt * dt + (dt * contact[2] if contact else 0))
        v = v + _cg(A, diag, b, free)
        return x + dt * v, v * free[:, None], None
    if integrator == "position":
        al, be = RAYLEIGH
        _, _, H0 = mesh.terms(s.material, s.mu, s.lam, torch.zeros_like(x))
        b = (1 / dt - al) * m * v + be * mesh.mul(H0, v) + R + force
        extra = (lambda y: be / dt * mesh.mul(H0, y), be / dt * mesh.diag(H0))
        A, diag = system(x, 1.0, 1 / dt ** 2 - al / dt, He, extra, hit, 1 + (contact[2] / dt if contact else 0))
        x = x + _cg(A, diag, b, free)
        return x, (x - old) / dt * free[:, None], None
    a0, a1, a2 = 4 / dt ** 2, 4 / dt, 1.0
    for _ in range(10):
        _, f, He = mesh.terms(s.material, s.mu, s.lam, x)
        b = (m * (a0 * (x - old) - a1 * v) - mesh.sum(f) - force) * free[:, None]
        A, diag = system(x, 1.0, a0, He)
        x = x - _cg(A, diag, b, free)
        if float((b * b).sum()) <= 1e-7:
            break
    dx = x - old
    return x, (2 / dt * dx - v) * free[:, None], (a0 * dx - a1 * v) * free[:, None]


def _diag(self, He):
    blocks = He.reshape(-1, 4, 3, 4, 3).diagonal(dim1=1, dim2=3).permute(0, 3, 1, 2)  # [n, 4, 3, 3]
    out = torch.zeros(len(self.rest), 3, 3, dtype=He.dtype, device=He.device)
    return out.index_add_(0, self.tets.reshape(-1), blocks.reshape(-1, 3, 3))


_Mesh.diag = _diag


def _np(a):
    return a.cpu().numpy().reshape(-1)


def exact(case, seed):
    path = case["path"]
    if path == "material":
        mu, lam = scenes.lame(1e4, 0.45)
        P, H = _energy(case["material"], mu, lam, _t(_gradients(case["n"], seed)))
        return {"P": P.cpu().numpy(), "H": H.cpu().numpy()}
    if path == "elements":
        s = _body(case["N"], case["material"], seed)
        mesh = _Mesh(s.rest, s.tets, 1.0)
        F, f, He = mesh.terms(s.material, s.mu, s.lam, _t(s.x0))
        n = len(F)
        return {"F": _flat(F).cpu().numpy(), "Sigma": _svd(F)[1].cpu().numpy(),
                "force": f.reshape(n, 12).cpu().numpy(), "hessian": -He.reshape(n, 144).cpu().numpy()}
    if path == "solve":
        s = _body(case["N"], case["material"], seed)
        group, integ, contact = [s], case["integrator"], None
    elif path == "serve":
        out = []
        for s, steps, c in _jobs(case, seed):
            mesh, x, v = _Mesh(s.rest, s.tets, s.density), _t(s.x0), _t(s.v0)
            force = mesh.mass[:, None] * _t(s.gravity)
            for _ in range(steps):
                x, v, _ = _exact_step(mesh, s, "velocity", x, v, force, None if c is None else (*c, False))
            out.append({"x": _np(x), "v": _np(v)})
        return out
    else:
        group, integ = _scenes(case, seed), case["integrator"]
        contact = (CONTACT["eps"], CONTACT["stiffness"], CONTACT["damping_beta"], True) if case["scene"] == "contact" else None
    parts = []
    for s in group:
        mesh = _Mesh(s.rest, s.tets, s.density)
        parts.append(_exact_step(mesh, s, integ, _t(s.x0), _t(s.v0), mesh.mass[:, None] * _t(s.gravity), contact))
    out = {"x": np.concatenate([_np(p[0]) for p in parts]), "v": np.concatenate([_np(p[1]) for p in parts])}
    if path == "solve" and integ == "newmark":
        out["a"] = _np(parts[0][2])
    return out

"""Timed cases of the library: field evaluation, batches, plans and assembly.

The ranges are those of the repository's own configurations: quad and triangle
meshes of 20 to 20,480 cells, k in [0.5, 20], observation points from a handful
to 20,000 with and without points close to the surface, 1 to 64 right-hand
sides, FP64 and mixed precision, single-pass and adaptive quadrature, real and
complex k. `exact` restates the operators in 64-bit torch.
"""
import math
import weakref

import numpy as np
import torch

from bielcc_b200 import abi, gpu
from bielcc_b200 import workloads as W

NEAR = 3.0  # default near-zone radius of the library, in cell diameters


# ---------------------------------------------------------------- cases
def listed():
    return [
        # a single scattering check from a host program: the smallest call, latency counts
        dict(name="host_small_fp64", kind="host", shape="ico", size=1, points=100, near=0.0, k=2.0, rhs=1,
             precision="fp64", n_start=8, p_max=1, incident=True),
        # host program, triangles, odd point count, two polarisations, total field, error report
        dict(name="host_ragged_mixed", kind="host", shape="torus_tri", size=23, points=4997, near=0.05, k=5.0, rhs=2,
             precision="mixed", n_start=8, p_max=1, incident=True),
        # near and far field of a PEC sphere on device buffers: the headline workload
        dict(name="field_mixed", kind="field", shape="sphere", size=64, points=20000, near=0.1, k=6.283185307179586,
             rhs=1, precision="mixed", n_start=8, p_max=1, incident=False),
        # the parity form of the same evaluation on a perturbed triangle mesh, odd point count
        dict(name="field_fp64", kind="field", shape="ico", size=4, points=6001, near=0.1, k=6.283185307179586, rhs=1,
             precision="fp64", n_start=8, p_max=1, incident=True),
        # dielectric body in a lossy medium: electric and magnetic currents, complex k
        dict(name="full_lossy_mixed", kind="full", shape="spheroid", size=30, points=3001, near=0.05, k=4.0, k_im=0.3,
             rhs=1, precision="mixed", n_start=8, p_max=1, incident=True),
        # adaptive quadrature, two passes
        dict(name="adaptive2_mixed", kind="field", shape="sphere", size=64, points=2000, near=0.1,
             k=6.283185307179586, rhs=1, precision="mixed", n_start=8, p_max=2, incident=False),
        # adaptive quadrature, three passes, parity form
        dict(name="adaptive3_fp64", kind="field", shape="sphere", size=40, points=1000, near=0.1,
             k=6.283185307179586, rhs=1, precision="fp64", n_start=8, p_max=3, incident=False),
        # monostatic sweep: one body, many incidence directions
        dict(name="sweep_mixed", kind="field", shape="spheroid", size=45, points=2000, near=0.0, k=8.0, rhs=24,
             precision="mixed", n_start=8, p_max=1, incident=False),
        # many bodies of uneven sizes in one launch
        dict(name="batch_mixed", kind="batch", meshes=12, cells_min=200, cells_max=12000, points=2000, rhs=64,
             precision="mixed", n_start=8, p_max=1),
        # iterative use of a planned batch: new currents, fixed geometry
        dict(name="replay_mixed", kind="replay", meshes=6, cells_min=200, cells_max=6000, points=2000, rhs=64,
             precision="mixed", n_start=8, p_max=1),
        # collocation matrix for a solver, complex64
        dict(name="assemble_mixed", kind="assemble", shape="ico", size=5, k=12.566370614359172, precision="mixed",
             layout="tau2", c64=True, n_start=8, p_max=1),
        # parity matrix of 3x3 blocks on quads, complex128
        dict(name="assemble_fp64", kind="assemble", shape="sphere", size=30, k=6.0, precision="fp64", layout="full3",
             c64=False, n_start=8, p_max=1),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["host", "field", "field", "field", "full", "batch", "replay", "assemble"])
    prec = rng.choice(["mixed", "mixed", "fp64"])
    case = dict(kind=kind, precision=prec, n_start=8, p_max=1)
    if kind in ("batch", "replay"):
        case.update(meshes=rng.randint(1, 12 if kind == "batch" else 6), cells_min=200,
                    cells_max=int(_log(rng, 400, 12000 if kind == "batch" else 6000)),
                    points=int(_log(rng, 33, 2000)), rhs=rng.randint(1, 64), precision="mixed")
        return case
    shape = rng.choice(["sphere", "ico", "torus_tri", "torus", "spheroid", "cube"])
    k = round(_log(rng, 0.5, 20.0), 4)
    if kind == "assemble":
        size = rng.randint(1, 4) if shape == "ico" else int(_log(rng, 4, 22 if shape.startswith("torus") else 35))
        case.update(shape=shape, size=size, k=k, layout=rng.choice(["tau2", "full3"]), c64=prec == "mixed")
        return case
    size = rng.randint(0, 4) if shape == "ico" else int(_log(rng, 4, 28 if shape.startswith("torus") else 60))
    if kind == "field":
        case["p_max"] = rng.choice([1, 1, 2, 3])
        case["n_start"] = rng.choice([8, 8, 4, 10]) if case["p_max"] == 1 else rng.choice([8, 4])
    cap = 1.6e8 if prec == "mixed" else 3e7
    cap /= {1: 1, 2: 5, 3: 20}[case["p_max"]]
    if kind == "full":
        cap /= 4
        case["k_im"] = round(_log(rng, 0.01, 0.5), 4) if rng.random() < 0.7 else 0.0
    points = int(_log(rng, 33, 20000))
    points = max(33, min(points, int(cap / _cells_about(shape, size))))
    rhs = rng.choice([1, 1, 1, 2, 3, 16]) if kind == "field" and case["p_max"] == 1 else 1
    case.update(shape=shape, size=size, points=points, near=rng.choice([0.0, 0.05, 0.1]), k=k, rhs=rhs,
                incident=rng.random() < 0.5)
    return case


def _cells_about(shape, size):
    if shape == "ico":
        return 20 * 4 ** size
    return {"torus": 3, "torus_tri": 6}.get(shape, 2) * size * size


# ---------------------------------------------------------------- inputs
def _rotation(rng):
    q, r = np.linalg.qr(rng.standard_normal((3, 3)))
    return q * np.sign(np.diag(r)) * np.sign(np.linalg.det(q * np.sign(np.diag(r))))


def _cells(shape, size, rng):
    if shape == "sphere":
        c = W.uv_sphere(size, 2 * size)
    elif shape == "ico":
        c = W.perturbed_icosphere(level=size, seed=int(rng.integers(1 << 30)), smooth_iters=4) if size >= 1 \
            else np.array(W.icosphere(0)[0])[W.icosphere(0)[1]]
    elif shape == "spheroid":
        c = W.spheroid(size, 2 * size, 1.0, 2.0)
    elif shape == "cube":
        c = W.rounded_cube(size)
    else:
        c = W.torus(3 * size, size, 1.5, 0.5)
        if shape == "torus_tri":
            c = W.triangulate(c)
    # another position and size for every seed
    return np.ascontiguousarray((c @ _rotation(rng).T) * rng.uniform(0.95, 1.05))


def _points(cells, m, near, rng):
    ext = float(np.max(np.linalg.norm(cells.reshape(-1, 3), axis=1)))
    n_near = int(near * m)
    p = W.shell_points(m - n_near, 2.0 * ext, 5.0 * ext, rng)
    if n_near:
        p = np.concatenate([p, W.near_points(cells, n_near, 0.02, 0.1, rng)])
    return np.ascontiguousarray(p)


def _inputs(case, seed):
    """Host inputs of a case as numpy arrays: one dict per mesh."""
    rng = np.random.default_rng([seed, 7])
    if case["kind"] in ("batch", "replay"):
        out = []
        # sizes, k and the number of currents belong to the case, the rest to the seed
        plan = np.random.default_rng([case["meshes"], case["cells_max"], case["rhs"], case["points"]])
        for i in range(case["meshes"]):
            target = math.exp(plan.uniform(math.log(case["cells_min"]), math.log(case["cells_max"])))
            if i == 0:
                target = case["cells_max"]
            half = (i // 3) % 2 == 1
            t = target / (2 if half else 1)
            shape = ("spheroid", "cube", "torus")[i % 3]
            size = max(4, int(round((t / (3 if shape == "torus" else 2)) ** 0.5)))
            k = math.exp(plan.uniform(math.log(0.5), math.log(20.0)))
            S = int(plan.integers(1, case["rhs"] + 1))
            cells = _cells(shape, size, rng)
            cells = W.triangulate(cells) if half else cells
            out.append(dict(cells=cells, k=k, J=W.po_currents(cells, k, directions=S, seed=int(rng.integers(1 << 30))),
                            pts=_points(cells, case["points"], 0.0, rng)))
        return out
    cells = _cells(case["shape"], case["size"], rng)
    k = complex(case["k"], case.get("k_im", 0.0))
    d = dict(cells=cells, k=k)
    if case["kind"] == "assemble":
        return [d]
    J = W.po_currents(cells, k.real, directions=case["rhs"], seed=int(rng.integers(1 << 30)))
    d["J"] = J
    if case["kind"] == "full":
        n = W.normals(cells)
        d["JM"] = np.cross(n[None], J) * (0.3 + 0.4j) + 0.1 * J
    d["pts"] = _points(cells, case["points"], case["near"], rng)
    d["mult"] = complex(0.0, 0.7) if case["kind"] == "full" else 1.0
    d["multH"] = complex(0.1, 0.9)
    if case.get("incident"):
        direction = rng.standard_normal(3)
        direction /= np.linalg.norm(direction)
        e0 = np.cross(direction, rng.standard_normal(3))
        e0 /= np.linalg.norm(e0)
        d["inc"] = (k.real * direction, e0, 1.0 / k.real)
    return [d]


_ctx = None


def _context():
    global _ctx
    if _ctx is None:
        _ctx = gpu.Context(0)
    return _ctx


class _State(dict):
    """A dict that can be weakly referenced, so that its meshes go with it."""
    __hash__ = object.__hash__


def _dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _close(mesh_list, plan):
    if plan is not None:
        plan.close()
    for m in mesh_list:
        m.close()


def _numparam(case):
    if case["p_max"] == 1:
        return abi.NumParam.default(n_start=case["n_start"])
    return abi.NumParam.default(n_start=case["n_start"], p_max=case["p_max"], p_max_seg=2)


def prepare(case, seed):
    ctx = _context()
    st = _State(case=case, ctx=ctx, np=_numparam(case))
    ins = _inputs(case, seed)
    meshes = [ctx.mesh(d["cells"]) for d in ins]
    plan = None
    st["mesh"] = meshes[0]
    d = ins[0]
    st["k"] = d["k"]
    inc = d.get("inc")
    st["inc"] = abi.PlaneWave.make(inc[0], inc[1], inc[2], add_E=True, add_H=True) if inc is not None else None
    kind = case["kind"]
    if kind == "host":
        S, M = case["rhs"], case["points"]
        st["J"], st["pts"] = d["J"], d["pts"]
        st["out"] = (np.zeros((S, M, 3), np.complex128), np.zeros((S, M, 3), np.complex128))
    elif kind in ("field", "full"):
        S, M = case["rhs"], case["points"]
        st["J"], st["pts"] = _dev(d["J"]), _dev(d["pts"])
        if kind == "full":
            st["JM"] = _dev(d["JM"])
            st["mult"], st["multH"] = d["mult"], d["multH"]
        st["E"] = torch.zeros((S, M, 3), dtype=torch.complex128, device="cuda")
        st["H"] = torch.zeros_like(st["E"])
    elif kind in ("batch", "replay"):
        specs, keep = [], []
        for d, m in zip(ins, meshes):
            J, pts = _dev(d["J"]), _dev(d["pts"])
            E = torch.zeros((J.shape[0], pts.shape[0], 3), dtype=torch.complex128, device="cuda")
            H = torch.zeros_like(E)
            specs.append(dict(mesh=m, n_rhs=J.shape[0], n_pts=pts.shape[0], J=J.data_ptr(), pts=pts.data_ptr(),
                              E=E.data_ptr(), H=H.data_ptr(), k=d["k"]))
            keep.append((J, pts, E, H))
        st["jobs"], st["keep"] = ctx.make_jobs(specs), keep
        if kind == "replay":
            st["J_new"] = [b[0].clone() for b in keep]
            for b in keep:
                b[0].zero_()
            plan = ctx.batch_plan(st["jobs"], numparam=st["np"], precision=case["precision"], stream=_stream())
            st["plan"] = plan
    else:
        n = (2 if case["layout"] == "tau2" else 3) * meshes[0].n_cells
        st["A"] = torch.zeros((n, n), dtype=torch.complex64 if case["c64"] else torch.complex128, device="cuda")
    weakref.finalize(st, _close, meshes, plan)
    return st


def _stream():
    return torch.cuda.current_stream().cuda_stream


def run(state):
    case, ctx = state["case"], state["ctx"]
    kind = case["kind"]
    if kind == "host":
        E, H, _ = ctx.field_EH(state["mesh"], state["J"], state["k"], state["pts"], numparam=state["np"],
                               inc=state["inc"], precision=case["precision"], out=state["out"])
        return [E, H]
    if kind == "field":
        ctx.field_EH_device(state["mesh"], state["J"].data_ptr(), state["k"], state["pts"].data_ptr(),
                            state["E"].data_ptr(), state["H"].data_ptr(), case["rhs"], case["points"],
                            numparam=state["np"], inc=state["inc"], precision=case["precision"], stream=_stream(),
                            report=False)
        return [state["E"], state["H"]]
    if kind == "full":
        ctx.field_EH_full_device(state["mesh"], state["J"].data_ptr(), state["JM"].data_ptr(), state["k"],
                                 state["pts"].data_ptr(), state["E"].data_ptr(), state["H"].data_ptr(), case["rhs"],
                                 case["points"], multE=state["mult"], multH=state["multH"], inc=state["inc"],
                                 numparam=state["np"], precision=case["precision"], stream=_stream())
        return [state["E"], state["H"]]
    if kind == "batch":
        ctx.field_EH_batch(state["jobs"], numparam=state["np"], precision=case["precision"], stream=_stream(),
                           report=False)
        return [t for b in state["keep"] for t in b[2:]]
    if kind == "replay":
        for b, j in zip(state["keep"], state["J_new"]):
            b[0].copy_(j)
        state["plan"].launch(stream=_stream())
        return [t for b in state["keep"] for t in b[2:]]
    layout = abi.LAYOUT_TAU2 if case["layout"] == "tau2" else abi.LAYOUT_FULL3
    ctx.assemble_K_device(state["mesh"], state["k"], state["A"].data_ptr(), numparam=state["np"], layout=layout,
                          c64=case["c64"], precision=case["precision"], stream=_stream())
    return state["A"]


# ---------------------------------------------------------------- what a pass cannot do without
def work(case):
    """Inputs read once, outputs written once; one evaluation of the kernel and
    its gradient per (point, cell) pair (130 flops, as one node of the
    quadrature) and one contraction per right-hand side (114 flops)."""
    def field(n, nv, S, P):
        return 24 * nv * n + 48 * S * n + 24 * P + 96 * S * P, n * P * (130 + 114 * S)

    if case["kind"] in ("batch", "replay"):
        b = f = 0
        for d in _inputs_sizes(case):
            x = field(*d)
            b += x[0]
            f += x[1] if case["kind"] == "batch" else x[1] - 130 * d[0] * d[3]
        return {"bytes": b, "flops": f}
    n = _cells_about(case["shape"], case["size"])
    nv = 3 if case["shape"] in ("ico", "torus_tri") else 4
    if case["kind"] == "assemble":
        m = 2 if case["layout"] == "tau2" else 3
        return {"bytes": 24 * nv * n + (8 if case["c64"] else 16) * (m * n) ** 2, "flops": n * n * (130 + 90)}
    S = case["rhs"] * (2 if case["kind"] == "full" else 1)
    b, f = field(n, nv, S, case["points"])
    return {"bytes": b, "flops": f}


def _inputs_sizes(case):
    """(cells, vertices, right-hand sides, points) of a batch's jobs: expected sizes of the distribution."""
    lo, hi = case["cells_min"], case["cells_max"]
    mean = (hi - lo) / math.log(hi / lo) if hi > lo else hi
    for i in range(case["meshes"]):
        yield (hi if i == 0 else int(mean)), (3 if (i // 3) % 2 else 4), (case["rhs"] + 1) // 2, case["points"]


def tolerance(case):
    """About four times what the forms differ from the 64-bit evaluation
    (mixed up to 2.3e-7; FP64 up to 5e-15, a little more where k r is large)."""
    return {"rel": 1e-6} if case["precision"] == "mixed" else {"rel": 5e-14}


# ---------------------------------------------------------------- 64-bit evaluation
# The operators written out in torch complex128 on whole tensors of pairs.
EPS0 = 2.220446049250313e-16
PI4 = 4.0 * math.pi
ANALYTIC, RS, RS_SEG, ACC = 3.0, 2.0, 2.0, 1e-6


def _lens(a):
    return torch.sqrt((a * a).sum(-1))


def _cross(a, b):
    return torch.linalg.cross(a, b, dim=-1)


def _geometry(v):
    """Centre, diameter, unit normal of cells v [N][nv][3]."""
    c = v.mean(1)
    nv = v.shape[1]
    seg = [v[:, (s + 1) % nv] - v[:, s] for s in range(nv)]
    if nv == 4:
        n = _cross(v[:, 2] - v[:, 0], v[:, 3] - v[:, 1])
        seg += [v[:, 2] - v[:, 0], v[:, 3] - v[:, 1]]
    else:
        n = _cross(v[:, 1] - v[:, 0], v[:, 2] - v[:, 0])
    diam = torch.stack([_lens(s) for s in seg], 0).max(0).values
    return c, diam, n / _lens(n)[:, None]


def _basis(v):
    if v.shape[1] == 4:
        base = (v[:, 2] + v[:, 3] - v[:, 0] - v[:, 1]) / 2
        other = (v[:, 3] + v[:, 0] - v[:, 1] - v[:, 2]) / 2
    else:
        base, other = v[:, 1] - v[:, 0], v[:, 2] - v[:, 0]
    n = _cross(base, other)
    n = n / _lens(n)[:, None]
    t1 = base / _lens(base)[:, None]
    t2 = _cross(n, t1)
    return torch.stack([t1, t2 / _lens(t2)[:, None]], 1)


def _nodes(v, n):
    """Midpoint rule of the n x n split: points [N][n^2][3], weights [N][n^2]."""
    dev = v.device
    if v.shape[1] == 4:
        t = torch.arange(n + 1, dtype=torch.float64, device=dev) / n
        p, q = t[:, None, None], t[None, :, None]
        a, b, c, d = [v[:, i, None, None, :] for i in range(4)]
        g = p * (q * c + (1 - q) * d) + (1 - p) * (q * b + (1 - q) * a)
        c1, c2, c3, c4 = g[:, :-1, :-1], g[:, :-1, 1:], g[:, 1:, 1:], g[:, 1:, :-1]
        y = (c1 + c2 + c3 + c4) / 4
        w = _lens(_cross((c2 + c3 - c1 - c4) / 2, (c3 + c4 - c1 - c2) / 2))
        return y.flatten(1, 2), w.flatten(1, 2)
    i, j = torch.meshgrid(torch.arange(n, device=dev), torch.arange(n, device=dev), indexing="ij")
    up, dn = i + j <= n - 1, i + j <= n - 2
    i, j = i.to(torch.float64), j.to(torch.float64)
    s = torch.cat([i[up] + 1 / 3, i[dn] + 2 / 3]) / n
    t = torch.cat([j[up] + 1 / 3, j[dn] + 2 / 3]) / n
    e1, e2 = v[:, 1] - v[:, 0], v[:, 2] - v[:, 0]
    y = v[:, None, 0] + s[None, :, None] * e1[:, None] + t[None, :, None] * e2[:, None]
    area = _lens(_cross(e1, e2)) / 2 / n ** 2
    return y, area[:, None].expand(y.shape[:2])


def _grad_weight(r, R):
    t = r / R
    return torch.where(t < 1, (3 - 2 * t) / (r * R * R), 1 / (r * r * r))


def _pot_weight(r, R):
    t = r / R
    return torch.where(t < 1, t * (3 - 2 * t) / R, 1 / r)


def _adaptive(one_pass, n, p_max, R, Rmin):
    """The refinement loop for all pairs at once: one_pass(n, R) -> [M][idim]."""
    active = torch.ones(len(R), dtype=torch.bool, device=R.device)
    prev = out = None
    R = R.clone()
    for p in range(p_max):
        val = one_pass(n, R)
        if prev is None:
            prev, out = torch.zeros_like(val), torch.zeros_like(val)
        if p:
            stop = active & ((val - prev).abs().pow(2).sum(-1) < ACC * ACC)
            out[stop] = val[stop]
            active &= ~stop
        prev = torch.where(active[:, None], val, prev)
        for _ in range(val.shape[1]):
            R = torch.where(active & (R > Rmin), R / 2, R)
        n *= 2
    out[active] = prev[active]
    return out, R


def _near_matrices(v, x, k, n_start, p_max, p_seg, analytic):
    """Near operators of pairs (cell v[m], point x[m]): K [M][3][3] and, for the
    field, G [M][3] with R = G x J; analytic: K_RotRot_HS_Colloc."""
    diam, nrm = _geometry(v)[1:]
    M, nv = len(v), v.shape[1]
    one = torch.ones(M, dtype=torch.float64, device=v.device)

    def dist(n):
        y, w = _nodes(v, n)
        d = x[:, None] - y
        return d, _lens(d), w

    if analytic:
        def hm1(n, R):
            _, r, w = dist(n)
            tiny = abs(k) * r < 1e-7
            f = torch.where(tiny, 1j * k - k * k * r / 2, (torch.exp(1j * k * r) - 1) / torch.where(tiny, 1.0, r))
            return (f * w).sum(1, keepdim=True)

        surf = _adaptive(hm1, n_start, p_max, EPS0 * one, EPS0 * one)[0][:, 0]
        surf = surf + _inv_r(v[:, :3], x)
        if nv == 4:
            surf = surf + _inv_r(v[:, [2, 3, 0]], x)
        R, Rmin = EPS0 * one, EPS0 * one
    else:
        def pot(n, R):
            _, r, w = dist(n)
            return (torch.exp(1j * k * r) * _pot_weight(r, R[:, None]) * w).sum(1, keepdim=True)

        surf = _adaptive(pot, n_start, p_max, RS * diam / n_start, ACC * one)[0][:, 0]
        R, Rmin = RS_SEG * diam / 10, ACC * one
    K = torch.zeros((M, 3, 3), dtype=torch.complex128, device=v.device)
    for s in range(nv):
        a, b = v[:, s], v[:, (s + 1) % nv]

        def seg(n, R):
            t = (torch.arange(n, dtype=torch.float64, device=v.device) + 0.5) / n
            d = x[:, None] - (a[:, None] + t[None, :, None] * (b - a)[:, None])
            r = _lens(d)
            f = torch.exp(1j * k * r) * (1j * k * r - 1) * _grad_weight(r, R[:, None])
            return torch.einsum("mq,mqg->mg", f, d.to(f.dtype)) * (_lens(b - a) / n)[:, None]

        ks, R = _adaptive(seg, 10, p_seg, R, Rmin)
        nu = _cross(b - a, nrm)
        ln = _lens(nu)[:, None]
        nu = torch.where(ln > EPS0, nu / torch.where(ln > EPS0, ln, 1.0), nu)
        K -= ks[:, :, None] * nu[:, None, :]
    K += (surf * k * k)[:, None, None] * torch.eye(3, dtype=K.dtype, device=v.device)
    if analytic:
        return K / PI4, None

    def grad(n, R):
        d, r, w = dist(n)
        f = torch.exp(1j * k * r) * (1j * k * r - 1) * _grad_weight(r, R[:, None]) * w
        return torch.einsum("mq,mqg->mg", f, d.to(f.dtype))

    G = _adaptive(grad, n_start, p_max, RS * diam / n_start, diam / 100)[0]
    return K / PI4, G / PI4


def _inv_r(tri, x):
    """Integral of 1/|x - y| over triangles (closed form, Wilton et al. 1984)."""
    e1, e2 = tri[:, 1] - tri[:, 0], tri[:, 2] - tri[:, 0]
    n = _cross(e1, e2)
    nl = _lens(n)
    flat = nl <= 1e-13 * _lens(e1) * _lens(e2)
    n = n / torch.where(flat, 1.0, nl)[:, None]
    h = ((x - tri[:, 0]) * n).sum(-1)
    ah, foot = h.abs(), x - h[:, None] * n
    total = torch.zeros_like(h)
    for e in range(3):
        A, B = tri[:, e], tri[:, (e + 1) % 3]
        L = _lens(B - A)
        l = (B - A) / torch.where(L > 0, L, 1.0)[:, None]
        u = _cross(l, n)
        P0, lm, lp = ((A - foot) * u).sum(-1), ((A - foot) * l).sum(-1), ((B - foot) * l).sum(-1)
        Rm, Rp = _lens(x - A), _lens(x - B)
        R02 = P0 * P0 + h * h
        num, den = Rp + lp, Rm + lm
        good = (num > 0) & (den > 0)
        term = torch.where(good, P0 * torch.log(torch.where(good, num, 1.0) / torch.where(good, den, 1.0)), 0.0)
        term = term - ah * (torch.atan2(P0 * lp, R02 + ah * Rp) - torch.atan2(P0 * lm, R02 + ah * Rm))
        total += torch.where((L > 0) & (P0.abs() > 1e-14 * (L + Rm + Rp)), term, 0.0)
    return torch.where(flat, 0.0, total)


def _far_matrices(y, w, x, k, with_G=True):
    """Raw far moments of every (point, cell): K [P][N][3][3] = A1 I + T and G [P][N][3]."""
    d = [x[:, None, None, g] - y[None, :, :, g] for g in range(3)]
    ir = torch.rsqrt(d[0] * d[0] + d[1] * d[1] + d[2] * d[2])
    e = torch.exp(1j * k / ir) * w[None]
    f2 = e * (3 * ir ** 3 - 3j * k * ir ** 2 - k * k * ir) * ir ** 2
    A1 = (e * (-(ir ** 3) + 1j * k * ir ** 2 + k * k * ir)).sum(-1)
    K = torch.empty(A1.shape + (3, 3), dtype=torch.complex128, device=x.device)
    for a in range(3):
        fd = f2 * d[a]
        for b in range(a, 3):
            K[..., a, b] = (fd * d[b]).sum(-1)
            K[..., b, a] = K[..., a, b]
        K[..., a, a] += A1
    if not with_G:
        return K, None
    f = e * (1j * k / ir - 1) * ir ** 3
    return K, torch.stack([(f * d[g]).sum(-1) for g in range(3)], -1)


def _near_table(c, diam, x):
    """Near decision per (point, cell) with the reference's rounding."""
    d = [x[:, None, g] - c[None, :, g] for g in range(3)]
    return torch.sqrt(d[0] * d[0] + d[1] * d[1] + d[2] * d[2]) < ANALYTIC * diam[None]


def _sums(d, case, sources):
    """Sums over the cells of K[J] and R[J] for each current set in `sources`."""
    v, x, k = _dev(d["cells"]), _dev(d["pts"]), complex(d["k"])
    c, diam, _ = _geometry(v)
    n0, p_max = case["n_start"], case["p_max"]
    p_seg = 1 if p_max == 1 else 2
    ns = [n0 << (p_max - 1)] if p_max <= 2 else [n0 << p for p in range(p_max)]
    tabs = [_nodes(v, n) for n in ns]
    Js = [_dev(j) for j in sources]
    out = [(torch.zeros((j.shape[0], len(x), 3), dtype=torch.complex128, device="cuda"),
            torch.zeros((j.shape[0], len(x), 3), dtype=torch.complex128, device="cuda")) for j in Js]
    N, nn = len(v), ns[-1] ** 2
    cc = max(1, min(N, 4_000_000 // nn))
    pc = max(1, 24_000_000 // (nn * cc))
    for p0 in range(0, len(x), pc):
        xs = x[p0:p0 + pc]
        for c0 in range(0, N, cc):
            sl = slice(c0, c0 + cc)
            far = ~_near_table(c[sl], diam[sl], xs)
            mats = [_far_matrices(y[sl], w[sl], xs, k) for y, w in tabs]
            for (E, H), J in zip(out, Js):
                j = J[:, sl]
                if len(mats) == 1:
                    K, G = mats[0]
                    E[:, p0:p0 + pc] += torch.einsum("pcab,scb->spa", K * far[..., None, None], j) / PI4
                    G = G * far[..., None]
                    gj = torch.einsum("pca,scb->spab", G, j)
                    H[:, p0:p0 + pc] += torch.stack([gj[..., 1, 2] - gj[..., 2, 1], gj[..., 2, 0] - gj[..., 0, 2],
                                                     gj[..., 0, 1] - gj[..., 1, 0]], -1) / PI4
                    continue
                # one refinement loop per integral: F . J for each right-hand side, grad F
                KJ = [torch.einsum("pcab,scb->spca", m[0], j) for m in mats]
                stop = (KJ[1] - KJ[0]).abs().pow(2).sum(-1, keepdim=True) < ACC * ACC
                E[:, p0:p0 + pc] += (torch.where(stop, KJ[1], KJ[2]) * far[None, :, :, None]).sum(2) / PI4
                G = [m[1] for m in mats]
                stop = (G[1] - G[0]).abs().pow(2).sum(-1, keepdim=True) < ACC * ACC
                G = torch.where(stop, G[1], G[2]) * far[..., None]
                H[:, p0:p0 + pc] += _cross(G[None].expand(len(j), *G.shape), j[:, None].expand(
                    -1, len(xs), -1, -1)).sum(2) / PI4
    # near pairs
    for p0 in range(0, len(x), 512):
        near = _near_table(c, diam, x[p0:p0 + 512])
        pi_all, ci_all = near.nonzero(as_tuple=True)
        for q in range(0, len(pi_all), 16384):
            pi, ci = pi_all[q:q + 16384] + p0, ci_all[q:q + 16384]
            K, G = _near_matrices(v[ci], x[pi], k, n0, p_max, p_seg, False)
            for (E, H), J in zip(out, Js):
                E.index_add_(1, pi, torch.einsum("mab,smb->sma", K, J[:, ci]))
                H.index_add_(1, pi, _cross(G[None].expand(J.shape[0], -1, -1), J[:, ci]))
    return out


def _add_incident(d, E, H):
    if d.get("inc") is None:
        return
    kv, e0, hs = (torch.as_tensor(np.asarray(t, np.float64)).cuda() for t in d["inc"])
    ph = torch.exp(1j * (_dev(d["pts"]) @ kv))[:, None]
    E += ph * e0
    H += ph * (hs * _cross(kv, e0))


def exact(case, seed):
    ins = _inputs(case, seed)
    if case["kind"] == "assemble":
        return _exact_matrix(case, ins[0])
    if case["kind"] == "full":
        d = ins[0]
        (KE, RE), (KM, RM) = _sums(d, case, [d["J"], d["JM"]])
        E, H = d["mult"] * KE - RM, d["multH"] * KM + RE
        _add_incident(d, E, H)
        return [E, H]
    res = []
    for d in ins:
        (E, H), = _sums(d, case, [d["J"]])
        _add_incident(d, E, H)
        res += [E, H]
    return [t.cpu().numpy() for t in res] if case["kind"] == "host" else res


def _exact_matrix(case, d):
    v, k = _dev(d["cells"]), complex(d["k"])
    N = len(v)
    if N > 8192:
        return None
    c, diam, _ = _geometry(v)
    tau2 = case["layout"] == "tau2"
    m = 2 if tau2 else 3
    base = _basis(v).to(torch.complex128) if tau2 else \
        torch.eye(3, dtype=torch.complex128, device="cuda").expand(N, 3, 3)
    A = torch.empty((N, m, N, m), dtype=torch.complex128, device="cuda")
    y, w = _nodes(v, case["n_start"])
    step = max(1, 12_000_000 // (N * y.shape[1]))
    for p0 in range(0, N, step):
        rows = slice(p0, p0 + step)
        K = _far_matrices(y, w, c[rows], k, with_G=False)[0] / PI4
        pi, ci = _near_table(c, diam, c[rows]).nonzero(as_tuple=True)
        K[pi, ci] = _near_matrices(v[ci], c[rows][pi], k, case["n_start"], 1, 1, True)[0]
        A[rows] = torch.einsum("pax,pcxy,cby->pacb", base[rows], K, base)
    return A.reshape(m * N, m * N)

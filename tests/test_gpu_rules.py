"""Compressed rules of the far pass (csrc/rules.cu): the field from the shortest
rule that a distance, cell and k allow equals the oracle's full n x n sum, over
the splits where levels appear, and on cells where the Jacobian is no polynomial
(twisted, reversed corner), vanishes (collapsed edge) or is strongly graded.

Tolerances: a pair's truncation is at most 3e-17 (FP64) / 1e-8 (mixed) of
sum w |F|; what remains is rounding, an ulp or so per operation: 1e-14 for
the few cells summed here in FP64, plus the rounding of the phase, k r ulps on
either side, and 1.5e-7 rms per pair in FP32."""
import numpy as np
import pytest

import oracle
from bielcc_b200 import abi
from bielcc_b200 import workloads as W
from conftest import rel_l2

pytestmark = pytest.mark.gpu
TOL = {"fp64": 2e-14, "mixed": 5e-7}
R_MAX = 100.0  # largest distance of _points

QUADS = np.array([
    [[0, 0, 0], [1, 0, 0], [1, 1, 0], [0, 1, 0]],                        # square
    [[0, 0, 0], [3, 0, 0], [3, 1, 0], [0, 1, 0]],                        # rectangle
    [[-1.1, -1, 0], [1.1, -1, 0], [0.9, 1, 0], [-0.9, 1, 0]],            # trapezoid
    [[0, 0, 0], [1, 0, 0], [0.5, 2, 0], [0.5, 2, 0]],                    # collapsed edge
    [[0, 0, 0], [1, 0, 0.2], [1.2, 1, -0.1], [0, 1, 0.15]],              # twisted
    [[0, 0, 0], [1, 0, 0], [0.35, 0.35, 0.05], [0, 1, 0]],               # reversed corner
], dtype=float)
TRIS = np.array([
    [[0, 0, 0], [1, 0, 0], [0.5, 0.866, 0]],
    [[0, 0, 0], [1, 0, 0], [0, 1, 0.3]],
    [[0, 0, 0], [1, 0, 0], [0.3, 0.03, 0]],                              # needle
], dtype=float)


def _cells(nv):
    c = QUADS if nv == 4 else TRIS
    off = 0.4 * np.arange(len(c))[:, None, None] * np.array([1.0, 0.3, 0.5])
    return np.ascontiguousarray(0.1 * c + off)


def _points(m, seed):
    rng = np.random.default_rng(seed)
    d = rng.standard_normal((m, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    # from just outside the near zone to a thousand radii, sorted and not
    r = 0.3 + 1.2 * np.exp(rng.uniform(np.log(0.02), np.log(80.0), size=(m, 1)))
    p = d * r + np.array([0.9, 0.3, 0.5])
    return p if seed % 2 else p[np.argsort(r[:, 0])]


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("nv", [3, 4])
@pytest.mark.parametrize("n_start,k", [(3, 1.0), (4, 1.0), (5, 2.0 + 0.3j), (7, 3.0), (8, 0.0), (8, 1.0), (8, 7.0),
                                       (8, 30.0), (8, 4.0 + 0.3j), (10, 3.0), (16, 3.0), (17, 6.0), (20, 20.0)])
def test_rules_equal_full_sum(gctx, n_start, k, nv, precision):
    # Im k <= 0.3: e^{-Im k R_MAX} >= 1e-13, so that the FP32 products (>= 1e-3 times
    # that) stay normal numbers; below 2^-126 the mixed form has no relative accuracy
    cells = _cells(nv)
    rng = np.random.default_rng(7)
    J = rng.standard_normal((1, len(cells), 3)) + 1j * rng.standard_normal((1, len(cells), 3))
    npm = abi.NumParam.default(n_start=n_start)
    m = gctx.mesh(cells)
    for pts in (_points(1, 3), _points(33, 4), _points(160, 5), _points(160, 6)):
        E, H, rep = gctx.field_EH(m, J, k, pts, numparam=npm, precision=precision)
        Eo, Ho = oracle.field_EH(cells, J, k, pts, npm)
        # per point: a distant point's small field must be as good as a near one's
        for a, b in ((E, Eo), (H, Ho)):
            err = np.linalg.norm(a - b, axis=-1) / np.linalg.norm(b, axis=-1)
            assert np.sqrt(np.mean(err ** 2)) < TOL[precision] + 2.0 ** -52 * abs(k) * R_MAX
    m.close()


@pytest.mark.parametrize("n_lat,points", [(2, 1), (3, 31), (4, 32), (6, 33), (5, 129), (24, 40), (24, 700)])
@pytest.mark.parametrize("precision,tol", [("fp64", 2e-14), ("mixed", 5e-7)])
def test_grids_of_small_problems(gctx, n_lat, points, precision, tol):
    """32-point tiles whose warps share the cells, 8- and 16-cell splits that write
    bytes of a near-mask word, and the first size with whole-warp sweeps."""
    cells = W.uv_sphere(n_lat, 2 * n_lat)
    J = W.po_currents(cells, 2.0, directions=2, seed=1)
    rng = np.random.default_rng(points)
    pts = np.concatenate([W.shell_points(points, 1.6, 5.0, rng), W.near_points(cells, points // 8, 0.05, 0.3, rng)])
    m = gctx.mesh(cells)
    E, H, rep = gctx.field_EH(m, J, 2.0, pts, precision=precision)
    Eo, Ho = oracle.field_EH(cells, J, 2.0, pts)
    assert rel_l2(E, Eo) < tol and rel_l2(H, Ho) < tol
    d = np.linalg.norm(pts[:, None] - W.centres(cells)[None], axis=2)
    assert rep.n_near_pairs == int((d < 3.0 * W.diameters(cells)[None]).sum())
    m.close()


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_non_finite_points_reach_the_result(gctx, precision):
    cells = W.uv_sphere(8, 16)
    J = W.po_currents(cells, 2.0)
    pts = W.sphere_points(70, 3.0, 0)
    pts[5, 1] = np.nan
    pts[40] = np.inf
    m = gctx.mesh(cells)
    E, H, rep = gctx.field_EH(m, J, 2.0, pts, precision=precision, check=False)
    bad = ~np.isfinite(E[0]).all(axis=1)
    assert bad[5] and bad[40] and bad.sum() == 2 and rep.n_nonfinite == 2
    keep = ~bad
    Eo, _ = oracle.field_EH(cells, J, 2.0, pts[keep])
    assert rel_l2(E[0][keep], Eo[0]) < (1e-12 if precision == "fp64" else 1e-6)
    m.close()


@pytest.mark.parametrize("p_max", [1, 2])
@pytest.mark.parametrize("nv", [3, 4])
@pytest.mark.parametrize("n_start,k", [(3, 0.5), (8, 0.5), (8, 5.0), (7, 60.0), (8, 5.0 + 2.0j), (5, 0.3 + 0.1j), (8, 0.0)])
def test_near_pairs_all_phase_forms(gctx, n_start, k, nv, p_max):
    """Near pairs where |k| r, only |k| (r - r0) or neither stays below 1/2, inside and
    outside the smoothing radius. Points lie within a diameter of every cell, at least
    h = 0.01 off its nodes, whose positions (|y| < 4) carry 2 ulps on either side: 3 of
    that over h for the 1/r^3 terms, and an ulp or so per operation."""
    cells = _cells(nv)
    n, h = len(cells), 0.01
    rng = np.random.default_rng(11)
    J = rng.standard_normal((1, n, 3)) + 1j * rng.standard_normal((1, n, 3))
    ctr = cells.mean(axis=1)
    nrm = np.cross(cells[:, 1] - cells[:, 0], cells[:, 2] - cells[:, 0])
    nrm /= np.linalg.norm(nrm, axis=1, keepdims=True)
    pts = np.concatenate([ctr + s * nrm for s in (0.05, 0.02 + h, 0.11)])
    npm = abi.NumParam.default(n_start=n_start, p_max=p_max)
    m = gctx.mesh(cells)
    E, H, rep = gctx.field_EH(m, J, k, pts, numparam=npm, precision="fp64")
    assert rep.n_near_pairs >= n
    Eo, Ho = oracle.field_EH(cells, J, k, pts, npm)
    tol = 3 * 4 * 2.0 ** -52 * 4 / h + 2e-14
    assert rel_l2(E, Eo) < tol and rel_l2(H, Ho) < tol
    if k != 0.0:
        A, _ = gctx.assemble_K(m, k, numparam=npm, layout=abi.LAYOUT_FULL3)
        assert rel_l2(A, oracle.assemble_K(cells, k, npm, layout=abi.LAYOUT_FULL3)) < tol
    m.close()


# Truncation seen apart from rounding: the errors of a cluster of points share the
# truncation of one row (they lie within 1 % of each other's distance and direction)
# while their rounding is independent, so the cluster's mean keeps the first and
# loses the second: m points leave 1.5e-7 (mixed; FP64: an ulp of the phase |k| r
# on either side) / sqrt(m) of it.
def _clusters(r, n_dirs, m, rng):
    d = rng.standard_normal((n_dirs, 1, 3))
    d = d / np.linalg.norm(d, axis=2, keepdims=True) + 0.005 * rng.uniform(-1, 1, (n_dirs, m, 3))
    d /= np.linalg.norm(d, axis=2, keepdims=True)
    return (d * r * rng.uniform(0.995, 1.005, (n_dirs, m, 1))).reshape(-1, 3)


def _cluster_rms(a, ref, m):
    """Per-cluster |mean relative error|, rms over clusters; rows of a, ref: points."""
    e = (a - ref) / np.linalg.norm(ref, axis=-1, keepdims=True)
    e = e.reshape(e.shape[:-2] + (-1, m, 3)).mean(axis=-2)
    return np.sqrt((np.abs(e) ** 2).sum(-1).mean())


def _unit_cells(shape):
    """Centred on the vertex mean, largest vertex distance 1."""
    c = np.array(shape, dtype=float)
    c -= c.mean(axis=0)
    return c / np.linalg.norm(c, axis=1).max()


@pytest.mark.parametrize("form", ["fused", "split", "tensor"])
def test_batch_pairs_take_a_row_both_cells_allow(gctx, form):
    """A collapsed quad (as at a sphere's pole) allows 16 nodes here but not the next
    level's 20, which its partner, a square, needs: the pair takes the first row that
    both allow. With 20 nodes the collapsed quads' truncation is up to 2.2e-7. One
    right-hand side per cell; tolerance: 1.5e-7 / sqrt(32) of rounding (2.7e-8), the
    allowed truncation 1e-8 and half of their sum again for the spread of 64 clusters."""
    torch = pytest.importorskip("torch")
    k, r, m = 0.96, 13.4, 32
    pole = _unit_cells([[-3.5, -1, 0], [3.5, -1, 0], [0.59, 1, 0], [0.59, 1, 0]])
    square = 1.4 * _unit_cells([[0, 0, 0], [1, 0, 0], [1, 1, 0], [0, 1, 0]])
    cells = np.stack([pole] * 4 + [square] * 4)
    J = np.zeros((8, 8, 3), np.complex128)
    for c in range(8):
        J[c, c, c % 2] = 1.0  # in the cells' plane
    pts = _clusters(r, 64, m, np.random.default_rng(3))
    Eo, Ho = oracle.field_EH(cells, J, k, pts)
    mesh = gctx.mesh(cells)
    dev = [torch.from_numpy(a).cuda() for a in (J, pts)]
    E, H = (torch.zeros((8, len(pts), 3), dtype=torch.complex128, device="cuda") for _ in range(2))
    jobs = gctx.make_jobs([dict(mesh=mesh, n_rhs=8, n_pts=len(pts), J=dev[0].data_ptr(), pts=dev[1].data_ptr(),
                                E=E.data_ptr(), H=H.data_ptr(), k=k)])
    if form == "tensor":
        gctx.set_batch_tensor_cores(True)
    try:
        if form == "split":
            plan = gctx.batch_plan(jobs, precision="mixed", stream=0)
            plan.launch(stream=0)
            torch.cuda.synchronize()
            plan.close()
        else:
            gctx.field_EH_batch(jobs, precision="mixed", stream=0)
    finally:
        gctx.set_batch_tensor_cores(False)
    torch.cuda.synchronize()
    tol = 1.5 * (1.5e-7 / np.sqrt(m) + 1e-8)
    for c in range(8):
        assert _cluster_rms(E[c].cpu().numpy(), Eo[c], m) < tol, c
        assert _cluster_rms(H[c].cpu().numpy(), Ho[c], m) < tol, c
    mesh.close()


@pytest.mark.parametrize("arg", [0.0, 0.25, 0.5])  # of k, in half turns
@pytest.mark.parametrize("precision,shape,kappa,theta", [
    ("fp64", QUADS[0], 0.472, 0.0408),  # the limits of 28 nodes
    ("fp64", QUADS[0], 0.400, 0.0400),
    ("fp64", TRIS[0], 0.760, 0.0820),   # of 33 nodes
    ("fp64", TRIS[0], 0.394, 0.0490),   # of 25
    ("mixed", TRIS[0], 1.285, 0.1640),  # of 16
    ("mixed", QUADS[0], 0.788, 0.0935)])  # of 12
def test_truncation_with_loss_at_the_limits(gctx, precision, shape, kappa, theta, arg):
    """A cell at a distance and |k| where both limits of a level for real k are reached:
    with Im k the level is not allowed there (its error was up to 1.7e-15 in FP64 and
    2.5e-7 in the mixed form). Copies of the problem at several scales, k scaled along,
    share the truncation and not the FP32 rounding, which points at one distance have in
    common. Tolerance: the allowed truncation (1.8 times 3e-17; 1e-8) and 1.5 times what
    the averages leave of the rounding: FP64, the exponent's |k| r ulps on either side
    and a few of the sums over 128 points; mixed, 1.5e-7 per pair over 16 scales."""
    m, dirs, n_scales = 128, 16, 1 if precision == "fp64" else 16
    rho = 1 - 1 / 8  # of the nodes of the 8-split of a square or triangle of radius 1
    k = kappa / rho * np.exp(1j * np.pi * arg)
    cell = _unit_cells(shape)[None]
    J = np.zeros((2, 1, 3), np.complex128)
    J[0, 0, 0] = J[1, 0, 1] = 1.0
    pts = _clusters(rho / theta, dirs, m, np.random.default_rng(5))
    err = []
    for scale in np.geomspace(1, 4, n_scales, endpoint=False):
        mesh = gctx.mesh(scale * cell)
        out = gctx.field_EH(mesh, J, k / scale, scale * pts, precision=precision)[:2]
        ref = oracle.field_EH(scale * cell, J, k / scale, scale * pts)
        mesh.close()
        err.append([((a - b) / np.linalg.norm(b, axis=-1, keepdims=True)).reshape(2, dirs, m, 3).mean(axis=2)
                    for a, b in zip(out, ref)])
    tol = (5.4e-17 + 1.5 * (kappa / theta + 4) * 2.0 ** -53 / np.sqrt(m) if precision == "fp64"
           else 1e-8 + 1.5 * 1.5e-7 / np.sqrt(n_scales))
    e = np.mean(err, axis=0)  # [E, H][right-hand side][cluster][3]
    assert np.sqrt((np.abs(e) ** 2).sum(-1).mean(axis=(1, 2))).max() < tol


@pytest.mark.parametrize("p_max", [1, 2, 3])
@pytest.mark.parametrize("nv", [3, 4])
def test_rules_are_built_in_the_rows_that_calls_read(gctx, nv, p_max):
    """A mesh holds the rules of the precisions that its calls used; whichever came
    first, a later call gives the bits of a first call on a mesh of its own."""
    cells = W.perturbed_icosphere(2, seed=1) if nv == 3 else W.uv_sphere(12, 24)
    J = W.po_currents(cells, 3.0)
    pts = W.shell_points(200, 1.7, 4.0, np.random.default_rng(2))
    npm = abi.NumParam.default(p_max=p_max)

    torch = pytest.importorskip("torch")
    Jd, Pd = torch.from_numpy(J).cuda(), torch.from_numpy(pts).cuda()

    def call(m, precision):  # without a report: no FP64 error sample in the mixed form
        E, H = (torch.zeros((len(J), len(pts), 3), dtype=torch.complex128, device="cuda") for _ in range(2))
        gctx.field_EH_device(m, Jd.data_ptr(), 3.0, Pd.data_ptr(), E.data_ptr(), H.data_ptr(), len(J), len(pts),
                             numparam=npm, precision=precision, stream=0, report=False)
        torch.cuda.synchronize()
        return np.concatenate([E.cpu().numpy(), H.cpu().numpy()])

    alone, mem = {}, {}
    for precision in ("fp64", "mixed"):
        m0 = gctx.mem_used()
        m = gctx.mesh(cells)
        alone[precision] = call(m, precision)
        m1 = gctx.mem_used()
        m.close()
        mem[precision] = m1 - gctx.mem_used()  # of the mesh alone
    if p_max == 1:  # FP64 rows are twice the bytes of FP32 rows
        assert mem["mixed"] < mem["fp64"]
    for order in (("fp64", "mixed", "fp64"), ("mixed", "fp64", "mixed")):
        m = gctx.mesh(cells)
        for precision in order:
            assert np.array_equal(call(m, precision), alone[precision])
        m1 = gctx.mem_used()
        m.close()
        if p_max == 1:
            assert m1 - gctx.mem_used() > max(mem.values())

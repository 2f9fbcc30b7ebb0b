"""Parallel-beam kernels (through the C ABI) against the oracle and the
reference's golden vectors.  Tolerance: relative L2 <= 1e-5 (float32 kernels
vs the reference's float64), dot test <= 1e-6 relative."""
import numpy as np
import pytest
import torch

from oracle import oracle as O
from tests.conftest import relL2

pytestmark = pytest.mark.gpu
TOL = 1e-5


def plan_for(shape, angles):
    from vamtoolbox_b200.projector.Projector3DParallel import ParallelPlan

    return ParallelPlan(shape[0], shape[1], shape[2], angles)


def dev(a):
    return torch.as_tensor(np.ascontiguousarray(a, dtype=np.float32), device="cuda")


@pytest.mark.parametrize("tag", ["even", "odd"])
def test_forward_backward_match_reference_golden(golden, tag):
    P = golden["parallel"]
    x, ang = P[f"{tag}_x"], P[f"{tag}_angles"]
    p = plan_for(x.shape, ang)
    b = p.forward(dev(x)).cpu().numpy()
    assert relL2(b, P[f"{tag}_fwd"]) < TOL
    xb = p.backward_ref(dev(P[f"{tag}_b"])).cpu().numpy()
    assert relL2(xb, P[f"{tag}_bwd"]) < TOL


def test_occlusion_matches_reference_golden(golden):
    P = golden["parallel"]
    p = plan_for(P["occ_x"].shape, P["occ_angles"])
    p.set_occlusion(P["occ_insert"])
    occ = p.occlusion_sinogram().cpu().numpy()
    ref = P["occ_sino"]
    assert np.array_equal(np.isnan(occ), np.isnan(ref))
    assert np.nanmax(np.abs(occ - ref)) == 0.0
    assert relL2(p.forward(dev(P["occ_x"])).cpu().numpy(), P["occ_fwd"]) < TOL
    assert relL2(p.backward_ref(dev(P["occ_b"])).cpu().numpy(), P["occ_bwd"]) < TOL


@pytest.mark.parametrize("shape,na", [((32, 32, 8), 24), ((33, 33, 5), 17), ((40, 40, 1), 30),
                                      ((24, 24, 12), 9), ((48, 48, 64), 12), ((20, 20, 3), 360)])
def test_against_oracle_shapes(shape, na):
    rng = np.random.default_rng(sum(shape) + na)
    ang = np.sort(rng.uniform(0, 360, na))
    ang[0] = 0.0
    x = rng.uniform(0, 1, shape)
    b = rng.uniform(0, 1, (shape[0], na, shape[2]))
    p = plan_for(shape, ang)
    assert relL2(p.forward(dev(x)).cpu().numpy(), O.parallel_forward(x, ang)) < TOL
    assert relL2(p.backward_ref(dev(b)).cpu().numpy(), O.parallel_backward_ref(b, ang)) < TOL
    assert relL2(p.adjoint(dev(b)).cpu().numpy(), O.parallel_adjoint(b, ang)) < TOL


def test_exact_angles_and_binary_target():
    """Multiples of 90 degrees put samples on integer coordinates (floor == ceil)."""
    n = 64
    yy, xx = np.mgrid[:n, :n] - n / 2
    x = ((xx ** 2 + yy ** 2) < 20 ** 2).astype(float)[:, :, None] * np.ones((1, 1, 4))
    ang = np.array([0.0, 45.0, 90.0, 180.0, 270.0, 359.5])
    p = plan_for(x.shape, ang)
    assert relL2(p.forward(dev(x)).cpu().numpy(), O.parallel_forward(x, ang)) < TOL
    bb = O.parallel_forward(x, ang)
    assert relL2(p.backward_ref(dev(bb)).cpu().numpy(), O.parallel_backward_ref(bb, ang)) < TOL


@pytest.mark.parametrize("absn", [None, "ray", "mask"])
def test_adjoint_dot_product(absn):
    rng = np.random.default_rng(3)
    shape, na = (36, 36, 8), 20
    ang = np.linspace(0, 360, na, endpoint=False) + 0.3
    p = plan_for(shape, ang)
    mask = None
    if absn == "ray":
        p.set_absorption("ray", alpha_per_px=0.03, radius_px=15.0)
        oabs = ("ray", 0.03, 15.0)
    elif absn == "mask":
        mask = rng.uniform(0.2, 1.0, shape[:2])
        p.set_absorption("mask", mask=mask)
        oabs = ("mask", mask)
    else:
        oabs = None
    x = rng.uniform(0, 1, shape)
    y = rng.uniform(0, 1, (shape[0], na, shape[2]))
    Ax = p.forward(dev(x)).double()
    Aty = p.adjoint(dev(y)).double()
    lhs = float((Ax * dev(y).double()).sum())
    rhs = float((dev(x).double() * Aty).sum())
    assert abs(lhs - rhs) <= 1e-6 * abs(lhs)
    # signed inputs: error relative to the sum of magnitudes
    xs, ys = dev(rng.standard_normal(shape)), dev(rng.standard_normal((shape[0], na, shape[2])))
    a1 = p.forward(xs).double() * ys.double()
    a2 = xs.double() * p.adjoint(ys).double()
    assert abs(float(a1.sum() - a2.sum())) <= 1e-6 * float(a1.abs().sum())
    assert relL2(Ax.cpu().numpy(), O.parallel_forward(x, ang, absorption=oabs)) < TOL
    assert relL2(p.backward_ref(dev(y)).cpu().numpy(), O.parallel_backward_ref(y, ang, absorption=oabs)) < TOL


def test_occlusion_adjoint_is_transpose(golden):
    P = golden["parallel"]
    p = plan_for(P["occ_x"].shape, P["occ_angles"])
    p.set_occlusion(P["occ_insert"])
    rng = np.random.default_rng(5)
    x = rng.standard_normal(P["occ_x"].shape)
    y = rng.standard_normal(P["occ_fwd"].shape)
    lhs = float((p.forward(dev(x)).double() * dev(y).double()).sum())
    rhs = float((dev(x).double() * p.adjoint(dev(y)).double()).sum())
    assert abs(lhs - rhs) <= 1e-5 * abs(lhs)


def test_mask_matches_reference_mask(golden):
    from vamtoolbox_b200 import geometry

    P = golden["parallel"]
    px, a, R = P["mask_params"]
    tg = geometry.TargetGeometry(target=np.ones((24, 24, 2)))
    pg = geometry.ProjectionGeometry(np.array([0.0]), "parallel", projector_pixel_size=px, absorption_coeff=a,
                                     container_radius=R)
    pg.calcAbsorptionMask(tg)
    assert np.array_equal(pg.absorption_mask[:, :, 0], P["mask"])


def test_projector_class_numpy_roundtrip(golden):
    from vamtoolbox_b200 import geometry
    from vamtoolbox_b200.projector.Projector3DParallel import Projector3DParallel

    P = golden["parallel"]
    x, ang = P["even_x"], P["even_angles"]
    tg = geometry.TargetGeometry(target=x.copy(), clip_to_circle=False)
    pg = geometry.ProjectionGeometry(ang, "parallel", CUDA=True)
    A = Projector3DParallel(tg, pg)
    b = A.forward(x)
    assert isinstance(b, np.ndarray) and b.dtype == np.float64 and b.shape == P["even_fwd"].shape
    assert relL2(b, P["even_fwd"]) < TOL
    assert relL2(A.backward(P["even_b"]), P["even_bwd"]) < TOL
    t = A.forward(torch.as_tensor(x, device="cuda", dtype=torch.float32))
    assert t.is_cuda and t.dtype == torch.float32


def test_deterministic_gather_kernels():
    rng = np.random.default_rng(11)
    shape, ang = (40, 40, 16), np.linspace(0, 180, 33)
    x, y = dev(rng.uniform(size=shape)), dev(rng.uniform(size=(40, 33, 16)))
    p = plan_for(shape, ang)
    for f, a in ((p.forward, x), (p.backward_ref, y), (p.adjoint, y)):
        assert torch.equal(f(a), f(a))


def test_bad_inputs_raise():
    from vamtoolbox_b200._lib import VamError

    p = plan_for((16, 16, 4), np.linspace(0, 180, 8))
    with pytest.raises(ValueError):
        p.forward(torch.zeros((16, 16, 5), device="cuda"))
    with pytest.raises(TypeError):
        p.forward(torch.zeros((16, 16, 4), device="cuda", dtype=torch.float64))
    with pytest.raises(VamError):
        p.set_absorption("ray", alpha_per_px=float("nan"), radius_px=3.0)


FAST_CASES = [
    ((32, 32, 128), np.linspace(0, 360, 24, endpoint=False)),     # even N, all angles paired, VZ=4
    ((33, 33, 256), np.linspace(0, 360, 20, endpoint=False)),     # odd N, paired, VZ=8
    ((30, 30, 128), None),                                        # unpaired random angles
    ((28, 28, 192), np.concatenate([np.linspace(0, 180, 7, endpoint=False), [200.0, 380.0]])),  # mixed
]


@pytest.mark.parametrize("shape,ang", FAST_CASES)
@pytest.mark.parametrize("absn", [None, "mask", "ray"])
def test_fast_paths_against_oracle(shape, ang, absn):
    rng = np.random.default_rng(shape[2] + shape[0])
    if ang is None:
        ang = np.sort(rng.uniform(0, 360, 17))
    x = rng.uniform(0, 1, shape)
    b = rng.uniform(0, 1, (shape[0], ang.size, shape[2]))
    p = plan_for(shape, ang)
    oabs = None
    if absn == "mask":
        m = rng.uniform(0.3, 1.0, shape[:2])
        p.set_absorption("mask", mask=m)
        oabs = ("mask", m)
    elif absn == "ray":
        p.set_absorption("ray", alpha_per_px=0.04, radius_px=shape[0] / 2 - 1.5)
        oabs = ("ray", 0.04, shape[0] / 2 - 1.5)
    assert relL2(p.forward(dev(x)).cpu().numpy(), O.parallel_forward(x, ang, absorption=oabs)) < TOL
    assert relL2(p.backward_ref(dev(b)).cpu().numpy(), O.parallel_backward_ref(b, ang, absorption=oabs)) < TOL
    assert relL2(p.adjoint(dev(b)).cpu().numpy(), O.parallel_adjoint(b, ang, absorption=oabs)) < TOL
    # dot test <Ax, y> = <x, A^T y>
    Ax = p.forward(dev(x)).double()
    lhs = float((Ax * dev(b).double()).sum())
    rhs = float((dev(x).double() * p.adjoint(dev(b)).double()).sum())
    assert abs(lhs - rhs) <= 1e-6 * abs(lhs)


@pytest.mark.parametrize("absn", [None, "ray"])
def test_adjoint_without_weight_table(absn):
    """The on-the-fly matched transpose (used when the table is not built or is too large)."""
    rng = np.random.default_rng(9)
    shape, ang = (30, 30, 128), np.linspace(0, 360, 18, endpoint=False) + 0.7
    p = plan_for(shape, ang)
    p.adj_table_limit_bytes = 0
    oabs = None
    if absn == "ray":
        p.set_absorption("ray", alpha_per_px=0.04, radius_px=13.0)
        oabs = ("ray", 0.04, 13.0)
    b = rng.uniform(0, 1, (30, 18, 128))
    assert relL2(p.adjoint(dev(b)).cpu().numpy(), O.parallel_adjoint(b, ang, absorption=oabs)) < TOL
    assert not p._adj_ready


TUNINGS = [dict(forward_vz=fv, backward_vz=bv, backward_batch=bb, adjoint_vz=av, adjoint_table=at, backward_table=bt)
           for fv, (bv, bb, bt), (av, at) in [(4, (4, 1, 0), (4, 1)), (8, (8, 1, 0), (8, 1)), (4, (4, 2, 0), (4, 0)),
                                              (8, (8, 2, 0), (8, 0)), (4, (4, 4, 0), (8, 1)), (1, (1, 1, 0), (1, 0)),
                                              (8, (8, 2, 1), (8, 1))]]


@pytest.mark.parametrize("tuning", TUNINGS, ids=lambda t: "-".join(str(v) for v in t.values()))
@pytest.mark.parametrize("absn", [None, "ray"])
def test_every_launch_shape_matches_oracle(tuning, absn):
    """Each launch shape the autotuner can pick (vector width, angle batch, table) gives the oracle's result,
    including an angle count that is not a multiple of the batch and paired + unpaired angles."""
    rng = np.random.default_rng(77)
    shape = (29, 29, 256)
    ang = np.concatenate([np.linspace(0, 360, 14, endpoint=False), [7.3, 101.9, 250.1]])
    x = rng.uniform(0, 1, shape)
    b = rng.uniform(0, 1, (shape[0], ang.size, shape[2]))
    p = plan_for(shape, ang)
    oabs = None
    if absn == "ray":
        p.set_absorption("ray", alpha_per_px=0.05, radius_px=12.5)
        oabs = ("ray", 0.05, 12.5)
    p.set_tuning(tuning)
    if tuning["backward_table"]:
        assert p.prepare_backward()
    got = p.get_tuning()
    assert {k: got[k] for k in tuning} == tuning
    assert relL2(p.forward(dev(x)).cpu().numpy(), O.parallel_forward(x, ang, absorption=oabs)) < TOL
    assert relL2(p.backward_ref(dev(b)).cpu().numpy(), O.parallel_backward_ref(b, ang, absorption=oabs)) < TOL
    assert relL2(p.adjoint(dev(b)).cpu().numpy(), O.parallel_adjoint(b, ang, absorption=oabs)) < TOL


def test_autotune_caches_winner(tmp_path, monkeypatch):
    monkeypatch.setenv("VAMTOOLBOX_B200_TUNE_CACHE", str(tmp_path / "tune.json"))
    from vamtoolbox_b200 import autotune as AT

    p = plan_for((40, 40, 128), np.linspace(0, 180, 30, endpoint=False))
    first = p.autotune()
    d = AT._load(str(tmp_path / "tune.json"))
    key = AT.problem_key(p)
    assert d[key]["tuning"] == first and set(d[key]["ms"]) == {"forward", "backward", "adjoint"}
    q = plan_for((40, 40, 128), np.linspace(0, 180, 30, endpoint=False))
    assert q.autotune() == first
    with pytest.raises(Exception):
        q.set_tuning({"backward_batch": 3})


@pytest.mark.parametrize("n,na", [(40, 30), (33, 17), (128, 180), (257, 90)])
@pytest.mark.parametrize("absn", [None, "mask", "ray"])
@pytest.mark.parametrize("path", ["tiles", "generic"])
def test_single_slice_paths_against_oracle(n, na, absn, path):
    """2-D slices: the shared-memory tile kernels (default) and the generic kernels both match the oracle."""
    rng = np.random.default_rng(n + na)
    ang = np.sort(rng.uniform(0, 360, na))
    ang[0] = 0.0
    x = rng.uniform(0, 1, (n, n, 1))
    b = rng.uniform(0, 1, (n, na, 1))
    p = plan_for(x.shape, ang)
    oabs = None
    if absn == "mask":
        m = rng.uniform(0.3, 1.0, (n, n))
        p.set_absorption("mask", mask=m)
        oabs = ("mask", m)
    elif absn == "ray":
        p.set_absorption("ray", alpha_per_px=0.02, radius_px=n / 2 - 1.5)
        oabs = ("ray", 0.02, n / 2 - 1.5)
    if path == "generic":
        p.set_tuning({"forward_vz": 1, "backward_vz": 1, "adjoint_vz": 1})
    else:
        p.set_tuning({"forward_vz": 4, "backward_vz": 4})  # tiles at every size
    assert relL2(p.forward(dev(x)).cpu().numpy(), O.parallel_forward(x, ang, absorption=oabs)) < TOL
    assert relL2(p.backward_ref(dev(b)).cpu().numpy(), O.parallel_backward_ref(b, ang, absorption=oabs)) < TOL


@pytest.mark.parametrize("nz", [1, 8])
def test_ray_absorption_disk_known_answer(nz):
    """Per-ray absorption, centred uniform disk of radius rho inside a container of radius R: the
    weight exp(-alpha (s - s_entry)), s_entry = -sqrt(R^2 - t^2), integrates over the disk's chord
    to b(t) = exp(-alpha sqrt(R^2 - t^2)) 2 sinh(alpha sqrt(rho^2 - t^2)) / alpha (straight-ray
    transmission); with alpha -> 0 it is the chord 2 sqrt(rho^2 - t^2)."""
    from vamtoolbox_b200.projector.Projector3DParallel import ParallelPlan

    n, rho, R, alpha = 128, 40.0, 56.0, 0.02
    yy, xx = np.mgrid[:n, :n] - n // 2
    disk = np.zeros((n, n))
    for dy in np.linspace(-0.5, 0.5, 8, endpoint=False) + 1 / 16:
        for dx in np.linspace(-0.5, 0.5, 8, endpoint=False) + 1 / 16:
            disk += ((xx + dx) ** 2 + (yy + dy) ** 2 <= rho ** 2)
    disk /= 64
    angles = np.array([0.0, 37.0, 90.0, 211.0])
    p = ParallelPlan(n, n, nz, angles)
    p.set_absorption("ray", alpha_per_px=alpha, radius_px=R)
    x = torch.as_tensor(np.repeat(disk[:, :, None], nz, axis=2), dtype=torch.float32, device="cuda").contiguous()
    b = p.forward(x).cpu().numpy().astype(np.float64)
    t = np.arange(n) - n // 2
    inner = np.abs(t) < rho - 2
    Lr, Lc = np.sqrt(np.clip(R ** 2 - t ** 2.0, 0, None)), np.sqrt(np.clip(rho ** 2 - t ** 2.0, 0, None))
    want = np.exp(-alpha * Lr) * 2 * np.sinh(alpha * Lc) / alpha
    rel = np.abs(b[inner] - want[inner, None, None]) / want[inner, None, None]
    assert rel.max() < 0.01
    for k in range(1, nz):
        assert np.array_equal(b[:, :, k], b[:, :, 0])


def _proj2d(x, ang, occ=None):
    from vamtoolbox_b200 import geometry
    from vamtoolbox_b200.projector.Projector2DParallel import Projector2DParallel

    tg = geometry.TargetGeometry(target=x.copy())
    pg = geometry.ProjectionGeometry(ang, "parallel", CUDA=True, occlusion=None if occ is None else occ.copy())
    return Projector2DParallel(tg, pg)


@pytest.mark.parametrize("tag", ["even", "odd", "wrap"])
def test_occlusion_2d_matches_reference_golden(golden, tag):
    """The 2-D class's digitised occlusion on the device: the occlusion sinogram bit for bit (float64
    minima, NaN pattern), the shadowed forward and backprojection within the projector tolerance; "wrap"
    has occluders below the first detector bin at some angles (the reference's shifted bin pairing)."""
    G = golden["occ2d"]
    A = _proj2d(G[f"{tag}_x"], G[f"{tag}_angles"], G[f"{tag}_occ"])
    sino = A.occ_sinogram
    assert np.array_equal(sino, G[f"{tag}_sino"], equal_nan=True)
    assert relL2(A.forward(G[f"{tag}_x"].copy()), G[f"{tag}_fwd"]) < TOL
    assert relL2(A.backward(G[f"{tag}_b"].copy()), G[f"{tag}_bwd"]) < TOL
    if tag != "wrap":
        assert relL2(A.backward(G[f"{tag}_b"].copy(), clipping=False), G[f"{tag}_bwd_noclip"]) < TOL


def test_occlusion_2d_raises_where_the_reference_raises(golden):
    G = golden["occ2d"]
    with pytest.raises(ValueError, match="shape mismatch"):
        _proj2d(G["clash_x"], G["clash_angles"], G["clash_occ"])
    with pytest.raises(ValueError, match="zero-size array"):
        _proj2d(G["even_x"], G["even_angles"], np.zeros_like(G["even_occ"]))


def test_occlusion_2d_adjoint_is_transpose(golden):
    G = golden["occ2d"]
    n, ang = G["wrap_x"].shape[0], G["wrap_angles"]
    p = plan_for((n, n, 1), ang)
    p.set_occlusion_2d(G["wrap_occ"])
    rng = np.random.default_rng(6)
    x, y = rng.standard_normal((n, n, 1)), rng.standard_normal((n, ang.size, 1))
    lhs = float((p.forward(dev(x)).double() * dev(y).double()).sum())
    rhs = float((dev(x).double() * p.adjoint(dev(y)).double()).sum())
    assert abs(lhs - rhs) <= 1e-5 * abs(lhs)


@pytest.mark.parametrize("n", [40, 363])
def test_backward_without_clipping_matches_oracle(n):
    """backward(b, clipping=False) of the 2-D class without occlusion: every pixel, inside the circle or
    not, against the oracle's unclipped np.interp backprojection."""
    rng = np.random.default_rng(n)
    ang = np.linspace(0, 360, 90, endpoint=False) + 0.25
    A = _proj2d(rng.uniform(size=(n, n)), ang)
    b = rng.uniform(size=(n, ang.size))
    got = A.backward(b.copy(), clipping=False)
    ref = O.parallel_backward_2d_occluded(b, ang, np.full((n, ang.size), np.nan), clipping=False)
    assert relL2(got, ref) < TOL
    assert np.abs(got[~O.circle_mask((n, n))]).max() > 0  # pixels outside the circle are not clipped
    assert relL2(A.backward(b.copy()), O.clip_to_circle(ref)) < TOL


def test_released_plan_is_reused_reset():
    """A plan whose ParallelPlan object was released is handed to the next plan of the same geometry with no
    absorption, no occlusion and the default launch shapes; its results equal a fresh plan's."""
    import gc

    from vamtoolbox_b200.projector import Projector3DParallel as P3

    P3.clear_plan_pool()
    shape, ang = (40, 40, 64), np.linspace(0, 360, 24, endpoint=False)
    rng = np.random.default_rng(12)
    x, b = rng.uniform(size=shape), rng.uniform(size=(40, 24, 64))
    p = plan_for(shape, ang)
    ref_fwd, ref_bwd = p.forward(dev(x)).cpu().numpy(), p.backward_ref(dev(b)).cpu().numpy()
    first = p.handle.value
    p.set_absorption("ray", alpha_per_px=0.05, radius_px=15.0)
    p.set_occlusion(np.zeros(shape))
    p.set_tuning({"forward_vz": 1, "backward_table": 0})
    del p
    gc.collect()
    q = plan_for(shape, ang)
    assert q.handle.value == first
    assert q.get_tuning() == P3._DEFAULT_TUNING
    assert np.array_equal(q.forward(dev(x)).cpu().numpy(), ref_fwd)
    assert np.array_equal(q.backward_ref(dev(b)).cpu().numpy(), ref_bwd)
    other = plan_for((40, 40, 64), ang + 1.0)  # different angles: a new plan
    assert other.handle.value != first
    q.close()
    P3.clear_plan_pool()


@pytest.mark.parametrize("ny,nx,na", [(256, 256, 90), (384, 384, 45), (363, 363, 60), (258, 258, 37)])
@pytest.mark.parametrize("mode", ["none", "mask", "ray"])
def test_tma_staged_slice_forward_matches_plain_loads_and_oracle(ny, nx, na, mode):
    """The 2-D tile forward stages its footprint boxes with TMA tensor copies; an image whose rows are not a
    multiple of 16 bytes, one at an address off a 16-byte boundary, and a masked image are first copied into
    the plan's padded image.  Every route gives the plain-load staging's sums bit for bit, those are the
    oracle's, and the plan records no timeout."""
    rng = np.random.default_rng(ny * nx)
    ang = np.linspace(0, 360, na, endpoint=False) + 0.4
    x = rng.uniform(0, 1, (ny, nx, 1))
    p = plan_for((ny, nx, 1), ang)
    oabs = None
    if mode == "mask":
        m = rng.uniform(0.2, 1.0, (ny, nx))
        p.set_absorption("mask", mask=m)
        oabs = ("mask", m)
    elif mode == "ray":
        p.set_absorption("ray", alpha_per_px=0.01, radius_px=min(nx, ny) / 2.0)
        oabs = ("ray", 0.01, min(nx, ny) / 2.0)
    aligned = dev(x)
    buf = torch.zeros(ny * nx + 1, device="cuda")
    buf[1:] = aligned.reshape(-1)
    misaligned = buf[1:].reshape(ny, nx, 1)  # 4 bytes past a 16-byte boundary
    assert aligned.data_ptr() % 16 == 0 and misaligned.data_ptr() % 16 == 4
    a = p.forward(aligned).cpu().numpy()
    b = p.forward(misaligned).cpu().numpy()
    p.set_tuning({"forward_tma": 0})
    c = p.forward(aligned).cpu().numpy()
    d = p.forward(misaligned).cpu().numpy()
    assert np.array_equal(a, b) and np.array_equal(a, c) and np.array_equal(a, d)
    assert relL2(a, O.parallel_forward(x, ang, absorption=oabs)) < TOL
    assert p.status() == 0


@pytest.mark.parametrize("shape,na,mode", [((64, 64, 256), 90, None), ((63, 63, 128), 47, "mask"),
                                           ((40, 40, 512), 33, None), ((34, 34, 64), 40, None),
                                           ((37, 37, 200), 25, "mask"), ((30, 30, 12), 19, None)])
def test_backprojection_table_bitwise_and_oracle(shape, na, mode):
    """The backprojection from the plan's 2 x 2 block bin table, with four and with eight slices per lane,
    gives the computed-bin kernel's sums bit for bit, and the oracle's within float32 tolerance: odd widths
    (partial blocks and tiles), several z chunks and partial ones (nZ not a multiple of 128 or 256), angle
    counts that are not multiples of 32 (partial entry chunks), mask absorption."""
    rng = np.random.default_rng(sum(shape) + na)
    ang = np.linspace(0, 360, na, endpoint=False) + 0.7
    p = plan_for(shape, ang)
    oabs = None
    if mode == "mask":
        m = rng.uniform(0.2, 1.0, shape[:2])
        p.set_absorption("mask", mask=m)
        oabs = ("mask", m)
    b = rng.uniform(0, 1, (shape[0], na, shape[2]))
    p.set_tuning({"backward_vz": 8, "backward_table": 0})
    computed = p.backward_ref(dev(b))
    assert p.prepare_backward()
    for vz in (4, 8):
        p.set_tuning({"backward_table": 1, "backward_vz": vz})
        tabled = p.backward_ref(dev(b))
        assert torch.equal(computed, tabled), vz
    assert relL2(tabled.cpu().numpy(), O.parallel_backward_ref(b, ang, absorption=oabs)) < TOL
    assert p.status() == 0


@pytest.mark.parametrize("shape,na,absn,vz", [((33, 33, 192), 29, None, 6), ((24, 24, 384), 36, "ray", 6),
                                              ((30, 30, 192), 40, "mask", 6), ((28, 28, 160), 31, None, 5),
                                              ((26, 26, 320), 24, "mask", 5), ((22, 22, 160), 30, "ray", 5)])
def test_six_slice_lanes_bitwise(shape, na, absn, vz):
    """Six / five slices per lane (a float4 and a float2 / a float per lane: 192- / 160-slice chunks fill
    every lane where 256-slice ones would not) give the eight-slice kernels' sums bit for bit: the forward
    (paired and unpaired angles, per-ray and mask absorption) and the block-table backprojection, and the
    oracle's."""
    rng = np.random.default_rng(sum(shape) + na)
    ang = np.linspace(0, 360, na, endpoint=False) + 0.9
    x = rng.uniform(0, 1, shape)
    b = rng.uniform(0, 1, (shape[0], na, shape[2]))
    p = plan_for(shape, ang)
    oabs = None
    if absn == "ray":
        p.set_absorption("ray", alpha_per_px=0.04, radius_px=shape[0] / 2 - 1.0)
        oabs = ("ray", 0.04, shape[0] / 2 - 1.0)
    elif absn == "mask":
        m = rng.uniform(0.2, 1.0, shape[:2])
        p.set_absorption("mask", mask=m)
        oabs = ("mask", m)
    p.set_tuning({"forward_vz": 8})
    f8 = p.forward(dev(x))
    p.set_tuning({"forward_vz": vz})
    f6 = p.forward(dev(x))
    p.set_tuning({"forward_vz": 0})
    f0 = p.forward(dev(x))
    assert torch.equal(f6, f8) and torch.equal(f0, f8)
    assert relL2(f6.cpu().numpy(), O.parallel_forward(x, ang, absorption=oabs)) < TOL
    if absn != "ray":
        p.set_tuning({"backward_vz": 8, "backward_table": 0})
        computed = p.backward_ref(dev(b))
        assert p.prepare_backward()
        p.set_tuning({"backward_vz": 0, "backward_table": 1})  # automatic: six / five slices per lane
        assert torch.equal(p.backward_ref(dev(b)), computed)
    assert p.status() == 0


@pytest.mark.parametrize("n,nz", [(5, 9), (12, 16), (17, 5), (24, 64), (33, 17), (31, 65), (20, 128), (21, 130),
                                  (26, 132), (16, 256), (15, 261), (41, 12), (64, 33)])
@pytest.mark.parametrize("absn", [None, "mask", "ray"])
def test_forward_strips_at_their_edges(n, nz, absn):
    """The strip forward against the oracle and the generic kernel: strips past the last detector bin, slice
    counts around the lanes of one chunk (float4 rows and single slices), paired and unpaired angles, rays along
    rows, columns and diagonals.  A strip sums batches of at most 32 pixels and then the batches, at most
    32 + 2.3 n / 25 additions of 2^-24 each: 2.3e-6 at the sizes here.  An infinity and a NaN reach exactly the
    bins that sample their pixels."""
    rng = np.random.default_rng(n * nz)
    ang = np.array([0.0, 30.0, 45.0, 62.5, 90.0, 133.3, 180.0, 210.0, 242.5, 270.0, 301.0])
    x = rng.uniform(-0.2, 1, (n, n, nz))
    p = plan_for(x.shape, ang)
    oabs = None
    if absn == "mask":
        m = rng.uniform(0.2, 1.0, (n, n))
        p.set_absorption("mask", mask=m)
        oabs = ("mask", m)
    elif absn == "ray":
        p.set_absorption("ray", alpha_per_px=0.03, radius_px=n / 2 - 1.5)
        oabs = ("ray", 0.03, n / 2 - 1.5)
    ref = O.parallel_forward(x, ang, absorption=oabs)
    got = p.forward(dev(x)).cpu().numpy()
    assert np.abs(got - ref).max() <= 2.3e-6 * O.parallel_forward(np.abs(x), ang, absorption=oabs).max()
    if n < 8:
        return
    xi = x.copy()
    xi[n // 2, n // 3, nz // 2], xi[n // 3, n // 2, 0] = np.inf, np.nan
    skew = np.delete(ang, [0, 4, 6, 9])  # (a tap of weight 1e-17 on an axis is read or not by rounding)
    q = plan_for(x.shape, skew)
    if absn == "mask":
        q.set_absorption("mask", mask=m)
    elif absn == "ray":
        q.set_absorption("ray", alpha_per_px=0.03, radius_px=n / 2 - 1.5)
    strip = q.forward(dev(xi)).cpu().numpy()
    q.set_tuning({"forward_vz": 1})
    plain = q.forward(dev(xi)).cpu().numpy()
    # an angle's partner 180 degrees away is sampled from the same lattice, mirrored (the generic kernel forms
    # its coordinates anew, and a weight of one rounding more or less than zero decides about an infinity)
    mirror = plain.copy()
    rows = np.arange(2 * (n // 2) - n + 1, n)
    for a, b in ((0, 4), (2, 5)) if absn != "ray" else ():  # 30 and 210, 62.5 and 242.5 (unpaired with "ray")
        mirror[2 * (n // 2) - rows, b] = plain[rows, a]
    assert np.array_equal(np.isnan(strip), np.isnan(mirror)) and np.array_equal(np.isinf(strip), np.isinf(mirror))
    ok = np.isfinite(plain) & np.isfinite(mirror)
    assert not ok.all() and np.abs(strip[ok] - plain[ok]).max() <= 4.6e-6 * np.abs(plain[ok]).max()


@pytest.mark.parametrize("n,nz", [(9, 9), (12, 16), (17, 5), (24, 64), (33, 17), (31, 65), (20, 128), (21, 130),
                                  (26, 132), (16, 256), (15, 261), (40, 70)])
@pytest.mark.parametrize("absn", [None, "mask", "ray"])
def test_transpose_blocks_and_padded_rows_at_their_edges(n, nz, absn):
    """The block kernel of the matched transpose against the oracle: blocks past the image's edge, slice counts
    around the lanes of one chunk, angle counts around its batches of six.  A pixel sums at most 2.6 rows per
    angle: 2.6 * 13 additions of 2^-24 each, 2.1e-6.  A slice count that is not a multiple of four is padded to
    one: forward and transpose equal the same kernels on the unpadded rows bit for bit, the backprojection from
    its bin table the oracle's.  An infinity reaches exactly the pixels its row touches."""
    from vamtoolbox_b200 import _lib

    rng = np.random.default_rng(n * nz + 1)
    ang = np.array([0.0, 17.3, 45.0, 62.5, 90.0, 133.3, 180.0, 197.3, 222.2, 242.5, 270.0, 301.0, 333.3])
    p = plan_for((n, n, nz), ang)
    p.pad_from = p.pad_backward_from = 0  # (from any size on)
    oabs = None
    if absn == "mask":
        m = rng.uniform(0.2, 1.0, (n, n))
        p.set_absorption("mask", mask=m)
        oabs = ("mask", m)
    elif absn == "ray":
        p.set_absorption("ray", alpha_per_px=0.03, radius_px=n / 2 - 1.5)
        oabs = ("ray", 0.03, n / 2 - 1.5)
    x, b = rng.uniform(-0.2, 1, (n, n, nz)), rng.uniform(-0.2, 1, (n, ang.size, nz))
    got = p.adjoint(dev(b))
    scale = O.parallel_adjoint(np.abs(b), ang, absorption=oabs).max()
    assert np.abs(got.cpu().numpy() - O.parallel_adjoint(b, ang, absorption=oabs)).max() <= 2.1e-6 * scale
    if nz % 4:
        assert p._pads(_lib.OP_FORWARD) and p._pads(_lib.OP_ADJOINT)
        for op, src, name in (("forward", dev(x), "vam_parallel_forward"), ("adjoint", dev(b), "vam_parallel_adjoint")):
            padded = getattr(p, op)(src)
            plain = torch.empty_like(padded)
            _lib.call(name, p.handle, _lib.ptr(src), _lib.ptr(plain), p._stream())
            assert torch.equal(padded, plain)
        back = p.backward_ref(dev(b)).cpu().numpy()
        assert relL2(back, O.parallel_backward_ref(b, ang, absorption=oabs)) < TOL
    bi = b.copy()
    bi[n // 2, 3, nz // 2] = np.inf  # angle 62.5 degrees
    inf = torch.isinf(p.adjoint(dev(bi))).cpu().numpy()
    touched = np.zeros((n, ang.size, nz))
    touched[n // 2, 3, nz // 2] = 1.0
    assert np.array_equal(inf, O.parallel_adjoint(touched, ang, absorption=oabs) > 1e-6)


@pytest.mark.parametrize("n", [31, 32, 33, 64, 65, 100])
@pytest.mark.parametrize("na", [1, 63, 64, 70])
def test_slice_backprojection_tiles_at_their_edges(n, na):
    """The 2-D backprojection tiles (32 x 8 pixels, 64 staged angles, four groups of angles): partial tiles and
    angle blocks, rays along the axes (coordinates on integers and at the detector's ends), against the oracle.
    A weight is good to 2^-23 and a group adds at most 18 terms, together below 20 2^-24 of the largest sum:
    1.2e-6.  An infinity reaches the pixels the generic kernel's does."""
    rng = np.random.default_rng(n + na)
    ang = np.concatenate([[0.0, 90.0, 180.0, 270.0, 45.0], rng.uniform(0, 360, 70)])[:na] if na > 1 else np.array([33.3])
    p = plan_for((n, n, 1), ang)
    p.set_tuning({"backward_vz": 4})
    b = rng.uniform(-0.2, 1, (n, ang.size, 1))
    ref = O.parallel_backward_ref(b, ang)
    got = p.backward_ref(dev(b)).cpu().numpy()
    assert np.abs(got - ref).max() <= 1.2e-6 * np.abs(O.parallel_backward_ref(np.abs(b), ang)).max()
    b[n // 2, ang.size - 1, 0] = np.inf
    got = p.backward_ref(dev(b))
    p.set_tuning({"backward_vz": 1})
    assert torch.equal(torch.isinf(got), torch.isinf(p.backward_ref(dev(b))))


@pytest.mark.parametrize("n", [31, 62, 63, 64, 65, 127, 128])
@pytest.mark.parametrize("absn", [None, "mask", "ray"])
def test_slice_forward_tiles_with_paired_angles_at_their_edges(n, absn):
    """The 2-D forward tiles sum an angle and the one 180 degrees from it from one lattice: lattice rows and
    samples at the ends of a tile of 64 (row N alone in its tile for n = 64 and 128), odd and even sizes, paired
    and unpaired angles, rays along the axes, both stagings.  A weight is good to 4e-5 (coordinates within 2e-5
    pixel) in a mean of n samples, which with the additions stays below 1e-4 of the largest sum; a wrong or
    missing sample is 1 / n of a bin."""
    rng = np.random.default_rng(n)
    ang = np.array([0.0, 33.0, 90.0, 180.0, 213.0, 270.0, 45.0, 77.7, 257.7])
    x = rng.uniform(0.5, 1, (n, n, 1))
    p = plan_for((n, n, 1), ang)
    oabs = None
    if absn == "mask":
        oabs = ("mask", rng.uniform(0.2, 1.0, (n, n)))
        p.set_absorption("mask", mask=oabs[1])
    elif absn == "ray":
        oabs = ("ray", 0.01, n / 2.0)
        p.set_absorption("ray", alpha_per_px=0.01, radius_px=n / 2.0)
    p.set_tuning({"forward_vz": 4})
    got = p.forward(dev(x)).cpu().numpy()
    ref = O.parallel_forward(x, ang, absorption=oabs)
    assert np.abs(got - ref).max() <= 1e-4 * ref.max()
    p.set_tuning({"forward_tma": 0})
    assert np.array_equal(p.forward(dev(x)).cpu().numpy(), got)


@pytest.mark.parametrize("n", [63, 64])
@pytest.mark.parametrize("absn", [None, "ray"])
def test_slice_forward_tiles_spread_no_infinity(n, absn):
    """An infinite pixel reaches the bins of the 2-D forward tiles that it reaches in the generic kernel: those it
    has a weight for, not those whose zero weight it would turn into NaN (angles off the axes, where the pixel is
    on no sample's edge to rounding, and 0 and 90 degrees, whose samples are pixels)."""
    ang = np.array([0.0, 17.3, 90.0, 197.3, 61.9])
    x = np.random.default_rng(n).uniform(0.5, 1, (n, n, 1))
    x[n // 3, n // 2, 0] = np.inf
    p = plan_for((n, n, 1), ang)
    if absn == "ray":
        p.set_absorption("ray", alpha_per_px=0.01, radius_px=n / 2.0)
    p.set_tuning({"forward_vz": 4})
    got = p.forward(dev(x))
    p.set_tuning({"forward_vz": 1})
    ref = p.forward(dev(x))
    assert torch.equal(torch.isinf(got), torch.isinf(ref)) and torch.equal(torch.isnan(got), torch.isnan(ref))
    assert 0 < int(torch.isinf(got).sum()) < 20


@pytest.mark.parametrize("n,nz", [(40, 33), (33, 66), (24, 130), (21, 165)])
@pytest.mark.parametrize("absn", [None, "mask", "ray"])
def test_padded_backprojection_under_every_tuning(n, nz, absn):
    """A slice count that is not a multiple of four under every backprojection tuning, direct and in a batch, against
    the oracle: a pixel adds at most 2 values per angle, 26 roundings of 2^-24 of the largest sum, 1.6e-6; guard
    values around the output stay as they were."""
    from vamtoolbox_b200.batch import ProjectionBatch

    rng = np.random.default_rng(n * nz + 2)
    ang = np.array([0.0, 17.3, 45.0, 62.5, 90.0, 133.3, 180.0, 197.3, 222.2, 242.5, 270.0, 301.0, 333.3])
    p = plan_for((n, n, nz), ang)
    p.pad_from = p.pad_backward_from = 0  # (from any size on)
    oabs = None
    if absn == "mask":
        oabs = ("mask", rng.uniform(0.2, 1.0, (n, n)))
        p.set_absorption("mask", mask=oabs[1])
    elif absn == "ray":
        oabs = ("ray", 0.03, n / 2 - 1.5)
        p.set_absorption("ray", alpha_per_px=0.03, radius_px=n / 2 - 1.5)
    b = rng.uniform(0, 1, (n, ang.size, nz))
    ref = O.parallel_backward_ref(b, ang, absorption=oabs)
    bound = 1.6e-6 * ref.max()
    if nz >= 64:
        p._prepare_padded()
    bd, guard = dev(b), torch.full((n * n * nz + 64,), -3.0, device="cuda")
    out = guard[32:32 + n * n * nz].view(n, n, nz)
    batch = ProjectionBatch()
    for vz in (0, 1, 4, 8):
        for nb, table in ((1, 0), (2, 0), (4, 0), (2, 1)):
            p.set_tuning({"backward_vz": vz, "backward_batch": nb, "backward_table": table})
            direct = p.backward_ref(bd)
            assert np.abs(direct.cpu().numpy() - ref).max() <= bound, (vz, nb, table)
            batch.submit([(p, "backward_ref", bd, out)])
            assert torch.equal(out, direct), (vz, nb, table)
            assert bool((guard[:32] == -3).all()) and bool((guard[-32:] == -3).all()), (vz, nb, table)


def test_autotune_of_a_padded_slice_count(tmp_path, monkeypatch):
    """Autotuning a plan whose slice count is not a multiple of four times every candidate and leaves the results
    the oracle's (two roundings for each of 30 angles)."""
    monkeypatch.setenv("VAMTOOLBOX_B200_TUNE_CACHE", str(tmp_path / "tune.json"))
    rng = np.random.default_rng(4)
    ang = np.linspace(0, 360, 30, endpoint=False) + 0.3
    p = plan_for((48, 48, 67), ang)
    p.pad_from = p.pad_backward_from = 0
    p._prepare_padded()
    p.autotune()
    x, b = rng.uniform(0, 1, p.shape_vol), rng.uniform(0, 1, p.shape_sino)
    ref = O.parallel_backward_ref(b, ang)
    assert np.abs(p.backward_ref(dev(b)).cpu().numpy() - ref).max() <= 60 * 2.0 ** -24 * ref.max()
    assert relL2(p.forward(dev(x)).cpu().numpy(), O.parallel_forward(x, ang)) < TOL
    assert relL2(p.adjoint(dev(b)).cpu().numpy(), O.parallel_adjoint(b, ang)) < TOL


@pytest.mark.parametrize("n,nz", [(24, 65), (33, 67), (40, 117), (21, 130), (31, 165), (26, 201), (17, 261)])
@pytest.mark.parametrize("absn", [None, "mask"])
def test_padded_table_backprojection_is_as_exact_as_the_generic_kernel(n, nz, absn):
    """Padded rows summed from the bin table against the generic kernel, whose lanes share a pixel's angles: bins on
    integers, the detector's ends (angles on the axes), every slice of the last chunk.  A run adds at most 16 values, each
    interpolated with three roundings, and the sum of the runs and the mask's product round once: 21 2^-24 of the
    sum of the magnitudes.  The error's norm is no larger than the generic kernel's but for the last rounding of
    either (2^-25.5 in the mean).  An infinity and a NaN reach the pixels they reach there (an infinite lower row
    gives an infinity as in np.interp, where the generic kernel's r0 + w (r1 - r0) gives a NaN)."""
    from vamtoolbox_b200 import _lib

    rng = np.random.default_rng(n * nz + 3)
    ang = np.concatenate([np.array([0.0, 45.0, 90.0, 180.0, 270.0, 359.9]), rng.uniform(0, 360, 33)])
    p = plan_for((n, n, nz), ang)
    p.pad_backward_from = 0
    p._prepare_padded()
    assert p.has_backward_table and p._pads(_lib.OP_BACKWARD_REF)
    oabs = None
    if absn == "mask":
        oabs = ("mask", rng.uniform(0.2, 1.0, (n, n)).astype(np.float32).astype(np.float64))
        p.set_absorption("mask", mask=oabs[1])
    b = rng.uniform(-0.3, 1, (n, ang.size, nz)).astype(np.float32)
    bi = b.copy()
    bi[n // 2, 0, nz // 2], bi[n // 3, 7, 0], bi[n - 1, 2, nz - 1], bi[n // 2 + 1, 1, 1] = np.inf, np.nan, np.inf, -np.inf
    ref = O.parallel_backward_ref(b.astype(np.float64), ang, absorption=oabs)
    size = O.parallel_backward_ref(np.abs(b).astype(np.float64), ang, absorption=oabs)

    def generic(src):
        out = torch.empty(p.shape_vol, device="cuda")
        _lib.call("vam_parallel_backward_ref", p.handle, _lib.ptr(src), _lib.ptr(out), p._stream())
        return out

    for vz in (0, 4, 8):
        p.set_tuning({"backward_vz": vz})
        got = p.backward_ref(dev(b)).cpu().numpy()
        assert (np.abs(got - ref) <= 21 * 2.0 ** -24 * size + 1e-30).all(), vz
        assert relL2(got, ref) <= relL2(generic(dev(b)).cpu().numpy(), ref) + 2.0 ** -25.5, vz
        assert torch.equal(p.backward_ref(dev(bi)).isfinite(), generic(dev(bi)).isfinite()), vz


def test_small_slices_build_no_padded_table():
    """Slices of few pixels with an odd slice count keep the generic kernel (its rows padded), which their few blocks
    do not leave waiting as the bin table's kernel."""
    from vamtoolbox_b200 import _lib

    ang = np.linspace(0, 360, 90, endpoint=False)
    small, large = plan_for((32, 32, 67), ang), plan_for((96, 96, 101), ang)
    assert not small.has_backward_table and small._pads(_lib.OP_BACKWARD_REF)
    assert large.has_backward_table and large._pads(_lib.OP_BACKWARD_REF)
    assert not plan_for((40, 40, 117), ang)._pads(_lib.OP_BACKWARD_REF)


@pytest.mark.parametrize("nz", [12, 33, 36, 40, 48, 65, 71])
@pytest.mark.parametrize("absn", [None, "mask", "ray"])
def test_strips_and_blocks_as_exact_as_the_generic_kernels(nz, absn):
    """Slice counts of which the generic kernels share a bin's samples, or a pixel's angles, among many lanes: the
    strips' and blocks' sums are as exact.  The error's norm relative to float64 exceeds the generic kernel's by less
    than a sixth of the last rounding (2^-27; a result's own rounding is 2^-25 / sqrt 3 in the mean)."""
    rng = np.random.default_rng(nz)
    n, ang = 64, np.linspace(0, 360, 90, endpoint=False)
    p = plan_for((n, n, nz), ang)
    oabs = None
    if absn == "mask":
        oabs = ("mask", rng.uniform(0.2, 1.0, (n, n)).astype(np.float32).astype(np.float64))
        p.set_absorption("mask", mask=oabs[1])
    elif absn == "ray":
        oabs = ("ray", 0.03, n / 2.0)
        p.set_absorption("ray", alpha_per_px=0.03, radius_px=n / 2.0)
    x, b = rng.uniform(-0.2, 1, p.shape_vol).astype(np.float32), rng.uniform(-0.2, 1, p.shape_sino).astype(np.float32)
    rf = O.parallel_forward(x.astype(np.float64), ang, absorption=oabs)
    ra = O.parallel_adjoint(b.astype(np.float64), ang, absorption=oabs)
    err = []
    for vz in (4, 1):
        p.set_tuning({"forward_vz": vz, "adjoint_vz": vz})
        err.append((relL2(p.forward(dev(x)).cpu().numpy(), rf), relL2(p.adjoint(dev(b)).cpu().numpy(), ra)))
    assert err[0][0] <= err[1][0] + 2.0 ** -27 and err[0][1] <= err[1][1] + 2.0 ** -27, err


@pytest.mark.parametrize("n", [112, 128, 160, 192, 256])
@pytest.mark.parametrize("absn", [None, "mask", "ray"])
def test_slice_tiles_as_exact_as_the_generic_kernels(n, absn):
    """The tiles' sums of a slice: the error's norm relative to float64 exceeds the generic kernels', whose 32 lanes
    share a bin's samples or a pixel's angles, by less than a sixth of the last rounding (2^-27)."""
    rng = np.random.default_rng(n)
    ang = np.linspace(0, 360, 240, endpoint=False)
    p = plan_for((n, n, 1), ang)
    oabs = None
    if absn == "mask":
        oabs = ("mask", rng.uniform(0.2, 1.0, (n, n)).astype(np.float32).astype(np.float64))
        p.set_absorption("mask", mask=oabs[1])
    elif absn == "ray":
        oabs = ("ray", 0.01, n / 2.0)
        p.set_absorption("ray", alpha_per_px=0.01, radius_px=n / 2.0)
    x, b = rng.uniform(-0.2, 1, p.shape_vol).astype(np.float32), rng.uniform(-0.2, 1, p.shape_sino).astype(np.float32)
    rf = O.parallel_forward(x.astype(np.float64), ang, absorption=oabs)
    rb = O.parallel_backward_ref(b.astype(np.float64), ang, absorption=oabs)
    err = []
    for vz in (4, 1):
        p.set_tuning({"forward_vz": vz, "backward_vz": 0 if absn == "ray" else vz})
        err.append((relL2(p.forward(dev(x)).cpu().numpy(), rf), relL2(p.backward_ref(dev(b)).cpu().numpy(), rb)))
    assert err[0][0] <= err[1][0] + 2.0 ** -27 and err[0][1] <= err[1][1] + 2.0 ** -27, err


@pytest.mark.parametrize("n,deg,bound", [(2048, 111.7, 11 * 2.0 ** -26), (4090, 328.5, 3 * 2.0 ** -25)])
def test_slice_backprojection_weights_of_wide_slices(n, deg, bound):
    """One angle's backprojection of alternating -1 and 1: a weight w gives 1 - 2 w, so its error is seen twice, and
    one rounding of the result adds 2^-25.  Up to 2048 pixels a weight carries its rounding (2^-25), that of the
    fraction (2^-26) and three of the low part (2^-27 each): twice 9 2^-27 and 2^-25, 11 2^-26.  Above it is formed in
    float64 and rounded once."""
    p = plan_for((n, n, 1), np.array([deg]))
    b = np.where(np.arange(n) % 2, 1.0, -1.0)
    got = p.backward_ref(dev(b.reshape(n, 1, 1))).cpu().numpy()[:, :, 0].astype(np.float64)
    r, C = deg * (np.pi / 180.0), n // 2
    t = (np.arange(n) - C)[None, :] * np.cos(r) - (np.arange(n) - C)[:, None] * np.sin(r)
    j, w = np.floor(t).astype(int) + C, t - np.floor(t)
    lin = np.linspace(-1, 1, n)
    inside = (lin[:, None] ** 2 + lin[None, :] ** 2 <= 1) & (j >= 0) & (j < n - 1)
    ref = np.where(inside, (1 - w) * b[j.clip(0, n - 1)] + w * b[(j + 1).clip(0, n - 1)], 0.0)
    safe = inside & (w > 1e-9) & (w < 1 - 1e-9)
    assert np.abs(got - ref)[safe].max() <= bound


@pytest.mark.parametrize("nz", [5, 13, 25, 26, 27, 53, 55, 109, 111])
@pytest.mark.parametrize("absn", [None, "mask", "ray"])
def test_padded_generic_backprojection_shares_angles_as_before(nz, absn):
    """The generic kernel on padded rows spreads a pixel's angles over as many lanes as on unpadded ones: where the
    float4s of a row would take twice the lanes, the results are the unpadded call's bits."""
    from vamtoolbox_b200 import _lib

    rng = np.random.default_rng(nz)
    p = plan_for((50, 50, nz), np.linspace(0, 360, 45, endpoint=False))
    p.pad_backward_from = 0
    assert p._pads(_lib.OP_BACKWARD_REF) and not p.has_backward_table
    if absn == "mask":
        p.set_absorption("mask", mask=rng.uniform(0.2, 1.0, (50, 50)))
    elif absn == "ray":
        p.set_absorption("ray", alpha_per_px=0.03, radius_px=23.5)
    b, plain = dev(rng.uniform(-0.2, 1, p.shape_sino)), torch.empty(p.shape_vol, device="cuda")
    _lib.call("vam_parallel_backward_ref", p.handle, _lib.ptr(b), _lib.ptr(plain), p._stream())
    assert torch.equal(p.backward_ref(b), plain)


@pytest.mark.parametrize("n,nz,na", [(48, 36, 61), (64, 9, 120), (64, 20, 90), (64, 40, 90), (40, 57, 60), (50, 63, 100),
                                     (96, 33, 60), (96, 16, 90)])
@pytest.mark.parametrize("value", [1.0, 0.3337])
def test_strips_as_exact_as_the_generic_kernel_on_solid_parts(n, nz, na, value):
    """Inside a solid part every sample is the part's value, which the generic kernel's few-lane sums add (nearly)
    without rounding.  The strips' sums carry what their rounding drops to the end, so their error's norm is no larger
    there either."""
    ang = np.linspace(0, 360, na, endpoint=False)
    p = plan_for((n, n, nz), ang)
    i, j, k = np.ogrid[:n, :n, :nz]
    r = np.hypot(i - n / 2.0 + 0.5, j - n / 2.0 + 0.5)
    x = np.where((r < 0.42 * n) & (r > 0.1 * n + 0.1 * k * n / nz), np.float32(value), np.float32(0))
    ref = O.parallel_forward(x.astype(np.float64), ang)
    err = []
    for vz in (4, 1):
        p.set_tuning({"forward_vz": vz})
        err.append(relL2(p.forward(dev(x)).cpu().numpy(), ref))
    assert err[0] <= err[1], err

"""Kernels and dispatch at the sizes where their tilings end: image tiles, line padding, layout
copies, footprint columns and splat lattices, against the oracle."""
import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu

# float32 sums of a few hundred terms in another order than the oracle's, the parity bound of the
# projectors
PARITY = 1e-5


def _apply(torch, proj, data, adjoint):
    d = torch.from_numpy(np.ascontiguousarray(data, np.float32).ravel()).cuda()
    out = torch.full((proj.domain_size if adjoint else proj.range_size,), float("nan"),
                     device="cuda")
    s = torch.cuda.current_stream().cuda_stream
    (proj.apply_adjoint_ptr if adjoint else proj.apply_ptr)(d.data_ptr(), out.data_ptr(), s)
    torch.cuda.synchronize()
    return out.cpu().numpy()


def _fill_memory(torch, leave):
    """Tensors that leave `leave` bytes (to 16 MiB) of the device's memory free."""
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    full = []
    for piece in (1 << 30, 1 << 26, 1 << 24):
        while torch.cuda.mem_get_info()[0] > leave + piece:
            full.append(torch.empty(piece, dtype=torch.uint8, device="cuda"))
    return full


def _problem(oracle, vol, views, det, arc=360, seed=3):
    n = max(vol)
    poses, det = oracle.circle_trajectory(vol, views, arc, 5.0 * n, 1.5 * n, det)
    rng = np.random.default_rng(seed)
    x = rng.uniform(0, 1, int(np.prod(vol))).astype(np.float32)
    y = rng.uniform(0, 1, int(np.prod(det))).astype(np.float32)
    return poses, det, x, y


@pytest.mark.parametrize("vol,views,det", [
    ((1, 1), 3, [3]), ((31, 33), 5, [31]), ((32, 32), 7, [33]), ((65, 40), 9, [64]),
    ((127, 1), 4, [140]), ((256, 257), 6, [321]), ((300, 290), 11, [401]), ((1, 70), 8, [97]),
    ((128, 128), 73, [182]), ((128, 128), 74, [182]), ((33, 31), 1200, [45])])
def test_joseph_2d_tiles(cuda, oracle, vol, views, det):
    """Tiles of 32 and 64 pixels, remainders, one-pixel edges, from the image and from its padded
    lines; views around 45 degrees mix both driving axes."""
    import elsa_b200
    poses, det, x, y = _problem(oracle, vol, views, det)
    proj = elsa_b200.Projector(elsa_b200.PROJECTOR_JOSEPH, vol, det, poses)
    for threads in (64, 256, 512):
        proj.set_knob(elsa_b200.KNOB_FORWARD_THREADS, threads)
        assert rel_l2(_apply(cuda, proj, x, False), oracle.joseph(x, vol, det, poses)) <= PARITY
    ref = oracle.joseph_adjoint(y, vol, det, poses)
    first = _apply(cuda, proj, y, True)
    assert rel_l2(first, ref) <= PARITY
    assert np.array_equal(first, _apply(cuda, proj, y, True))
    proj.set_knob(elsa_b200.KNOB_ADJOINT_CHUNKS, 1)
    assert rel_l2(_apply(cuda, proj, y, True), ref) <= PARITY


@pytest.mark.parametrize("vol,views,det", [((40, 37), 6, [50]), ((140, 137), 9, [200]),
                                           ((100, 60), 210, [150])])
def test_joseph_2d_non_finite(cuda, oracle, vol, views, det):
    """An infinity reaches exactly the pixels whose rays meet it, as in the oracle, from the image
    and from its padded lines."""
    import elsa_b200
    poses, det, x, _ = _problem(oracle, vol, views, det)
    x[20 + vol[0] * 11] = np.inf
    proj = elsa_b200.Projector(elsa_b200.PROJECTOR_JOSEPH, vol, det, poses)
    got = _apply(cuda, proj, x, False)
    ref = np.asarray(oracle.joseph(x, vol, det, poses))
    assert np.array_equal(np.isfinite(got), np.isfinite(ref))
    assert np.array_equal(np.isinf(got), np.isinf(ref))


@pytest.mark.parametrize("kind", ["SIDDON", "BINARY"])
@pytest.mark.parametrize("vol,views,det", [
    ((1, 1, 1), 3, [3, 3]), ((33, 31, 35), 7, [40, 33]), ((64, 5, 32), 8, [70, 9]),
    ((1, 34, 67), 5, [90, 50]), ((33, 65), 9, [80]), ((1, 40), 6, [60]),
    ((64, 60, 70), 100, [96, 100]), ((131, 40, 37), 120, [140, 60])])
def test_siddon_forward_layouts(cuda, oracle, vol, views, det, kind):
    """Rays read from the volume or, with rays enough, from a copy with another axis contiguous: the
    same visits and sums, bit for bit."""
    import elsa_b200
    poses, det, x, _ = _problem(oracle, vol, views, det)
    proj = elsa_b200.Projector(getattr(elsa_b200, "PROJECTOR_" + kind), vol, det, poses)
    assert proj.info(6) == (2 if views >= 100 else 1)  # launches of a forward
    fn = oracle.siddon if kind == "SIDDON" else oracle.binary
    ref = np.asarray(fn(x, vol, det, poses), np.float32)
    assert np.array_equal(_apply(cuda, proj, x, False), ref)


@pytest.mark.parametrize("kind", ["RAY_BLOB", "RAY_BSPLINE"])
@pytest.mark.parametrize("vol,views,det", [((1, 1, 1), 2, [2, 2]), ((17, 9, 21), 6, [24, 11]),
                                           ((3, 12, 2), 5, [9, 20]), ((33, 5), 7, [40])])
def test_ray_lut_layouts(cuda, oracle, vol, views, det, kind):
    """The forward sums every ray in the reference's order, bit for bit, whatever its leading
    axis; the adjoint's fixed-point sums do not depend on which copy a ray adds to."""
    import elsa_b200
    poses, det, x, y = _problem(oracle, vol, views, det)
    proj = elsa_b200.Projector(getattr(elsa_b200, "PROJECTOR_" + kind), vol, det, poses)
    if kind == "RAY_BLOB":
        lut, radius = oracle.blob_lut(), 2.0
    else:
        lut, radius = oracle.bspline_lut(len(vol), 2), oracle.bspline_support(2)
    ref = np.asarray(oracle.lut_project(False, x, vol, det, poses, lut, radius, 2), np.float32)
    assert np.array_equal(_apply(cuda, proj, x, False), ref)
    ref = oracle.lut_project(True, y, vol, det, poses, lut, radius, 2)
    assert rel_l2(_apply(cuda, proj, y, True), ref) <= PARITY


VOXEL_KINDS = [("blob", (2.0, 10.83, 2)), ("bspline", (3,)), ("phase_blob", (2.0, 10.83, 2)),
               ("phase_bspline", (3,))]
VOXEL_CODES = {"blob": 2, "bspline": 3, "phase_blob": 4, "phase_bspline": 5}


def _voxel_reference(oracle, kind, params, dim):
    if kind.endswith("blob"):
        return oracle.voxel_lut(kind, dim, *params)
    return oracle.voxel_lut(kind, dim, order=params[0])


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("kind,params", [
    ("blob", (2.0, 10.83, 2)), ("blob", (0.55, 10.83, 2)), ("blob", (3.7, 8.0, 1)),
    ("blob", (9.0, 10.83, 2)), ("blob", (1.3, 2.0, 0)), ("bspline", (0,)), ("bspline", (5,)),
    ("phase_blob", (3.1, 10.83, 2)), ("phase_bspline", (3,))])
@pytest.mark.parametrize("vol,views,det", [((13, 21, 9), 7, [17, 12]), ((50, 6, 49), 5, [70, 31]),
                                           ((200, 7), 6, [90]), ((60, 41), 11, [70]),
                                           ((700, 500), 3, [900])])
def test_voxel_footprints(cuda, oracle, vol, views, det, kind, params, mode):
    """Footprints of one pixel to more than six columns, detector patches that do not fit, tables
    that do not end in 0, voxels projected off the detector (the small problems' forward). The
    default adjoint visits exactly the pixels of the exact one: its weights differ by a few ulp
    (an edge pixel more or less would show as 1e-4)."""
    import elsa_b200
    codes = {"blob": 2, "bspline": 3, "phase_blob": 4, "phase_bspline": 5}
    poses, det, x, y = _problem(oracle, vol, views, det)
    x[::3] = 0.0
    proj = elsa_b200.Projector(codes[kind], vol, det, poses, tuple(map(float, params)) + (mode,))
    if kind.endswith("blob"):
        lut, support, wk = oracle.voxel_lut(kind, len(vol), *params)
    else:
        lut, support, wk = oracle.voxel_lut(kind, len(vol), order=params[0])
    args = (vol, det, poses, lut, support, wk, mode)
    ref = oracle.voxel_project(False, x, *args)
    assert rel_l2(_apply(cuda, proj, x, False), ref) <= PARITY
    fast = _apply(cuda, proj, y, True)
    proj.set_knob(elsa_b200.KNOB_EXACT_WEIGHTS, 1)
    exact = _apply(cuda, proj, y, True)
    assert np.array_equal(exact, np.asarray(oracle.voxel_project(True, y, *args), np.float32))
    # phase-contrast sums cancel: weights of both signs, relative to their magnitude
    assert rel_l2(fast, exact) <= (PARITY if kind.startswith("phase") else 2e-6)


# voxels times poses above the small problems', which have a forward of their own
LATTICE = [((50, 60, 49), 41, [70, 61]), ((200, 37), 90, [250]), ((60, 75), 110, [80]),
           ((20, 400), 60, [560])]


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("kind,params", [
    ("blob", (2.0, 10.83, 2)), ("blob", (3.7, 8.0, 1)), ("blob", (0.55, 10.83, 2)),
    ("bspline", (5,)), ("phase_blob", (3.1, 10.83, 2))])
@pytest.mark.parametrize("vol,views,det", LATTICE)
def test_voxel_lattice(cuda, oracle, vol, views, det, kind, params, mode):
    """The forward of larger problems: lattices of several tiles and rows of 32, 16, 8 and 4
    voxels, patches clipped by the detector."""
    import elsa_b200
    poses, det, x, _ = _problem(oracle, vol, views, det)
    x[::3] = 0.0
    proj = elsa_b200.Projector(VOXEL_CODES[kind], vol, det, poses,
                               tuple(map(float, params)) + (mode,))
    ref = oracle.voxel_project(False, x, vol, det, poses,
                               *_voxel_reference(oracle, kind, params, len(vol)), mode)
    for _ in range(2):  # the second one starts from what the first left in its counter
        assert rel_l2(_apply(cuda, proj, x, False), ref) <= PARITY


@pytest.mark.parametrize("kind,params", VOXEL_KINDS)
@pytest.mark.parametrize("offset", [(0.0, 0.0), (40.0, 0.0), (-25.0, 70.0), (400.0, 0.0)])
@pytest.mark.parametrize("s2c,c2d", [(400.0, 100.0), (55.0, 40.0), (-300.0, 800.0), (20.0, 60.0)])
@pytest.mark.parametrize("vol,views,det", [((50, 60, 49), 41, [24, 17]), ((200, 150), 16, [70])])
def test_voxel_lattice_on_a_small_detector(cuda, oracle, vol, views, det, s2c, c2d, offset, kind,
                                           params):
    """Detectors that see a part of the volume or none of it: the ends of the lattice that project
    off them are left out, from near and far sources, behind them and around them."""
    import elsa_b200
    one, origin, sino = [1.0] * len(vol), [0.5 * v for v in vol], [0.5 * d for d in det] + [0.0]
    angles = np.linspace(0.0, 6.0, views)
    if len(vol) == 3:
        poses = [elsa_b200.pose_3d(s2c, c2d, one, origin, one, sino, g, pp_offset=offset)
                 for g in angles]
    else:
        poses = [elsa_b200.pose_2d(s2c, c2d, g, one, origin, one, sino, pp_offset=offset[0])
                 for g in angles]
    poses, det = np.concatenate(poses), det + [views]
    x = np.random.default_rng(6).uniform(0, 1, int(np.prod(vol))).astype(np.float32)
    proj = elsa_b200.Projector(VOXEL_CODES[kind], vol, det, poses,
                               tuple(map(float, params)) + (0,))
    ref = oracle.voxel_project(False, x, vol, det, poses,
                               *_voxel_reference(oracle, kind, params, len(vol)), 0)
    assert rel_l2(_apply(cuda, proj, x, False), ref) <= PARITY


@pytest.mark.parametrize("radius", [6.0, 9.0])
@pytest.mark.parametrize("vol,views,det", LATTICE)
def test_voxel_lattice_of_wide_footprints(cuda, oracle, vol, views, det, radius):
    """Lattices that do not fit their patch or overlap (shared atomics), against the adjoint of the
    same weights: <A x, y> = <x, A^T y>."""
    import elsa_b200
    poses, det, x, y = _problem(oracle, vol, views, det)
    proj = elsa_b200.Projector(elsa_b200.PROJECTOR_BLOB, vol, det, poses, (radius, 10.83, 2.0, 1.0))
    ax = _apply(cuda, proj, x, False).astype(np.float64)
    aty = _apply(cuda, proj, y, True).astype(np.float64)
    assert abs(ax @ y - x @ aty) <= 1e-6 * (ax @ y)


def test_voxel_adjoint_same_footprints_at_size(cuda, oracle):
    """10^8 footprints: one ulp in a centre or a scaling would move the edges of about a thousand
    of them and the sums by 1e-5 and more."""
    import elsa_b200
    vol = (128, 128, 64)
    poses, det = oracle.circle_trajectory(vol, 96, 360, 1280.0, 320.0, [192, 96])
    proj = elsa_b200.Projector(elsa_b200.PROJECTOR_BLOB, vol, det, poses)
    y = np.random.default_rng(1).uniform(0, 1, int(np.prod(det))).astype(np.float32)
    fast = _apply(cuda, proj, y, True)
    proj.set_knob(elsa_b200.KNOB_EXACT_WEIGHTS, 1)
    assert rel_l2(fast, _apply(cuda, proj, y, True)) <= 5e-7


FORWARDS = [("JOSEPH", (300, 280), [401]), ("JOSEPH", (120, 100), [150]),
            ("SIDDON", (60, 50, 70), [90, 80]), ("BLOB", (40, 50, 45), [60, 70]),
            ("RAY_BLOB", (24, 20, 28), [40, 30])]


@pytest.mark.parametrize("kind,vol,det", FORWARDS)
@pytest.mark.parametrize("count", [2, 7])
def test_forwards_on_several_streams(cuda, oracle, kind, vol, det, count):
    """The forwards' scratch is not shared between streams: that of the first one, kept buffers of
    others and, of the seven, temporary ones. Longer views and queues than a call takes to enqueue,
    so that the streams overlap."""
    import elsa_b200
    torch = cuda
    poses, det, x, _ = _problem(oracle, vol, 150, det)
    make = lambda: elsa_b200.Projector(getattr(elsa_b200, "PROJECTOR_" + kind), vol, det, poses)
    proj, other, repeats = make(), make(), 10
    xs = [torch.from_numpy(x * np.float32(k + 1)).cuda() for k in range(count)]
    ref = [_apply(torch, other, v.cpu().numpy(), False) for v in xs]
    streams = [torch.cuda.Stream() for _ in range(count)]
    outs = torch.zeros((count, repeats, proj.range_size), device="cuda")
    # the streams' work waits for this product, so that all of it is enqueued by then
    big = torch.zeros((8192, 8192), device="cuda")
    torch.cuda.synchronize()
    for _ in range(4):
        big = big @ big
    start = torch.cuda.Event()
    start.record()
    for s in streams:
        s.wait_event(start)
    for i in range(repeats):
        for k, s in enumerate(streams):
            proj.apply_ptr(xs[k].data_ptr(), outs[k][i].data_ptr(), s.cuda_stream)
    torch.cuda.synchronize()
    bound = 1e-6 if kind == "BLOB" else 0.0  # the voxel forward's atomics reorder its sums
    for k in range(count):
        for got in outs[k].cpu().numpy():
            assert rel_l2(got, ref[k]) <= bound


def test_forwards_on_streams_that_come_and_go(cuda, oracle):
    """A program that makes a stream for every call keeps a bounded amount of scratch."""
    import elsa_b200
    torch = cuda
    vol = (160, 150, 170)
    poses, det, x, _ = _problem(oracle, vol, 20, [220, 220])
    proj = elsa_b200.Projector(elsa_b200.PROJECTOR_SIDDON, vol, det, poses)
    assert proj.info(6) > 1  # with a copy
    ref = _apply(torch, proj, x, False)
    d = torch.from_numpy(x).cuda()
    y = torch.empty(proj.range_size, device="cuda")
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    for i in range(24):
        s = torch.cuda.ExternalStream(_new_stream(torch))
        y.zero_()
        torch.cuda.synchronize()
        proj.apply_ptr(d.data_ptr(), y.data_ptr(), s.cuda_stream)
        if i % 3 == 0:
            torch.cuda.synchronize()
            assert np.array_equal(y.cpu().numpy(), ref)
    torch.cuda.synchronize()
    # four kept buffers of a copy, and what the device's pool takes at a time
    assert before - torch.cuda.mem_get_info()[0] <= 4 * 4 * x.size + (96 << 20)


def _new_stream(torch):
    import ctypes
    rt = ctypes.CDLL("libcudart.so.12")
    s = ctypes.c_void_p()
    assert rt.cudaStreamCreateWithFlags(ctypes.byref(s), 1) == 0
    return s.value


@pytest.mark.parametrize("kind", ["SIDDON", "RAY_BLOB"])
def test_forward_without_room_for_a_copy(cuda, oracle, kind):
    """On a stream for which no scratch is left the volume itself is read."""
    import elsa_b200
    torch = cuda
    vol = (300, 280, 320)
    poses, det, x, _ = _problem(oracle, vol, 4, [400, 400] if kind == "SIDDON" else [24, 20])
    proj = elsa_b200.Projector(getattr(elsa_b200, "PROJECTOR_" + kind), vol, det, poses)
    assert proj.info(6) > 1  # with a copy
    ref = _apply(torch, proj, x, False)
    d = torch.from_numpy(x).cuda()
    y = torch.full((proj.range_size,), float("nan"), device="cuda")
    s = torch.cuda.Stream()
    full = _fill_memory(torch, 48 << 20)
    try:
        proj.apply_ptr(d.data_ptr(), y.data_ptr(), s.cuda_stream)
        torch.cuda.synchronize()
    finally:
        del full
        torch.cuda.empty_cache()
    assert np.array_equal(y.cpu().numpy(), ref)


@pytest.mark.parametrize("vol", [(20, 17, 23), (40, 33)])
@pytest.mark.parametrize("kind", ["JOSEPH", "SIDDON", "BINARY", "BLOB", "RAY_BLOB"])
def test_no_ray_meets_the_volume(cuda, kind, vol):
    """A detector far off the volume: zeros in both directions, written over what the output held,
    through every entry point."""
    import elsa_b200
    torch = cuda
    dim, n = len(vol), max(vol)
    det = [30, 24, 6][:dim - 1] + [6]
    origin = [0.5 * v for v in vol]
    sino = [0.5 * v for v in det[:-1]]
    one = [1.0] * dim
    if dim == 3:
        poses = [elsa_b200.pose_3d(5.0 * n, 1.5 * n, one, origin, one, sino + [0.0], g,
                                   pp_offset=(30.0 * n, 0.0)) for g in np.linspace(0.0, 3.0, 6)]
    else:
        poses = [elsa_b200.pose_2d(5.0 * n, 1.5 * n, g, one, origin, [1.0, 1.0], sino + [0.0],
                                   pp_offset=30.0 * n) for g in np.linspace(0.0, 3.0, 6)]
    proj = elsa_b200.Projector(getattr(elsa_b200, "PROJECTOR_" + kind), vol, det,
                               np.concatenate(poses))
    rng = np.random.default_rng(2)
    x = rng.uniform(1, 2, int(np.prod(vol))).astype(np.float32)
    y = rng.uniform(1, 2, int(np.prod(det))).astype(np.float32)
    assert not _apply(torch, proj, x, False).any()
    scatters = [0, 1] if kind in ("JOSEPH", "SIDDON", "BINARY") else [None]
    for scatter in scatters:
        if scatter is not None:
            proj.set_knob(elsa_b200.KNOB_ADJOINT_SCATTER, scatter)
        assert not _apply(torch, proj, y, True).any()
        assert not proj.apply_adjoint_host(y).any()
        s = torch.cuda.current_stream().cuda_stream
        ys = torch.from_numpy(np.stack([y, y])).cuda()
        xs = torch.full((2, proj.domain_size), float("nan"), device="cuda")
        proj.apply_adjoint_batch_ptr(ys.data_ptr(), proj.range_size, xs.data_ptr(),
                                     proj.domain_size, 2, s)
        torch.cuda.synchronize()
        assert not xs.cpu().numpy().any()


def test_batched_solve_with_an_operator_that_meets_nothing(cuda, oracle):
    """Its normal equations are 0 x = 0; the other instances are not disturbed."""
    import elsa_b200
    torch = cuda
    n = 24
    vol, one = (n, n, n), [1.0] * 3
    poses, det, _, y = _problem(oracle, vol, 8, [36, 36])
    off = np.concatenate([elsa_b200.pose_3d(5.0 * n, 1.5 * n, one, [0.5 * n] * 3, one,
                                            [18.0, 18.0, 0.0], g, pp_offset=(30.0 * n, 0.0))
                          for g in np.linspace(0.0, 3.0, 8)])
    ops = [elsa_b200.Projector(elsa_b200.PROJECTOR_JOSEPH, vol, det, p) for p in (poses, off)]
    b = [torch.from_numpy(y).cuda() for _ in ops]
    xs = [torch.zeros(n ** 3, device="cuda") for _ in ops]
    s = torch.cuda.current_stream().cuda_stream
    batch = elsa_b200.BatchCGNE(ops, [t.data_ptr() for t in b], [t.data_ptr() for t in xs], s)
    batch.iterate(1, s)
    single = torch.zeros(n ** 3, device="cuda")
    solver = elsa_b200.Solver(elsa_b200.SOLVER_CGNE, ops[0], b[0].data_ptr(), single.data_ptr(),
                              stream=s)
    solver.iterate(1, s)
    torch.cuda.synchronize()
    assert torch.equal(xs[0], single)
    assert not batch.squared_residuals(s)[1] > 0.0  # 0 / 0 afterwards, as in a solve of its own


@pytest.mark.parametrize("kind,params", VOXEL_KINDS)
@pytest.mark.parametrize("s2c,c2d", [(-100.0, 300.0), (-40.0, 90.0), (-90.0, 30.0), (6.0, 20.0)])
@pytest.mark.parametrize("vol,views,det", [((13, 21, 9), 5, [17, 12]), ((30, 23), 5, [41]),
                                           ((60, 50), 160, [70]), ((46, 48, 50), 55, [60, 62])])
def test_voxel_source_in_front_or_inside(cuda, oracle, vol, views, det, s2c, c2d, kind, params):
    """A volume behind the source projects as well (quotients of two negative numbers), also with
    a negative source-detector distance, and around a source inside the volume."""
    import elsa_b200
    poses, det = elsa_b200.circle_trajectory(vol, views, 300.0, s2c, c2d, det)
    rng = np.random.default_rng(4)
    x = rng.uniform(0, 1, int(np.prod(vol))).astype(np.float32)
    y = rng.uniform(0, 1, int(np.prod(det))).astype(np.float32)
    proj = elsa_b200.Projector(VOXEL_CODES[kind], vol, det, poses,
                               tuple(map(float, params)) + (1,))
    args = (vol, det, poses, *_voxel_reference(oracle, kind, params, len(vol)), 1)
    assert rel_l2(_apply(cuda, proj, x, False), oracle.voxel_project(False, x, *args)) <= PARITY
    assert rel_l2(_apply(cuda, proj, y, True), oracle.voxel_project(True, y, *args)) <= PARITY


@pytest.mark.parametrize("vol,det", [((13, 21, 9), [17, 12]), ((30, 23), [41]),
                                     ((400, 390), [500]), ((130, 128, 126), [170, 166])])
def test_voxel_pose_of_nan(cuda, oracle, vol, det):
    """A pose that is not a number spoils its own view and no other."""
    import elsa_b200
    poses, det, x, _ = _problem(oracle, vol, 3, det)
    size = int(np.prod(det[:-1]))
    ref = _apply(cuda, elsa_b200.Projector(elsa_b200.PROJECTOR_BLOB, vol, det, poses), x, False)
    poses = np.array(poses, np.float32).reshape(3, -1)
    poses[1] = np.nan
    got = _apply(cuda, elsa_b200.Projector(elsa_b200.PROJECTOR_BLOB, vol, det, poses.ravel()), x,
                 False)
    for view in (0, 2):
        part = slice(view * size, (view + 1) * size)
        assert rel_l2(got[part], ref[part]) <= 1e-6  # the forward's atomics reorder its sums


@pytest.mark.parametrize("adjoint", [False, True])
@pytest.mark.parametrize("kind,vol,det", [("JOSEPH", (120, 100), [150]),
                                          ("JOSEPH", (40, 36, 44), [60, 60]),
                                          ("SIDDON", (60, 50, 70), [90, 80]),
                                          ("BLOB", (40, 50, 45), [60, 70]),
                                          ("RAY_BLOB", (24, 20, 28), [40, 30])])
def test_host_threads_on_one_stream(cuda, oracle, kind, vol, det, adjoint):
    """Host threads that apply one projector on one stream: every result is that of its own
    input."""
    import threading
    import elsa_b200
    torch = cuda
    poses, det, x, y = _problem(oracle, vol, 110, det)
    proj = elsa_b200.Projector(getattr(elsa_b200, "PROJECTOR_" + kind), vol, det, poses)
    base = y if adjoint else x
    count, repeats = 4, 60
    data = [torch.from_numpy(base * (k + 1)).cuda() for k in range(count)]
    ref = [_apply(torch, proj, base * np.float32(k + 1), adjoint) for k in range(count)]
    size = proj.domain_size if adjoint else proj.range_size
    outs = [torch.empty((repeats, size), device="cuda") for _ in range(count)]
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    apply = proj.apply_adjoint_ptr if adjoint else proj.apply_ptr
    gate, failed = threading.Barrier(count), []

    def work(k):
        try:
            gate.wait()
            for i in range(repeats):
                apply(data[k].data_ptr(), outs[k][i].data_ptr(), stream.cuda_stream)
        except Exception as e:  # reported below, in the main thread
            failed.append(e)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(count)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert not failed, failed
    # (the voxel forward's atomics and the Siddon scatter reorder their sums)
    bound = 1e-6 if kind == "BLOB" and not adjoint else 0.0
    for k in range(count):
        for got in outs[k].cpu().numpy():
            assert rel_l2(got, ref[k]) <= bound


@pytest.mark.parametrize("kind,vol,det", FORWARDS)
def test_captured_forwards_next_to_others(cuda, oracle, kind, vol, det):
    """Replays of captured forwards next to one another and to applies on the stream that they were
    captured on: scratch is not shared between them."""
    import elsa_b200
    torch = cuda
    poses, det, x, _ = _problem(oracle, vol, 150, det)
    make = lambda: elsa_b200.Projector(getattr(elsa_b200, "PROJECTOR_" + kind), vol, det, poses)
    proj, other, repeats = make(), make(), 12
    xs = [torch.from_numpy(x * np.float32(k + 1)).cuda() for k in range(3)]
    ref = [_apply(torch, other, v.cpu().numpy(), False) for v in xs]
    outs = torch.zeros((3, 2, proj.range_size), device="cuda")
    a, b, c = (torch.cuda.Stream() for _ in range(3))
    torch.cuda.synchronize()
    proj.apply_ptr(xs[0].data_ptr(), outs[0][0].data_ptr(), a.cuda_stream)
    graphs = []
    for k in (1, 2):
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=a):
            for i in range(2):  # two calls of one capture
                proj.apply_ptr(xs[k].data_ptr(), outs[k][i].data_ptr(), a.cuda_stream)
        graphs.append(g)
    torch.cuda.synchronize()
    bound = 1e-6 if kind == "BLOB" else 0.0  # the voxel forward's atomics reorder its sums
    for _ in range(repeats):
        outs.zero_()
        torch.cuda.synchronize()
        for i in range(2):
            for s, g in zip((b, c), graphs):
                with torch.cuda.stream(s):
                    g.replay()
            proj.apply_ptr(xs[0].data_ptr(), outs[0][i].data_ptr(), a.cuda_stream)
        torch.cuda.synchronize()
        for k in range(3):
            for got in outs[k].cpu().numpy():
                assert rel_l2(got, ref[k]) <= bound


def test_captures_reuse_scratch(cuda, oracle):
    """The scratch of a destroyed graph serves the next capture."""
    import time
    import elsa_b200
    torch = cuda
    vol = (160, 150, 170)
    poses, det, x, _ = _problem(oracle, vol, 20, [220, 220])
    proj = elsa_b200.Projector(elsa_b200.PROJECTOR_SIDDON, vol, det, poses)
    assert proj.info(6) > 1  # with a copy
    d = torch.from_numpy(x).cuda()
    y = torch.empty(proj.range_size, device="cuda")
    s = torch.cuda.Stream()

    def capture():
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s):
            proj.apply_ptr(d.data_ptr(), y.data_ptr(), s.cuda_stream)
        g.replay()
        torch.cuda.synchronize()
        del g
        time.sleep(0.05)  # (references are dropped asynchronously)

    capture()
    free = torch.cuda.mem_get_info()[0]
    for _ in range(20):
        capture()
    assert free - torch.cuda.mem_get_info()[0] <= 4 * 4 * x.size  # four of 20 captures' copies


def test_siddon_copies_leave_the_adjoint_its_tables(cuda):
    """Where the adjoint's tables just fit its rule (half of what is free beside the rays), the
    forward's volume copy does not turn it to the scatter."""
    import elsa_b200
    torch = cuda
    n, pixels = 512, 1000
    one = [1.0] * 3
    pose = elsa_b200.pose_3d(5.0 * n, 5.0 * n, one, [0.5 * n] * 3, one,
                             [0.5 * pixels, 0.5 * pixels, 0.0], 0.5 * np.pi)  # drives along x
    make = lambda: elsa_b200.Projector(elsa_b200.PROJECTOR_SIDDON, (n,) * 3,
                                       [pixels, pixels, 1], pose)
    torch.cuda.synchronize()
    x = torch.rand(n ** 3, device="cuda")
    y = torch.empty(pixels * pixels, device="cuda")
    out = []
    for limited in (False, True):
        rays = pixels * pixels
        tables, setup, copy = 20 * rays * (n // 16 + 3), 128 * rays, 4 * n ** 3
        full = _fill_memory(torch, 2 * tables + setup + copy // 2) if limited else []
        try:
            proj = make()
            assert proj.knob(elsa_b200.KNOB_ADJOINT_SCATTER) == 0
            assert proj.info(6) == 2 or limited  # with a copy
            proj.apply_ptr(x.data_ptr(), y.data_ptr(), torch.cuda.current_stream().cuda_stream)
            torch.cuda.synchronize()
        finally:
            del full
        out.append(y.cpu().numpy())
        proj.close()
        torch.cuda.empty_cache()
    assert np.array_equal(*out)


def test_fast_joseph_2d_with_little_room_for_checkpoints(cuda, oracle):
    """The forward of the `fast` operator, whose adjoint has no use for the checkpoint table, then
    takes deeper slabs."""
    import elsa_b200
    torch = cuda
    vol = (1000, 980)
    poses, det, x, _ = _problem(oracle, vol, 1000, [1400])
    make = lambda: elsa_b200.Projector(elsa_b200.PROJECTOR_JOSEPH, vol, det, poses, (1.0,))
    proj = make()
    ref = _apply(torch, proj, x, False)
    proj.close()
    d = torch.from_numpy(x).cuda()
    y = torch.full((ref.size,), float("nan"), device="cuda")
    # 45 MB of rays, 202 MB of checkpoints (one slab: 34 MB)
    full = _fill_memory(torch, 160 << 20)
    try:
        proj = make()
        proj.apply_ptr(d.data_ptr(), y.data_ptr(), torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
    finally:
        del full
        torch.cuda.empty_cache()
    got = y.cpu().numpy()
    assert rel_l2(got, ref) <= PARITY
    assert not np.array_equal(got, ref)  # (the slabs' sums were added in another order)


@pytest.mark.parametrize("kind", ["SIDDON", "BINARY"])
@pytest.mark.parametrize("gamma", [0.0, 0.5 * np.pi])  # rays along z and along x
def test_siddon_forward_beyond_32_bit_offsets(cuda, oracle, kind, gamma):
    """A volume of 2^32 words and more, rays through its last planes: the same visits and sums, bit
    for bit. (The host copy is zero pages but for a few planes.)"""
    import elsa_b200
    torch = cuda
    vol, det = (1700, 1600, 1600), [12, 9, 1]
    if torch.cuda.mem_get_info()[0] < 60 << 30:
        pytest.skip("needs 60 GB of device memory")
    one = [1.0] * 3
    pose = elsa_b200.pose_3d(9000.0, 2000.0, one, [850.5, 800.25, 1594.0], one, [6.0, 4.5, 0.0],
                             gamma)
    planes = [0, 1, 900, 1590, 1591, 1592, 1593, 1594, 1595, 1596, 1597, 1598, 1599]
    size = vol[0] * vol[1]
    assert size * vol[2] > 2 ** 32 > size * planes[2]
    x = np.zeros(size * vol[2], np.float32)
    d = torch.zeros(x.size, device="cuda")
    rng = np.random.default_rng(8)
    for k in planes:
        part = rng.uniform(0.5, 1, size).astype(np.float32)
        x[k * size:(k + 1) * size] = part
        d[k * size:(k + 1) * size] = torch.from_numpy(part).cuda()
    proj = elsa_b200.Projector(getattr(elsa_b200, "PROJECTOR_" + kind), vol, det, pose)
    y = torch.full((proj.range_size,), float("nan"), device="cuda")
    proj.apply_ptr(d.data_ptr(), y.data_ptr(), torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    fn = oracle.siddon if kind == "SIDDON" else oracle.binary
    ref = np.asarray(fn(x, vol, det, pose), np.float32)
    assert np.count_nonzero(ref) > ref.size // 2  # (rays along x at the volume's end may miss it)
    assert np.array_equal(y.cpu().numpy(), ref)
    del d
    torch.cuda.empty_cache()

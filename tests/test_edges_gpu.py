"""GPU: the kernels at the sizes where their tiles and dispatches can go
wrong -- planes that no column tile divides, the smallest box, odd level
counts (the two eliminations of the W system meet on face nz / 2), columns so
deep that the tile narrows, level counts that no block of the microphysics
divides, views with ghost cells, row tiles of the network.

Bars: FP64 against the oracle, relative L2 <= 1e-10 per field (the bar of the
parity tests: rounding, amplified by a few steps); the FP32-bulk form against
the oracle <= 1e-4 on flat grids (its increments carry 24 bits), over terrain
the bars stated there; the network's BF16 products
<= 1e-2 as in test_mlp_gpu."""
import ctypes

import numpy as np
import pytest

import oracle
from erf_b200 import cases, config as C, terrain as T
from helpers import compare_states, rel_l2

pytestmark = pytest.mark.gpu
TOL = 1e-10
# the mixed form over terrain, two steps: ten times the largest error measured on these planes (w, smallest of
# the winds, 1.4e-6; v 2.1e-7; u 2.3e-8)
MIXED_TERRAIN = {"rho": 2.4e-8, "rhotheta": 7.4e-9, "rhoKE": 5.2e-7, "theta": 2.2e-8, "u": 2.3e-7, "v": 2.2e-6,
                 "w": 1.4e-5}


def _advance(case, base, state, steps, precision):
    from erf_b200 import Dycore
    cfg = case.cfg.copy()
    cfg.precision = precision
    dy = Dycore(cfg)
    dy.set_base_state(base)
    got = dy.advance_host(*state, steps)
    assert dy.status() == 0
    dy.close()
    return got


def _marches(nx, ny, nz):
    """Whether the tiled passes take several levels per block: more 32 x 8 tiles x levels than a wave of
    256-thread blocks (8 fit an SM at most, 148 SMs)."""
    return -(-nx // 32) * -(-ny // 8) * nz > 8 * 148


@pytest.mark.parametrize("size", [(4, 4, 4), (5, 7, 9), (36, 5, 13), (33, 31, 17), (8, 4, 150), (101, 75, 41)])
@pytest.mark.parametrize("flow,dyc,dry,moist", [("abl", C.UPWIND_5TH, C.UPWIND_5TH, C.WENO_5),
                                                ("bubble", C.UPWIND_3RD, C.UPWIND_3RD, C.WENO_3)])
def test_step(size, flow, dyc, dry, moist):
    nx, ny, nz = size
    assert _marches(nx, ny, nz) == (nx > 100)
    case = cases.abl_dry(nx=nx, ny=ny, nz=nz) if flow == "abl" else cases.moist_bubble(nx=nx, ny=ny, nz=nz)
    c = case.cfg
    if nz > 80:
        c.dz = c.dz * 80 / nz
        c.dt = 0.5 * c.dt
    c.dycore_horiz_adv = c.dycore_vert_adv = dyc
    c.dryscal_horiz_adv = c.dryscal_vert_adv = dry
    c.moistscal_horiz_adv = c.moistscal_vert_adv = moist
    case.pert.update({"vel_noise_amp": 0.5})
    base = oracle.make_base_state(c, case)
    state = case.build_state(base[0])
    ref = oracle.advance(c, base, *state, 2)
    for precision, tol in ((C.PREC_FP64, TOL), (C.PREC_MIXED, 1e-4)):
        errs = compare_states(_advance(case, base, state, 2, precision), ref)
        bad = {k: e for k, e in errs.items() if not e <= tol}
        assert not bad, (precision, errs)


@pytest.mark.parametrize("nx,ny,nz,dyc", [(4, 4, 4, C.UPWIND_5TH), (13, 9, 33, C.UPWIND_5TH), (9, 5, 150, C.UPWIND_5TH),
                                           (101, 75, 41, C.UPWIND_5TH), (101, 75, 41, C.UPWIND_3RD)])
def test_terrain_substeps(nx, ny, nz, dyc):
    from erf_b200 import Dycore
    assert _marches(nx, ny, nz) == (nx > 100)   # the larger planes run the tiled passes on ragged tiles
    case = T.abl_terrain(nx=nx, ny=ny, nz=nz, dx=25.0, dz0=320.0 / nz, stretch=1.01, h0=30.0, r0=100.0,
                         amp=5.0)
    case.cfg.dt *= min(1.0, 16.0 / nz)
    case.cfg.dycore_horiz_adv = case.cfg.dycore_vert_adv = dyc
    ref = None
    for precision in (C.PREC_FP64, C.PREC_MIXED):
        cfg = case.cfg.copy()
        cfg.precision = precision
        dy = Dycore(cfg)
        dy.set_terrain(case.z_nd)
        if ref is None:
            base = dy.make_base_state_terrain(case)
            cons, u, v, w = case.build_state(base[0])
            v = v + 2.0 * np.sin(2.0 * np.pi * np.arange(ny + 1) / ny)[None, :, None]
            v[:, ny] = v[:, 0]
            ref = oracle.advance_terrain(case.cfg, case.z_nd, base, cons, u, v, w, 2)
        dy.set_base_state(base)
        got = dy.advance_host(cons, u, v, w, 2)
        assert dy.status() == 0
        dy.close()
        errs = compare_states(got, ref)
        print("terrain", (nx, ny, nz), dyc, precision, errs)
        bars = {k: TOL for k in errs} if precision == C.PREC_FP64 else MIXED_TERRAIN
        assert all(e <= bars[k] for k, e in errs.items()), errs


def test_terrain_momentum_accumulates_in_fp64():
    """Uniform flow over flat ground, no gravity, a constant force: nothing but
    the force acts, so a step adds dt F to the momenta whatever the number of
    substeps.  The mixed form stores F in FP32 but accumulates the state in
    FP64: each of the ~150 substeps rounds to 2^-53 of a momentum of the size
    of dt F (bar 1e-13 of the velocity); increments carried in 24 bits left
    1.7e-7."""
    from erf_b200 import Dycore
    nx, ny, nz = 8, 6, 8
    cfg = T.abl_terrain(nx=nx, ny=ny, nz=nz, les="smagorinsky").cfg
    cfg.les_type, cfg.zlo_bc, cfg.gravity, cfg.use_coriolis = C.LES_NONE, C.BC_SLIP_WALL, 0.0, 0
    cfg.precision, cfg.mri_ratio, cfg.dt = C.PREC_MIXED, 100, 1.5
    cfg.abl_geo_forcing[:] = [0.7, -0.3, 0.0]
    rho, theta, u0, v0 = 1.1, 300.0, 1.0, -0.5
    pi = (C.R_D * rho * theta / 1.0e5) ** (T.GAMMA * C.R_D / cfg.c_p)
    p = 1.0e5 * (C.R_D * rho * theta / 1.0e5) ** T.GAMMA
    dy = Dycore(cfg)
    dy.set_terrain(T.btf_nodes(T.zlevels(nz, cfg.dz), np.zeros((ny + 1, nx + 1))))
    dy.set_base_state([np.full((nz + 2) * ny * nx, b) for b in (rho, p, pi, theta)])
    cons = np.zeros((5, nz, ny, nx))
    cons[0], cons[1] = rho, rho * theta
    got = dy.advance_host(cons, np.full((nz, ny, nx + 1), u0), np.full((nz, ny + 1, nx), v0), np.zeros((nz + 1, ny, nx)), 1)
    assert dy.status() == 0
    dy.close()
    for vel, start, a in ((got[1], u0, 0.7), (got[2], v0, -0.3)):
        want = start + cfg.dt * float(np.float32(rho * a)) / rho
        assert np.max(np.abs(vel - want)) <= 1e-13 * abs(want), np.max(np.abs(vel - want))


@pytest.mark.parametrize("nx,ny,nz", [(12, 4, 7), (24, 7, 33), (37, 23, 9), (67, 29, 12), (61, 41, 20), (101, 75, 32)])
@pytest.mark.parametrize("precision", [C.PREC_FP64, C.PREC_MIXED])
def test_moving_terrain_substeps(nx, ny, nz, precision):
    """Column tiles of 2 (the first two planes), 4, 8 and 16 columns, the last
    tile ragged, and a plane whose slow passes march ragged x-y tiles; a wind
    that varies in y, and a scalar.  FP64 <= 1e-10; mixed
    (FP32 tendencies and averages) <= 1e-6, w, the smallest wind, <= 1e-5."""
    assert _marches(nx, ny, nz) == (nx > 100)
    case = T.moving_terrain(nx=nx, ny=ny, nz=nz, Lx=5.0 * nx, Ly=5.0 * ny, H=5.0 * nz, ampl=0.05, wavelength=2.5 * nx,
                            substeps=True, dt=0.02)
    case.cfg.mri_ratio = 6
    case.cfg.precision = precision
    from erf_b200 import Dycore
    cons, u, v, w = case.build_state()
    y = 2.0 * np.pi * np.arange(ny + 1)[None, :, None] / ny
    x = 2.0 * np.pi * np.arange(nx)[None, None, :] / nx
    v = v + 0.2 * np.sin(y) * (1.0 + 0.3 * np.cos(x)) * np.linspace(1.0, 0.5, nz)[:, None, None]
    v[:, ny] = v[:, 0]
    cons[4] = cons[0] * (1.0 + 0.1 * np.cos(x + y[:, :ny]))
    dy = Dycore(case.cfg)
    dy.set_base_state(case.base)
    got = dy.advance_host(cons, u, v, w, 3)
    _, z, r0, p0 = dy.moving_terrain_state()
    assert dy.status() == 0
    dy.close()
    ref = oracle.advance_moving_terrain(case.cfg, 0.0, case.base, cons, u, v, w, 3)
    errs = {"rho": rel_l2(got[0][0], ref[0][0]), "rhotheta": rel_l2(got[0][1], ref[0][1]),
            "scalar": rel_l2(got[0][4], ref[0][4]), "u": rel_l2(got[1], ref[1]), "v": rel_l2(got[2], ref[2]),
            "w": rel_l2(got[3], ref[3]), "z": rel_l2(z, ref[4]), "r0": rel_l2(r0, ref[5]), "p0": rel_l2(p0, ref[6])}
    print("moving", (nx, ny, nz), precision, errs)
    if precision == C.PREC_FP64:
        assert all(e <= TOL for e in errs.values()), errs
    else:
        assert errs.pop("w") <= 1e-5 and all(e <= 1e-6 for e in errs.values()), errs


def _held(which):
    """(case, bytes that a context may hold).  Flat grids: the state three
    times and its fast sum, two sets of velocities and the stage's arrays, as
    cells and z faces of FP64 and of the bulk type; terrain: the same with
    the metric tables, as measured when the substeps were separate horizontal
    and vertical kernels."""
    n, f = 24 * 20 * 32, 24 * 20 * 33
    if which == "dry":
        return cases.abl_dry(nx=24, ny=20, nz=32), 8 * (57 * n + 15 * f)
    if which == "moist":
        return cases.moist_bubble(nx=24, ny=20, nz=32), 8 * (75 * n + 15 * f)
    if which == "mixed":
        case = cases.abl_dry(nx=24, ny=20, nz=32)
        case.cfg.precision = C.PREC_MIXED
        return case, 8 * (32 * n + 6 * f) + 4 * (25 * n + 9 * f)
    if which == "terrain":
        return T.abl_terrain(nx=64, ny=64, nz=64, dt=0.25, h0=30.0, r0=200.0, amp=2.0), 253505056
    return T.moving_terrain(substeps=True), 31041904


@pytest.mark.parametrize("which", ["dry", "moist", "mixed", "terrain", "moving"])
def test_memory_of_a_context(which):
    """The largest grid that fits the card is set by what a context holds."""
    from erf_b200 import Dycore
    case, most = _held(which)
    dy = Dycore(case.cfg)
    held = dy.scratch_bytes()
    dy.close()
    assert held <= most, (held, most)


@pytest.mark.parametrize("size,ghost,rain", [((24, 20, 40), 2, True), ((13, 9, 17), 1, True), ((13, 9, 17), 2, False),
                                             ((33, 4, 8), 0, False)])
def test_kessler_views(size, ghost, rain):
    import torch
    from erf_b200 import Dycore, dycore
    from test_zz_no_alloc import ghost_fab
    nx, ny, nz = size
    case = cases.moist_bubble(nx=nx, ny=ny, nz=nz)
    cfg = case.cfg
    if not rain:
        cfg.moisture, cfg.ncomp, cfg.buoyancy_type = C.MOIST_KESSLER_NORAIN, 7, 1
    base = oracle.make_base_state(cfg, case)
    cons = np.ascontiguousarray(case.build_state(base[0])[0][:cfg.ncomp])
    rng = np.random.default_rng(3)
    cons[5] *= 1.0 + 0.3 * rng.random(cons[5].shape)
    cons[6] = cons[0] * 2.0e-3 * rng.random(cons[0].shape)
    if rain:
        cons[7] = cons[0] * 1.0e-3 * rng.random(cons[0].shape) * (rng.random(cons[0].shape) > 0.3)
    ref = oracle.kessler(cfg, cons, cfg.dt)
    g = ghost
    x = np.full((cfg.ncomp, nz + 2 * g, ny + 2 * g, nx + 2 * g), -7.0)
    inner = np.s_[:, g:g + nz, g:g + ny, g:g + nx]
    x[inner] = cons
    dy = Dycore(cfg)
    t = torch.from_numpy(x).cuda()
    f = ghost_fab(t, g, nx, ny, nz, cfg.ncomp)
    torch.cuda.synchronize()
    assert dycore.load_library().erf_b200_kessler_advance(dy.ctx, ctypes.byref(f), cfg.dt) == 0
    assert dy.status() == 0
    dy.close()
    got = t.cpu().numpy()
    for n in range(cfg.ncomp):
        assert rel_l2(got[inner][n], ref[n]) <= TOL, n
    # ghosts: periodic laterally, the nearest level vertically
    want = np.pad(np.pad(got[inner], ((0, 0), (0, 0), (g, g), (g, g)), mode="wrap"), ((0, 0), (g, g), (0, 0), (0, 0)),
                  mode="edge")
    assert np.array_equal(got, want)


@pytest.mark.parametrize("n", [1, 127, 129, 128 * 5 * 148 + 77])
def test_network_row_tiles(n):
    """One row, ragged tiles, and more tiles than resident blocks (a block's later tiles)."""
    import torch
    from erf_b200.closure import MLP
    from oracle import mlp as ref
    p = ref.init_params(4)
    x = np.random.default_rng(n).standard_normal((n, 13)).astype(np.float32)
    m = MLP()
    m.set_params(p)
    m.set_normalization(np.zeros(13), np.ones(13), np.zeros(9), np.ones(9))
    y = torch.full((n + 1, 9), -7.0, device="cuda")
    m.infer(torch.from_numpy(x).cuda(), y, n)
    m.close()
    y = y.cpu().numpy()
    rows = np.unique(np.r_[0:min(n, 300), max(0, n - 300):n])
    yr = ref.forward(p.astype(np.float64), x[rows].astype(np.float64), bf=True)
    assert rel_l2(y[rows], yr) <= 1e-2
    assert np.all(y[n] == -7.0) and np.all(y[:n] != -7.0)


def test_training_step_is_adam_on_the_gradient():
    """One minibatch: the parameters move by Adam's first step on the gradient
    that erf_b200_mlp_gradient returns (FP32: 1e-6), and the packed tiles
    follow (the second gradient is that of the moved parameters)."""
    import torch
    from erf_b200.closure import MLP
    from oracle import mlp as ref
    n, lr = 700, 1e-3
    rng = np.random.default_rng(2)
    x = torch.from_numpy(rng.standard_normal((n, 13)).astype(np.float32)).cuda()
    t = torch.from_numpy(rng.standard_normal((n, 9)).astype(np.float32)).cuda()
    p = ref.init_params(6)
    a, b = MLP(), MLP()
    for m in (a, b):
        m.set_params(p)
        m.set_normalization(np.zeros(13), np.ones(13), np.zeros(9), np.ones(9))
    loss, g = a.gradient(x, t, n)
    assert abs(b.train(x, t, n, n, 1, lr) - loss) <= 1e-6 * loss
    q = b.get_params()
    g64 = g.astype(np.float64)
    want = p - lr * g64 / (np.abs(g64) + 1e-8)
    # eps against the gradient's own rounding where a gradient is near 0
    ok = (np.abs(g64) > 1e-6) | (g64 == 0.0)
    assert np.max(np.abs(q - want)[ok]) <= 1e-3 * lr
    _, g1 = b.gradient(x, t, n)
    a.set_params(q)
    _, g2 = a.gradient(x, t, n)
    a.close()
    b.close()
    assert np.array_equal(g1, g2)

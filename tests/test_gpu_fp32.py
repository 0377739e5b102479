"""The FP32 precision form: flux and reconstruction arithmetic in FP32, state,
RK sums and the time step in FP64.  Its results are compared with the FP64
path (bitwise the reference) on the same inputs; the bounds below are the
accepted error of the form and are written into the test."""
import numpy as np
import pytest

import oracle as orc
import wenofd
from conftest import fixture_id, fixture_paths, load_fixture

pytestmark = pytest.mark.gpu

RHS_REL_TOL = 2e-4      # max |rhs32 - rhs64| / max |rhs64|
STATE_REL_TOL = 1e-5    # max |U32 - U64| / max |U64| after the fixture's steps


def _config(meta, precision):
    cfg = {"TESTCASE": meta["testcase"], "ELEMNUMX": meta["nx"], "ELEMNUMY": meta["ny"],
           "RKMETH": meta["rk"], "CFL": meta["cfl"], "SCHEME": meta["scheme"], "SEED": meta["seed"],
           "PRECISION": precision}
    if meta.get("t_end") is not None:
        cfg["TEND"] = meta["t_end"]
    return cfg


@pytest.mark.parametrize("path", fixture_paths("rhs_"), ids=fixture_id)
def test_fp32_rhs_close_to_reference(path):
    fx = load_fixture(path)
    m = fx["meta"]
    with wenofd.Solver(_config(m, wenofd.FP32)) as s:
        s.set_state(fx["init"])
        rhs = s.get_flux()
    assert np.all(np.isfinite(rhs))
    err = np.max(np.abs(rhs - fx["rhs"])) / np.max(np.abs(fx["rhs"]))
    assert err <= RHS_REL_TOL, err


@pytest.mark.parametrize("path", fixture_paths("run_"), ids=fixture_id)
def test_fp32_steps_close_to_reference(path):
    fx = load_fixture(path)
    m = fx["meta"]
    with wenofd.Solver(_config(m, wenofd.FP32)) as s:
        s.set_state(fx["init"])
        n = s.advance(max_steps=m["steps"] if m["t_end"] is None else -1)
        U = s.get_state()
    assert n == m["steps"]
    assert np.all(np.isfinite(U))
    err = np.max(np.abs(U - fx["state"])) / np.max(np.abs(fx["state"]))
    assert err <= STATE_REL_TOL, err


@pytest.mark.parametrize("scheme", [orc.WENOJS, orc.WENOZ, orc.WENOZP, orc.WENOZPI])
def test_fp32_shear_layer_stays_finite_and_close(scheme):
    """The shear layer has flat stencils next to jumps (beta = 0 beside a
    large tau), the case that overflows unguarded FP32 weights."""
    n, steps = 256, 40
    p = orc.Problem(orc.SHEAR, n, n, scheme, 2, 0.7, seed=5)
    init = p.interior()
    out = {}
    for prec in (wenofd.FP64, wenofd.FP32):
        with wenofd.Solver({"TESTCASE": 5, "ELEMNUMX": n, "ELEMNUMY": n, "RKMETH": 2, "CFL": 0.7,
                            "SCHEME": scheme, "SEED": 5, "PRECISION": prec}) as s:
            s.set_state(init)
            assert s.advance(max_steps=steps) == steps
            out[prec] = s.get_state()
    assert np.all(np.isfinite(out[wenofd.FP32]))
    rho32, rho64 = out[wenofd.FP32][0], out[wenofd.FP64][0]
    assert np.mean(np.abs(rho32 - rho64)) <= 1e-5
    assert np.max(np.abs(rho32 - rho64)) <= 1e-3


@pytest.mark.parametrize("tc,n,steps", [(orc.RIEMANN_SEEDED, 300, 0), (orc.RIEMANN_SEEDED, 300, 15),
                                        (orc.SHEAR, 256, 5), (orc.SMOOTH, 120, 3), (orc.RTI, 64, 5),
                                        (orc.RIEMANN1, 200, 10)])
def test_two_pass_time_step_equals_fp64_reduction(tc, n, steps):
    """The FP32 forms reduce the time step in two passes (FP32 screen with an
    error bound, FP64 only where a node can hold the maximum); the result
    must equal the FP64 form's single FP64 pass bit for bit.  Constant
    quadrants (step 0) make whole regions tie for the maximum."""
    p = orc.Problem(tc, n, n, orc.WENOZ, 2, 0.7, seed=19)
    p.run(max_steps=steps)
    U = p.interior()
    dts = []
    for prec in (wenofd.FP64, wenofd.FP32, wenofd.LEARNED):
        with wenofd.Solver({"TESTCASE": tc, "ELEMNUMX": n, "ELEMNUMY": n, "RKMETH": 2, "CFL": 0.7,
                            "SCHEME": 1, "SEED": 19, "PRECISION": prec}) as s:
            s.set_state(U)
            dts.append(s.calc_dt())
    assert dts[0] == dts[1] == dts[2] == p.calc_dt()


@pytest.mark.parametrize("precision", [wenofd.FP32, wenofd.LEARNED])
@pytest.mark.parametrize("tile_i", [0, 31])
def test_fused_screen_steps_equal_separate_steps(precision, tile_i):
    """Inside wenofd_advance the last RK stage of a step also screens the
    next time step per stage tile, and the reduction then refines only the
    tiles that can hold the maximum.  The steps must equal, bit for bit,
    steps driven one call at a time (calc_dt: full screen + refine; rk_step)."""
    import mlp_oracle

    n, steps = 200, 8
    cfg = {"TESTCASE": 5, "ELEMNUMX": n, "ELEMNUMY": n + 17, "RKMETH": 2, "CFL": 0.7, "SCHEME": 1, "SEED": 5,
           "PRECISION": precision, "TILE_I": tile_i}
    params = mlp_oracle.init_params(3)

    def make():
        s = wenofd.Solver(cfg)
        s.initialize()
        if precision == wenofd.LEARNED:
            s.set_indicator(params, 0.5)
        return s

    with make() as a:
        assert a.advance(max_steps=steps) == steps
        Ua, ta = a.get_state(), a.info().now
    with make() as b:
        now = 0.0
        for _ in range(steps):
            dt = b.calc_dt()
            b.rk_step(dt)
            now += dt
            b.set_time(now)
        Ub = b.get_state()
    assert ta == now
    assert np.array_equal(Ua, Ub)


@pytest.mark.parametrize("nx,ny", [(6, 6), (7, 32), (8, 33), (14, 64), (15, 97), (300, 300), (307, 321)])
@pytest.mark.parametrize("precision", [wenofd.FP32, wenofd.LEARNED])
def test_short_tiles_of_small_grids_equal_the_default_height(nx, ny, precision):
    """Grids whose 7-row tiles are resident at once take those (300^2: 430 of
    456 FP32 tiles; 307 x 321: 484, past the FP32 form's limit and within the
    learned form's); every node's operations are those of the 15-row tile, so
    the states and the times are the same bits."""
    import mlp_oracle

    got = []
    for tile_i in (0, 15):
        with wenofd.Solver({"TESTCASE": 5, "ELEMNUMX": nx, "ELEMNUMY": ny, "RKMETH": 2, "CFL": 0.5, "SCHEME": 1,
                            "SEED": 8, "PRECISION": precision, "TILE_I": tile_i}) as s:
            s.initialize()
            if precision == wenofd.LEARNED:
                s.set_indicator(mlp_oracle.init_params(3), 0.5)
            assert s.advance(max_steps=6) == 6
            got.append((s.info().now, s.get_state()))
    assert got[0][0] == got[1][0]
    assert np.all(np.isfinite(got[0][1])) and np.array_equal(got[0][1], got[1][1])


@pytest.mark.parametrize("bc", [(0, 0, 0), (1, 3, 1), (3, 1, 0), (0, 0, 3), (2, 1, 3), (3, 2, 1), (0, 0, 2), (2, 2, 2),
                                (1, 1, 2)])
@pytest.mark.parametrize("rk", [0, 1, 2])
@pytest.mark.parametrize("precision", [wenofd.FP32, wenofd.LEARNED])
def test_steps_of_the_time_loop_equal_host_driven_steps(bc, rk, precision):
    """The time loop's stages write the ghosts of their results, the last block
    of a step's last stage ends the step and the last block of the refinement
    forms dt; host-driven steps launch a ghost fill per stage and a kernel for
    each of the others.  Same bits, on every boundary kind, on grids whose edge
    nodes image to both sides, on several tiles, and on the large grids' tile;
    a second call starts from the ghosts of the first."""
    import mlp_oracle

    sizes = [(6, 6), (7, 9), (9, 40), (33, 65)] + ([(33, 9800)] if precision == wenofd.LEARNED and rk == 2 else [])
    for nx, ny in sizes:
        cfg = {"TESTCASE": 4, "ELEMNUMX": nx, "ELEMNUMY": ny, "RKMETH": rk, "CFL": 0.4, "SCHEME": 1, "SEED": 6,
               "PRECISION": precision, "BC_LEFT": bc[0], "BC_RIGHT": bc[1], "BC_BOTTOM": bc[2], "BC_TOP": bc[2]}

        def make():
            s = wenofd.Solver(cfg)
            s.initialize()
            if precision == wenofd.LEARNED:
                s.set_indicator(mlp_oracle.init_params(3), 0.5)
            return s

        with make() as a:
            assert a.advance(max_steps=2) == 2
            assert a.advance(max_steps=3) == 3
            Ua, ta = a.get_state(), a.info().now
        with make() as b:
            for _ in range(5):
                b.step()
            Ub, tb = b.get_state(), b.info().now
        assert ta == tb, (nx, ny)
        assert np.array_equal(Ua, Ub, equal_nan=True), (nx, ny)
        assert np.all(np.isfinite(Ua)), (nx, ny)


@pytest.mark.parametrize("nx,ny", [(6, 6), (7, 9), (16, 31), (33, 65), (100, 7)])
@pytest.mark.parametrize("tile_i", [15, 31])
def test_tma_tiles_on_small_and_ragged_grids(nx, ny, tile_i):
    """The per-solve FP32 tiles take their halo and flags by TMA in boxes of
    40 x (TI + 6) nodes and 48 x (TI + 4) flag bytes: on grids smaller than a
    box or not a multiple of the tile the boxes run past the arrays (zero
    fill) and past the tiles' last nodes.  The batched kernel runs the same
    tile arithmetic with per-thread 128-bit loads instead, so the two must
    agree (to the last bit here), on every boundary kind.  On the smallest
    Riemann grids a shock crosses most nodes and FP32 rounding grows: the FP32
    form sits up to ~3e-4 from FP64 there, and the learned form with every
    node flagged (the WENO list for every face, whose four lanes group the
    arithmetic differently) up to ~2e-4 from the FP32 form; both are held to
    1e-3."""
    for tc in (orc.RIEMANN_SEEDED, orc.RIEMANN1, orc.SMOOTH):
        cfg = {"TESTCASE": tc, "ELEMNUMX": nx, "ELEMNUMY": ny, "RKMETH": 2, "CFL": 0.5, "SCHEME": 1, "SEED": 4}

        def run(precision, params=None, batched=False):
            with wenofd.Solver(dict(cfg, PRECISION=precision, TILE_I=tile_i)) as s:
                s.initialize()
                if params is not None:
                    s.set_indicator(params, 0.5)
                if batched:
                    with wenofd.Batch([s]) as b:
                        b.configure(tile_i=tile_i)
                        assert b.advance(5) == 5
                else:
                    assert s.advance(max_steps=5) == 5
                return s.get_state()

        U64 = run(wenofd.FP64) if tile_i == 15 else None
        U32 = run(wenofd.FP32)
        scale = np.max(np.abs(U32))
        assert np.all(np.isfinite(U32))
        assert np.max(np.abs(U32 - run(wenofd.FP32, batched=True))) <= 1e-12 * scale, (tc, nx, ny)
        every = np.zeros(wenofd.MLP_PARAMS, dtype=np.float32)
        every[2720] = 50.0
        Ul = run(wenofd.LEARNED, every)
        if U64 is not None:
            assert np.max(np.abs(U32 - U64)) <= 1e-3 * scale, (tc, nx, ny)
        assert np.max(np.abs(Ul - U32)) <= 1e-3 * scale, (tc, nx, ny)


@pytest.mark.parametrize("nx,ny", [(6, 9), (15, 32), (16, 33), (31, 64), (46, 97)])
@pytest.mark.parametrize("scheme", [orc.WENOJS, orc.WENOZ])
@pytest.mark.parametrize("tile_i", [0, 31])
def test_fp32_rhs_of_a_smooth_flow_is_fp64_to_rounding(nx, ny, scheme, tile_i):
    """Where the reconstruction's weights are well conditioned (the smooth
    wave; a stencil that is flat up to roundoff has weights of 0/0) the FP32 RHS
    differs from FP64's by rounding alone: a face flux is a few dozen operations
    on values of at most max(|F| + (|u| + c) |U|), so 32 roundings of 2^-24 each
    of that on two faces per direction bound it."""
    rhs = {}
    for prec in (wenofd.FP64, wenofd.FP32):
        cfg = {"TESTCASE": orc.SMOOTH, "ELEMNUMX": nx, "ELEMNUMY": ny, "RKMETH": 2, "CFL": 0.5, "SCHEME": scheme,
               "PRECISION": prec, "TILE_I": tile_i if prec == wenofd.FP32 else 0}
        with wenofd.Solver(cfg) as s:
            s.initialize()
            U, info = s.get_state(), s.info()
            rhs[prec] = s.get_flux()
    u, v = U[1] / U[0], U[2] / U[0]
    p = (info.gamma - 1) * (U[3] - 0.5 * U[0] * (u * u + v * v))
    c = np.sqrt(info.gamma * p / U[0])
    speed = np.max(np.abs(u)) + np.max(np.abs(v)) + np.max(c)
    largest = speed * max(np.max(np.abs(U)), np.max(U[3] + p)) * 2
    bound = 32 * 2.0 ** -24 * largest * (2 / info.dx + 2 / info.dy)
    assert np.max(np.abs(rhs[wenofd.FP32] - rhs[wenofd.FP64])) <= bound

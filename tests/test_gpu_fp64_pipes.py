"""The FP64 parity tile forms products, quotients and roots on the integer
pipes where its operands lie in a wide range of exponents and leaves the rest to
the FP64 instructions.  Both, and tiles that mix them, are the oracle's bits:
states scaled to the ranges' edges and past them, zeros, roundoff-sized momenta,
exact powers of two, on tiles of one node, full tiles and remainders."""
import numpy as np
import pytest

import oracle as orc
import wenofd
from conftest import assert_same

pytestmark = pytest.mark.gpu


def _state(p, kind):
    U = p.interior()
    rng = np.random.default_rng(3)
    if kind == "zeros":
        U[1:3] = 0.0
    elif kind == "roundoff":
        U[2] = 1e-17 * rng.standard_normal(U[2].shape)
    elif kind == "tiny":  # momenta below 2^-200 in part of the grid
        U[1][::3] = 1e-70
        U[2][:, ::5] = -1e-90
    elif kind == "dense":  # above the range: every value times 2^70
        U *= 2.0 ** 70
    elif kind == "thin":  # below it: every value times 2^-80
        U *= 2.0 ** -80
    elif kind == "edge":  # pressure jumps across the upper bound
        U[3][U.shape[1] // 2:] *= 2.0 ** 59
    elif kind == "binary":  # exact powers of two: quotients and roots are exact
        U[0], U[1], U[2], U[3] = 2.0, 0.5, -0.25, 4.0
        U[0][::2], U[3][:, ::4] = 8.0, 16.0
    return U


@pytest.mark.parametrize("nx,ny", [(6, 7), (15, 32), (16, 33), (31, 65), (47, 70)])
@pytest.mark.parametrize("kind", ["zeros", "roundoff", "tiny", "dense", "thin", "edge", "binary"])
def test_rhs_and_steps_equal_the_oracle_at_every_range(nx, ny, kind):
    for tc in (orc.RIEMANN_SEEDED, orc.SMOOTH):
        for scheme in (orc.WENOJS, orc.WENOZ, orc.WENOZP):
            p = orc.Problem(tc, nx, ny, scheme, 2, 0.3, seed=2)
            U = _state(p, kind)
            p.set_interior(U)
            with wenofd.Solver({"TESTCASE": tc, "ELEMNUMX": nx, "ELEMNUMY": ny, "RKMETH": 2, "CFL": 0.3,
                                "SCHEME": scheme, "SEED": 2}) as s:
                s.set_state(U)
                rhs = s.get_flux()
                s.set_state(U)
                dt = s.calc_dt()
                s.rk_step(dt)
                got = s.get_state()
            want = p.assemble_rhs()
            p.set_interior(U)
            assert dt == p.calc_dt()
            p.rk_step(dt)
            if scheme == orc.WENOZP:  # pow(x, 2) of the C library: to rounding
                assert np.max(np.abs(rhs - want)) <= 1e-12 * np.max(np.abs(want))
                continue
            assert_same(rhs, want, f"rhs {kind} tc {tc} scheme {scheme}")
            assert_same(got, p.interior(), f"state {kind} tc {tc} scheme {scheme}")


def test_nan_and_infinity_spread_as_in_the_oracle():
    nx, ny = 40, 45
    for bad in (np.nan, np.inf):
        p = orc.Problem(orc.SMOOTH, nx, ny, orc.WENOZ, 2, 0.3, seed=2)
        U = p.interior()
        U[3, 20, 21] = bad
        p.set_interior(U)
        with wenofd.Solver({"TESTCASE": orc.SMOOTH, "ELEMNUMX": nx, "ELEMNUMY": ny, "RKMETH": 2, "CFL": 0.3,
                            "SCHEME": orc.WENOZ}) as s:
            s.set_state(U)
            assert_same(s.get_flux(), p.assemble_rhs(), f"rhs with {bad}")


@pytest.mark.parametrize("nx,ny", [(6, 6), (17, 40), (100, 100), (121, 481), (300, 33), (40, 900)])
@pytest.mark.parametrize("batched", [False, True])
def test_split_of_small_grids_changes_no_bit(nx, ny, batched):
    """TILE_I = 0 picks the FP64 tiles' rows, and whether two lanes share a
    face, from the grid and the number of SMs; 15 and 7 are fixed."""
    got = []
    for tile in (15, 7, 0):
        cfg = {"TESTCASE": 4, "ELEMNUMX": nx, "ELEMNUMY": ny, "RKMETH": 2, "CFL": 0.5, "SCHEME": 1, "SEED": 4}
        with wenofd.Solver(cfg if batched else dict(cfg, TILE_I=tile)) as s:
            s.initialize()
            if batched:
                with wenofd.Batch([s]) as b:
                    b.configure(tile_i=tile)
                    assert b.advance(3) == 3
            else:
                assert s.advance(max_steps=3) == 3
            got.append(s.get_state())
    assert np.array_equal(got[0], got[1]) and np.array_equal(got[0], got[2])


def _speed_states(nx, ny):
    """Conserved states whose time step goes through every branch: ties, one
    maximum, values that FP32 or the integer forms do not hold, pressure left
    over from a cancellation of 20 bits."""
    rng = np.random.default_rng(nx * 1000 + ny)
    rho = rng.uniform(0.5, 2.0, (nx, ny))
    u, v, p = rng.uniform(-1, 1, (nx, ny)), rng.uniform(-1, 1, (nx, ny)), rng.uniform(0.5, 2.0, (nx, ny))

    def state(rho, u, v, p):
        return np.stack([rho, rho * u, rho * v, p / 0.4 + 0.5 * rho * (u * u + v * v)])

    yield "random", state(rho, u, v, p)
    half = np.where(np.arange(nx)[:, None] < nx // 2, 1.0, 0.125) * np.ones((nx, ny))
    yield "ties", state(half, 0 * u, 0 * v, 1.6 * half)
    yield "tiny", state(rho, u, v, p) * 2.0 ** -150
    yield "huge", state(rho, u, v, p) * 2.0 ** 140
    yield "cancelling", state(rho, 30 * u, 30 * v, 1e-3 * p)
    mixed = state(rho, u, v, p)
    mixed[:, nx // 2, ny // 3] *= 2.0 ** -90
    mixed[1:3, nx // 3, ny // 2] *= 2.0 ** 35  # (kinetic energy below the energy: a positive pressure)
    mixed[3, nx // 3, ny // 2] *= 2.0 ** 75
    yield "mixed", mixed


@pytest.mark.parametrize("nx,ny", [(6, 6), (33, 65), (257, 193), (700, 411)])
@pytest.mark.parametrize("precision", [wenofd.FP64, wenofd.FP32])
def test_time_step_is_the_exact_maximum(nx, ny, precision):
    """calc_dt, and the batched kernel's time step, against the formula in
    float64 in the reference's operation order, bit for bit: the screen may
    only drop nodes that do not hold the maximum and the integer forms round
    as FP64 does."""
    cfg = {"TESTCASE": 4, "ELEMNUMX": nx, "ELEMNUMY": ny, "RKMETH": 2, "CFL": 0.6, "SCHEME": 1, "SEED": 2,
           "PRECISION": precision}
    for name, U in _speed_states(nx, ny):
        with wenofd.Solver(cfg) as s:
            s.initialize()
            inf = s.info()
            with np.errstate(all="ignore"):
                u, v = U[1] / U[0], U[2] / U[0]
                p = (inf.gamma - 1.0) * (U[3] - 0.5 * U[0] * (u * u + v * v))
                c = np.sqrt(inf.gamma * p / U[0])
                dt = np.min(0.6 / ((np.abs(u) + c) / inf.dx + (np.abs(v) + c) / inf.dy))
            assert np.isfinite(dt)
            want = min(1.0, dt, inf.t_end)
            s.set_state(U)
            assert s.calc_dt() == want, name
            if name in ("random", "ties", "cancelling"):
                with wenofd.Batch([s]) as b:
                    assert b.advance(1) == 1
                assert s.info().now == want, name


@pytest.mark.parametrize("nx,ny", [(6, 6), (33, 65), (257, 193), (300, 411)])
@pytest.mark.parametrize("precision", [wenofd.FP64, wenofd.FP32, wenofd.LEARNED])
def test_batched_time_step_outside_the_integer_domain(nx, ny, precision):
    """The first time step of a batch whose member holds values outside the
    integer forms' exponents, against the formula as above, bit for bit: the FP64
    instructions that take over round every operation, also in the units that
    may contract multiply-adds."""
    cfg = {"TESTCASE": 4, "ELEMNUMX": nx, "ELEMNUMY": ny, "RKMETH": 2, "CFL": 0.6, "SCHEME": 1, "SEED": 2,
           "PRECISION": precision}
    states = dict(_speed_states(nx, ny))
    for name, U in (("huge", states["huge"]), ("mixed", states["mixed"]), ("cancelling", states["cancelling"] * 2.0 ** 140),
                    ("thin", states["cancelling"] * 2.0 ** -150)):
        with wenofd.Solver(cfg) as s:
            s.initialize()
            inf = s.info()
            with np.errstate(all="ignore"):
                u, v = U[1] / U[0], U[2] / U[0]
                c = np.sqrt(inf.gamma * ((inf.gamma - 1.0) * (U[3] - 0.5 * U[0] * (u * u + v * v))) / U[0])
                want = min(1.0, np.min(0.6 / ((np.abs(u) + c) / inf.dx + (np.abs(v) + c) / inf.dy)), inf.t_end)
            s.set_state(U)
            with wenofd.Batch([s]) as b:
                assert b.advance(1) == 1
            assert s.info().now == want, name

"""Both forms of the per-mode solves, the line solver (line_solver.cu) and the sweeps
(wavespace_split.cu), and the mean lines (k_mean), against the numpy oracle at the sizes where they can go
wrong: the smallest ny that a spline order takes (the first and last rows' wide profiles overlap), the
edges of the staged chunks (ny = bw + 24 c and one more), even ny, mode counts that are no multiple of a
tile, every band width (2 to 7), one and two scalars, control, both time step rules and both precisions;
and tall grids: one block of the line solver an SM (ny of 140 and more at band width 4), its last ny (367)
and the sweeps that take over, the mean lines in global memory (ny of 568 and more).  Tolerances: FP64
1e-11 of the field as the other trajectory tests, mixed 1e-5; above ny = 129, the tallest of those tests,
1e-11 times (ny / 129)^2, as the rounding of the second derivatives goes with the inverse square of the
spacing."""
import ctypes

import numpy as np
import pytest

from channel_passive_b200 import Channel, KmmError
from channel_passive_b200 import _lib
from oracle import kmm as okmm
from tests.helpers import STATE_SLOTS, STATE_SLOTS2, make_pair, oracle_ctrl, rel_l2, seeded_state, with_scalar2

pytestmark = pytest.mark.gpu

SIZES = [  # labs_k, ny
    (6, 18), (6, 19), (6, 28), (6, 29), (6, 52), (6, 77), (4, 10), (4, 26), (4, 51), (5, 14), (5, 40), (7, 18),
    (7, 30), (8, 22), (8, 33), (10, 26), (10, 45), (11, 31), (11, 32), (12, 55)]
SOLVERS = ["lines", "sweeps"]


def _compare(cfg, p, nsteps, tol, scalars=1, solver="auto", expect=None):
    ops = okmm.make_operators(p)
    U = seeded_state(cfg, ops.y)
    if scalars == 2:
        U = with_scalar2(U, U[6] * 0.5)
    RK = okmm.set_initial_data_uvw(U.copy(), ops, p)
    Uo, RKo, dt = U.copy(), RK.copy(), 0.01
    for _ in range(nsteps):
        dt, sc = okmm.rk3_step(Uo, RKo, ops, p, dt, ctrl=oracle_ctrl(ops, p))
    with Channel(cfg, solver=solver) as ch:
        assert ch.solver == (expect or solver)
        ch.set_initial_data_uvw(U, 0.01)
        out = ch.step(nsteps)
        Ug, RKg = ch.download_state(U.shape[0])
    for s in STATE_SLOTS2 if scalars == 2 else STATE_SLOTS:
        assert rel_l2(Ug[s], Uo[s]) < tol, s
    assert rel_l2(RKg[: RKo.shape[0]], RKo) < 10 * tol
    assert abs(out["dt"] - dt) <= tol * dt
    assert abs(out["wall_shear_stress"] - sc.wall_shear_stress) <= 10 * tol * abs(sc.wall_shear_stress)


@pytest.mark.parametrize("solver", SOLVERS)
@pytest.mark.parametrize("labs_k,ny", SIZES)
def test_lines_match_oracle(labs_k, ny, solver):
    cfg, p = make_pair(nx=12, ny=ny, nz=18, control_amp=-0.7, fixed_dt=ny % 2, labs_k=labs_k)
    p.labs_k = labs_k
    _compare(cfg, p, 2, 1e-11, solver=solver)


@pytest.mark.parametrize("solver", SOLVERS)
@pytest.mark.parametrize("ny", [33, 53])
@pytest.mark.parametrize("precision", [0, 1])
def test_two_scalars_match_oracle(ny, precision, solver):
    cfg, p = make_pair(nx=16, ny=ny, nz=16, control_amp=-0.7, fixed_dt=0, precision=precision, n_scalar=2)
    _compare(cfg, p, 2, 1e-5 if precision else 1e-11, scalars=2, solver=solver)


@pytest.mark.parametrize("ny,scalars,expect", [
    (139, 1, "lines"), (140, 1, "lines"), (193, 1, "lines"), (367, 1, "lines"), (368, 1, "sweeps"),
    (568, 1, "sweeps"), (80, 2, "lines"), (141, 2, "lines"), (261, 2, "lines"), (262, 2, "sweeps"), (426, 2, "sweeps")])
def test_tall_grids_match_oracle(ny, scalars, expect):
    cfg, p = make_pair(nx=8, ny=ny, nz=10, control_amp=-0.7, fixed_dt=ny % 2, n_scalar=scalars)
    _compare(cfg, p, 1, 1e-11 * max(1.0, ny / 129) ** 2, scalars=scalars, expect=expect)


def test_the_caller_can_choose_the_solver():
    cfg, p = make_pair(nx=16, ny=368, nz=16)
    with Channel(cfg, solver="sweeps") as ch:
        assert ch.solver == "sweeps"
    with pytest.raises(KmmError) as e:
        Channel(cfg, solver="lines")
    assert e.value.code == _lib.KMM_ERR_CONFIG


def test_kept_factors_carry_their_own_time_step():
    """A substep that ends between the factorisation and the solves (a device wait that gives up) leaves
    the factors of its dt behind: a caller that goes back to the former dt gets that dt's operators.  The
    factorisation alone is the internal launcher's (no public call ends there on purpose)."""
    torch = pytest.importorskip("torch")
    cfg, p = make_pair(nx=32, ny=33, nz=32, control_amp=-1.0)
    U = seeded_state(cfg, okmm.make_operators(p).y)
    out = []
    for interrupted in (False, True):
        with Channel(cfg) as ch:
            ch.set_initial_data_uvw(U, 0.01)
            ch.step(1)
            if interrupted:
                factor = getattr(ch._lib, "_ZN3kmm18launch_line_factorERNS_6HandleEiPKdP11CUstream_st")
                factor.argtypes = [ctypes.c_void_p, ctypes.c_int, ctypes.c_void_p, ctypes.c_void_p]
                other = torch.tensor([0.02], dtype=torch.float64, device="cuda")
                for s in (1, 2, 3):
                    assert factor(ch._h, s, other.data_ptr(), None) == 0
                torch.cuda.synchronize()
            ch.step(1)
            out.append(ch.download_state(10))
    for f in STATE_SLOTS:
        assert np.array_equal(out[0][0][f], out[1][0][f]), f
    assert np.array_equal(out[0][1], out[1][1])


@pytest.mark.parametrize("nx,ny,nz,kw,expect", [
    (128, 97, 128, dict(fixed_dt=1), "lines"), (128, 225, 128, dict(fixed_dt=0), "lines"),
    (128, 257, 128, dict(fixed_dt=0), "sweeps"), (128, 257, 128, dict(fixed_dt=1), "lines"),
    (144, 257, 144, dict(fixed_dt=1), "sweeps"), (160, 65, 160, dict(fixed_dt=1), "sweeps"),
    (128, 65, 128, dict(n_scalar=2), "lines"), (128, 129, 128, dict(n_scalar=2), "sweeps"),
    (128, 33, 128, dict(fixed_dt=1, labs_k=10), "sweeps"), (128, 193, 128, dict(fixed_dt=0, labs_k=10), "lines")])
def test_the_faster_solver_is_the_default(nx, ny, nz, kw, expect):
    """One grid on each side of the rule's lines (line_modes); the figures stand there."""
    cfg, _ = make_pair(nx=nx, ny=ny, nz=nz, **kw)
    with Channel(cfg) as ch:
        assert ch.solver == expect

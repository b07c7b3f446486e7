"""tlq_set_winds again on a context that has winds (its buffers are kept), with
steps in flight: the steps before take the winds before, the steps after the
new ones.  Plain FP64 is the oracle's bits; both forms give the bits of a run
that waits for its steps and drops the winds before each new set."""
import numpy as np
import pytest

from oracle.oracle import Run
from tests.helpers import face_ghost_mask, interior, oracle_params
from tests.test_gpu_step import smooth_state
from tests.test_host_winds import set_winds
from tlaloque_gb300 import tlq

pytestmark = pytest.mark.gpu


def drifting_winds(cfg):
    """Winds that drift by a third of a cell a set; in some sets a second one,
    and once a larger one (more and larger tables, then fewer)."""
    w, h = cfg.winds[0], (cfg.xr - cfg.xl) / cfg.nx

    def at(q, x=0.0, r=0.0):
        return tlq.Wind(**{**w.__dict__, "xc": w.xc + x * h + q * h / 3, "yc": w.yc - q * h / 5, "radius": w.radius + r * h})

    return [[at(0)], [at(1), at(1, x=1.0)], [at(2), at(2, x=1.0, r=1.0), at(2, x=2.0)], [at(3, r=0.5)], [at(4)]]


def case():
    """A light wind in a smooth medium (a strong wind that moves into cells of
    another density makes the scheme's own next step negative)."""
    cfg = tlq.Config(nx=40, ny=37, nz=35, xl=-1.0, xr=1.0, yl=-0.9, yr=0.95, zl=-0.8, zr=0.95)
    cfg.winds = [tlq.Wind(radius=4.0 * cfg.dx, mdot=0.25, vinf=0.5, temp=1.2e-8, mu=1.0)]
    return cfg, smooth_state(cfg, seed=5, mach=0.5)


STEPS = 3


def oracle_run():
    cfg, U0 = case()
    run = None
    for winds in drifting_winds(cfg):
        new = Run(oracle_params(tlq.Config(**{**cfg.__dict__, "winds": winds})), U0)
        if run is not None:
            for k in new.arrays:
                new.arrays[k][...] = run.arrays[k]
            new.st.t, new.st.dt, new.st.it = run.st.t, run.st.dt, run.st.it
        run = new
        for _ in range(STEPS):
            run.run(1)
            assert interior(run.U)[0].min() > 0.0
    return run


@pytest.mark.parametrize("precision", [tlq.PREC_FP64, tlq.PREC_MIXED])
def test_winds_move_behind_steps_in_flight(gpu_lib, precision):
    cfg, U0 = case()
    cfg = tlq.Config(**{**cfg.__dict__, "precision": precision})

    def run(wait):
        U = U0.copy(order="F")
        with tlq.Context(cfg) as ctx:
            ctx.borders(U, 1)
            ctx.upload(U)
            for winds in drifting_winds(cfg):
                if wait:
                    ctx.synchronize()
                    set_winds(ctx, [])
                set_winds(ctx, winds)
                if wait:
                    ctx.synchronize()
                ctx.advance(STEPS)  # (returns before the steps have run)
            return ctx.state()[0], ctx.time()

    U, tm = run(False)
    V, tv = run(True)
    assert tm == tv and tm[3] == tlq.OK
    np.testing.assert_array_equal(interior(U), interior(V))
    if precision == tlq.PREC_FP64:
        ref, m = oracle_run(), face_ghost_mask(cfg)
        assert tm[:3] == (ref.t, ref.it, ref.dt)
        np.testing.assert_array_equal(U[:, m], ref.U[:, m])

"""Every instance of the stage kernels (van Leer with HLLC, with HLL, every
other limiter) on chunks of the default's one or two planes, of 8 planes, and
on one chunk of all planes (long enough that each landing slot of the plane
ring is used several times): plain FP64 is the oracle's bits, the mixed form's
bits do not depend on the split."""
import numpy as np
import pytest

from oracle.oracle import Run
from tests.helpers import face_ghost_mask, interior, oracle_params
from tests.test_gpu_step import smooth_state
from tests.test_gpu_tiling import BC
from tlaloque_gb300 import tlq

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("limiter,solver", [(tlq.LIMITER_VANLEER, tlq.SOLVER_HLLC), (tlq.LIMITER_VANLEER, tlq.SOLVER_HLL),
                                            (tlq.LIMITER_MINMOD, tlq.SOLVER_HLLC), (tlq.LIMITER_MINMOD, tlq.SOLVER_HLL)])
@pytest.mark.parametrize("shape", [(16, 8, 41), (19, 11, 26)])
def test_instances_on_every_split(gpu_lib, shape, limiter, solver):
    nx, ny, nz = shape
    cfg = tlq.Config(nx=nx, ny=ny, nz=nz, xl=0.0, xr=1.0, yl=0.0, yr=0.6, zl=0.0, zr=0.7, limiter=limiter,
                     solver=solver, bc=BC)
    U0 = smooth_state(cfg, seed=nz, mach=0.8)
    steps = 3
    ref = Run(oracle_params(cfg), U0)
    ref.run(steps)
    m = face_ghost_mask(cfg)
    for precision in (tlq.PREC_FP64, tlq.PREC_MIXED):
        ran, first = [], None
        for zlen in (None, 8, nz):
            U1 = U0.copy(order="F")
            with tlq.Context(tlq.Config(**{**cfg.__dict__, "precision": precision})) as ctx:
                if zlen:
                    ctx.set_tiling(zlen)
                ran.append(ctx.running_tiling())
                ctx.borders(U1, 1)
                ctx.upload(U1)
                ctx.advance(steps)
                t, it, dt, rc = ctx.time()
                U = ctx.state()[0]
            assert rc == tlq.OK and it == steps
            if precision == tlq.PREC_FP64:
                assert (t, dt) == (ref.t, ref.dt)
                np.testing.assert_array_equal(U[:, m], ref.U[:, m])
            else:
                first = first or (U, t, dt)
                assert (t, dt) == first[1:]
                np.testing.assert_array_equal(interior(U), interior(first[0]))
        assert ran[0] < 3 and ran[1:] == [8, nz]

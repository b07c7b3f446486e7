"""The stage kernels at the edges of their tiles and at every way z is split:
the default (meshes too small to fill the GPU run chunks below 8 planes), the
shortest choice and a single chunk.  Plain FP64 is the oracle's bits; the
mixed form's bits do not depend on the split."""
import numpy as np
import pytest

from oracle.oracle import Run
from tests.helpers import face_ghost_mask, interior, oracle_params
from tests.test_gpu_step import smooth_state
from tlaloque_gb300 import tlq

pytestmark = pytest.mark.gpu

BC = (tlq.BC_REFLECTIVE, tlq.BC_OUTFLOW, tlq.BC_PERIODIC, tlq.BC_PERIODIC, tlq.BC_OUTFLOW, tlq.BC_REFLECTIVE)
PAIRS = [(tlq.LIMITER_VANLEER, tlq.SOLVER_HLLC), (tlq.LIMITER_MINMOD, tlq.SOLVER_HLL)]  # both kernel instances


def run(cfg, U0, zlen, steps):
    U1 = U0.copy(order="F")
    with tlq.Context(cfg) as ctx:
        if zlen:
            ctx.set_tiling(zlen)
            assert ctx.tiling() == min(zlen, cfg.nz)
        ctx.borders(U1, 1)
        ctx.upload(U1)
        ctx.advance(steps)
        t, it, dt, rc = ctx.time()
        assert rc == tlq.OK and it == steps
        return ctx.state()[0], (t, dt)


@pytest.mark.parametrize("shape", [(2, 2, 2), (3, 5, 1 + 1), (16, 8, 9), (17, 9, 17), (15, 7, 23), (33, 20, 25)])
@pytest.mark.parametrize("limiter,solver", PAIRS)
def test_every_split_gives_the_same_bits(gpu_lib, shape, limiter, solver):
    nx, ny, nz = shape
    cfg = tlq.Config(nx=nx, ny=ny, nz=nz, xl=0.0, xr=1.0, yl=0.0, yr=0.6, zl=0.0, zr=0.7, limiter=limiter,
                     solver=solver, bc=BC)
    U0 = smooth_state(cfg, seed=nx, mach=0.8)
    steps = 3
    ref = Run(oracle_params(cfg), U0)
    ref.run(steps)
    m = face_ghost_mask(cfg)
    mixed = tlq.Config(**{**cfg.__dict__, "precision": tlq.PREC_MIXED})
    first = None
    for zlen in (0, 8, nz):
        U, (t, dt) = run(cfg, U0, zlen, steps)
        assert (t, dt) == (ref.t, ref.dt)
        np.testing.assert_array_equal(U[:, m], ref.U[:, m])
        V, tm = run(mixed, U0, zlen, steps)
        first = first or (V, tm)
        assert tm == first[1]
        np.testing.assert_array_equal(interior(V), interior(first[0]))

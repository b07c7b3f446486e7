"""Set-up calls that copy from the host and launch a kernel on the context's
stream (which waits for no other stream) leave no copy that the kernel does
not wait for.  Host side only, on a fake CUDA runtime."""
import numpy as np
import pytest

from tests import fakecuda
from tests.test_host_winds import set_winds, wind
from tlaloque_gb300 import problems, tlq


@pytest.fixture(scope="module")
def fake_lib(tmp_path_factory):
    return fakecuda.link(tmp_path_factory.mktemp("fakecuda"))


@pytest.mark.parametrize("precision", [tlq.PREC_FP64, tlq.PREC_MIXED])
def test_set_up_copies_are_ordered(fake_lib, precision):
    T, logL = problems.synthetic_cooling_table()
    cooling = tlq.COOL_MLP if precision == tlq.PREC_MIXED else tlq.COOL_EXACT
    cfg = tlq.Config(nx=32, ny=32, nz=32, precision=precision, cooling=cooling, cool_T=T, cool_logL=logL,
                     masses=np.array([[0.0, 0.0, 0.0, 1.0]]), winds=[wind(0.0)])
    with fakecuda.loaded(fake_lib) as fake:
        ctx = tlq.Context(cfg)
        if cooling == tlq.COOL_MLP:
            ctx.set_cooling_surrogate(np.zeros(8641, np.float32), np.ones(6, np.float32), [0, 1, 0, 1, 0, 1])
        ctx.upload(np.ones(cfg.shape, order="F"))
        ctx.advance(1)
        set_winds(ctx, [wind(0.1), wind(0.2)])
        ctx.advance(1)
        assert fake.launches() and fake.calls("fake_unordered") == 0
        ctx.close()

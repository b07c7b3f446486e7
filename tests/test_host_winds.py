"""tlq_set_winds called again and again (a program that moves its winds each
step): buffers kept while they are large enough, one launch, one wait.  Host
side only, on a fake CUDA runtime."""
import pytest

from tests import fakecuda
from tlaloque_gb300 import tlq


@pytest.fixture(scope="module")
def fake_lib(tmp_path_factory):
    return fakecuda.link(tmp_path_factory.mktemp("fakecuda"))


def set_winds(ctx, winds):
    arr = (tlq.CWind * max(1, len(winds)))()
    for q, w in enumerate(winds):
        for f, _ in tlq.CWind._fields_:
            setattr(arr[q], f, float(getattr(w, f)))
    ctx._check(ctx.L.tlq_set_winds(ctx.h, arr, len(winds)), "set_winds")


def wind(x, radius=0.2):
    return tlq.Wind(xc=x, radius=radius, mdot=1.0, vinf=1.0)


@pytest.mark.parametrize("precision", [tlq.PREC_FP64, tlq.PREC_MIXED])
def test_winds_set_again(fake_lib, precision):
    with fakecuda.loaded(fake_lib) as fake:
        before = fake.bytes()
        ctx = tlq.Context(tlq.Config(nx=48, ny=48, nz=48, precision=precision))
        none = fake.bytes()
        set_winds(ctx, [wind(0.0), wind(0.3), wind(0.5)])
        some = fake.bytes()
        assert some > none
        for winds in ([wind(0.1), wind(0.2), wind(0.4)], [wind(-0.2)], [wind(0.0, 0.1), wind(0.2)]):
            fake.reset()
            set_winds(ctx, winds)
            assert fake.calls("cudaMalloc", "cudaFree", "cudaHostAlloc") == 0
            assert fake.calls("cudaMemcpy", "cudaMemcpyAsync") == 1
            assert fake.calls("cudaStreamSynchronize", "cudaDeviceSynchronize", "cudaEventSynchronize") == 1
            assert len(fake.launches()) == 1
            assert fake.bytes() == some
        set_winds(ctx, [wind(0.0, 0.5)] * 5)  # larger tables, more winds
        assert fake.bytes() > some
        set_winds(ctx, [])
        assert fake.bytes() == none
        ctx.close()
        assert fake.bytes() == before

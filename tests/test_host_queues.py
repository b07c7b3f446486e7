"""What the surrogate's cooling queues take: one word a cell in a single
context, two in a batch member (whose sort pass fills the second).  Host side
only, on a fake CUDA runtime."""
import numpy as np
import pytest

from tests import fakecuda
from tlaloque_gb300 import problems, tlq


@pytest.fixture(scope="module")
def fake_lib(tmp_path_factory):
    return fakecuda.link(tmp_path_factory.mktemp("fakecuda"))


def test_queue_memory(fake_lib):
    T, logL = problems.synthetic_cooling_table()
    n = 40

    def config(cooling):
        return tlq.Config(nx=n, ny=n, nz=n, precision=tlq.PREC_MIXED, cooling=cooling, cool_T=T, cool_logL=logL)

    with fakecuda.loaded(fake_lib) as fake:
        start = fake.bytes()

        def taken(make):
            obj = make()
            size = fake.bytes() - start
            obj.close()
            assert fake.bytes() == start
            return size

        plain, net = (taken(lambda: tlq.Context(config(c))) for c in (tlq.COOL_EXACT, tlq.COOL_MLP))
        assert net - plain == 4 * n**3 + 3 * 4
        plain, net = (taken(lambda: tlq.Batch([config(c)])) for c in (tlq.COOL_EXACT, tlq.COOL_MLP))
        assert net - plain == 8 * n**3 + 3 * 4


def test_batch_member_alone(fake_lib):
    """A batch member stepped by itself takes the single launch."""
    T, logL = problems.synthetic_cooling_table()
    cfg = tlq.Config(nx=32, ny=32, nz=32, precision=tlq.PREC_MIXED, cooling=tlq.COOL_MLP, cool_T=T, cool_logL=logL)
    with fakecuda.loaded(fake_lib) as fake:
        b = tlq.Batch([cfg])
        m = b.members[0]
        m.set_cooling_surrogate(np.zeros(8641, np.float32), np.ones(6, np.float32), [0, 1, 0, 1, 0, 1])
        m.upload(np.ones(cfg.shape, order="F"))
        fake.reset()
        m.advance(1)
        b.run(1)
        names = [k for k in ("k_cool_all", "k_cool_sort", "k_cool_net", "k_cool_dt") if fake.launches(k)]
        assert names == ["k_cool_all", "k_cool_sort", "k_cool_net", "k_cool_dt"]
        b.close()

"""The self-gravity solver's launches on several devices of one process
(tlq_config.device): what a kernel may use belongs to the device.  Host side
only, on a fake CUDA runtime with two devices."""
import numpy as np
import pytest

from tests import fakecuda
from tlaloque_gb300 import problems, tlq


@pytest.fixture(scope="module")
def fake_lib(tmp_path_factory):
    return fakecuda.link(tmp_path_factory.mktemp("fakecuda"))


def solve(device, n):
    cfg, U = problems.gravitating_cloud(n, grav_bc=tlq.GBC_ZERO)
    with tlq.Context(tlq.Config(**{**cfg.__dict__, "device": device})) as ctx:
        ctx.upload(np.asfortranarray(U))
        ctx.advance(2)


@pytest.mark.parametrize("n", [16, 64])
def test_plane_relax_on_a_second_device(fake_lib, n):
    """A 64-cell level's plane takes more than 48 KB of shared memory: an
    attribute of the kernel on each device."""
    with fakecuda.loaded(fake_lib) as fake:
        for device in (0, 1, 0):
            fake.reset()
            solve(device, n)
            planes = [d for k, g, d in fake.launches("k_mg_relax_plane") if g[0] == n]
            assert planes and set(planes) == {device}
            assert not fake.launches("k_mg_relax_pipe")


def test_refused_plane_launch_falls_back(fake_lib):
    """A relax whose launch is refused runs in another form, and the solve
    does not report the refusal."""
    with fakecuda.loaded(fake_lib) as fake:
        fake.fail("k_mg_relax_plane")
        solve(0, 32)
        assert not fake.launches("k_mg_relax_plane")
        assert fake.launches("k_mg_relax_pipe")

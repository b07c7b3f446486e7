"""The z-chunk length: a length that is set is the one that runs, the default
is split for meshes too small to fill the GPU, and the autotuners try the
default beside the lengths.  Host side only, on a fake CUDA runtime whose
launches take a time set per number of blocks."""
import json

import numpy as np
import pytest

from tests import fakecuda
from tlaloque_gb300 import problems, tlq


@pytest.fixture(scope="module")
def fake_lib(tmp_path_factory):
    return fakecuda.link(tmp_path_factory.mktemp("fakecuda"))


def config(shape, precision=tlq.PREC_FP64):
    nx, ny, nz = shape
    return tlq.Config(nx=nx, ny=ny, nz=nz, precision=precision)


def uploaded(cfg):
    ctx = tlq.Context(cfg)
    ctx.upload(np.ones(cfg.shape, order="F"))
    return ctx


def chunks(fake, ctx):
    """The z extent of the two stages' grids in one step."""
    fake.lib.fake_reset()
    ctx.advance(1)
    z = {g[2] for k, g, _ in fake.launches("stage_kernel")}
    assert len(z) == 1 and len(fake.launches("stage_kernel")) == 2
    return z.pop()


@pytest.mark.parametrize("precision", [tlq.PREC_FP64, tlq.PREC_MIXED])
@pytest.mark.parametrize("shape", [(16, 8, 9), (33, 20, 25), (48, 48, 48), (64, 64, 70), (150, 150, 150)])
def test_a_length_that_is_set_runs(fake_lib, shape, precision):
    nz = shape[2]
    with fakecuda.loaded(fake_lib) as fake:
        ctx = uploaded(config(shape, precision))
        run = ctx.running_tiling()
        assert chunks(fake, ctx) == -(-nz // run)
        assert ctx.tiling() >= run and ctx.tiling() >= min(8, nz)
        assert run < 8 or shape[0] >= 100
        for z in (8, 16, nz, nz + 5):
            ctx.set_tiling(z)
            assert ctx.tiling() == ctx.running_tiling() == min(z, nz)
            assert chunks(fake, ctx) == -(-nz // min(z, nz))
        for z in (-1, 0, 1, 7):
            with pytest.raises(tlq.TlqError):
                ctx.set_tiling(z)
        ctx.close()


def blocks(shape, z):
    return -(-shape[0] // 16) * -(-shape[1] // 8) * -(-shape[2] // z)


@pytest.mark.parametrize("shape", [(48, 48, 48), (150, 150, 150)])
@pytest.mark.parametrize("winner", ["default", 8, 16, 32])
def test_autotune_tries_the_default(fake_lib, tmp_path, shape, winner):
    cache = str(tmp_path / "tune.json")
    with fakecuda.loaded(fake_lib) as fake:
        ctx = uploaded(config(shape, tlq.PREC_MIXED))
        default, nominal = ctx.running_tiling(), ctx.tiling()
        run = default if winner == "default" else winner
        ctx.set_tiling(shape[2])  # (not where the tuner starts from)
        fake.set_cost(blocks(shape, run), 0.25)
        got = ctx.autotune(cache, steps=2)
        assert ctx.running_tiling() == run
        assert got == ctx.tiling() == (nominal if winner == "default" else winner)
        (entry,) = json.load(open(cache))["tuned"].values()
        assert entry["zlen"] == winner
        ctx.close()
        ctx = uploaded(config(shape, tlq.PREC_MIXED))
        fake.lib.fake_reset()
        assert ctx.autotune(cache, steps=2) == got and ctx.running_tiling() == run
        assert not fake.launches("stage_kernel")  # (from the cache)
        ctx.close()


@pytest.mark.parametrize("winner", ["default", 8, 16])
def test_batch_autotune_tries_the_default(fake_lib, tmp_path, winner):
    cache = str(tmp_path / "tune.json")
    shapes = [(48, 48, 48), (32, 32, 32), (48, 48, 48)]
    with fakecuda.loaded(fake_lib) as fake:
        def batch():
            b = tlq.Batch([config(s, tlq.PREC_MIXED) for s in shapes])
            for m in b.members:
                m.upload(np.ones(m.cfg.shape, order="F"))
            return b

        b = batch()
        default = b.running_tiling()
        assert max(default) < 8 and b.tiling() == [8, 8, 8]
        wins = default if winner == "default" else [winner] * 3
        fake.set_cost(sum(blocks(s, z) for s, z in zip(shapes, wins)), 0.25)
        got = b.autotune(cache, steps=2)
        assert got == b.tiling() == ([8] * 3 if winner == "default" else [winner] * 3)
        assert b.running_tiling() == (default if winner == "default" else [winner] * 3)
        assert {e["zlen"] for e in json.load(open(cache))["tuned"].values()} == {winner}
        b.set_tiling(1, 16)
        assert b.tiling()[1] == b.running_tiling()[1] == 16
        fake.lib.fake_reset()
        b.run(1)
        items = {g[0] for k, g, _ in fake.launches("stage_kernel_mixed_batch")}
        assert items == {sum(blocks(s, z) for s, z in zip(shapes, b.running_tiling()))}
        b.close()
        b = batch()
        fake.lib.fake_reset()
        assert b.autotune(cache, steps=2) == got
        assert not fake.launches("stage_kernel")
        b.close()


def stages(fake):
    return len(fake.launches("stage_kernel"))


def test_equal_launches_are_timed_once(fake_lib, tmp_path):
    """Each running length once (64 planes: the default is one of the lengths),
    nothing timed or cached where there is one, and a hopeless candidate left
    after its first step."""
    cache = tmp_path / "tune.json"
    with fakecuda.loaded(fake_lib) as fake:
        ctx = uploaded(config((128, 128, 128), tlq.PREC_MIXED))
        assert ctx.running_tiling() == 8
        fake.lib.fake_reset()
        ctx.autotune(str(cache), steps=4)
        # captured per candidate and parity, launched 1 + 4 times
        assert stages(fake) == 5 * 2 * 2 and len({g for _, g, _ in fake.launches("stage_kernel")}) == 5
        ctx.close()
        ctx = uploaded(config((512, 256, 8)))
        assert ctx.running_tiling() == 8
        fake.lib.fake_reset()
        assert ctx.autotune(str(tmp_path / "none.json"), steps=4) == 8
        assert stages(fake) == 0 and not (tmp_path / "none.json").exists()
        ctx.close()
        shape = (48, 48, 48)
        b = tlq.Batch([config(shape, tlq.PREC_MIXED)])
        b.members[0].upload(np.ones(b.members[0].cfg.shape, order="F"))
        default = b.running_tiling()[0]
        fake.lib.fake_reset()
        fake.set_cost(blocks(shape, default), 0.25)
        fake.set_cost(blocks(shape, 16), 0.45)
        b.autotune(None, steps=4)
        # the default: 1 + 4 steps; 8, 16 and 32 planes: 1 step
        assert b.running_tiling() == [default] and stages(fake) == 2 * (5 + 1 + 1 + 1)
        b.close()


@pytest.mark.parametrize("share,kept", [(0.995, True), (0.985, False), (0.9, False)])
def test_batch_keeps_the_default_for_a_small_gain(fake_lib, share, kept):
    shape = (48, 48, 48)
    with fakecuda.loaded(fake_lib) as fake:
        b = tlq.Batch([config(shape, tlq.PREC_MIXED)])
        b.members[0].upload(np.ones(b.members[0].cfg.shape, order="F"))
        default = b.running_tiling()[0]
        fake.set_cost(blocks(shape, 16), share)
        b.autotune(None, steps=3)
        assert b.running_tiling() == [default if kept else 16]
        b.close()


def test_batch_is_timed_with_all_members(fake_lib, tmp_path):
    """Every timed launch holds all members' tiles; after one length for all
    sizes, a size may take half or twice of it; a size in the cache keeps its."""
    cache = tmp_path / "tune.json"
    shapes = [(64, 64, 64), (32, 32, 32), (48, 48, 48)]

    def items(z):
        return sum(blocks(s, q) for s, q in zip(shapes, z))

    with fakecuda.loaded(fake_lib) as fake:
        b = tlq.Batch([config(s, tlq.PREC_MIXED) for s in shapes])
        for m in b.members:
            m.upload(np.ones(m.cfg.shape, order="F"))
        default = b.running_tiling()
        fake.set_cost(items([16, 16, 16]), 0.5)
        fake.set_cost(items([32, 16, 16]), 0.25)
        fake.set_cost(items([16, 8, 16]), 0.4999)  # (not gain enough)
        before = len(fake.launches("stage_kernel"))
        assert b.autotune(str(cache), steps=2) == [32, 16, 16] == b.running_tiling()
        timed = {g[0] for k, g, _ in fake.launches("stage_kernel")[before:]}
        lengths = [default] + [[min(z, s[2]) for s in shapes] for z in (8, 16, 32, 64)]
        lengths += [[16, 8, 16], [16, 32, 16], [16, 16, 8], [16, 16, 32], [8, 16, 16], [32, 16, 16]]
        assert timed == {items(z) for z in lengths}
        b.close()
        doc = json.load(open(cache))
        del doc["tuned"]["48x48x48/batch_mixed"]
        lines = ",\n".join(f'    "{k}": {{"zlen": {v["zlen"]}, "ms_per_step": {v["ms_per_step"]:.6f}}}'
                           for k, v in doc["tuned"].items())
        cache.write_text('{\n  "gpu": "fake",\n  "tuned": {\n' + lines + "\n  }\n}\n")
        fake.reset()
        fake.set_cost(items([32, 16, 8]), 0.25)
        b = tlq.Batch([config(s, tlq.PREC_MIXED) for s in shapes])
        for m in b.members:
            m.upload(np.ones(m.cfg.shape, order="F"))
        assert b.autotune(str(cache), steps=2) == [32, 16, 8]
        b.close()

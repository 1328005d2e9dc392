"""The mixed state's device layout ([block][half][cell][4], its correction
[block][interior cell][8]) as seen from outside: restart files keep their
[block][variable][cell] order, and blocks split over several CTAs give the
unsplit step's bits."""
import numpy as np
import pytest

import falcon_gb300 as fg
from falcon_gb300 import config, synth

pytestmark = pytest.mark.gpu

HEADER = 80   # bytes before the arrays of a restart file


@pytest.mark.parametrize("block,tiles", [(8, (1, 2, 6)), (16, (1, 1, 3))])
def test_restart_file_holds_the_state_variable_by_variable(tmp_path, block, tiles):
    cfg = config.make_config(block=(block,) * 3, root_tiles=tiles, radial_levels=1, amr=(), precision=config.PREC_MIXED)
    f = fg.Falcon(cfg)
    u = synth.initial_state(cfg, f.block_ranges(), f.block_flags(), seed=77)
    f.upload_state(u)
    path = str(tmp_path / "run.rst")
    f.save_restart(path)
    u = f.download_state()[:, :8]
    raw = np.fromfile(path, dtype=np.uint8)[HEADER:]
    hi = raw[:u.size * 4].view(np.float32).reshape(u.shape)
    lo = raw[u.size * 4:].view(np.int8)[:u.shape[0] * 8 * block ** 3].reshape(u.shape[0], 8, block, block, block)
    assert np.array_equal(hi, u.astype(np.float32))
    inner = (slice(None), slice(None)) + (slice(2, -2),) * 3
    e = (hi[inner].view(np.int32) >> 23) & 0xff
    unit = np.where(e >= 32, np.ldexp(1.0, e - 158), 0.0)
    assert np.any(lo)
    assert np.array_equal(hi[inner].astype(np.float64) + lo * unit, u[inner])
    g = fg.Falcon(cfg)
    g.load_restart(path)
    assert np.array_equal(g.download_state()[:, :8], u)


@pytest.mark.parametrize("tiles", [(1, 1, 3), (1, 2, 6), (1, 3, 9), (2, 3, 9)])
def test_split_blocks_step_as_whole_ones(tiles):
    """Grids of few 16^3 blocks run several CTAs per block (2 to 8 parts in these
    grids of 12 to 216 blocks); the persistent step never splits."""
    cfg = config.make_config(block=(16, 16, 16), root_tiles=tiles, radial_levels=1, radial_option=1, amr=(),
                             precision=config.PREC_MIXED)
    a, b = fg.Falcon(cfg), fg.Falcon(cfg)
    b.set_step_mode(fg.STEP_PERSISTENT)
    u = synth.initial_state(cfg, a.block_ranges(), a.block_flags(), seed=78)
    for x in (a, b):
        x.upload_state(u)
        x.exchange()
    assert [a.advance_rk4() for _ in range(3)] == [b.advance_rk4() for _ in range(3)]
    ua = a.download_state()
    assert np.isfinite(ua).all()
    assert np.array_equal(ua, b.download_state())


@pytest.mark.parametrize("block,tiles", [(8, (1, 2, 6)), (16, (1, 1, 3))])
def test_denormal_fields_stay_small(block, tiles):
    """The limiter's quotient flushes a denormal jump: its flux stays of the size of
    the jumps themselves. A field of noise below the smallest normal number
    (jumps to 4e-39) takes fluxes of at most 8 times three jumps and the step's
    CFL number below 1, so it stays below 1e-36."""
    cfg = config.make_config(block=(block,) * 3, root_tiles=tiles, radial_levels=1, amr=(), precision=config.PREC_MIXED)
    f = fg.Falcon(cfg)
    u = synth.initial_state(cfg, f.block_ranges(), f.block_flags(), seed=79)
    rng = np.random.default_rng(79)
    u[:, 4:7] = rng.uniform(-2e-39, 2e-39, u[:, 4:7].shape)
    f.upload_state(u)
    f.exchange()
    for _ in range(2):
        f.advance_rk4()
    out = f.download_state()
    assert np.isfinite(out).all()
    assert np.abs(out[:, 4:7]).max() < 1e-36

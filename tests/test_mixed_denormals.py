"""The mixed diffusion on a field whose jumps lie below FP32's normal range: the limiter
acts on them as on any jump (both slopes are 0 there, phi = 1)."""
import numpy as np
import pytest

import falcon_gb300 as fg
import oracle
from falcon_gb300 import config

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("block,tiles", [(8, (1, 2, 6)), (16, (1, 1, 3))])
def test_diffusion_of_denormal_jumps_is_the_oracles(built_lib, oracle_lib, block, tiles):
    mk = lambda **kw: config.make_config(block=(block,) * 3, root_tiles=tiles, radial_levels=1, amr=(), **kw)
    f, o = fg.Falcon(mk(precision=config.PREC_MIXED)), oracle.Oracle(mk(device=-1))
    u = np.zeros(f.shape)
    # whole multiples of 2^-149, below 2^-126: FP32 holds the values exactly
    u[:, 7] = np.random.default_rng(5).integers(-(1 << 22), 1 << 22, u[:, 7].shape) * 2.0 ** -149
    f.upload_state(u)
    o.set_state(u)
    for x in (f, o):
        x.exchange()
        x.exchange()
    f.step_phase(0)
    o.phase(0)
    f.step_phase(5)
    o.phase(5)
    g, r = f.download_state()[:, 7, 2:-2, 2:-2, 2:-2], o.get_state()[:, 7, 2:-2, 2:-2, 2:-2]
    moved = np.abs(r - u[:, 7, 2:-2, 2:-2, 2:-2]).max()
    assert moved > 1e5 * 2.0 ** -149   # the diffusion acts
    # a ghost is rounded to 2^-149 and a cell's flux sum and update round some ten times; dt
    # and the geometry are FP32 values (2^-24 of 2^22 units, some ten of them): below 100 units
    assert np.abs(g - r).max() <= 100 * 2.0 ** -149
    f.close()

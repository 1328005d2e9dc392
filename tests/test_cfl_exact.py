"""The FP64 CFL minimum: cells are screened by an FP32 estimate of their ratio, the dt is
the oracle's bits whatever the speeds: even ones, one fast cell, values beyond FP32's
range on either side, ratios that differ in their last bits."""
import numpy as np
import pytest

import falcon_gb300 as fg
import oracle
from falcon_gb300 import config

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("block,tiles", [(8, (1, 2, 6)), (16, (1, 1, 3))])
@pytest.mark.parametrize("kind", ["zero", "even", "one", "binades", "large", "small"])
def test_timestep_is_the_oracles(built_lib, oracle_lib, block, tiles, kind):
    mk = lambda **kw: config.make_config(block=(block,) * 3, root_tiles=tiles, radial_levels=1, amr=(), **kw)
    f, o = fg.Falcon(mk()), oracle.Oracle(mk(device=-1))
    rng = np.random.default_rng(17)
    u = np.zeros(f.shape)
    s = u[:, 1:7]
    if kind == "even":
        s[:] = 0.25 * (1.0 + 1e-15 * rng.integers(-4, 5, s.shape))
    elif kind == "one":
        s[:] = 0.01
        s[s.shape[0] // 2, :, 5, 6, 7] = 3.0
    elif kind == "binades":
        s[:] = rng.standard_normal(s.shape) * 2.0 ** rng.integers(-200, 20, s.shape)
    elif kind == "large":
        s[:] = rng.standard_normal(s.shape) * 1e30
    elif kind == "small":
        s[:] = rng.standard_normal(s.shape) * 1e-160
    f.upload_state(u)
    o.set_state(u)
    assert f.timestep() == o.timestep()

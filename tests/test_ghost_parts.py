"""The FP64 exchange with one, two and four threads per interpolated entry (by the length of
the list) against the oracle, bit for bit."""
import numpy as np
import pytest

import falcon_gb300 as fg
import oracle
from falcon_gb300 import config

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tiles,most", [((1, 2, 6), 100000), ((2, 3, 9), 320000), ((2, 3, 18), 1 << 30)])
def test_exchange_is_the_oracles_with_any_number_of_threads(built_lib, oracle_lib, tiles, most):
    mk = lambda **kw: config.make_config(block=(8,) * 3, root_tiles=tiles, radial_levels=1, amr=(), **kw)
    f, o = fg.Falcon(mk()), oracle.Oracle(mk(device=-1))
    n = f.ghost_list_sizes()["trilinear"]
    assert n <= most and (most == 100000 or n > (100000 if most == 320000 else 320000))
    rng = np.random.default_rng(12)
    u = np.zeros(f.shape)
    u[:, :8] = rng.standard_normal(u[:, :8].shape) * 2.0 ** rng.integers(-20, 20, u[:, :8].shape)
    f.upload_state(u)
    o.set_state(u)
    f.exchange()
    o.exchange()
    assert np.array_equal(f.download_state(), o.get_state())
    f.close()

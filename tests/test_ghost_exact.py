"""The FP64 ghost fill forms the products with weights within 1e-13 of 0 and 1 by integer
arithmetic on the significands; its results are the CPU oracle's bits whatever the
values: smooth, noise over many binades, next to powers of two, zeros, denormals."""
import numpy as np
import pytest

import falcon_gb300 as fg
import oracle
from falcon_gb300 import config

pytestmark = pytest.mark.gpu


def _values(kind, shape, rng):
    if kind == "smooth":
        return 1.5 + 1e-6 * rng.standard_normal(shape)
    if kind == "noise":
        return rng.standard_normal(shape) * 2.0 ** rng.integers(-60, 60, shape)
    if kind == "binade":
        return 2.0 ** rng.integers(-3, 3, shape) * (1.0 + rng.integers(-40, 40, shape) * 2.0 ** -53)
    if kind == "ties":
        return 1.25 + rng.integers(-3, 4, shape) * 2.0 ** -52
    return np.where(rng.random(shape) < 0.5, 0.0, rng.standard_normal(shape) * 10.0 ** rng.choice([-320.0, -300.0, 0.0, 300.0], shape))


@pytest.mark.parametrize("block,tiles", [(8, (1, 2, 6)), (16, (1, 1, 3))])
@pytest.mark.parametrize("kind", ["smooth", "noise", "binade", "ties", "extremes"])
def test_exchange_is_the_oracles_for_any_values(built_lib, block, tiles, kind):
    mk = lambda **kw: config.make_config(block=(block,) * 3, root_tiles=tiles, radial_levels=1,
                                         amr=((0, 1, 1),) if block == 8 else (), **kw)
    f, o = fg.Falcon(mk()), oracle.Oracle(mk(device=-1))
    rng = np.random.default_rng(91)
    u = np.zeros(f.shape)
    u[:, :8] = _values(kind, u[:, :8].shape, rng)
    f.upload_state(u)
    o.set_state(u)
    f.exchange()
    o.exchange()
    assert np.array_equal(f.download_state()[:, :8], o.get_state()[:, :8], equal_nan=True)

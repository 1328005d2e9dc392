"""The FP64 kernels' short forms (integer minmod selector, faces that skip
their division, quotients by reciprocals, shared point fields) on states that
reach their edges: constant regions, single extrema, differences at the
selector's threshold, magnitudes over hundreds of binades. Every phase must
leave the oracle's bits."""
import numpy as np
import pytest

import falcon_gb300 as fg
import oracle
from falcon_gb300 import config, synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built(built_lib):
    return built_lib


def _rough(shape, kind, seed):
    rs = np.random.default_rng(seed)
    u = np.zeros(shape)
    s = u[:, :8]
    if kind == "constant":
        s[:] = rs.integers(-1, 2, size=s.shape)
    elif kind == "threshold":     # |a| |b|^2 |c| about 1e-40
        s[:] = 2.0 ** -33 * rs.uniform(-1, 1, size=s.shape) * 2.0 ** rs.integers(-2, 3, size=s.shape)
    elif kind == "extremum":
        s[:] = 3.0
        s[:, :, ::3, ::4, ::5] = rs.uniform(-5, 5, size=s[:, :, ::3, ::4, ::5].shape)
    else:
        s[:] = rs.uniform(-1, 1, size=s.shape) * 2.0 ** rs.integers(-270, 120, size=s.shape)
    return u


@pytest.mark.parametrize("block,tiles", [(8, (1, 2, 6)), (16, (1, 1, 3))])
@pytest.mark.parametrize("kind", ["constant", "threshold", "extremum", "binades"])
def test_diffusion_of_rough_states_is_the_oracles(block, tiles, kind):
    mk = lambda **kw: config.make_config(block=(block,) * 3, root_tiles=tiles, radial_levels=1, amr=(), **kw)
    f, o = fg.Falcon(mk()), oracle.Oracle(mk(device=-1))
    u = _rough(f.shape, kind, 11)
    f.upload_state(u)
    o.set_state(u)
    for x in (f, o):
        x.exchange()
        x.exchange()
    f.step_phase(0)
    o.phase(0)
    f.step_phase(5)
    o.phase(5)
    assert np.array_equal(f.download_state(), o.get_state())
    f.close()


@pytest.mark.parametrize("block,tiles,divb", [(8, (1, 2, 6), 0), (8, (1, 2, 6), 1), (16, (1, 1, 3), 0), (16, (1, 1, 3), 2)])
def test_steps_from_noise_are_the_oracles(block, tiles, divb):
    mk = lambda **kw: config.make_config(block=(block,) * 3, root_tiles=tiles, radial_levels=1, amr=(), divb_option=divb, **kw)
    f, o = fg.Falcon(mk()), oracle.Oracle(mk(device=-1))
    u = synth.initial_state(mk(), o.block_ranges(), o.block_flags(), seed=3, psi_amp=1e-3 if divb == 1 else 0.0)
    u[:, 1:4] += 1e3 * np.random.default_rng(4).standard_normal(u[:, 1:4].shape)
    f.upload_state(u)
    o.set_state(u)
    for x in (f, o):
        x.exchange()
        x.exchange()
    for _ in range(2):
        assert f.advance_rk4() == o.step()
        assert np.array_equal(f.download_state(), o.get_state())
    f.close()

"""The clear-sky kernels against the oracle at the edges of their tiles: profile
counts around the groups of 4 and 8 profiles and the CTAs of 16 and 32, channel
counts around the 32- and 64-channel tiles, layer counts at both ends of the
range, ragged batches.  Tolerances as in test_gpu_parity: FP64 form 1e-4 K and
1e-6 of the largest Jacobian, mixed form 0.01 K and 1e-3 (absorbers ten times
that)."""
import numpy as np
import pytest

from crtmv3_gb300 import synthetic as sy

pytestmark = pytest.mark.gpu

BT_TOL = {0: 1e-4, 1: 1e-2}
JAC_TOL = {0: 1e-6, 1: 1e-3}


def _rel(a, b):
    return np.abs(a - b).max() / max(np.abs(b).max(), 1e-300)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("sensor,channels,profiles,layers", [
    ("mwsynth_c22", 0, 3, (40, 40)), ("mwsynth_c22", 5, 17, (60, 137)),
    ("irsynth_c616", 31, 33, (90, 110)), ("irsynth_c616", 33, 9, (100, 100)), ("irsynth_c616", 65, 8, (127, 129)),
    ("irsynth_c616", 64, 4, (30, 200)), ("irsynth_c616", 0, 2, (199, 200))])
def test_tile_edges_match_oracle(gpu_lib, coeff_dir, sensor, channels, profiles, layers, precision):
    from oracle.pyoracle import Oracle
    rng = np.random.default_rng(channels + 100 * profiles)
    nl = rng.integers(layers[0], layers[1] + 1, profiles)
    nl[0], nl[-1] = layers
    atm, sfc, geo, opt = sy.clear_sky_workload(sensor, profiles, nl, 4000 + profiles)
    ref = Oracle(coeff_dir, sensor).k_matrix(atm, sfc, geo, opt)
    h = gpu_lib.CRTM([sensor], coeff_dir, precision)
    pos = slice(None)
    if channels:
        pos = np.sort(rng.choice(sy.SENSORS[sensor][1], channels, replace=False))
        h.set_channel_subset(0, pos)
        opt.emissivity = np.ascontiguousarray(opt.emissivity[:, pos])
    rts = h.forward(atm, sfc, geo, opt)
    assert np.abs(rts.brightness_temperature - ref["bt"][:, pos]).max() < BT_TOL[precision]
    km, rts = h.k_matrix(atm, sfc, geo, opt)
    assert (rts.status == 0).all()
    assert np.abs(rts.brightness_temperature - ref["bt"][:, pos]).max() < BT_TOL[precision]
    assert _rel(km.temperature, ref["temperature_k"][:, pos]) < JAC_TOL[precision]
    for j in range(atm.n_absorbers):
        assert _rel(km.absorber[:, :, j], ref["absorber_k"][:, pos, j]) < JAC_TOL[precision] * 10
    assert _rel(km.water_temperature, ref["water_temperature_k"][:, pos]) < JAC_TOL[precision]
    assert _rel(km.surface_emissivity, ref["surface_emissivity_k"][:, pos]) < JAC_TOL[precision]
    seed = rng.normal(size=rts.radiance.shape)
    ad, _ = h.adjoint(atm, sfc, geo, opt, seed)
    kt = np.einsum("pl,plk->pk", seed, km.temperature)
    assert _rel(ad["temperature"], kt) < (1e-5 if precision else 1e-10)


def test_too_few_layers_refused(gpu_lib, coeff_dir):
    """Two layers: more reference layers in a user layer than its band holds."""
    atm, sfc, geo, opt = sy.clear_sky_workload("mwsynth_c16", 1, np.array([2]), 4001)
    with pytest.raises(RuntimeError, match="0x8"):
        gpu_lib.CRTM(["mwsynth_c16"], coeff_dir, 0).forward(atm, sfc, geo, opt)

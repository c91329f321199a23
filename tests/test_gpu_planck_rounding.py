"""The FP64 form's layer Planck radiance, read where it is an output by itself: the
overcast radiance of the topmost layer (a black cloud there: nothing above it),
against 80-bit or longer arithmetic on the same FP64 constants (band coefficients
0 and 1, so that the effective temperature is the layer's).

B = c1 / (exp(x) - 1), x = c2 / te, u = 2^-53, r = e^x / (e^x - 1).  One rounding
of x leaves an error uniform within half its spacing s, rms s / sqrt(12), times r
in B; the exponential's is 2 u at most, times r; the subtraction's and the
division's have rms u / sqrt(3) at most each.  So over the samples
rms(dB / B)^2 <= mean(r^2 (s^2 / 12 + 4 u^2) + 2 u^2 / 3).  The channels are those
with x from 10 on, where a second rounding of x would show (twice the first term).
"""
import os

import numpy as np
import pytest

from crtmv3_gb300 import coefficients as co, synthetic as sy

pytestmark = pytest.mark.gpu

U = 2.0 ** -53


@pytest.mark.parametrize("call", ["forward", "k_matrix"])
def test_layer_planck_radiance_rounds_its_exponent_once(gpu_lib, tmp_path, call):
    sensor, P = "irsynth_c2211", 60
    sy.write_sensor_files(str(tmp_path), sensor)
    f = os.path.join(tmp_path, f"{sensor}.SpcCoeff.bin")
    spc = co.read_spccoeff(f)
    spc.band_c1[:], spc.band_c2[:] = 0.0, 1.0
    co.write_spccoeff(f, spc)
    atm, sfc, geo, opt = sy.clear_sky_workload(sensor, P, 40, 41)
    rng = np.random.default_rng(8)
    atm.temperature[:, 0] = rng.uniform(190.0, 300.0, P)
    h = gpu_lib.CRTM([sensor], str(tmp_path), 0)
    if call == "forward":
        rts = h.forward(atm, sfc, geo, opt, components=True)
    else:
        rts = h.k_matrix(atm, sfc, geo, opt, components=True)[1]
    got = rts.upwelling_overcast_radiance[:, :, 0]
    LD = np.longdouble
    assert np.finfo(LD).nmant >= 63
    x = LD(spc.planck_c2)[None] / LD(atm.temperature[:, :1])
    ref = LD(spc.planck_c1)[None] / np.expm1(x)
    x = x.astype(np.float64)
    ok = x >= 10.0
    assert ok.sum() > 2000
    err = ((LD(got) - ref) / ref).astype(np.float64)[ok]
    r = 1.0 / -np.expm1(-x[ok])
    bound = np.sqrt(np.mean(r ** 2 * (np.spacing(x[ok]) ** 2 / 12.0 + 4.0 * U ** 2) + 2.0 / 3.0 * U ** 2))
    assert np.sqrt(np.mean(err ** 2)) <= bound


def test_overflowing_exponential_is_zero_radiance(gpu_lib, coeff_dir):
    """A layer so cold that e^x has no finite value emits nothing: c1 / inf = 0."""
    sensor, P = "irsynth_c2211", 3
    spc = co.read_spccoeff(os.path.join(coeff_dir, f"{sensor}.SpcCoeff.bin"))
    atm, sfc, geo, opt = sy.clear_sky_workload(sensor, P, 40, 43)
    atm.temperature[:, 0] = [1.0, 2.0, 250.0]
    x = spc.planck_c2[None] / (spc.band_c1[None] + spc.band_c2[None] * atm.temperature[:, :1])
    assert (x > 711.0).any(axis=1).tolist() == [True, True, False]
    rts = gpu_lib.CRTM([sensor], coeff_dir, 0).forward(atm, sfc, geo, opt, components=True)
    got = rts.upwelling_overcast_radiance[:, :, 0]
    assert (got[x > 711.0] == 0.0).all() and (got[x < 700.0] > 0.0).all()
    assert np.isfinite(rts.radiance).all() and np.isfinite(rts.brightness_temperature).all()

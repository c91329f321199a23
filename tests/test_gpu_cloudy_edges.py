"""Mixed-form scattering: a (profile, channel)'s results do not depend on what
shares its warps, teams and lists.  A batch of ragged profiles, some clear, of
several stream counts against each profile by itself, and all channels against
subsets around the teams of 8, 4 and 2 channels a warp: the same bits."""
import copy

import numpy as np
import pytest

from crtmv3_gb300 import synthetic as sy

pytestmark = pytest.mark.gpu

FIELDS = ("temperature", "absorber", "water_temperature", "surface_emissivity", "cloud_water_content",
          "cloud_effective_radius")


@pytest.fixture(scope="module")
def cloud_dir(coeff_dir):
    sy.write_cloud_files(coeff_dir)
    return coeff_dir


def _take(batch, i):
    """Profile i of a batch's arrays (by their first dimension)."""
    b = copy.copy(batch)
    for k, v in vars(batch).items():
        if isinstance(v, np.ndarray) and v.ndim and k not in ("absorber_id", "absorber_units"):
            setattr(b, k, np.ascontiguousarray(v[i:i + 1]))
    return b


@pytest.mark.parametrize("sensor,streams,channels", [
    ("mwsynth_c16", None, (1, 7, 9)), ("mwsynth_c16", (16, 8, 16, 8, 8), (1, 3, 5)),
    ("irsynth_c616", None, (1, 31, 33)), ("irsynth_c616", (8, 16, 8, 16, 16), (3, 17, 65))])
def test_results_independent_of_the_batch(gpu_lib, cloud_dir, sensor, streams, channels):
    nl = np.array([60, 101, 33, 101, 97])
    atm, sfc, geo, opt = sy.cloudy_workload(sensor, 5, nl, 777, wc_scale=50.0, n_streams=streams)
    atm.n_clouds[2] = 0
    h = gpu_lib.CRTM([sensor], cloud_dir, 1)
    km, rts = h.k_matrix(atm, sfc, geo, opt)
    fw = h.forward(atm, sfc, geo, opt)
    assert np.isfinite(km.temperature).all() and (rts.status == 0).all()
    for i in (0, 1, 2, 4):
        one = [_take(x, i) for x in (atm, sfc, geo, opt)]
        k1, r1 = h.k_matrix(*one)
        assert np.array_equal(r1.radiance[0], rts.radiance[i])
        assert np.array_equal(h.forward(*one).radiance[0], fw.radiance[i])
        for f in FIELDS:
            assert np.array_equal(getattr(k1, f)[0], getattr(km, f)[i]), (i, f)
    rng = np.random.default_rng(3)
    for n in channels:
        pos = np.sort(rng.choice(rts.radiance.shape[1], n, replace=False))
        hs = gpu_lib.CRTM([sensor], cloud_dir, 1)
        hs.set_channel_subset(0, pos)
        so = copy.copy(opt)
        so.emissivity = np.ascontiguousarray(opt.emissivity[:, pos])
        ks, rs = hs.k_matrix(atm, sfc, geo, so)
        assert np.array_equal(rs.radiance, rts.radiance[:, pos])
        for f in FIELDS:
            assert np.array_equal(getattr(ks, f), getattr(km, f)[:, pos]), (n, f)


def test_static_scratch_without_room_for_the_lists(gpu_lib, cloud_dir):
    """The largest profile that the static scratch takes leaves no room for the
    layers' lists; its layers are then taken in order, with the same bits."""
    import torch
    import bench
    dev = torch.device("cuda")
    sensor = "irsynth_c2211"
    h = gpu_lib.CRTM([sensor], cloud_dir, 1)
    L, stream = h.n_channels[0], torch.cuda.current_stream().cuda_stream

    def call(K, static):
        atm, sfc, geo, opt = sy.cloudy_workload(sensor, 1, K, 778, wc_scale=50.0)
        b, keep, t = bench.scatter_device_inputs(torch, h, atm, sfc, geo, opt, dev)
        out = bench.k_outputs(torch, 1, L, K, atm.n_absorbers, dev)
        h.k_matrix_device(b, out, None, 0, stream, static_scratch=static)
        torch.cuda.synchronize()
        return {f: v.cpu().numpy() for f, v in out.items() if v is not None}

    taken = []
    for K in range(60, 140):
        try:
            taken.append((K, call(K, True)))
        except RuntimeError as e:
            assert "static scratch holds" in str(e)
            break
    assert 60 < taken[-1][0] < 139
    for K, got in taken[-3:]:
        ref = call(K, False)
        for f in ref:
            assert np.array_equal(got[f], ref[f]), (K, f)

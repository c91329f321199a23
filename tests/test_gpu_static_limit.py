"""What crtm_gpu_k_matrix_device_static takes and refuses, at the limit, and that
a refused call launches nothing and leaves its outputs as they were.

The FP64 limit counts a profile's K-matrix intermediates as the entry point was
released with: predictors, partials, bands, reference and user layer arrays,
each rounded up to 256 bytes (counted out below for 100 reference layers of an
absorber group with 21 predictors and 29 partials).  14000 channels and 6
absorber Jacobians: 130 layers are the most that 128 MiB take."""
import os

import numpy as np
import pytest

from crtmv3_gb300 import coefficients as co, synthetic as sy

pytestmark = pytest.mark.gpu

SID, L, K = "wide_c14000", 14000, 100


def _counted(layers, nv):
    def up(n):
        return (n + 255) // 256 * 256
    n = up(16 * K * 21 * 8) + up(16 * K * 29 * 8) + 2 * up(4 * K) + up(8 * K * 32)
    n += 2 * up(4 * (layers + 1)) + up(8 * (layers + 1)) + 2 * up(4 * (K + 1))
    n += 2 * up(4 * layers) + up(8 * layers * 16) + up(8 * 4) + up(4)
    return n + up(8 * K * L) + 3 * up(8 * layers * L) + up(8 * L) + up(8 * nv * K * L) + up(4 * 6)


@pytest.fixture(scope="module")
def wide(gpu_lib, tmp_path_factory):
    d = str(tmp_path_factory.mktemp("wide"))
    tc = sy.generate_odps(3, L, 5, SID, co.INFRARED_SENSOR, max_predictors_per_channel=1)
    co.write_odps(os.path.join(d, f"{SID}.TauCoeff.bin"), tc)
    co.write_spccoeff(os.path.join(d, f"{SID}.SpcCoeff.bin"), sy.generate_spccoeff(SID, co.INFRARED_SENSOR, L, 6))
    sy.write_cloud_files(d)
    return gpu_lib.CRTM([SID], d, 0)


def _call(h, atm, sfc, geo, static, species=0):
    import torch
    import bench
    dev = torch.device("cuda")
    P, Km, J = atm.n_profiles, atm.max_layers, atm.n_absorbers
    opt = sy.OptionsBatch(emissivity=sy.emissivity_for(co.INFRARED_SENSOR, P, L, 10))
    b, keep, t = bench.scatter_device_inputs(torch, h, atm, sfc, geo, opt, dev)
    out = {k: v.fill_(-7) for k, v in bench.k_outputs(torch, P, L, Km, J, dev).items()}
    if species:
        for f in ("cloud_water_content_k", "cloud_effective_radius_k"):
            out[f] = torch.full((P, L, species, Km), -7.0, dtype=torch.float64, device=dev)
    try:
        h.k_matrix_device(b, out, None, 0, torch.cuda.current_stream().cuda_stream, static_scratch=static)
        return out, None
    except RuntimeError as e:
        return out, str(e)
    finally:
        torch.cuda.synchronize()


def test_limit(wide):
    assert _counted(130, 7) <= 128 << 20 < _counted(131, 7)
    atm, sfc, geo = sy.generate_profiles(1, 130, sy.absorber_set(1), 9)
    assert atm.n_absorbers == 6
    out, err = _call(wide, atm, sfc, geo, True)
    assert err is None
    ref, _ = _call(wide, atm, sfc, geo, False)
    for f in ref:
        assert bool((out[f] == ref[f]).all()), f
    atm, sfc, geo = sy.generate_profiles(1, 131, sy.absorber_set(1), 9)
    launches = wide.launch_count()
    out, err = _call(wide, atm, sfc, geo, True)
    assert "static scratch holds" in err and f" {_counted(131, 7)} bytes" in err
    assert wide.launch_count() == launches


@pytest.mark.parametrize("clear", [(0, 1), (0,)])
def test_refused_call_leaves_outputs_alone(wide, clear):
    """Cloud arrays with clear profiles beside a cloudy one, and clear ones alone."""
    atm, sfc, geo = sy.generate_profiles(2, 200, sy.absorber_set(1), 9)
    sy.add_clouds(atm, (co.WATER_CLOUD, co.ICE_CLOUD), 12)
    atm.n_clouds[list(clear)] = 0
    launches = wide.launch_count()
    out, err = _call(wide, atm, sfc, geo, True, species=atm.cloud_type.shape[1])
    assert "static scratch holds" in err
    assert wide.launch_count() == launches
    for f, v in out.items():
        assert bool((v == -7).all()), f


@pytest.mark.parametrize("clear", [(0, 1), (0,)])
def test_clear_profiles_scattering_jacobians_are_zero(gpu_lib, coeff_dir, clear):
    """Of device and of host calls, into buffers that hold something else."""
    import torch
    import bench
    sy.write_cloud_files(coeff_dir)
    sensor, dev = "mwsynth_c16", torch.device("cuda")
    atm, sfc, geo, opt = sy.cloudy_workload(sensor, 2, 60, 31, wc_scale=50.0)
    atm.n_clouds[list(clear)] = 0
    for precision in (0, 1):
        h = gpu_lib.CRTM([sensor], coeff_dir, precision)
        km, _ = h.k_matrix(atm, sfc, geo, opt)
        b, keep, t = bench.scatter_device_inputs(torch, h, atm, sfc, geo, opt, dev)
        out = bench.k_outputs(torch, 2, 16, 60, atm.n_absorbers, dev)
        NC = atm.cloud_type.shape[1]
        for f in ("cloud_water_content", "cloud_effective_radius"):
            out[f + "_k"] = torch.full((2, 16, NC, 60), -7.0, dtype=torch.float64, device=dev)
        h.k_matrix_device(b, out, None, 0, torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
        for f in ("cloud_water_content", "cloud_effective_radius"):
            got = out[f + "_k"].cpu().numpy()
            assert np.array_equal(got, getattr(km, f)), f
            for p in range(2):
                assert (got[p] == 0.0).all() == (p in clear), (f, p)

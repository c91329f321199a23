"""What crtm_gpu_k_matrix_device_static takes and refuses, at the limit.

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
    return gpu_lib.CRTM([SID], d, 0)


def _call(h, atm, sfc, geo, static):
    import torch
    import bench
    dev = torch.device("cuda")
    P, Km, J = atm.n_profiles, atm.max_layers, atm.n_absorbers
    opt = sy.OptionsBatch(emissivity=sy.emissivity_for(co.INFRARED_SENSOR, P, L, 10))
    b, keep, t = bench.scatter_device_inputs(torch, h, atm, sfc, geo, opt, dev)
    out = {k: v.fill_(-7) for k, v in bench.k_outputs(torch, P, L, Km, J, dev).items()}
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

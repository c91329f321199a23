"""The trajectory's contractions (crtm_gpu_tangent_linear_apply,
crtm_gpu_adjoint_apply) against the K-matrix contracted on the host, where
their blocks end: channel counts around 8, 64 and 256, profiles that fill the
layer stride and profiles that do not.  The terms are the same FP64 products
in another order: at most 400 of them, so 400 roundings of 1.1e-16 each against
the sum of their sizes, held to 1e-12."""
import numpy as np
import pytest

from crtmv3_gb300 import synthetic as sy

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("channels,layers", [(1, (40, 40)), (7, (30, 101)), (9, (101, 101)), (65, (64, 64)),
                                             (255, (33, 33)), (616, (31, 32))])
def test_contractions_match_k_matrix(gpu_lib, coeff_dir, channels, layers):
    import torch
    import bench
    dev = torch.device("cuda")
    sensor, P = "irsynth_c616", 3
    rng = np.random.default_rng(channels)
    nl = np.array([layers[1], layers[0], layers[1]])
    atm, sfc, geo, opt = sy.clear_sky_workload(sensor, P, nl, 600 + channels)
    h = gpu_lib.CRTM([sensor], coeff_dir, 0)
    if channels < 616:
        pos = np.sort(rng.choice(616, channels, replace=False))
        h.set_channel_subset(0, pos)
        opt.emissivity = np.ascontiguousarray(opt.emissivity[:, pos])
    km, rts = h.k_matrix(atm, sfc, geo, opt)
    L, K = rts.radiance.shape[1], atm.max_layers
    f64 = dict(dtype=torch.float64, device=dev)
    b, keep, t = bench.scatter_device_inputs(torch, h, atm, sfc, geo, opt, dev)
    h.linearize_device(b, dict(radiance=torch.zeros((P, L), **f64), bt=torch.zeros((P, L), **f64)))
    # the stride beyond a profile's layers may hold anything
    dt = rng.normal(size=(P, K))
    dw, de = rng.normal(size=P), rng.uniform(-0.01, 0.01, (P, L))
    bt = torch.zeros((P, L), **f64)
    h.tangent_linear_apply_device({"temperature": torch.from_numpy(dt).to(dev),
                                   "water_temperature": torch.from_numpy(dw).to(dev),
                                   "emissivity": torch.from_numpy(de).to(dev)}, bt)
    torch.cuda.synchronize()
    terms = [km.temperature * dt[:, None, :], (km.water_temperature * dw[:, None])[:, :, None],
             (km.surface_emissivity * de)[:, :, None]]
    ref = sum(x.sum(axis=2) for x in terms)
    size = sum(np.abs(x).sum(axis=2) for x in terms)
    assert (np.abs(bt.cpu().numpy() - ref) <= 1e-12 * size).all()
    seed = rng.normal(size=(P, L))
    out = {"temperature_ad": torch.zeros((P, K), **f64), "absorber_ad": torch.zeros((P, atm.n_absorbers, K), **f64),
           "water_temperature_ad": torch.zeros((P,), **f64)}
    h.adjoint_apply_device(torch.from_numpy(seed).to(dev), out)
    torch.cuda.synchronize()
    x = km.temperature * seed[:, :, None]
    assert (np.abs(out["temperature_ad"].cpu().numpy() - x.sum(axis=1)) <= 1e-12 * np.abs(x).sum(axis=1)).all()
    x = km.water_temperature * seed
    assert (np.abs(out["water_temperature_ad"].cpu().numpy() - x.sum(axis=1)) <= 1e-12 * np.abs(x).sum(axis=1)).all()

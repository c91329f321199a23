"""The trajectory's contractions with its multi-row block, the absorbers, in both
directions and with several blocks at once: profiles that fill the layer stride
(their rows run on as one index) and profiles that do not, against the K-matrix
contracted on the host.  Each side sums n products in FP64 in its own order: within
n 2^-53 of the sum of their sizes each, so 2 n 2^-53 apart at most (n: layers x
(1 + absorbers) + 1 in the tangent linear, the channels in the adjoint)."""
import numpy as np
import pytest

from crtmv3_gb300 import synthetic as sy

pytestmark = pytest.mark.gpu

U = 2.0 ** -53


@pytest.mark.parametrize("sensor,channels,layers", [
    ("irsynth_c616", 1, (40, 40)), ("irsynth_c616", 9, (31, 101)), ("irsynth_c616", 65, (101, 101)),
    ("irsynth_c616", 616, (33, 34)), ("mwsynth_c22", 22, (60, 100)), ("mwsynth_c22", 7, (97, 97))])
def test_absorber_blocks_match_k_matrix(gpu_lib, coeff_dir, sensor, channels, layers):
    import torch
    import bench
    dev = torch.device("cuda")
    P = 3
    rng = np.random.default_rng(channels)
    nl = np.array([layers[1], layers[0], layers[1]])
    atm, sfc, geo, opt = sy.clear_sky_workload(sensor, P, nl, 650 + channels)
    h = gpu_lib.CRTM([sensor], coeff_dir, 0)
    if channels < h.n_channels[0]:
        pos = np.sort(rng.choice(h.n_channels[0], channels, replace=False))
        h.set_channel_subset(0, pos)
        opt.emissivity = np.ascontiguousarray(opt.emissivity[:, pos])
    km, rts = h.k_matrix(atm, sfc, geo, opt)
    L, K, J = rts.radiance.shape[1], atm.max_layers, atm.n_absorbers
    assert J > 1 and np.abs(km.absorber).max() > 0.0
    f64 = dict(dtype=torch.float64, device=dev)
    b, keep, t = bench.scatter_device_inputs(torch, h, atm, sfc, geo, opt, dev)
    h.linearize_device(b, dict(radiance=torch.zeros((P, L), **f64), bt=torch.zeros((P, L), **f64)))
    dt, dw = rng.normal(size=(P, K)), rng.normal(size=P)
    da = atm.absorber * rng.normal(0.0, 0.1, atm.absorber.shape)
    live = (np.arange(K)[None] < nl[:, None]).astype(float)
    tl = {"temperature": dt, "absorber": da, "water_temperature": dw}
    bt = torch.full((P, L), np.nan, **f64)
    h.tangent_linear_apply_device({k: torch.from_numpy(np.ascontiguousarray(v)).to(dev) for k, v in tl.items()}, bt)
    torch.cuda.synchronize()
    terms = np.concatenate([(km.temperature * (dt * live)[:, None]).reshape(P, L, -1),
                            (km.absorber * (da * live[:, None])[:, None]).reshape(P, L, -1),
                            (km.water_temperature * dw[:, None])[:, :, None]], axis=2)
    n = K * (1 + J) + 1
    assert (np.abs(bt.cpu().numpy() - terms.sum(axis=2)) <= 2 * n * U * np.abs(terms).sum(axis=2)).all()
    seed = rng.normal(size=(P, L))
    out = {"temperature_ad": torch.full((P, K), np.nan, **f64), "absorber_ad": torch.full((P, J, K), np.nan, **f64),
           "water_temperature_ad": torch.full((P,), np.nan, **f64)}
    h.adjoint_apply_device(torch.from_numpy(seed).to(dev), out)
    torch.cuda.synchronize()
    for f, k in (("temperature_ad", km.temperature), ("absorber_ad", km.absorber),
                 ("water_temperature_ad", km.water_temperature)):
        x = k * seed.reshape((P, L) + (1,) * (k.ndim - 2))
        assert (np.abs(out[f].cpu().numpy() - x.sum(axis=1)) <= 2 * L * U * np.abs(x).sum(axis=1)).all(), f

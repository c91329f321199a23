"""The calls that a user of the library times: forward, K-matrix, adjoint and
trajectory calls through the public Python API, from one profile to thousands.

A case is a dict: ``call`` (which entry point), ``sensor`` and ``channels``
(0: all; else that many, evenly spread, through the channel subset),
``profiles``, ``layers_lo`` .. ``layers_hi`` (layer counts uniform between
them), ``precision`` ("fp64", the handle's default, or "mixed"), ``sky``
("clear", "cloudy", "aerosol": clouds and three aerosols), ``cloudy_percent``
(profiles that have clouds) and ``streams`` ("rule", or "options": a share of
the cloudy profiles with Options%n_Streams 8 / 16).

Coefficients and profiles are the repository's synthetic ones
(crtmv3_gb300.synthetic), drawn from the seed.
"""
from __future__ import annotations

import math
import os
import tempfile

import numpy as np
import torch

# A cloudy infrared K-matrix keeps 0.3 - 1.3 GB of intermediates per profile:
# programs that run those raise the work space from its 8 GB default.
os.environ.setdefault("CRTM_GPU_WORKSPACE_MB", "32768")

from crtmv3_gb300 import api, coefficients as co, synthetic as sy  # noqa: E402
from crtmv3_gb300.api import ChannelInfo, CRTM_Forward  # noqa: E402

MW22, MW16, IR616, IR2211 = "mwsynth_c22", "mwsynth_c16", "irsynth_c616", "irsynth_c2211"
IR_CLOUDS = (co.WATER_CLOUD, co.ICE_CLOUD)
MW_CLOUDS = (co.WATER_CLOUD, co.ICE_CLOUD, co.RAIN_CLOUD, co.SNOW_CLOUD, co.GRAUPEL_CLOUD)


def _case(name, call, sensor, profiles, layers_lo, layers_hi, precision, channels=0, sky="clear",
          cloudy_percent=0, streams="rule"):
    c = dict(call=call, sensor=sensor, channels=channels, profiles=profiles, layers_lo=layers_lo,
             layers_hi=layers_hi, precision=precision, sky=sky, cloudy_percent=cloudy_percent, streams=streams)
    return c if name is None else dict(name=name, **c)


def listed():
    return [
        # one sounding as it arrives: the operator inside a retrieval or a column model
        _case("forward_mw_one", "forward", MW22, 1, 100, 100, "fp64"),
        # a granule line of a microwave sounder through the reference-named host call (numpy in, numpy out)
        _case("host_forward_mw", "host_forward", MW22, 100, 100, 100, "fp64"),
        # observation minus background of a hyperspectral sounder, the channel subset a weather centre assimilates
        _case("forward_ir_subset", "forward", IR2211, 1500, 101, 101, "mixed", channels=431),
        # microwave K-matrix of a ragged batch (1D-Var over a scan)
        _case("k_mw_ragged", "k_matrix", MW22, 333, 60, 137, "fp64"),
        # clear-sky hyperspectral K-matrix, every channel: the framework's headline in clear sky
        _case("k_ir_clear", "k_matrix", IR2211, 1000, 101, 101, "mixed"),
        # the same call in the default, all-FP64 form
        _case("k_ir_clear_fp64", "k_matrix", IR616, 250, 100, 100, "fp64"),
        # 4D-Var gradient: the adjoint of a clear-sky infrared batch
        _case("adjoint_ir_clear", "adjoint", IR616, 700, 90, 100, "mixed"),
        # inner loop of a variational analysis: tangent linear and adjoint about one trajectory
        _case("trajectory_ir", "trajectory", IR616, 500, 101, 101, "mixed"),
        # cloudy microwave adjoint, five cloud types, some profiles with more streams
        _case("adjoint_mw_cloudy", "adjoint", MW16, 2000, 100, 100, "mixed", sky="cloudy", cloudy_percent=100,
              streams="options"),
        # all-sky infrared simulation for monitoring, default precision
        _case("forward_ir_cloudy", "forward", IR616, 64, 80, 120, "fp64", sky="cloudy", cloudy_percent=70),
        # all-sky infrared K-matrix with liquid and ice clouds and three aerosols
        _case("k_ir_allsky", "k_matrix", IR616, 120, 100, 100, "mixed", sky="aerosol", cloudy_percent=100),
        # the ragged stress batch of one hyperspectral sensor: 30 % cloudy, 60 - 137 layers, mixed streams
        _case("k_ir_ragged", "k_matrix", IR2211, 150, 60, 137, "mixed", sky="cloudy", cloudy_percent=30,
              streams="options"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: one of the listed kinds with its sizes drawn over their range."""
    kind = rng.choice(["forward_mw", "host", "forward_ir", "k_mw", "k_ir", "k_ir_fp64", "adjoint_ir", "trajectory",
                       "adjoint_mw_cloudy", "forward_cloudy", "k_allsky", "k_ragged"])
    lo = rng.randint(60, 110)
    hi = rng.randint(lo, 137)
    if kind == "forward_mw":
        return _case(None, "forward", MW22, _log_int(rng, 1, 3000), lo, hi, rng.choice(["fp64", "mixed"]))
    if kind == "host":
        return _case(None, "host_forward", rng.choice([MW22, MW16]), _log_int(rng, 1, 1000), 100, 100, "fp64")
    if kind == "forward_ir":
        return _case(None, "forward", IR2211, _log_int(rng, 1, 1500), lo, hi, "mixed",
                     channels=rng.choice([0, 137, 431, 616]))
    if kind == "k_mw":
        return _case(None, "k_matrix", MW22, _log_int(rng, 1, 3000), lo, hi, rng.choice(["fp64", "mixed"]))
    if kind == "k_ir":
        return _case(None, "k_matrix", rng.choice([IR2211, IR616]), _log_int(rng, 2, 800), lo, min(hi, lo + 10), "mixed",
                     channels=rng.choice([0, 0, 137, 431]))
    if kind == "k_ir_fp64":
        return _case(None, "k_matrix", IR616, _log_int(rng, 1, 250), lo, min(hi, 110), "fp64",
                     channels=rng.choice([0, 137]))
    if kind == "adjoint_ir":
        return _case(None, "adjoint", IR616, _log_int(rng, 1, 700), lo, hi, rng.choice(["mixed", "mixed", "fp64"]),
                     channels=rng.choice([0, 137]))
    if kind == "trajectory":
        return _case(None, "trajectory", rng.choice([IR616, MW22]), _log_int(rng, 5, 500), lo, hi, "mixed")
    if kind == "adjoint_mw_cloudy":
        return _case(None, "adjoint", MW16, _log_int(rng, 10, 2000), lo, hi, rng.choice(["mixed", "mixed", "fp64"]),
                     sky="cloudy", cloudy_percent=rng.randint(20, 100), streams=rng.choice(["rule", "options"]))
    if kind == "forward_cloudy":
        sensor = rng.choice([IR616, MW16])
        return _case(None, "forward", sensor, _log_int(rng, 2, 64 if sensor == IR616 else 1000), lo, hi,
                     rng.choice(["fp64", "mixed"]), sky="cloudy", cloudy_percent=rng.randint(20, 100),
                     streams=rng.choice(["rule", "options"]))
    if kind == "k_allsky":
        return _case(None, "k_matrix", IR616, _log_int(rng, 2, 100), lo, min(hi, lo + 20), "mixed", sky="aerosol",
                     cloudy_percent=rng.randint(50, 100), channels=rng.choice([0, 137]))
    return _case(None, "k_matrix", rng.choice([IR2211, IR616]), _log_int(rng, 4, 120), lo, hi, "mixed", sky="cloudy",
                 cloudy_percent=rng.randint(10, 40), streams="options")


# ---------------------------------------------------------------------------
# what a program has before the call
# ---------------------------------------------------------------------------
_coeff_dir = None
_handles = {}


def _coefficients() -> str:
    """The synthetic coefficient files, written once per process."""
    global _coeff_dir
    if _coeff_dir is None:
        d = tempfile.mkdtemp(prefix="crtm_perf_")
        for sid in (MW22, MW16, IR616, IR2211):
            sy.write_sensor_files(d, sid)
        sy.write_cloud_files(d)
        sy.write_aerosol_files(d)
        _coeff_dir = d
    return _coeff_dir


def _positions(sensor: str, channels: int):
    L = sy.SENSORS[sensor][1]
    return None if channels in (0, L) else np.unique(np.linspace(0, L - 1, channels).astype(np.int32))


def _new_handle(sensor: str, channels: int, precision: str):
    h = api.CRTM([sensor], _coefficients(), api.MIXED if precision == "mixed" else api.FP64)
    pos = _positions(sensor, channels)
    if pos is not None:
        h.set_channel_subset(0, pos)
    return h


def _handle(sensor: str, channels: int, precision: str):
    """A program has one handle per sensor, channel selection and precision and keeps it."""
    key = (sensor, channels, precision)
    if key not in _handles:
        _handles[key] = _new_handle(*key)
    return _handles[key]


def _host_inputs(case, seed):
    """The batch as numpy structures."""
    P, sensor = case["profiles"], case["sensor"]
    rng = np.random.Generator(np.random.PCG64([seed, 1]))
    nl = rng.integers(case["layers_lo"], case["layers_hi"] + 1, P)
    nl[int(rng.integers(0, P))] = case["layers_hi"]   # the batch's layer stride is the same for every seed
    base = int(rng.integers(1, 1 << 30))
    atm, sfc, geo, opt = sy.clear_sky_workload(sensor, P, nl, base)
    pos = _positions(sensor, case["channels"])
    if pos is not None:
        opt.emissivity = np.ascontiguousarray(opt.emissivity[:, pos])
    if case["sky"] != "clear":
        sy.add_clouds(atm, MW_CLOUDS if sensor in (MW22, MW16) else IR_CLOUDS, base + 11)
        cloudy = rng.uniform(size=P) < case["cloudy_percent"] / 100.0
        if case["cloudy_percent"]:
            cloudy[int(rng.integers(0, P))] = True
        atm.n_clouds[~cloudy] = 0
        if case["sky"] == "aerosol":
            sy.add_aerosols(atm, sy.AEROSOL_TYPES, base + 12)
        if case["streams"] == "options":
            ns = np.where(cloudy, rng.choice(np.array([0, 8, 16], np.int32), size=P, p=[0.6, 0.2, 0.2]), 0)
            opt.use_n_streams, opt.n_streams = ns > 0, ns.astype(np.int32)
    return atm, sfc, geo, opt, rng


def _jacobians(atm):
    """The absorber Jacobians that a program asks for: water vapour and ozone."""
    ids = list(atm.absorber_id)
    return [ids.index(j) for j in (co.H2O_ID, co.O3_ID) if j in ids]


ATM_FIELDS = ("level_pressure", "pressure", "temperature", "absorber", "cloud_water_content",
              "cloud_effective_radius", "cloud_fraction", "aerosol_concentration", "aerosol_effective_radius")
INT_FIELDS = ("n_layers", "n_clouds", "cloud_type", "n_aerosols", "aerosol_type")
SFC_FIELDS = ("land_coverage", "water_coverage", "snow_coverage", "ice_coverage", "land_temperature",
              "water_temperature", "snow_temperature", "ice_temperature")
GEO_FIELDS = ("sensor_zenith_angle", "source_zenith_angle", "surface_altitude")


def _on_device(atm, sfc, geo, opt):
    t = {}
    for obj, fields, dt in ((atm, ATM_FIELDS, np.float64), (atm, INT_FIELDS, np.int32), (sfc, SFC_FIELDS, np.float64),
                            (geo, GEO_FIELDS, np.float64)):
        for f in fields:
            v = getattr(obj, f)
            if v is not None:
                t[f] = torch.from_numpy(np.ascontiguousarray(v, dt)).cuda()
    t["emissivity"] = torch.from_numpy(np.ascontiguousarray(opt.emissivity)).cuda()
    if opt.n_streams is not None:
        t["n_streams"] = torch.from_numpy(np.where(opt.use_n_streams, opt.n_streams, 0).astype(np.int32)).cuda()
    return t


def _empty(*shape, dtype=torch.float64):
    return torch.empty(shape, dtype=dtype, device="cuda")


def _outputs(case, atm, L, sel):
    P, K = atm.n_profiles, atm.max_layers
    out = dict(radiance=_empty(P, L), bt=_empty(P, L), status=_empty(P, dtype=torch.int32))
    NC = atm.cloud_type.shape[1] if atm.cloud_type is not None else 0
    NA = atm.aerosol_type.shape[1] if atm.aerosol_type is not None else 0
    if case["call"] == "k_matrix":
        lead, sfx = (P, L), "_k"
        out.update(temperature_k=_empty(P, L, K), absorber_k=_empty(P, L, len(sel), K),
                   water_temperature_k=_empty(P, L), surface_emissivity_k=_empty(P, L))
    elif case["call"] == "adjoint":
        lead, sfx = (P,), "_ad"
        out.update(temperature_ad=_empty(P, K), absorber_ad=_empty(P, atm.n_absorbers, K),
                   water_temperature_ad=_empty(P))
    else:
        return out
    if NC:
        out["cloud_water_content" + sfx] = _empty(*lead, NC, K)
        out["cloud_effective_radius" + sfx] = _empty(*lead, NC, K)
    if NA:
        out["aerosol_concentration" + sfx] = _empty(*lead, NA, K)
        out["aerosol_effective_radius" + sfx] = _empty(*lead, NA, K)
    return out


def _perturbations(atm, sfc, rng):
    """A background-error-like increment of temperature, absorbers and skin temperature."""
    live = (np.arange(atm.max_layers)[None] < atm.n_layers[:, None]).astype(np.float64)
    return dict(temperature=rng.normal(0.0, 1.0, atm.temperature.shape) * live,
                absorber=atm.absorber * rng.normal(0.0, 0.1, atm.absorber.shape) * live[:, None],
                water_temperature=rng.normal(0.0, 1.0, sfc.water_temperature.shape))


def prepare(case, seed):
    atm, sfc, geo, opt, rng = _host_inputs(case, seed)
    call = case["call"]
    st = dict(call=call)
    if call == "host_forward":
        h = _handle(case["sensor"], case["channels"], case["precision"])
        n = h.n_channels[0]
        st.update(atm=atm, sfc=sfc, geo=geo, opt=opt,
                  info=[ChannelInfo(case["sensor"], 0, n, h, np.arange(1, n + 1), np.ones(n, bool))])
        return st
    # a trajectory belongs to its handle: each analysis has its own
    h = (_new_handle if call == "trajectory" else _handle)(case["sensor"], case["channels"], case["precision"])
    L, P = h.n_channels[0], atm.n_profiles
    t = _on_device(atm, sfc, geo, opt)
    b, keep = h.device_batch(t, atm.absorber_id)
    sel = _jacobians(atm)
    st.update(h=h, batch=b, keep=(keep, t), sel=sel, out=_outputs(case, atm, L, sel))
    if call in ("adjoint", "trajectory"):
        st["seed"] = torch.from_numpy(rng.normal(0.0, 1.0, (P, L))).cuda()
    if call == "trajectory":
        st["tl"] = {k: torch.from_numpy(v).cuda() for k, v in _perturbations(atm, sfc, rng).items()}
        st["bt_tl"] = _empty(P, L)
        K = atm.max_layers
        st["ad"] = dict(temperature_ad=_empty(P, K), absorber_ad=_empty(P, atm.n_absorbers, K),
                        water_temperature_ad=_empty(P))
        torch.cuda.synchronize()
        h.linearize_device(b, st["out"], 0, torch.cuda.current_stream().cuda_stream)
    return st


def run(state):
    call = state["call"]
    if call == "host_forward":
        rts = []
        CRTM_Forward(state["atm"], state["sfc"], state["geo"], state["info"], rts, state["opt"])
        r = rts[0]
        return dict(bt=r.brightness_temperature, radiance=r.radiance, up=r.up_radiance, down=r.down_radiance,
                    layer_optical_depth=r.layer_optical_depth, upwelling=r.upwelling_radiance)
    h, stream = state["h"], torch.cuda.current_stream().cuda_stream
    if call == "forward":
        h.forward_device(state["batch"], state["out"], 0, stream)
    elif call == "k_matrix":
        h.k_matrix_device(state["batch"], state["out"], None, 0, stream, k_absorbers=state["sel"])
    elif call == "adjoint":
        h.adjoint_device(state["batch"], state["seed"], state["out"], 0, stream)
    else:
        h.tangent_linear_apply_device(state["tl"], state["bt_tl"], stream)
        h.adjoint_apply_device(state["seed"], state["ad"], stream)
        return dict(bt_tl=state["bt_tl"], **state["ad"])
    return state["out"]


# ---------------------------------------------------------------------------
# the work a pass cannot do without
# ---------------------------------------------------------------------------
_SLOTS = {1: (89, 118, 6), 2: (50, 64, 3), 3: (21, 26, 1)}   # predictors, their partials, absorbers
_COLUMN_FLOPS = 60        # Planck, transmittance and recursion of a layer of one channel
_LAYER_OPS = {5: 14550.0, 6: 24700.0, 10: 113600.0}   # reverse sweep of one scattering layer by its angles


def work(case):
    group, L_all, stype, _ = sy.SENSORS[case["sensor"]]
    pos = _positions(case["sensor"], case["channels"])
    L = L_all if pos is None else pos.size
    P, K = case["profiles"], case["layers_hi"]
    Km = 0.5 * (case["layers_lo"] + case["layers_hi"])
    ns, nnz, jm = _SLOTS[group]
    jm = 2 if case["sensor"] == MW22 else jm
    pc, cloudy = P * L, P * case["cloudy_percent"] / 100.0
    nc = 0 if case["sky"] == "clear" else (5 if case["sensor"] in (MW22, MW16) else 2)
    na = 3 if case["sky"] == "aerosol" else 0
    nin = P * 8.0 * (3 * K + 1 + jm * K + 11) + 8.0 * pc + P * 8.0 * (2 * nc + 2 * na + (1 if nc else 0)) * K
    coeff = 4.0 * 100 * ns * L
    active = 0.7 * ns            # predictors that a channel has, on average
    flops = pc * (2.0 * 100 * active + _COLUMN_FLOPS * Km)
    sel = 1 if group == 3 else 2
    call = case["call"]
    if call in ("forward", "host_forward"):
        nout = 16.0 * pc
        if call == "host_forward":
            nout = 8.0 * pc * (11 + 3 * K)
    elif call == "k_matrix":
        nout = 8.0 * pc * (4 + (1 + sel + 2 * nc + 2 * na) * K)
    elif call == "adjoint":
        nout = 16.0 * pc + 8.0 * P * (1 + jm + 2 * nc + 2 * na) * K
    else:
        # the stored Jacobians of temperature and every absorber, read by each of the two contractions
        return dict(bytes=2.0 * 8 * pc * (1 + jm) * K + 24.0 * pc, flops=4.0 * pc * (1 + jm) * Km)
    if call in ("k_matrix", "adjoint"):
        flops += pc * (2.0 * 100 * 0.7 * nnz + _COLUMN_FLOPS * Km)
    if nc:
        share = 1.0 - (1.0 - 0.15) ** nc      # layers with an active cloud
        layers = cloudy * L * Km * share + (P * L * Km * 0.2 if na else 0.0)
        per = _LAYER_OPS[5] if case["streams"] == "rule" else 0.6 * _LAYER_OPS[5] + 0.2 * _LAYER_OPS[6] + 0.2 * _LAYER_OPS[10]
        flops += layers * (per / 3.0 if call == "forward" else per)
    return dict(bytes=nin + coeff + nout, flops=flops)


# ---------------------------------------------------------------------------
# the clear-sky outputs in plain torch, 64 bits
# ---------------------------------------------------------------------------
_TZ_MAX, _R_EARTH, _OD_MAX, _EPS = 63.6122, 6370.0, 20.0, 2.220446049250313e-16
_C_TV = (28.9648 / 18.01528 - 1.0) / 1000.0
_C_H = 0.001 * (8.314472 / 28.9648e-3) / 9.80665


class _Tables:
    """One sensor's coefficients as dense torch arrays (C: layers x predictors x channels)."""

    def __init__(self, sensor, channels, dev):
        group, L, stype, seed = sy.SENSORS[sensor]
        tc = sy.generate_odps(group, L, seed, sensor, stype,
                              max_predictors_per_channel=20 if sensor == MW22 else None)
        sc = sy.generate_spccoeff(sensor, stype, L, seed + 100)
        pos = _positions(sensor, channels)
        pos = np.arange(L) if pos is None else pos
        mx = {1: (7, 18, 7, 11, 11, 14, 10, 11), 2: (7, 15, 7, 11, 10), 3: (7, 14)}[group]
        K = tc.ref_pressure.size
        C = np.zeros((K, sum(mx), pos.size))
        for i, l in enumerate(pos):
            off = 0
            for j, m in enumerate(mx):
                n = int(tc.n_predictors[j, l])
                if n > 0:
                    at = int(tc.pos_index[j, l]) - 1
                    C[:, off:off + n, i] = tc.c[at:at + n * K].reshape(n, K).T
                off += m
        self.group, self.K = group, K
        self.C = torch.from_numpy(C).to(dev)
        self.lev, self.p, self.t = tc.ref_level_pressure, tc.ref_pressure, tc.ref_temperature
        self.a, self.lo, self.hi = tc.ref_absorber, tc.min_absorber, tc.max_absorber
        self.ids = {1: (1, 3, 2, 4, 5, 6), 2: (1, 3, 2), 3: (1,)}[group]
        self.spec = [torch.from_numpy(np.ascontiguousarray(np.asarray(v, np.float64)[pos])).to(dev) for v in
                     (sc.planck_c1, sc.planck_c2, sc.band_c1, sc.band_c2, sc.cosmic_background_radiance)]


def _layer_weights(x1, x2):
    """Weights (reference layer, user layer) of the layer averaging of one profile; x1, x2 the ln p of both grids."""
    n1, n2 = x1.size, x2.size
    W = np.zeros((n1, n2))
    a, b = x2[:-1], x2[1:]
    j = np.arange(n2 - 1)
    for i in range(n1):
        z2 = x1[i]
        z1 = 2 * z2 - x1[i + 1] if i == 0 else x1[i - 1]
        z3 = min(2 * z2 - z1 if i == n1 - 1 else x1[i + 1], x2[-1])
        below = z2 >= x2[-1]
        if below:
            z2 = z3 = x2[-1]
        w = np.zeros(n2)
        hit_any = False
        for edge in (0, 1):
            za = z1 if edge == 0 else z3
            hit = (a <= z2) & (b > z1) if edge == 0 else (a < z3) & (b >= z2) & (not below)
            hit &= a <= z3
            if not hit.any():
                continue
            hit_any = True
            ya, yb = (z1, z2) if edge == 0 else (z2, z3)
            top, bot = a > ya, b < yb
            y1, y2 = np.where(top, a, ya), np.where(bot, b, yb)
            dy = y2 - y1
            with np.errstate(divide="ignore", invalid="ignore"):
                w1, w2 = (za - y1) / (za - z2) * dy, (za - y2) / (za - z2) * dy
            d = (b - z2) / (b - a)
            if edge == 0:
                move = hit & ~bot
                w1, w2 = np.where(move, w1 + w2 * d, w1), np.where(move, w2 * (1 - d), w2)
            else:
                move = hit & ~top
                w1, w2 = np.where(move, w1 * d, w1), np.where(move, w2 + w1 * (1 - d), w2)
            np.add.at(w, j[hit], w1[hit])
            np.add.at(w, j[hit] + 1, w2[hit])
        if not hit_any:
            over = np.nonzero(a > z3)[0]
            w[over[0] if over.size else n2 - 1] = 1.0
        W[i] = w / w.sum()
    return W


def _predictors(group, T, A, Tref, Aref, pdp, s):
    """The regression's predictors (..., K, slots) of mapped temperature T (..., K) and absorbers A[j] (..., K)."""
    dT, t = T - Tref, T / Tref
    t2, dT2 = t * t, dT * dT.abs()
    cum = lambda v: torch.cumsum(v, -1)  # noqa: E731
    tz, tzp = cum(T) / cum(Tref), cum(pdp * T) / cum(pdp * Tref)
    R = [a / r for a, r in zip(A, Aref)]
    gz = [cum(pdp * a) / cum(pdp * r) for a, r in zip(A, Aref)]
    gt = [cum(pdp * a * T) / cum(pdp * r * Tref) for a, r in zip(A, Aref)]
    S = s + 0 * t
    H = R[0]
    Ha = s * H
    Hr = Ha.sqrt()
    Hd = H / gt[0]
    dry = [S, s * t, s * t2, t, S * S, t2, tz]
    cont = [Ha / t, Ha / t * H, Ha / t2 * H / t2, Ha / t2, Ha / t2 * H, Ha / t2 ** 2, Ha]
    if group == 3:
        X = dry + cont + [Ha * dT, (s * gz[0]) ** 2, s * gz[0], S, Ha ** 3, Ha ** 4, Hd]
        return torch.stack(X, -1)
    O, C2 = R[1], R[2]
    Oa = s * O
    Or = Oa.sqrt()
    wlo = [Ha, Ha * dT, Ha ** 2, Ha * dT2, Hr.sqrt(), Ha ** 3, Hr, Hr * dT, Ha ** 4, Hd, Hr * Hd, (s * gz[0]) ** 2,
           s * gz[0], S, s * C2]
    ozo = [Oa, Oa * dT, Oa * O * gz[1], Oa ** 2, Oa * gz[1], Oa * (s * gz[1]).sqrt(), Or * dT, Or, Or * O / gz[1],
           s * gz[1], (s * gz[1]) ** 2]
    co2 = [s * t, s * t2, t, t2, S, s * C2, s * tzp, (s * gz[2]) ** 2, tzp ** 3, s * tzp * t.sqrt()]
    if group == 2:
        return torch.stack(dry + wlo + cont + ozo + co2, -1)
    N, Co, M = R[3], R[4], R[5]
    Na, Ca, Ma = s * N, s * Co, s * M
    Cr, Mr, Nr = Ca.sqrt(), Ma.sqrt(), Na.sqrt()
    Cc, Mz = Ca * Co / gz[4], s * gz[5]
    wlo += [Ma, Ma * Ma * dT, Ca]
    co2 += [Ca]
    n2o = [Na * dT, Nr, N * dT, Nr.sqrt(), Na, s * gz[3], s * gt[3], Na ** 2, gt[3], Nr * N / gz[3], Ma, Ma * gz[5],
           Ca, Ca * s * gz[4]]
    cop = [Ca, Ca * dT, Cr.sqrt(), Cr * dT, Ca ** 2, Cr, Ca * dT2, Cc, Cc / Cr, Cc * gz[4].sqrt()]
    ch4 = [Ma * dT, Mr, Ma ** 2, Ma, M * dT, Mz, Mz ** 2, Mr.sqrt(), gt[5], s * gt[5], Mr * M / gz[5]]
    return torch.stack(dry + wlo + cont + ozo + co2 + n2o + cop + ch4, -1)


def _column(tab, atm, sfc, geo, e, m, T, A, Ts, dev, per_channel):
    """One profile's clear column: T (..., Ku), A[j] (..., Ku), Ts and e (L); with ``per_channel`` the leading axis
    of T and A is the channel."""
    f8 = lambda v: torch.from_numpy(np.ascontiguousarray(v)).to(dev)  # noqa: E731
    K, Ku = tab.K, int(atm.n_layers[m])
    lev, lay = atm.level_pressure[m, :Ku + 1], atm.pressure[m, :Ku]
    W = f8(_layer_weights(np.log(tab.p), np.log(lay)))
    Tref = f8(tab.t)
    mapped = []
    for j, aid in enumerate(tab.ids):
        ref = f8(tab.a[:, j])
        if aid in A:
            v = (A[aid] @ W.T).clamp_min(_EPS)
            v = torch.minimum(torch.maximum(v, f8(tab.lo[:, j])), f8(tab.hi[:, j]))
        else:
            v = ref + 0 * Tref
            v = v.expand(*T.shape[:-1], K)
        mapped.append(v)
    pdp = np.empty(K)
    pdp[0] = tab.lev[0] * (tab.lev[1] - tab.lev[0])
    pdp[1:] = tab.lev[2:] * (tab.lev[2:] - tab.lev[1:-1])
    # slant path at each reference layer's height
    z = np.zeros(K + 1)
    h2o = tab.ids.index(1)
    for k in range(K, 0, -1):
        z[k - 1] = z[k] + _C_H * tab.t[k - 1] * (1 + _C_TV * tab.a[k - 1, h2o]) * math.log(tab.lev[k] / tab.lev[k - 1])
    zen, alt, psfc = math.radians(geo.sensor_zenith_angle[m]), float(geo.surface_altitude[m]), lev[-1]
    tzen = min(zen, math.radians(_TZ_MAX))
    lnl = np.log(tab.lev)
    if tab.lev[-1] >= psfc:
        i, frac = K, 0.0
        if tab.lev[-1] > psfc:
            i = int(np.nonzero(tab.lev < psfc)[0][-1]) + 1
            frac = (lnl[i] - math.log(psfc)) / (lnl[i] - lnl[i - 1])
        zoff = -(z[i] + frac * (z[i - 1] - z[i])) + alt
    else:
        zoff = _C_H * tab.t[-1] * math.log(1013.0 / tab.lev[-1])
    sa = (_R_EARTH + alt) * math.sin(tzen) / (_R_EARTH + z[1:] + zoff)
    s = f8(1.0 / np.sqrt(1.0 - sa * sa))
    X = _predictors(tab.group, T @ W.T, mapped, Tref, [f8(tab.a[:, j]) for j in range(len(tab.ids))], f8(pdp), s)
    od = torch.einsum("lks,ksl->lk" if per_channel else "ks,ksl->lk", X, tab.C).clamp(0.0, _OD_MAX)
    path = torch.cat([torch.zeros_like(od[:, :1]), od.cumsum(-1)], -1)
    # the path at the user's levels
    x, u = lnl, np.log(np.where(lev > 0, lev, lev[min(1, Ku)] / 2.0))
    hi = np.clip(np.searchsorted(x, u, side="left"), 1, K)
    fac = np.clip((u - x[hi - 1]) / (x[hi] - x[hi - 1]), 0.0, 1.0)
    hi_t, fac_t = torch.from_numpy(hi).to(dev), f8(fac)
    at = path[:, hi_t - 1] + (path[:, hi_t] - path[:, hi_t - 1]) * fac_t
    tau = (at[:, 1:] - at[:, :-1]) * math.cos(tzen)
    tr = torch.exp(-tau / math.cos(zen))
    c1, c2, b1, b2, cosmic = tab.spec
    planck = lambda v, k: k[0] / torch.expm1(k[1] / (k[2] + k[3] * v))  # noqa: E731
    col = [v[:, None] for v in (c1, c2, b1, b2)]
    B = planck(T if per_channel else T[None], col)
    down = cosmic
    for k in range(Ku):
        down = down * tr[:, k] + B[:, k] * (1 - tr[:, k])
    rad = e * planck(Ts, (c1, c2, b1, b2)) + (1 - e) * down
    for k in range(Ku - 1, -1, -1):
        rad = rad * tr[:, k] + B[:, k] * (1 - tr[:, k])
    return rad, (c2 / torch.log1p(c1 / rad) - b1) / b2


_EXACT_PAIRS = 40000      # profile-channel pairs of a K-matrix or adjoint that take under 20 s
_EXACT_FORWARD = 150      # profiles of a forward call


def exact(case, seed):
    """The clear-sky outputs by a plain torch model in 64 bits and its automatic derivatives.  None for the larger
    calls and for columns with clouds or aerosols, whose 64-bit solution (an eigenproblem per layer, channel and
    profile, and its derivatives) takes minutes."""
    call, P = case["call"], case["profiles"]
    L = sy.SENSORS[case["sensor"]][1] if case["channels"] == 0 else case["channels"]
    small = P <= _EXACT_FORWARD if call in ("forward", "host_forward") else P * L <= _EXACT_PAIRS and P <= 60
    if case["sky"] != "clear" or not small:
        return None
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    atm, sfc, geo, opt, rng = _host_inputs(case, seed)
    tab = _Tables(case["sensor"], case["channels"], dev)
    L, Km = tab.C.shape[2], atm.max_layers
    f8 = lambda v: torch.from_numpy(np.ascontiguousarray(v)).to(dev)  # noqa: E731
    derivs = call in ("k_matrix", "adjoint", "trajectory")
    J = atm.n_absorbers
    bt, rad = np.zeros((P, L)), np.zeros((P, L))
    kt, ka = np.zeros((P, L, Km)), np.zeros((P, L, J, Km))
    kw, ke = np.zeros((P, L)), np.zeros((P, L))
    for m in range(P):
        Ku = int(atm.n_layers[m])
        lead = (L,) if derivs else ()
        T = f8(atm.temperature[m, :Ku]).expand(*lead, Ku).clone().requires_grad_(derivs)
        A = {int(a): f8(atm.absorber[m, j, :Ku]).expand(*lead, Ku).clone().requires_grad_(derivs)
             for j, a in enumerate(atm.absorber_id)}
        ts = float(sum(getattr(sfc, c + "_coverage")[m] * getattr(sfc, c + "_temperature")[m]
                       for c in ("land", "water", "snow", "ice")))
        Ts = torch.full((L,), ts, dtype=torch.float64, device=dev, requires_grad=derivs)
        e = f8(opt.emissivity[m]).requires_grad_(derivs)
        r, b = _column(tab, atm, sfc, geo, e, m, T, A, Ts, dev, derivs)
        bt[m], rad[m] = b.detach().cpu().numpy(), r.detach().cpu().numpy()
        if derivs:
            g = torch.autograd.grad(b.sum(), [T, Ts, e] + list(A.values()), allow_unused=True)
            kt[m, :, :Ku], kw[m], ke[m] = (v.cpu().numpy() for v in g[:3])
            kw[m] *= sfc.water_coverage[m]
            for j, v in enumerate(g[3:]):
                if v is not None:
                    ka[m, :, j, :Ku] = v.cpu().numpy()
    if call == "host_forward":
        return dict(bt=bt, radiance=rad, up=None, down=None, layer_optical_depth=None, upwelling=None)
    if call == "forward":
        return dict(radiance=rad, bt=bt, status=np.zeros(P, np.int32))
    if call == "k_matrix":
        return dict(radiance=rad, bt=bt, status=np.zeros(P, np.int32), temperature_k=kt,
                    absorber_k=ka[:, :, _jacobians(atm)], water_temperature_k=kw, surface_emissivity_k=ke)
    w = rng.normal(0.0, 1.0, (P, L))
    ad = dict(temperature_ad=np.einsum("pl,plk->pk", w, kt), absorber_ad=np.einsum("pl,pljk->pjk", w, ka),
              water_temperature_ad=(w * kw).sum(1))
    if call == "adjoint":
        return dict(radiance=rad, bt=bt, status=np.zeros(P, np.int32), **ad)
    d = _perturbations(atm, sfc, rng)
    tl = (np.einsum("plk,pk->pl", kt, d["temperature"]) + np.einsum("pljk,pjk->pl", ka, d["absorber"]) +
          kw * d["water_temperature"][:, None])
    return dict(bt_tl=tl, **ad)

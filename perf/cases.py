"""Performance cases: the work a user of larndsim_gb300 runs, through the
public functions, from a single small event to the 64-event batch.

A case is a dict of plain values; ``kind`` names the path:

* ``predict``      LUTSimulation.predict: tracks to waveforms and hits
* ``wfs``          simulate_wfs: tracks to waveforms
* ``grad``         LUTChain.loss_and_grad_device: one fit step's loss and gradient
* ``hits``         simulate_stochastic: stored waveforms to hits, noise on
* ``param_wfs``    simulate_parametrized_wfs: the parametrised current's waveforms
* ``param_grad``   param_wfs_fn + fee_adc + SSE + backward: a parametrised fit step
* ``prob_values``  average_hit_values + backward: the probabilistic fit's front end
* ``prob_predict`` simulate_probabilistic: the full hit distributions
* ``loss``         mse_adc / nll_loss / chamfer_3d of hits against target hits + backward
* ``chop``         chop_tracks: segments to fixed-length steps

The LUT is the package's synthetic 45 x 45 x 1950 response with 100
long-diffusion templates, number_pix_neighbors = 4, signal length 150.
"""

import functools
import math
import sys
from pathlib import Path

import numpy as np
import torch

sys.path.insert(0, str(Path(__file__).resolve().parent.parent / "larnd-sim-jax_gb300"))

from larndsim_gb300 import consts, dataio, grad, losses, sim, strategies, workloads  # noqa: E402

MUON_SEGMENTS = 60        # segments per muon track of workloads.muon_event
PIXELS_PER_SEGMENT = 0.21  # simulated pixels per segment of the mixed events
HITS_PER_PIXEL = 4.5
TICKS = 2000
HITS = 10                 # MAX_ADC_VALUES
WINDOW = 152              # ticks one contribution touches
NEIGHBOURS = 320          # neighbour contributions per simulated pixel on the mixed events


def listed():
    return [
        # a few small cosmic events through the whole LUT chain: the smallest call, latency and launches
        {"name": "predict_muons", "kind": "predict", "events": 6, "muons": 2},
        # waveforms of a batch of 64 events, 1k to 50k segments each: the forward at its largest
        {"name": "wfs_64_events", "kind": "wfs", "events": 64, "lo": 1000, "hi": 50000},
        # one fit step on one ordinary event
        {"name": "grad_1_event", "kind": "grad", "events": 1, "lo": 5000, "hi": 5000},
        # one fit step on the 64-event batch: the package's headline workload
        {"name": "grad_64_events", "kind": "grad", "events": 64, "lo": 1000, "hi": 50000},
        # the self-trigger front end on stored waveforms with the default noise
        {"name": "hits_30000_rows", "kind": "hits", "rows": 30000},
        # parametrised mode, forward and one fit step
        {"name": "param_wfs_32_events", "kind": "param_wfs", "events": 32, "lo": 1000, "hi": 50000},
        {"name": "param_grad_16_events", "kind": "param_grad", "events": 16, "lo": 1000, "hi": 50000},
        # the probabilistic front end of a likelihood-style fit: expected hits and their gradient
        {"name": "prob_values_1500_rows", "kind": "prob_values", "rows": 1500},
        # its full distributions, as LUTProbabilisticSimulation returns them
        {"name": "prob_predict_1000_rows", "kind": "prob_predict", "rows": 1000},
        # the fitter's default loss on the hits of the 64-event batch, with its gradient
        {"name": "mse_adc_64_events", "kind": "loss", "fn": "mse_adc", "events": 64, "lo": 1000, "hi": 50000},
        # another hit-level loss on an ordinary batch
        {"name": "nll_8_events", "kind": "loss", "fn": "nll_loss", "events": 8, "lo": 1000, "hi": 20000},
        # the input side: a shower cut into 0.001 cm steps (the loader's default)
        {"name": "chop_200k_segments", "kind": "chop", "segments": 200000, "precision": 0.001},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["predict", "wfs", "grad", "hits", "param_wfs", "param_grad", "prob_values", "prob_predict",
                       "loss", "chop"])
    if kind == "predict":
        return {"kind": kind, "events": rng.randint(5, 12), "muons": rng.randint(1, 5)}
    if kind == "hits":
        return {"kind": kind, "rows": _log(rng, 300, 30000)}
    if kind == "prob_values":
        return {"kind": kind, "rows": _log(rng, 40, 1500)}
    if kind == "prob_predict":
        return {"kind": kind, "rows": _log(rng, 40, 1000)}
    if kind == "chop":
        return {"kind": kind, "segments": _log(rng, 1000, 200000), "precision": rng.choice([0.001, 0.003, 0.01])}
    top = {"wfs": 48, "grad": 48, "param_wfs": 32, "param_grad": 16, "loss": 24}[kind]
    lo = _log(rng, 300, 5000)
    c = {"kind": kind, "events": _log(rng, 1, top), "lo": lo, "hi": _log(rng, lo, 25000)}
    if kind == "loss":
        c["fn"] = rng.choice(["mse_adc", "nll_loss", "chamfer_3d"])
    return c


# ---------------------------------------------------------------- inputs

# The geometry of a case (its tracks) is fixed by its sizes, so that arrays keep
# their shapes from seed to seed; the seed draws the deposited energies, the
# order of events and rows, the noise, the hit charges and the fit parameters.

@functools.lru_cache(maxsize=1)
def _response():
    return workloads.synthetic_response(seed=0)    # the detector's calibration: the same for every input


def _params(**kw):
    base = dict(number_pix_neighbors=4, signal_length=150, RESET_NOISE_CHARGE=0, UNCORRELATED_NOISE_CHARGE=0)
    base.update(kw)
    return consts.Params(**base)


def _lut(params):
    templates, params = sim.load_lut(_response(), params)
    return sim.prepare_lut(templates, params), params


@functools.lru_cache(maxsize=4)
def _geometry(events, lo, hi):
    return workloads.batched_events(seed=events + 7 * lo + 13 * hi, n_events=events, min_segments=lo, max_segments=hi)


def _tracks(events, lo, hi, seed):
    """A batch whose deposited energies the seed scales, row by row."""
    t, fields = _geometry(events, lo, hi)
    t = t.copy()
    f = np.random.default_rng(seed).uniform(0.7, 1.3, t.shape[0]).astype(np.float32)
    for k in ("dE", "dEdx"):
        t[:, fields.index(k)] *= f
    return torch.from_numpy(t).cuda(), fields


def _muon_events(events, muons, seed):
    """Events of a few muons each, their order drawn by the seed."""
    parts = []
    for ev, source in enumerate(np.random.default_rng(seed).permutation(events)):
        t, fields = workloads.muon_event(seed=100 * muons + int(source), n_tracks=muons, event_id=ev)
        parts.append(t)
    return torch.from_numpy(np.concatenate(parts)).cuda(), fields


def _perturbed(params, seed):
    """Every fit parameter off by a few per cent, as in the middle of a fit."""
    rng = np.random.default_rng(seed + 77)
    return params.replace(**{k: float(getattr(params, k)) * (1 + 0.05 * rng.standard_normal())
                             for k in grad.GRAD_PARAMS})


def _rows(n, seed, params):
    """(waveforms, pixel ids) of n simulated pixels of 8k-segment events, the
    rows of one batch in an order drawn by the seed."""
    lut, params = _lut(params)
    t, fields = _tracks(-(-n // 1000), 8000, 8000, 0)
    sim.reset_size_history()
    wfs, unique = sim.simulate_wfs(params, lut, t, fields)
    at = (unique >= 0).nonzero()[:, 0]
    at = at[torch.linspace(0, at.shape[0] - 1, n, device="cuda").long()]
    at = at[torch.randperm(n, generator=_generator(seed), device="cuda")]
    return wfs[at].contiguous(), unique[at].contiguous(), params


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _jitter(t, seed, width):
    return t * (1 + width * torch.randn(t.shape, generator=_generator(seed), device="cuda"))


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if "lo" in case:
        batch = (case["events"], case["lo"], case["hi"])
    if kind == "predict":
        lut, s["params"] = _lut(_params())
        s["tracks"], s["fields"] = _muon_events(case["events"], case["muons"], seed)
        s["strategy"] = strategies.LUTSimulation(lut)
    elif kind == "wfs":
        s["lut"], s["params"] = _lut(_params())
        s["tracks"], s["fields"] = _tracks(*batch, seed)
    elif kind == "grad":
        lut, params = _lut(_params())
        tracks, fields = _tracks(*batch, seed)
        s["chain"] = grad.LUTChain(params, lut, tracks, fields, n_events=case["events"])
        s["target"] = s["chain"].target(params)
        s["params"] = _perturbed(params, seed)
    elif kind == "hits":
        s["wfs"], s["unique"], s["params"] = _rows(case["rows"], seed, _params(RESET_NOISE_CHARGE=900,
                                                                               UNCORRELATED_NOISE_CHARGE=500))
        # the noise goes with its row, so that the number of hits stays
        normals = torch.randn((case["rows"], 1 + 3 * HITS), generator=_generator(1), device="cuda")
        s["normals"] = normals[torch.randperm(case["rows"], generator=_generator(seed), device="cuda")]
    elif kind in ("param_wfs", "param_grad"):
        s["tracks"], s["fields"] = _tracks(*batch, seed)
        s["params"] = _params(number_pix_neighbors=0, mc_diff=True)
        s["offsets"] = torch.randn((s["tracks"].shape[0], 3), generator=_generator(2), device="cuda")
        if kind == "param_grad":
            with torch.no_grad():
                theta = grad.theta_of(s["params"], device="cuda")
                wfs, unique = sim.param_wfs_fn(theta, s["params"], s["tracks"], s["fields"], s["offsets"])
                s["target"], _ = sim.fee_adc(s["params"], wfs[unique >= 0])
            # the pixels stay the target's: the diffusion and drift parameters are not moved
            s["params"] = s["params"].replace(lifetime=s["params"].lifetime * 1.05, Ab=s["params"].Ab * 0.97)
    elif kind == "prob_values":
        s["wfs"], _, s["params"] = _rows(case["rows"], seed, _params(RESET_NOISE_CHARGE=900))
        s["cot"] = [torch.randn((case["rows"], HITS), generator=_generator(seed + k), device="cuda") for k in range(3)]
    elif kind == "prob_predict":
        s["wfs"], s["unique"], s["params"] = _rows(case["rows"], seed, _params(RESET_NOISE_CHARGE=900))
    elif kind == "loss":
        lut, params = _lut(_params())
        tracks, fields = _tracks(*batch, 0)
        chain = grad.LUTChain(params, lut, tracks, fields, n_events=case["events"])
        with torch.no_grad():
            for k, (name, p) in enumerate((("ref", params), ("pred", _perturbed(params, 0)))):
                q, x, y, z, *rest = (t.detach() for t in grad.predicted_hits(grad.theta_of(p, device="cuda"), chain, p))
                s[name] = [_jitter(q, seed + k, 0.1), x, y, _jitter(z, seed + 2 + k, 0.01), *rest]
        s["params"], s["fn"] = params, getattr(losses, case["fn"])
    else:
        t, s["fields"] = workloads.large_shower_event(seed=case["segments"], n_segments=case["segments"])
        s["tracks"] = torch.from_numpy(t[np.random.default_rng(seed).permutation(t.shape[0])]).cuda()
    return s


# ---------------------------------------------------------------- one pass

def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind in ("predict", "wfs", "param_wfs", "param_grad", "loss"):
        sim.reset_size_history()     # a pass's row counts do not depend on the passes before it
    if kind == "predict":
        return s["strategy"].predict(s["params"], s["tracks"], s["fields"], 0)
    if kind == "wfs":
        return sim.simulate_wfs(s["params"], s["lut"], s["tracks"], s["fields"])
    if kind == "grad":
        return s["chain"].loss_and_grad_device(s["params"], s["target"])
    if kind == "hits":
        return sim.simulate_stochastic(s["params"], s["wfs"], s["unique"], normals=s["normals"])
    if kind == "param_wfs":
        return sim.simulate_parametrized_wfs(s["params"], s["tracks"], s["fields"], offsets=s["offsets"])
    if kind == "param_grad":
        theta = grad.theta_of(s["params"], device="cuda").requires_grad_(True)
        wfs, unique = sim.param_wfs_fn(theta, s["params"], s["tracks"], s["fields"], s["offsets"])
        adc, _ = sim.fee_adc(s["params"], wfs[unique >= 0])
        loss = ((adc - s["target"]) ** 2).sum()
        loss.backward()
        return loss.detach(), theta.grad
    if kind == "prob_values":
        w = s["wfs"].detach().requires_grad_(True)
        out = sim.average_hit_values(s["params"], w)
        torch.autograd.backward(out, s["cot"])
        return [o.detach() for o in out], w.grad
    if kind == "prob_predict":
        return sim.simulate_probabilistic(s["params"], s["wfs"], s["unique"])
    if kind == "loss":
        q, x, y, z, t, hp, ev = s["pred"]
        q, z = q.detach().requires_grad_(True), z.detach().requires_grad_(True)
        loss, _ = s["fn"](s["params"], q, x, y, z, t, hp, ev, *s["ref"])
        loss.backward()
        return loss.detach(), q.grad, z.grad
    return dataio.chop_tracks(s["tracks"], s["fields"], case["precision"])


def _segments(case):
    if "muons" in case:
        return case["events"] * case["muons"] * MUON_SEGMENTS
    lo, hi = case["lo"], case["hi"]
    mean = lo if hi <= lo else (hi - lo) / math.log(hi / lo)    # of a log-uniform draw
    return case["events"] * mean


def work(case):
    kind = case["kind"]
    if kind in ("hits", "prob_values", "prob_predict"):
        n = case["rows"]
        if kind == "hits":     # the rows read, 8 hit columns written; a few operations per tick and hit
            return {"bytes": n * (4 * TICKS + 32 * HITS_PER_PIXEL), "flops": n * TICKS * (2 + 4 * HITS_PER_PIXEL)}
        # 20 paths x 10 steps per tick, five log_ndtr and the log-sum-exps of each (about 100 operations)
        f = n * TICKS * 20 * HITS * 100
        if kind == "prob_predict":
            return {"bytes": n * (4 * TICKS + 8 * TICKS * HITS), "flops": f}
        return {"bytes": n * (8 * TICKS + 24 * HITS), "flops": 3 * f}
    if kind == "chop":
        steps = case["segments"] * (0.1 / case["precision"] + 0.5)
        return {"bytes": 104 * (case["segments"] + steps), "flops": 30 * steps}
    seg = _segments(case)
    if kind in ("param_wfs", "param_grad"):
        pix = 0.12 * seg
        f = seg * 51 * 4 * 60     # four error-function edges per tick
        if kind == "param_wfs":
            return {"bytes": 64 * seg + 4 * TICKS * pix, "flops": f}
        return {"bytes": 64 * seg + 8 * HITS * pix, "flops": 5 * f}
    pix = PIXELS_PER_SEGMENT * seg
    if kind == "loss":
        hits = pix * HITS_PER_PIXEL
        per = hits / case["events"]
        pairs = {"mse_adc": 3, "nll_loss": 2, "chamfer_3d": 2}[case["fn"]] * hits * per
        return {"bytes": hits * (14 * 4 + 8), "flops": 12 * pairs}
    f = (pix * NEIGHBOURS + 2 * seg * 25) * WINDOW * 4
    if kind == "grad":
        return {"bytes": 52 * seg + 4 * HITS * pix, "flops": 2 * f}
    return {"bytes": 52 * seg + 4 * TICKS * pix, "flops": f}


# ---------------------------------------------------------------- in 64 bits

def exact(case, seed):
    """What ``run`` returns, in float64 on float32's own discrete decisions
    (bins, pixels, ticks, stacked coordinates).  None where a value follows
    from threshold crossings of the float32 cumulative charge (hits, and the
    gradients taken through them) and for the cases that would take long."""
    kind = case["kind"]
    if kind in ("wfs", "predict"):
        if _segments(case) > 30000:
            return None
        s = prepare(case, seed)
        wfs = _exact_lut_wfs(s["params"], s["tracks"], s["fields"])
        if kind == "wfs":
            return [wfs, None]
        keys = ("adcs", "pixel_x", "pixel_y", "pixel_z", "ticks", "hit_prob", "event", "hit_pixels", "unique_pixels")
        return {"wfs": wfs, **{k: None for k in keys}}
    if kind == "param_wfs":
        s = prepare(case, seed)
        return [_exact_param_wfs(s["params"], s["tracks"], s["fields"], s["offsets"]), None]
    if kind in ("prob_values", "prob_predict"):
        s = prepare(case, seed)
        if kind == "prob_values":
            return [list(_exact_prob(s["params"], s["wfs"], True)), None]
        log_prob, adc = _exact_prob(s["params"], s["wfs"], False)
        return [adc, None, None, log_prob, None]
    if kind == "loss":
        s = prepare(case, seed)
        return _exact_loss(case["fn"], s["pred"], s["ref"])
    if kind == "chop" and case["segments"] <= 200000:
        s = prepare(case, seed)
        return _exact_chop(s["tracks"], s["fields"], case["precision"])
    return None


def _f32(v):
    return torch.tensor(float(np.float32(v)), dtype=torch.float32, device="cuda")


def _drifted(params, tracks, fields):
    """Quench and drift of every segment: float64 values from the float32
    columns, and the float32 values that take the discrete decisions."""
    col = {f: tracks[:, i] for i, f in enumerate(fields)}
    b = torch.as_tensor(np.asarray(params.tpc_borders, np.float32), device="cuda")
    z = col["z"]
    m = params.size_margin
    inside = [((z >= b[i, 2].min() - m) & (z <= b[i, 2].max() + m)) for i in range(b.shape[0])]
    plane = torch.where(inside[0], 0, 1)
    mask = torch.zeros_like(inside[0])
    for i in range(b.shape[0]):
        mask |= (inside[i] & (col["x"] >= b[i, 0, 0] - m) & (col["x"] <= b[i, 0, 1] + m)
                 & (col["y"] >= b[i, 1, 0] - m) & (col["y"] <= b[i, 1, 1] + m))
    d = {k: v.double() for k, v in col.items()}
    v = consts.get_vdrift(params)
    za, zc = b[plane, 2, 0], b[plane, 2, 1]
    tdr = ((d["z"] - za.double()).abs() + 1e-6) / v
    ne = params.Ab / (1 + params.kb * d["dEdx"] / (params.eField * params.lArDensity)) * d["dE"] * params.MeVToElectrons
    ne = ne * torch.exp(-tdr / params.lifetime) * mask
    tdr32 = ((z - za).abs() + _f32(1e-6)) / _f32(v)
    return dict(col=col, d=d, b=b, plane=plane, ne=ne, tdr=tdr, tdr32=tdr32, za=za, zc=zc, v=v,
                event=col["eventID"].long())


def _floordiv32(a, w):
    m = torch.fmod(a, w)
    q = (a - m) / w
    q = torch.where((m != 0) & (m < 0), q - 1, q)
    return torch.where(q >= 0, torch.floor(q + 0.5), torch.ceil(q - 0.5)).long()


def _pixel_ids(params, px, py, plane, event):
    pid = ((event * params.tpc_borders.shape[0] + plane) * params.n_pixels_y + py) * params.n_pixels_x + px
    ok = (px >= 0) & (py >= 0) & (px < params.n_pixels_x) & (py < params.n_pixels_y)
    return torch.where(ok, pid, -1)


def _bank_window(params, L):
    """(windows [T][nx][ny][L + 1] from tick Nt - L - 1 on, cumulative sums of
    template 0 and of the 5 x 5 main positions) of the long-diffusion bank."""
    r = torch.as_tensor(_response(), device="cuda").double()
    nx, ny, nt = r.shape
    ext = params.long_diff_extent
    j = torch.arange(-ext, ext + 1, device="cuda", dtype=torch.float64)
    main = r[:5, :5].reshape(25, 1, nt)
    banks = [main[:, 0]]
    for sg in np.asarray(params.long_diff_template, np.float64)[1:]:
        g = torch.exp(-0.5 * (j / sg) ** 2)
        banks.append(torch.nn.functional.conv1d(main, (g / g.sum()).reshape(1, 1, -1), padding=ext)[:, 0])
    return r, torch.stack(banks).reshape(-1, 5, 5, nt)


def _exact_lut_wfs(params, tracks, fields):
    s = _drifted(params, tracks, fields)
    L, nb, n = params.signal_length, params.nb_sampling_bins_per_pixel, params.number_pix_neighbors
    NT = consts.n_ticks(params)
    r, main = _bank_window(params, L)
    nt = r.shape[2]
    c0, cmain = r.cumsum(2), main.cumsum(3)
    width = _f32(params.pixel_pitch / nb)
    frac_bin, bins, inte = {}, {}, {}
    sig = torch.sqrt(2 * s["tdr"] * params.tran_diff)
    edges = torch.as_tensor(consts.tran_diff_bin_edges(params), device="cuda").double()
    for a, k in ((0, "x"), (1, "y")):
        rel = s["col"][k] - s["b"][s["plane"], a, 0]
        bins[k] = _floordiv32(rel, width)
        m = torch.fmod(rel, width)
        x0 = torch.where((m != 0) & (m < 0), m + width, m).double()
        e = torch.erf((edges[None, 1:-1] - x0[:, None]) / (math.sqrt(2) * sig[:, None]))
        one = torch.ones_like(e[:, :1])
        inte[k] = 0.5 * torch.diff(torch.cat([-one, e, one], dim=1), dim=1)
    ft32 = ((s["col"]["z"] - s["zc"]).abs() / _f32(s["v"])) / _f32(params.t_sampling)
    cath = ft32.floor().clamp(0, nt - 1).long()
    frac = (s["d"]["z"] - s["zc"].double()).abs() / s["v"] / params.t_sampling - cath
    grid32 = torch.as_tensor(np.asarray(params.long_diff_template, np.float32), device="cuda")
    ld32 = (torch.sqrt((s["tdr32"] * 2) * _f32(params.long_diff)) / _f32(s["v"])) / _f32(params.t_sampling)
    idx = torch.searchsorted(grid32, ld32.contiguous()).clamp(1, grid32.shape[0] - 2)
    ld = torch.sqrt(2 * s["tdr"] * params.long_diff) / s["v"] / params.t_sampling
    X = [grid32.double()[idx + q] for q in (-1, 0, 1)]
    q3 = [(ld - X[1]) * (ld - X[2]) / ((X[0] - X[1]) * (X[0] - X[2])),
          (ld - X[0]) * (ld - X[2]) / ((X[1] - X[0]) * (X[1] - X[2])),
          (ld - X[0]) * (ld - X[1]) / ((X[2] - X[0]) * (X[2] - X[1]))]
    px, py = bins["x"].div(nb, rounding_mode="floor"), bins["y"].div(nb, rounding_mode="floor")
    pid = _pixel_ids(params, px, py, s["plane"], s["event"])
    unique = torch.unique(pid)
    has_m1 = bool((unique < 0).any())
    unique = unique[unique >= 0]
    rows = int((unique.shape[0] + has_m1 + 1) * 1.1 + 0.5)      # pad_size's bucket of a fresh history
    out = torch.zeros(rows * NT, dtype=torch.float64, device="cuda")
    k = torch.arange(L + 2, device="cuda")

    def lut_index(b, shift):
        return (b.remainder(nb) - nb // 2 + 0.5 - shift).abs().long()

    def add(pixel, win, corr, weight):
        """win (S, L): samples; corr (S,): the boundary term; per segment."""
        at = torch.searchsorted(unique, pixel).clamp(max=unique.shape[0] - 1)
        use = ((unique[at] == pixel) & (pixel >= 0)).nonzero()[:, 0]
        if use.numel() == 0:
            return
        w, cr, f = win(use) * weight[use, None], corr(use) * weight[use], frac[use, None]
        z = torch.zeros_like(w[:, :2])
        vals = torch.cat([z, w], 1) * (1 - f) + torch.cat([z[:, :1], w, z[:, :1]], 1) * f
        col = nt - L - cath[use, None] - 1 + k[None]
        vals = torch.where((col >= 2) & (col <= NT - 1), vals, 0.0)
        cc = torch.cat([cr[:, None] * f, cr[:, None] * (1 - f)], 1)
        vals[:, :2] += torch.where((col[:, :2] >= 1) & (col[:, :2] <= NT - 2), cc, 0.0)
        flat = (rows - unique.shape[0] + at[use, None]) * NT + col
        ok = (col >= 1) & (col <= NT - 1)
        out.index_add_(0, flat[ok], vals[ok])

    def lerp(cum, use):
        f, c = frac[use], cath[use]
        row = torch.arange(use.shape[0], device="cuda")
        return cum[row, nt - L] - (cum[row, c] * (1 - f) + cum[row, (c + 1).clamp(max=nt - 1)] * f)

    for dx in range(-n, n + 1):
        for dy in range(-n, n + 1):
            if dx == 0 and dy == 0:
                continue
            cx, cy = lut_index(bins["x"], dx * nb), lut_index(bins["y"], dy * nb)
            p = _pixel_ids(params, px + dx, py + dy, s["plane"], s["event"])
            add(p, lambda u: r[cx[u], cy[u], nt - L:], lambda u: lerp(c0[cx[u], cy[u]], u), s["ne"])
    for i in range(5):
        for j in range(5):
            bi, bj = bins["x"] + i - 2, bins["y"] + j - 2
            p = _pixel_ids(params, bi.div(nb, rounding_mode="floor"), bj.div(nb, rounding_mode="floor"), s["plane"],
                           s["event"])
            u_, v_ = lut_index(bi, 0), lut_index(bj, 0)

            def win(u):
                return sum(q[u, None] * main[idx[u] + o, u_[u], v_[u], nt - L:] for q, o in zip(q3, (-1, 0, 1)))

            # the boundary term of a main position is the central template's alone
            add(p, win, lambda u: lerp(cmain[idx[u], u_[u], v_[u]], u), s["ne"] * inte["x"][:, i] * inte["y"][:, j])
    return out.reshape(rows, NT)[:, 1:]


def _exact_param_wfs(params, tracks, fields, offsets):
    s = _drifted(params, tracks, fields)
    NT, n = consts.n_ticks(params), int(5 / params.t_sampling) + 1
    sT32 = torch.sqrt((s["tdr32"] * 2) * _f32(params.tran_diff))
    sT = torch.sqrt(2 * s["tdr"] * params.tran_diff)
    pix, dist = {}, {}
    pitch = _f32(params.pixel_pitch)
    for a, k in ((0, "x"), (1, "y")):
        b0 = s["b"][s["plane"], a, 0]
        pix[k] = _floordiv32((s["col"][k] + offsets[:, a] * sT32) - b0, pitch)
        centre = pix[k].double() * params.pixel_pitch + b0.double() + params.pixel_pitch / 2
        dist[k] = (s["d"][k] + offsets[:, a].double() * sT - centre).abs()
    t0_32 = (s["col"]["z"] - s["za"]).abs() / _f32(s["v"])
    tick = (t0_32 / _f32(params.t_sampling) + 0.5).long()
    t0 = (s["d"]["z"] - s["za"].double()).abs() / s["v"] - tick * params.t_sampling
    x, y = dist["x"], dist["y"]

    def quad(c):
        return c[0] + c[1] * x + c[2] * y + c[3] * x * y + c[4] * x * x + c[5] * y * y

    a = quad((1.060, -0.909, -0.909, 5.856, 0.207, 0.207)).clamp(max=1)
    rb = 1 / quad((0.679, -1.083, -1.083, 8.772, -5.521, -5.521))
    rc = 1 / quad((2.644, -9.174, -9.174, 13.483, 45.887, 45.887))
    loc = -(t0 + quad((2.948, -2.705, -2.705, 4.825, 20.814, 20.814)))
    sg = torch.sqrt(2 * s["tdr"] * params.long_diff) / s["v"]
    dt = 5.0 / (n - 1)
    t = -torch.linspace(0, 5, n, dtype=torch.float64, device="cuda")

    def edge(e, lam):
        lam, l, d = lam[:, None], loc[:, None], sg[:, None]
        # exp(u) erfc(v) of the exponentially modified Gaussian, v >= 0 through erfcx so that u may be large
        v = (l + lam * d * d - e) / (math.sqrt(2) * d)
        u = lam / 2 * (2 * l + lam * d * d - 2 * e)
        ee = torch.where(v > 0, torch.special.erfcx(v.clamp(min=0)) * torch.exp(u - v * v),
                         torch.exp(u.clamp(max=700)) * torch.erfc(v))
        return 0.5 * torch.erf((e - l) / (math.sqrt(2) * d)) - 0.5 * ee

    pid = _pixel_ids(params, pix["x"], pix["y"], s["plane"], s["event"])
    unique = torch.unique(pid)
    rows = int(unique.shape[0] * 1.025 + 0.5)
    unique = unique[unique >= 0]
    out = torch.zeros(rows * NT, dtype=torch.float64, device="cuda")
    at = torch.searchsorted(unique, pid).clamp(max=unique.shape[0] - 1)
    cur = 0.0
    for w, lam in ((a, rb), (1 - a, rc)):
        up, lo = edge((t + dt / 2)[None], lam), edge((t - dt / 2)[None], lam)
        cur = cur + w[:, None] * (up - lo) / (lo[:, :1] - up[:, -1:]) / dt
    tt = tick[:, None] - n + torch.arange(n, device="cuda")[None]
    ok = (tt >= 0) & (tt < NT - 1) & (pid >= 0)[:, None]
    flat = (rows - unique.shape[0] + at)[:, None] * NT + tt + 1
    out.index_add_(0, flat[ok], (cur * s["ne"][:, None])[ok])
    return out.reshape(rows, NT)[:, 1:]


def _exact_prob(params, wfs, values):
    """The beam search of the probabilistic front end in float64 (its own top-K choices)."""
    K, H, gap = params.fee_paths_scaling, params.MAX_ADC_VALUES, consts.fee_interval(params)
    zs, thr = 1.0 / params.RESET_NOISE_CHARGE, params.DISCRIMINATION_THRESHOLD
    P, T = wfs.shape
    t = torch.arange(T - 1, device="cuda")
    sh = (t + gap + 1).clamp(max=T - 1)
    fe, nx = (sh + gap + 1).clamp(max=T - 1), (sh + 1).clamp(max=T - 1)

    def softplus(v):
        return v.clamp(min=0) + torch.log1p(torch.exp(-v.abs()))

    def logdiff(a, b, la, lb):
        neg = -torch.expm1(torch.where(a > b, lb - la, -1.0))
        neg = 1e-30 + softplus((neg - 1e-30) * 1e10) / 1e10
        lt = -100 + softplus((torch.log(neg) + 100) * 10) / 10
        w = torch.sigmoid((a - b) * 1000)
        return w * (la + lt) + (1 - w) * -1000.0

    def digitize(c):
        v = ((c * params.GAIN + params.V_PEDESTAL - params.V_CM).clamp(min=0) * params.ADC_COUNTS
             / (params.V_REF - params.V_CM))
        return v.clamp(max=float(params.ADC_COUNTS))

    outs, lps = [], []
    state = []
    for i in range(0, P, 64):
        q = (wfs[i:i + 64].double() * params.t_sampling).cumsum(1)
        c = torch.zeros((q.shape[0], K), dtype=torch.float64, device="cuda")
        lp = torch.full_like(c, -1000.0)
        lp[:, 0] = 0
        esp = q[:, sh] + thr - 0.5 * (q[:, 1:] + q[:, :-1])
        gate = torch.sigmoid((esp - thr) * 10)[:, None]
        cm = q.cummax(1).values
        cr = q.flip(1).cummax(1).values.flip(1)
        hits, alive = [], []
        for _ in range(H):
            zm = (cm[:, None] - c[..., None] - thr) * zs
            lm = torch.special.log_ndtr(zm)
            lg = logdiff(zm[..., 1:], zm[..., :-1], lm[..., 1:], lm[..., :-1])
            zq = (q[:, None] - c[..., None] - thr) * zs
            lq = torch.special.log_ndtr(zq)
            le = torch.minimum(logdiff(zq[..., sh], zq[..., :-1], lq[..., sh], lq[..., :-1]), lg)
            le = -1000 + softplus(le + 1000)
            le = gate * le + (1 - gate) * -1000.0
            hit = torch.logsumexp(le + lp[..., None], 1)
            dist = torch.logsumexp(lg + lp[..., None], 1)
            sel = torch.logsumexp(lg + torch.special.log_ndtr((cr[:, fe] - q[:, nx] - thr) * zs)[:, None]
                                  + lp[..., None], 1)
            top = sel.topk(K, dim=1).indices
            lp, c = dist.gather(1, top), q.gather(1, nx[top])
            hits.append(hit)
            alive.append(torch.logsumexp(lp, 1).max())
        state.append(torch.stack(alive))
        hits = torch.stack(hits, 1)
        adc = digitize(esp)[:, None].expand(-1, H, -1)
        if values:
            p = hits.exp()
            lam = p.sum(2)
            den = lam.clamp(min=1e-10)
            outs.append(torch.stack([(p * t).sum(2) / den, (p * adc).sum(2) / den, lam]))
        else:
            outs.append(adc.clone())
            lps.append(hits)
    live = torch.stack(state).max(0).values > math.log(1e-9)      # the whole batch stops together
    steps = 1 + int(live.long().cumprod(0)[:-1].sum())
    if values:
        o = torch.cat(outs, 1)
        o[:, :, steps:] = 0
        return o[0], o[1], o[2]
    log_prob, adc = torch.cat(lps), torch.cat(outs)
    log_prob[:, steps:] = -1000.0
    adc[:, steps:] = digitize(torch.zeros((), dtype=torch.float64, device="cuda"))
    return log_prob, adc


def _exact_loss(fn, pred, ref):
    """Loss, dL/dQ and dL/dz on the float32 stacked coordinates, event by event."""
    Q, x, y, z, _, hp, ev = pred
    rQ, rx, ry, rz, _, rhp, rev = ref
    off = 1e5 if fn == "mse_adc" else 1e9
    A = torch.stack([(x + ev.float() * off), y, z], 1).double()
    B = torch.stack([(rx + rev.float() * off), ry, rz], 1).double()
    n_ev = int(max(ev.max(), rev.max())) + 1
    pairs = sum(float((ev == e).sum()) * float((rev == e).sum()) for e in range(n_ev))
    if pairs > 2.5e10 or fn == "chamfer_3d":     # nearest neighbours: a choice, and zero padding up to a bucket
        return None

    def sums(R, C, w, more=()):
        """sum_j w_j K_ij times 1, (z_i - z_j) and any further differences."""
        got = torch.zeros((2 + len(more), R.shape[0]), dtype=torch.float64, device="cuda")
        step = max(1, int(2e8 // max(1, C.shape[0])))
        for i in range(0, R.shape[0], step):
            r = R[i:i + step]
            d = (r[:, None, 0] - C[None, :, 0]).square_()
            for a in range(1, R.shape[1]):
                d += (r[:, None, a] - C[None, :, a]).square_()
            k = d.mul_(-0.5).exp_()
            got[0, i:i + step] = k @ w
            for m, a in enumerate((2,) + tuple(more)):
                got[1 + m, i:i + step] = r[:, a] * got[0, i:i + step] - k @ (w * C[:, a])
        return got

    f = [torch.zeros(Q.shape[0], dtype=torch.float64, device="cuda") for _ in range(6)]
    if fn == "mse_adc":
        w, v = (Q * hp).double(), (rQ * rhp).double()
        c = torch.zeros_like(v)
        for e in range(n_ev):
            i, j = (ev == e).nonzero()[:, 0], (rev == e).nonzero()[:, 0]
            if i.numel():
                f[0][i], f[1][i] = sums(A[i], A[i], w[i])
            if i.numel() and j.numel():
                f[2][i], f[3][i] = sums(A[i], B[j], v[j])
            if j.numel():
                c[j] = sums(B[j], B[j], v[j])[0]
        sw, sv = w.sum(), v.sum()
        aa, bb, cc = (w * f[0]).sum(), (w * f[2]).sum(), (v * c).sum()
        rel = (sw - sv) / (sv + 1e-6)
        loss = aa / sw ** 2 + cc / sv ** 2 - 2 * bb / (sw * sv) + rel ** 2
        gw = (2 * f[0] / sw ** 2 - 2 * aa / sw ** 3 - 2 * f[2] / (sw * sv) + 2 * bb / (sw ** 2 * sv)
              + 2 * rel / (sv + 1e-6))
        return [loss, gw * hp.double(), -2 * w * (f[1] / sw ** 2 - f[3] / (sw * sv))]
    A = torch.cat([A, (Q / 10).double()[:, None]], 1)
    B = torch.cat([B, (rQ / 10).double()[:, None]], 1)
    lam = torch.zeros(rQ.shape[0], dtype=torch.float64, device="cuda")
    for e in range(n_ev):
        i, j = (ev == e).nonzero()[:, 0], (rev == e).nonzero()[:, 0]
        if i.numel() and j.numel():
            lam[j] = sums(B[j], A[i], hp[i].double())[0]
    for e in range(n_ev):
        i, j = (ev == e).nonzero()[:, 0], (rev == e).nonzero()[:, 0]
        if i.numel() and j.numel():
            use = (rhp[j] > 0.5).double() / (lam[j] + 1e-10)
            f[0][i], f[1][i], f[2][i] = sums(A[i], B[j], use, (3,))
    loss = hp.double().sum() - torch.log(lam[rhp > 0.5] + 1e-10).sum()
    return [loss, hp * f[2] / 10, hp * f[1]]


def _exact_chop(tracks, fields, precision):
    """The reference's float32 step counts, float64 positions."""
    c = {f: i for i, f in enumerate(fields)}
    s = tracks[:, [c["x_start"], c["y_start"], c["z_start"]]]
    e = tracks[:, [c["x_end"], c["y_end"], c["z_end"]]]
    seg = e - s
    sq = seg * seg
    length = torch.sqrt((sq[:, 0] + sq[:, 1]) + sq[:, 2])
    n = torch.ceil(length / _f32(precision)).clamp(min=1).long()
    src = torch.repeat_interleave(torch.arange(n.shape[0], device="cuda"), n)
    first = n.cumsum(0) - n
    k = (torch.arange(src.shape[0], device="cuda") - first[src]).double()
    last = k == (n[src] - 1)
    d = (seg / (length + _f32(1e-10))[:, None]).double()
    out = tracks[src].double()
    for a, name in enumerate("xyz"):
        st = s[src, a].double() + k * precision * d[src, a]
        en = torch.where(last, e[src, a].double(), s[src, a].double() + (k + 1) * precision * d[src, a])
        out[:, c[name + "_start"]], out[:, c[name + "_end"]], out[:, c[name]] = st, en, 0.5 * (st + en)
    dE, l64 = tracks[src, c["dE"]].double(), length[src].double()
    out[:, c["dE"]] = torch.where(last, dE * (1 - precision * k / (l64 + 1e-10)), dE * precision / (l64 + 1e-10))
    out[:, c["dx"]] = torch.where(last, l64 - precision * k, precision)
    return out

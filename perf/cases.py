"""The work a user of this package has it do, as cases that can be timed.

Five kinds of call, each through the package's public entry points:

* ``photons``: propagate_photons on a setup -- the package's main call.  From
  the README example (one module, one wavelength, 1e5 photons) over the
  400-module detector at 1e7 and 1e8 photons to events of many emitters;
  water and deep ice, point, cascade and track emitters;
* ``tables``: surrogate.generate_tables -- expected hits and arrival-time
  histograms of many source-module pairs in one launch;
* ``detect``: detection.make_hits_device -- photon hits on the device to PMT
  hits, for every module model;
* ``train`` / ``gradient``: surrogate.train and MLP.loss_grad on training
  tables in device memory;
* ``infer``: MLP.infer -- expected counts and arrival-time PDFs of many pairs.

A case is a dict of plain values; listed() gives fixed ones, draw() others of
the same ranges.
"""
import math
import os

import numpy as np
import torch

import __graft_entry__ as entry

pp = entry.load()

N_FEATURES, N_KNOTS = 8, 600
PMT_AREA = 16 * math.pi * 0.0762 ** 2
MODULE_RADIUS = 0.2159
FLOPS_PER_STEP = 82        # FP32 operations of a photon step with one candidate sphere
MAX_TRAIN_BATCH = 8192


def listed():
    photons = dict(kind="photons", strings=20, per_string=20, medium="water", spectrum="cherenkov",
                   emitter="point", sources=1, steps=15)
    net = dict(hidden=256, layers=4, bins=64)
    return [
        # the README example: the smallest call, launch and host latency
        dict(photons, name="readme_1e5", photons=100_000, strings=1, per_string=1,
             spectrum="mono"),
        # one event in the 400-module detector: a flasher or a cascade vertex
        dict(photons, name="detector_1e7", photons=10_000_000),
        # the same at the size of one bright event: the benchmark's workload
        dict(photons, name="detector_1e8", photons=100_000_000),
        # an event of 256 emitters, half points and half cascades, uneven counts
        dict(photons, name="events_256", photons=40_000_000, emitter="mixed", sources=256),
        # a muon track through the detector in deep ice, an odd photon count
        dict(photons, name="ice_track", photons=3_000_001, medium="ice", emitter="track"),
        # a batch of surrogate training tables: 500 pairs, 1e5 photons each
        dict(kind="tables", name="tables_500", pairs=500, photons=100_000, steps=15),
        # hits of a long simulation onto 400 POMs, records streaming from HBM
        dict(kind="detect", name="detect_pom_5e7", module="pom", records=50_000_000),
        # the hits of one event on all module kinds, an odd count
        dict(kind="detect", name="detect_mixed_1e5", module="mixed", records=100_003),
        # a stretch of surrogate training at the standard batch, then a checkpoint
        dict(net, kind="train", name="train_8192", rows=65_536, batch=8192, steps=32),
        # loss and gradient of one ragged batch, for a caller's own optimiser
        dict(net, kind="gradient", name="gradient_1000", batch=1000),
        # serving: a million pairs with their time PDFs
        dict(net, kind="infer", name="infer_1e6", pairs=1_000_000, pdf=True),
        # serving: one event's modules, counts only
        dict(net, kind="infer", name="infer_997", pairs=997, pdf=False),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["photons"] * 4 + ["tables", "detect", "detect", "train", "gradient",
                                         "infer", "infer"])
    net = dict(hidden=rng.choice([128, 256, 256]), layers=rng.choice([3, 4, 4, 5]),
               bins=rng.choice([32, 64, 64]))
    if kind == "photons":
        return dict(kind=kind, photons=_log_int(rng, 1e4, 3e7), strings=rng.randint(1, 20),
                    per_string=rng.randint(1, 20), medium=rng.choice(["water", "water", "ice"]),
                    spectrum=rng.choice(["cherenkov", "cherenkov", "mono"]),
                    emitter=rng.choice(["point", "cascade", "track", "mixed"]),
                    sources=_log_int(rng, 1, 256), steps=rng.randint(10, 20))
    if kind == "tables":
        return dict(kind=kind, pairs=_log_int(rng, 10, 1000), photons=_log_int(rng, 1e4, 1e5),
                    steps=15)
    if kind == "detect":
        return dict(kind=kind, module=rng.choice(["pom", "pom", "dom", "multipmt", "mixed"]),
                    records=_log_int(rng, 1e3, 3e7))
    if kind == "train":
        return dict(net, kind=kind, rows=_log_int(rng, 1e4, 1e5),
                    batch=_log_int(rng, 500, MAX_TRAIN_BATCH), steps=rng.randint(8, 32))
    if kind == "gradient":
        return dict(net, kind=kind, batch=_log_int(rng, 1, MAX_TRAIN_BATCH))
    return dict(net, kind="infer", pairs=_log_int(rng, 1, 8e5), pdf=rng.random() < 0.7)


# ---- photons -----------------------------------------------------------------

_COLUMNS = dict(position="f4", direction="f4", initial_direction="f4", wavelength="f4",
                time="f8", dist_travelled="f4", module_id="i4", n_steps="i4", base_weight="f8",
                abs_weight="f8", total_weight="f8", photon_index="i8", source_index="i4")

_MEDIA = {}


def _medium(name):
    """A medium and its Frank-Tamm spectrum, made once by a user's program."""
    if name not in _MEDIA:
        m = pp.CascadiaMediumProperties(0.95, 0.2, 1.0, 1.0) if name == "water" else \
            pp.make_homogenous_clearice_properties()
        _MEDIA[name] = m, pp.make_cherenkov_spectrum((300.0, 800.0), m)
    return _MEDIA[name]


def _unit(rng, n):
    v = rng.normal(size=(n, 3))
    return v / np.linalg.norm(v, axis=1, keepdims=True)


def _detector(case):
    """Vertical strings at fixed places in a 500 m square, modules every 25 m; a
    single module stands 10 m above the origin, as in the README."""
    if case["strings"] * case["per_string"] == 1:
        return [pp.HomogeneousDetector(pp.Spherical([0.0, 0.0, 10.0], 0.3), PMT_AREA, 1)]
    xy = np.random.default_rng(1234).uniform(-250.0, 250.0, size=(case["strings"], 2))
    n = case["per_string"]
    z = 25.0 * (np.arange(n) - 0.5 * n)
    return [pp.HomogeneousDetector(pp.Spherical([float(x), float(y), float(z[k])], MODULE_RADIUS),
                                   PMT_AREA, s * n + k + 1)
            for s, (x, y) in enumerate(xy) for k in range(n)]


def _emitters(case, rng):
    n, total = case["sources"], case["photons"]
    if case["strings"] * case["per_string"] == 1:
        half = [2.0, 2.0, 2.0]
    else:
        half = [200.0, 200.0, 200.0] if n == 1 else [500.0, 500.0, 500.0]
    pos = rng.uniform(-1.0, 1.0, size=(n, 3)) * half
    dirs = _unit(rng, n)
    share = np.exp(rng.uniform(math.log(1e4), math.log(1e7), size=n))
    counts = np.maximum(1, np.floor(share / share.sum() * total)).astype(np.int64)
    counts[0] += max(0, total - int(counts.sum()))
    cascade = pp.LongitudinalParameterisation(2.0, 0.63, 0.36)
    out = []
    for i in range(n):
        p, d, c = [float(v) for v in pos[i]], [float(v) for v in dirs[i]], int(counts[i])
        e = case["emitter"]
        if e == "mixed":
            e = "point" if i % 2 == 0 else "cascade"
        if e == "point":
            out.append(pp.PointlikeIsotropicEmitter(p, 0.0, c))
        elif e == "cascade":
            out.append(pp.ExtendedCherenkovEmitter(p, d, 0.0, c, cascade))
        else:
            start = [p[a] - 150.0 * d[a] for a in range(3)]
            out.append(pp.CherenkovTrackEmitter(start, d, 0.0, 300.0, c))
    return out


def _prepare_photons(case, seed):
    rng = np.random.default_rng([seed, 1])
    medium, cherenkov = _medium(case["medium"])
    spectrum = cherenkov if case["spectrum"] == "cherenkov" else \
        pp.make_monochromatic_spectrum(450.0)
    setup = pp.PhotonPropSetup(_emitters(case, rng), _detector(case), medium, spectrum,
                               int(rng.integers(1, 1 << 30)))
    # the program's own hit columns, reused event after event
    rows = 2000 + case["photons"] // 200
    columns = {k: np.zeros((rows, 3) if k.endswith(("position", "direction")) else rows, dt)
               for k, dt in _COLUMNS.items()}
    return dict(setup=setup, buffers=pp.make_hit_buffers(), steps=case["steps"], columns=columns,
                filled=0)


def _run_photons(s):
    table = pp.propagate_photons(s["setup"], s["buffers"], s["steps"])
    # in photon order: the table lists the hits in the order they were found
    order = np.argsort(table["source_index"].astype(np.int64) << 40 | table["photon_index"])
    n = len(order)
    for k, column in s["columns"].items():
        column[:n] = table[k][order]
        column[n:s["filled"]] = 0
    s["filled"] = n
    return dict(s["columns"], hits=n, simulated=table.n_ph_sim)


# ---- tables --------------------------------------------------------------------

def _prepare_tables(case, seed):
    medium, spectrum = _medium("water")
    return dict(pairs=pp.surrogate.sample_pairs(case["pairs"], seed=seed), ctx=pp.Context(0),
                photons=case["photons"], steps=case["steps"], seed=seed % 100_003, medium=medium,
                spectrum=spectrum)


def _run_tables(s):
    return pp.surrogate.generate_tables(s["pairs"], s["photons"], seed=s["seed"], ctx=s["ctx"],
                                        medium=s["medium"], spectrum=s["spectrum"],
                                        n_steps=s["steps"], device_out=True)


# ---- detection ------------------------------------------------------------------

def _modules(kind):
    xy = np.random.default_rng(1234).uniform(-250.0, 250.0, size=(20, 2))
    acceptance = pp.dom.load_dom_acceptance()
    qe = pp.InterpQuantumEff(*pp.generic_multipmt.load_multipmt_qe())
    layout = pp.make_generic_multipmt_positions()
    out = []
    for i in range(400):
        p = [float(xy[i // 20, 0]), float(xy[i // 20, 1]), -250.0 + 25.0 * (i % 20)]
        k = ("pom", "dom", "multipmt", "homogeneous")[i % 4] if kind == "mixed" else kind
        if k == "pom":
            out.append(pp.POM.at(p, i + 1))
        elif k == "dom":
            out.append(pp.DOM(pp.Spherical(p, pp.dom.DOM_RADIUS), i + 1, acceptance=acceptance))
        elif k == "multipmt":
            out.append(pp.SphericalMultiPMTTarget(pp.Spherical(p, MODULE_RADIUS),
                                                  (0.0762 / 2) ** 2 * math.pi, layout, qe, i + 1))
        else:
            out.append(pp.HomogeneousDetector(pp.Spherical(p, MODULE_RADIUS), PMT_AREA, i + 1))
    return out


def _records(case, seed, targets):
    """Hit records as the propagation leaves them on the device: positions on the
    modules' surfaces, photons flying inwards, wavelengths of density
    1 / lambda^2 on 300-800 nm.  80 bytes each, as 20 words."""
    n = case["records"]
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    centre = torch.tensor(np.array([t.shape.position for t in targets], np.float32), device="cuda")
    radius = torch.tensor(np.array([t.shape.radius for t in targets], np.float32), device="cuda")
    rec = torch.zeros((n, 20), dtype=torch.float32, device="cuda")
    mi = torch.randint(0, len(targets), (n,), device="cuda", generator=g)
    v = torch.randn((n, 3), device="cuda", generator=g)
    v /= v.norm(dim=1, keepdim=True)
    rec[:, 0:3] = centre[mi] + radius[mi, None] * v
    d = torch.randn((n, 3), device="cuda", generator=g)
    d /= d.norm(dim=1, keepdim=True)
    rec[:, 4:7] = torch.where((d * v).sum(1, keepdim=True) > 0, -d, d)
    u = torch.rand(n, device="cuda", generator=g)
    rec[:, 3] = 1.0 / (1.0 / 300.0 - u * (1.0 / 300.0 - 1.0 / 800.0))
    rec[:, 7] = (mi + 1).to(torch.int32).view(torch.float32)
    return rec


def _prepare_detect(case, seed):
    targets = _modules(case["module"])
    rec = _records(case, seed, targets)
    n = case["records"]
    return dict(targets=targets, rec=rec, seed=seed,
                ids=torch.empty(n, dtype=torch.int32, device="cuda"),
                qe=torch.empty(n, dtype=torch.float32, device="cuda"))


def _run_detect(s):
    pp.detection.make_hits_device(s["rec"].data_ptr(), s["rec"].shape[0], s["targets"], s["seed"],
                                  s["ids"].data_ptr(), s["qe"].data_ptr())
    return s["ids"], s["qe"]


def _exact_detect(case, seed):
    """The QE weights: the tables' linear interpolation in 64 bits; the PMT
    numbers are whole."""
    data = os.path.join(entry.PKG_DIR, "data")
    pom = np.loadtxt(os.path.join(data, "pom_rel_qe.csv"), delimiter=",", skiprows=1)
    mpmt = np.loadtxt(os.path.join(data, "multipmt_qe.csv"), delimiter=",", skiprows=1)
    rec = _records(case, seed, _modules(case["module"]))
    wl = rec[:, 3].cpu().numpy().astype(np.float64)
    which = (rec[:, 7].view(torch.int32) - 1).cpu().numpy() % 4
    if case["module"] != "mixed":
        which[:] = ("pom", "dom", "multipmt").index(case["module"])
    qe = np.ones(len(wl))
    for k, t in ((0, pom), (2, mpmt)):
        rows = which == k
        qe[rows] = np.interp(wl[rows], t[:, 0], t[:, 1], left=0.0, right=0.0)
    return None, qe


# ---- the surrogate network ----------------------------------------------------------

def _up(n, k):
    return (n + k - 1) // k * k


def _layers(case):
    """(rows, cols, real rows, real cols) of the weight matrices, padded as the
    packed parameter vector holds them."""
    h, out = case["hidden"], case["bins"] + 1
    shapes = [(h, _up(N_FEATURES, 16), h, N_FEATURES)]
    shapes += [(h, h, h, h)] * (case["layers"] - 1)
    return shapes + [(_up(out, 16), h, out, h)]


def _weights(case, seed):
    """The packed parameter vector: per layer W (row-major) then b, each padded
    to a multiple of 8 values; He-uniform weights, a smaller head."""
    rng = np.random.default_rng([seed, 2])
    flat, shapes = [], _layers(case)
    for l, (r, c, rr, cc) in enumerate(shapes):
        a = math.sqrt(6.0 / cc) * (0.3 if l == len(shapes) - 1 else 1.0)
        w = np.zeros((r, c), np.float32)
        w[:rr, :cc] = rng.uniform(-a, a, size=(rr, cc))
        b = np.zeros(_up(r, 8), np.float32)
        b[:rr] = rng.uniform(-0.1, 0.1, size=rr)
        flat += [w.ravel(), b]
    return np.concatenate(flat)


def _split(case, flat):
    out, at = [], 0
    for r, c, _, _ in _layers(case):
        w = flat[at:at + r * c].reshape(r, c)
        at += _up(r * c, 8)
        out.append((w, flat[at:at + r]))
        at += _up(r, 8)
    return out


def _net(case, seed, max_batch):
    net = pp.surrogate.MLP(n_in=N_FEATURES, hidden=case["hidden"], n_layers=case["layers"],
                           n_bins=case["bins"], max_batch=max_batch)
    net.set_params(_weights(case, seed))
    return net


def _features(n, seed):
    pairs = pp.surrogate.sample_pairs(n, seed=seed)
    return pairs, torch.tensor(pp.surrogate.pair_features(pairs), device="cuda")


def _training_tables(n, bins, seed):
    """Features, expected hits and time histograms with the shape of the MC's
    tables: counts falling as exp(-d / 25 m) / d^2, arrival times spreading
    with distance."""
    pairs, x = _features(n, seed)
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    d = torch.tensor(pairs.distance.astype(np.float32), device="cuda")
    mean = 1e5 * MODULE_RADIUS ** 2 / (4.0 * d * d) * torch.exp(-d / 25.0)
    counts = torch.poisson(mean, generator=g)
    bin_no = torch.arange(bins, device="cuda", dtype=torch.float32)
    peak = (0.15 + 0.5 * torch.log10(d / 5.0) / 1.8)[:, None] * bins
    shape = torch.exp(-0.5 * ((bin_no - peak) / (0.1 * bins)) ** 2)
    hist = torch.poisson(counts[:, None] * shape / shape.sum(1, keepdim=True), generator=g)
    return x, counts, hist


def _prepare_train(case, seed):
    x, c, h = _training_tables(case["rows"], case["bins"], seed)
    return dict(net=_net(case, seed, MAX_TRAIN_BATCH), x=x, counts=c, hists=h,
                steps=case["steps"], batch=case["batch"], seed=seed)


def _run_train(s):
    pp.surrogate.train(s["net"], s["x"], s["counts"], s["hists"], s["steps"], s["batch"], lr=1e-4,
                       seed=s["seed"])
    return s["net"].params()


def _prepare_gradient(case, seed):
    x, c, h = _training_tables(case["batch"], case["bins"], seed)
    return dict(net=_net(case, seed, MAX_TRAIN_BATCH), x=x, counts=c, hists=h)


def _run_gradient(s):
    return s["net"].loss_grad(s["x"].data_ptr(), s["counts"].data_ptr(), s["hists"].data_ptr(),
                              s["x"].shape[0])


def _head(case, flat, x):
    """The network's head outputs for FP64 tensors."""
    y = torch.zeros((x.shape[0], _up(N_FEATURES, 16)), dtype=torch.float64, device=x.device)
    y[:, :N_FEATURES] = x
    layers = _split(case, flat)
    for w, b in layers[:-1]:
        y = torch.nn.functional.silu(y @ w.T + b)
    w, b = layers[-1]
    return y @ w.T + b


def _exact_gradient(case, seed):
    x, c, h = (t.double() for t in _training_tables(case["batch"], case["bins"], seed))
    flat = torch.tensor(_weights(case, seed), dtype=torch.float64, device="cuda",
                        requires_grad=True)
    o = _head(case, flat, x)
    log_p = torch.log_softmax(o[:, 1:case["bins"] + 1], dim=1)
    loss = (torch.exp(o[:, 0]) - c * o[:, 0] - (h * log_p).sum(1)).mean()
    loss.backward()
    return float(loss.detach()), flat.grad


def _prepare_infer(case, seed):
    n = case["pairs"]
    return dict(net=_net(case, seed, 128), x=_features(n, seed)[1],
                counts=torch.empty(n, dtype=torch.float32, device="cuda"),
                pdf=torch.empty((n, case["bins"]), dtype=torch.float32, device="cuda")
                if case["pdf"] else None)


def _run_infer(s):
    s["net"].infer(s["x"].data_ptr(), s["x"].shape[0], s["counts"].data_ptr(),
                   s["pdf"].data_ptr() if s["pdf"] is not None else 0)
    return s["counts"], s["pdf"]


def _exact_infer(case, seed):
    x = _features(case["pairs"], seed)[1].double()
    flat = torch.tensor(_weights(case, seed), dtype=torch.float64, device="cuda")
    counts, pdf = [], []
    for part in x.split(1 << 17):
        o = _head(case, flat, part)
        counts.append(torch.exp(o[:, 0]))
        if case["pdf"]:
            pdf.append(torch.softmax(o[:, 1:case["bins"] + 1], dim=1))
    return torch.cat(counts), torch.cat(pdf) if case["pdf"] else None


# ---- the interface ------------------------------------------------------------------

_PREPARE = dict(photons=_prepare_photons, tables=_prepare_tables, detect=_prepare_detect,
                train=_prepare_train, gradient=_prepare_gradient, infer=_prepare_infer)
_RUN = dict(photons=_run_photons, tables=_run_tables, detect=_run_detect, train=_run_train,
            gradient=_run_gradient, infer=_run_infer)


def prepare(case, seed):
    return dict(_PREPARE[case["kind"]](case, seed), kind=case["kind"])


def run(state):
    return _RUN[state["kind"]](state)


def exact(case, seed):
    """None for the Monte Carlo (its trajectories are chaotic: 64 bits give other
    photons) and for a stretch of training (Adam's first steps are signs)."""
    if case["kind"] == "detect":
        return _exact_detect(case, seed)
    if case["kind"] == "gradient":
        return _exact_gradient(case, seed)
    if case["kind"] == "infer":
        return _exact_infer(case, seed)
    return None


def work(case):
    kind = case["kind"]
    if kind == "photons":
        n = case["photons"]
        modules = case["strings"] * case["per_string"]
        return {"bytes": 96 * case["sources"] + 16 * modules + 80 * 1e-4 * n,
                "flops": FLOPS_PER_STEP * n * case["steps"]}
    if kind == "tables":
        n = case["pairs"]
        return {"bytes": (96 + 4 + 4 * 65) * n,
                "flops": FLOPS_PER_STEP * n * case["photons"] * case["steps"]}
    if kind == "detect":
        n = case["records"]
        return {"bytes": (32 + 4 + 4) * n, "flops": 16 * 20 * n}
    weights = sum(r * c for r, c, _, _ in _layers(case))
    params = len(_weights(case, 0))
    row = 4 * (N_FEATURES + 1 + case["bins"])
    if kind == "train":
        b = case["batch"] * case["steps"]
        return {"bytes": row * b + 2 * 12 * params, "flops": 6 * weights * b}
    if kind == "gradient":
        b = case["batch"]
        return {"bytes": row * b + 8 * params, "flops": 6 * weights * b}
    n = case["pairs"]
    return {"bytes": (4 * (N_FEATURES + 1) + (4 * case["bins"] if case["pdf"] else 0)) * n
            + 4 * params, "flops": 2 * weights * n}

"""Timed workloads of the sampler, through its public Python entry points.

A case is a dict of plain values; `prepare` makes what a program holds before
the call (a page-locked freeze-out surface, a handle, a page-locked buffer for
the hadrons), and `run` is one pass: hand over the surface, sample, read the
hadron lists back.  The surfaces are the synthetic ones of
iss_gb300.surfaces.  Every draw of the sampler is keyed by the seed, so a pass
gives the same hadrons whenever it is repeated.
"""
import math
import os
import tempfile

import numpy as np
import torch

from iss_gb300 import HADRON_DTYPE, iSS, native
from iss_gb300 import surfaces as S

# hadrons per event: of the boost-invariant surface as a whole, and per cell of
# the two 3+1D surfaces
IDEAL_PER_EVENT = 9400.0
PER_CELL = {"viscous": 0.222, "finite_density": 0.218}
# final hadrons per sampled one when the resonances decay
DECAY_GROWTH = 1.7
# weights of the proposal network that are not padding, and of its layers
NET_IN, NET_HIDDEN, NET_OUT, NET_LAYERS = 18, 128, 48, 5


# ---------------------------------------------------------------------------
# the cases

def listed():
    return [
        # one sample of one boost-invariant event: the smallest call, all latency
        dict(name="ideal_1_event", kind="sample", surface="ideal", dx=0.5, events=1),
        # the same surface oversampled, every pass a replay of the captured graph
        dict(name="ideal_100_events_graph", kind="sample", surface="ideal", dx=0.5, events=100, graph=True),
        # one sample of a 3+1D event, as an event-by-event hydro chain draws it
        dict(name="viscous_200k_1_event", kind="sample", surface="viscous", cells=200_000, events=1,
             bulk_kind=11),
        # the benchmark's surface oversampled, all hadrons to the host
        dict(name="viscous_200k_300_events", kind="sample", surface="viscous", cells=200_000, events=300,
             bulk_kind=11),
        # final-state hadrons: the resonances decay before the lists are read
        dict(name="viscous_decays", kind="sample", surface="viscous", cells=100_000, events=100,
             bulk_kind=11, decays=True),
        # finite baryon density: chemical potentials, baryon diffusion, SMASH species
        dict(name="finite_density", kind="sample", surface="finite_density", cells=100_000, events=40,
             bulk_kind=11),
        # charge conserved pair by pair, RTA bulk correction, ragged sizes
        dict(name="viscous_charge_pairs", kind="sample", surface="viscous", cells=37_211, events=37,
             bulk_kind=1, lcc=True),
        # the lab-frame sampler (MC_sampling = 2) with the parameter file's defaults
        dict(name="lab_frame", kind="sample", surface="viscous", cells=50_000, events=40, bulk_kind=1,
             mc_sampling=2),
        # a set of events of unequal sizes sampled by one call
        dict(name="batch_16", kind="batch", surfaces=16, cells_low=5_000, cells_high=40_000,
             events_low=10, events_high=100),
        # momenta proposed by the network, exact rejection
        dict(name="learned_sampler", kind="learned", cells=50_000, events=200),
        # the network by itself: outputs, loss and weight gradient of one batch
        dict(name="network_gradient", kind="network", rows=50_001),
        # the OSCAR text file an afterburner reads
        dict(name="oscar_file", kind="oscar", cells=50_000, events=20),
    ]


def _log_int(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(["ideal", "ideal", "viscous", "viscous", "viscous", "decays", "finite_density", "pairs",
                       "lab_frame", "batch", "learned", "network", "oscar"])
    if kind == "ideal":
        return dict(kind="sample", surface="ideal", dx=round(rng.uniform(0.25, 1.0), 3),
                    events=_log_int(rng, 1, 300), graph=rng.random() < 0.5)
    if kind in ("viscous", "decays", "pairs"):
        cells = _log_int(rng, 500, 200_000)
        events = _log_int(rng, 1, min(1000, 5e7 / cells))
        case = dict(kind="sample", surface="viscous", cells=cells, events=events,
                    bulk_kind=rng.choice([0, 1, 11, 21]))
        if case["bulk_kind"] == 21:   # the NEoS-BQS coefficients
            case["afterburner"] = 2
        if kind == "decays":
            case.update(bulk_kind=rng.choice([0, 1, 11]), decays=True, events=max(1, events // 2))
            case.pop("afterburner", None)
        if kind == "pairs":
            case.update(lcc=True, events=max(1, events // 2))
        return case
    if kind == "finite_density":
        cells = _log_int(rng, 2_000, 110_000)
        return dict(kind="sample", surface="finite_density", cells=cells, bulk_kind=11,
                    events=_log_int(rng, 1, min(400, 4e6 / cells)))
    if kind == "lab_frame":
        cells = _log_int(rng, 2_000, 50_000)
        return dict(kind="sample", surface="viscous", cells=cells, bulk_kind=1, mc_sampling=2,
                    events=_log_int(rng, 1, min(100, 2e6 / cells)))
    if kind == "batch":
        return dict(kind="batch", surfaces=rng.randint(2, 24), cells_low=rng.randint(500, 5_000),
                    cells_high=rng.randint(6_000, 40_000), events_low=rng.randint(1, 10),
                    events_high=rng.randint(11, 100))
    if kind == "learned":
        cells = _log_int(rng, 3_000, 50_000)
        return dict(kind="learned", cells=cells, events=_log_int(rng, 50, min(1000, 1e7 / cells)))
    if kind == "network":
        return dict(kind="network", rows=_log_int(rng, 500, 100_000))
    cells = _log_int(rng, 1_000, 50_000)
    return dict(kind="oscar", cells=cells, events=_log_int(rng, 1, min(100, 1e6 / cells)))


# ---------------------------------------------------------------------------
# inputs

_pool = []


def _finite_density(cells, seed):
    """Cells of a finite-density surface, drawn from 120,000 of them (the
    equation of state behind a surface takes seconds to tabulate)."""
    if not _pool:
        _pool.append(S.finite_density_3d(120_000, seed=3).fo_surf())
    rows = np.random.default_rng(seed).permutation(len(_pool[0]))[:cells]
    return _pool[0][rows]


def _surface(case, seed):
    if case["surface"] == "ideal":
        rng = np.random.default_rng(seed)
        return S.ideal_boost_invariant(T=rng.uniform(0.147, 0.153), tau=rng.uniform(9.0, 11.0), dx=case["dx"],
                                       umax=rng.uniform(0.5, 0.7)).fo_surf()
    if case["surface"] == "finite_density":
        return _finite_density(case["cells"], seed)
    return S.viscous_3d(case["cells"], seed=seed).fo_surf()


def _pinned(a):
    return torch.from_numpy(np.ascontiguousarray(a)).pin_memory().numpy()


def _hadron_buffer(n):
    return torch.zeros(int(n) * HADRON_DTYPE.itemsize, dtype=torch.uint8, pin_memory=True).numpy().view(HADRON_DTYPE)


def _parameters(case):
    p = dict(S.DEFAULT_PARAMETERS, hydro_mode=2, afterburner_type=0, quantum_statistics=1,
             dN_dy_sampling_model=30, number_of_repeated_sampling=case.get("events", 0))
    if case.get("surface") == "ideal":
        p.update(hydro_mode=1, include_deltaf_shear=0, include_deltaf_bulk=0)
    else:
        kind = case.get("bulk_kind", 11)
        p.update(include_deltaf_shear=1, include_deltaf_bulk=int(kind != 0), turn_on_bulk=int(kind != 0),
                 bulk_deltaf_kind=kind if kind else 11, afterburner_type=case.get("afterburner", 0))
    if case.get("surface") == "finite_density":
        p.update(afterburner_type=2, turn_on_rhob=1, turn_on_diff=1, include_deltaf_diffusion=1)
    if case.get("decays"):
        p["perform_decays"] = 1
    if case.get("lcc"):
        p["local_charge_conservation"] = 1
    if case.get("graph"):
        p["gpu_graph"] = 1
    if case.get("mc_sampling") == 2:
        p.update(MC_sampling=2, restrict_deltaf=1, deltaf_max_ratio=1.0, sample_pT_up_to=-1,
                 sample_y_minus_eta_s_range=3)
    return p


def _batch_sizes(case):
    """Cells and events of each surface of a batch: a property of the case, so
    that every seed has the same amount of work."""
    rng = np.random.default_rng(case["surfaces"] * 1_000_003 + case["cells_low"])
    low, high = case["cells_low"], case["cells_high"]
    cells = np.exp(rng.uniform(np.log(low), np.log(high), case["surfaces"])).astype(np.int64)
    events = np.exp(rng.uniform(np.log(case["events_low"]), np.log(case["events_high"]),
                                case["surfaces"])).astype(np.int32)
    return cells, events


def _hadrons(case):
    """Hadrons of a pass, about."""
    if case["kind"] == "batch":
        cells, events = _batch_sizes(case)
        return float((cells * events).sum()) * PER_CELL["viscous"]
    if case.get("surface") == "ideal":
        n = IDEAL_PER_EVENT * case["events"]
    else:
        n = PER_CELL[case.get("surface", "viscous")] * case["cells"] * case["events"]
    return n * (DECAY_GROWTH if case.get("decays") else 1.0)


def _room(case):
    """Hadrons that a pass has room for."""
    return int(1.6 * _hadrons(case)) + 20_000


def _network_inputs(case, seed):
    """Feature rows and (K, n) targets with the ranges they have on the viscous
    surface: temperature and chemical potential, shear, bulk, diffusion, the
    surface element, mass over temperature and statistics."""
    rng = np.random.default_rng(seed)
    n = case["rows"]
    f = np.zeros((n, NET_IN), dtype=np.float32)
    f[:, 0] = rng.uniform(-0.25, 0.25, n)
    f[:, 1] = rng.uniform(-0.5, 0.5, n)
    f[:, 2:7] = rng.normal(0.0, 0.7, (n, 5))
    f[:, 7] = rng.uniform(-2.0, 0.0, n)
    ds = np.concatenate([np.ones((n, 1)), rng.normal(0.0, 0.4, (n, 3))], axis=1)
    f[:, 12:16] = ds / (np.abs(ds[:, :1]) + np.linalg.norm(ds[:, 1:], axis=1, keepdims=True))
    f[:, 16] = rng.choice([0.093, 0.33, 0.52, 0.63, 0.74, 0.83], n)
    f[:, 17] = np.where(f[:, 16] > 0.6, 1.0, -1.0)
    t = np.zeros((n, 4), dtype=np.float32)
    t[:, 0] = rng.gamma(2.5, 1.0, n) + 1e-3
    v = rng.normal(size=(n, 3))
    t[:, 1:] = v / np.linalg.norm(v, axis=1, keepdims=True)
    return f, t


def _weights(seed):
    """A network as it starts its training: He-uniform layers, a small last
    layer, output biases that spread the mixture over K = 0.25 .. 6.7."""
    rng = np.random.default_rng(seed + 1)
    flat = []
    for i in range(NET_LAYERS):
        n_in = 32 if i == 0 else NET_HIDDEN
        n_out = 64 if i == NET_LAYERS - 1 else NET_HIDDEN
        fan = NET_IN if i == 0 else NET_HIDDEN
        last = i == NET_LAYERS - 1
        w = rng.uniform(-1.0, 1.0, (n_out, n_in)) * (0.1 * math.sqrt(3.0 / fan) if last else math.sqrt(6.0 / fan))
        b = np.zeros(n_out)
        if i == 0:
            w[:, NET_IN:] = 0.0
        if last:
            w[NET_OUT:] = 0.0
            b[8:16] = np.log(0.25 * 1.6 ** np.arange(8))
            b[16:24] = math.log(0.5)
            b[24:48] = rng.uniform(-0.1, 0.1, 24)
        flat += [w.ravel(), b]
    return np.concatenate(flat).astype(np.float32)


def prepare(case, seed):
    kind = case["kind"]
    s = iSS(".", inputfile="")
    state = {"case": case, "sampler": s}
    if kind == "network":
        state["features"], state["targets"] = _network_inputs(case, seed)
        s.learned_set_weights(_weights(seed))
        return state
    s.set_params(**_parameters(case))
    s.set_random_seed(seed)
    if kind == "batch":
        cells, events = _batch_sizes(case)
        state["cell_offsets"] = np.concatenate([[0], np.cumsum(cells)]).astype(np.int64)
        state["events"] = events
        state["surface"] = _pinned(np.concatenate([S.viscous_3d(int(c), seed=seed + 7919 * i).fo_surf()
                                                   for i, c in enumerate(cells)]))
    else:
        state["surface"] = _pinned(_surface(dict({"surface": "viscous"}, **case), seed))
    if kind == "learned":
        s.set_params(gpu_sampler=1, gpu_learned_alpha=0.8, gpu_learned_exact=1)
        s.learned_set_weights(_weights(seed))
    if kind == "oscar":
        # a RAM disk where there is one: the file system's own speed is not the sampler's
        where = "/dev/shm" if os.path.isdir("/dev/shm") and os.access("/dev/shm", os.W_OK) else None
        state["folder"] = tempfile.TemporaryDirectory(dir=where)
        state["file"] = os.path.join(state["folder"].name, "OSCAR.DAT")
        state["file_bytes"] = 300 * _room(case)
    else:
        state["out"] = _hadron_buffer(_room(case))
    return state


# ---------------------------------------------------------------------------
# one pass

def _lists(state, offsets):
    """The hadron lists as plain arrays, without a copy: the program's whole
    buffer (zero behind the last hadron) and where each event starts in it."""
    out = state["out"]
    return {"pid": out["pid"], "values": out.view(np.float32).reshape(-1, 10)[:, 1:], "offsets": offsets}


def run(state):
    case, s = state["case"], state["sampler"]
    kind = case["kind"]
    if kind == "network":
        out = s.learned_forward(state["features"])
        loss, grad = s.learned_loss_grad(state["features"], state["targets"])
        return {"out": out, "loss": np.float32(loss), "grad": grad}
    if kind == "batch":
        s.set_surface_batch_flat(state["surface"], state["cell_offsets"], state["events"])
    else:
        s.set_surface(state["surface"])
    if kind == "oscar":
        s.generate_samples()
        s.write_output(native.OUTPUT_OSCAR, state["file"])
        # a mapping of one length for every seed: zeros behind the text
        os.truncate(state["file"], state["file_bytes"])
        return {"file": np.memmap(state["file"], dtype=np.uint8, mode="r")}
    if case.get("graph"):
        s.generate_samples()
        return _lists(state, s.all_hadrons(state["out"])[1])
    return _lists(state, s.generate_into(state["out"])[1])


# ---------------------------------------------------------------------------
# what a pass cannot do without

def work(case):
    if case["kind"] == "network":
        weights = NET_IN * NET_HIDDEN + 3 * NET_HIDDEN * NET_HIDDEN + NET_HIDDEN * NET_OUT
        # forward twice, and two products of the same size per weight backward
        return {"bytes": case["rows"] * 4.0 * (2 * NET_IN + 64 + 4) + 4.0 * 2 * 62_016,
                "flops": 2.0 * 4 * weights * case["rows"]}
    hadrons = _hadrons(case)
    if case["kind"] == "batch":
        cells, events = (float(v.sum()) for v in _batch_sizes(case))
    else:
        cells = math.pi * (10.0 / case["dx"]) ** 2 if case.get("surface") == "ideal" else case["cells"]
        events = case["events"]
    per_hadron = 257 if case["kind"] == "oscar" else 40
    # a yield of every species in every cell (a few terms of a series each), and
    # a proposal, its weight and a boost for every hadron
    tries = 1900.0 if case.get("mc_sampling") == 2 else 2.0
    return {"bytes": 136.0 * cells + per_hadron * hadrons + 8.0 * events,
            "flops": cells * 319.0 * 20.0 + hadrons * (100.0 + 100.0 * tries)}


# ---------------------------------------------------------------------------
# the network in 64 bits (sampled hadrons have no such value)

def exact(case, seed):
    if case["kind"] != "network":
        return None
    features, targets = _network_inputs(case, seed)
    flat = torch.from_numpy(_weights(seed)).double().cuda().requires_grad_(True)
    n_in = [32] + [NET_HIDDEN] * (NET_LAYERS - 1)
    n_out = [NET_HIDDEN] * (NET_LAYERS - 1) + [64]
    h = torch.zeros(len(features), 32, dtype=torch.float64, device="cuda")
    h[:, :NET_IN] = torch.from_numpy(features).double()
    at = 0
    for i, (a, b) in enumerate(zip(n_in, n_out)):
        w = flat[at:at + a * b].reshape(b, a)
        bias = flat[at + a * b:at + a * b + b]
        at += a * b + b
        h = h @ w.T + bias
        if i < NET_LAYERS - 1:
            h = torch.relu(h)
    t = torch.from_numpy(targets).double().cuda()
    logits, mu, ls, v = h[:, :8], h[:, 8:16], h[:, 16:24].clamp(-4.0, 1.5), h[:, 24:48].reshape(-1, 8, 3)
    log_k = torch.log(t[:, :1])
    kappa = torch.sqrt((v * v).sum(-1) + 1e-300)
    # ln(kappa / (4 pi sinh kappa))
    small = kappa < 1e-3
    k1 = torch.where(small, torch.ones_like(kappa), kappa)
    log_norm = torch.where(small, -kappa ** 2 / 6.0,
                           -k1 + torch.log(2.0 * k1) - torch.log(-torch.expm1(-2.0 * k1))) - math.log(4.0 * math.pi)
    log_q = (torch.log_softmax(logits, 1) - ls - 0.5 * math.log(2.0 * math.pi)
             - 0.5 * ((log_k - mu) * torch.exp(-ls)) ** 2 + log_norm + (v * t[:, None, 1:]).sum(-1))
    loss = -(torch.logsumexp(log_q, 1) - log_k[:, 0]).mean()
    loss.backward()
    return {"out": h.detach(), "loss": loss.detach(), "grad": flat.grad}

"""The work this simulator is used for, as cases that can be timed and compared.

Two families, both through the package's public entry points:

  net    a spiking network advanced `steps` steps (`engine.Simulation`): the
         records of those steps are fetched and every membrane potential is
         read, as a program does that runs a network in stretches and keeps
         its state.  With `fresh` a pass is the whole call on a lowered model
         (create, initialise, run, fetch, close), as in a parameter sweep.
  grad   a fit of cable cells to recorded potentials (`CableGradient.apply`):
         one forward and one backward of the squared error.

The networks are drawn here from plain numbers, of the shapes
`eden_gb300.workloads` names: single HH cells with DC pulses, branching HH
cells with expTwo synapses and Poisson inputs, izhikevich2007 networks,
both together, HH cells joined by gap junctions, and ball-and-stick cables.
"""
import math

import numpy as np
import torch

from eden_gb300 import lowering
from eden_gb300.engine import MODE_BATCHED, MODE_PLAIN, Simulation
from eden_gb300.gradient import CableGradient, per_cell_density_map, with_weights
from eden_gb300.network import (SYN_EXPONE, SYN_EXPTWO, ChannelDensity, ElectricalProjection, EventSelection,
                                GapJunctionType, Izhikevich2007Cell, NetworkSpec, OutputColumn, PhysicalCell,
                                PoissonInputs, Population, Projection, PulseInputs, SpikeArrayCell, SynapseType,
                                TimedInputs, hh_channels)

G_HH = (0.3, 120.0, 36.0)            # leak, Na, K conductivities, mS/cm2
E_HH = (-54.387, 50.0, -77.0)        # their reversal potentials, mV
LONG_MS = 100000.0                   # an input that lasts the whole run
EXPTWO = dict(name="syn_e2", kind=SYN_EXPTWO, gbase=1.0, erev=0.0, tau_decay=5.0, tau_rise=0.5)


def listed():
    return [
        # a small model created, run and read from scratch: one point of a parameter sweep
        _net("sweep_hh_100", "hh", 100, steps=400, fresh=True),
        # single-compartment HH cells with one DC pulse each: the 1,000 cells of the
        # smallest configuration, and a large ragged count of them
        _net("hh_1000", "hh", 1000, steps=2000),
        _net("hh_30011", "hh", 30011, steps=1000),
        # branching cells with an HH soma, expTwo synapses and Poisson inputs: a model
        # that is worked on interactively, one with active dendrites and synapses all
        # over them, and the 10,000 cells of the batched-network configuration
        _net("trees_50", "trees", 50, in_degree=10, steps=1000),
        _net("trees_1200_dend", "trees", 1200, in_degree=100, steps=500, max_seg=200, dend_hh=0.2, dend_syn=True),
        _net("trees_10000", "trees", 10000, in_degree=100, steps=1000),
        # point and branching cells in one network, four to one
        _net("mixed_5000", "mixed", 5000, in_degree=100, steps=500, pois_hz=2.0),
        # a point-neuron network with ten million synapses
        _net("izh_100000", "izh", 100000, in_degree=100, steps=500),
        # cells coupled within the step
        _net("gap_600", "gap", 600, steps=400),
        # the same branching network step by step (the per-step kernels, which the
        # explicit cable update and the plastic synapses run too)
        _net("plain_1000", "trees", 1000, in_degree=100, steps=200, plain=True),
        # a fit of 256 cables' conductivities and axial resistivities, and one of
        # synaptic weights on longer cables
        _grad("grad_256", 256, dend=50, steps=600),
        _grad("grad_weights_60", 60, dend=110, steps=400, drive=8),
    ]


def _net(name, kind, cells, *, steps, in_degree=0, max_seg=500, pois_hz=5.0, dend_hh=0.0, dend_syn=False,
         plain=False, fresh=False):
    case = dict(family="net", kind=kind, cells=cells, steps=steps, in_degree=in_degree, max_seg=max_seg,
                pois_hz=pois_hz, dend_hh=dend_hh, dend_syn=dend_syn, plain=plain, fresh=fresh)
    return dict(case, name=name) if name else case


def _grad(name, cells, *, dend, steps, drive=0):
    case = dict(family="grad", cells=cells, dend=dend, steps=steps, drive=drive)
    return dict(case, name=name) if name else case


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    kind = rng.choice(["hh", "trees", "trees", "trees", "mixed", "izh", "gap", "grad", "grad", "sweep"])
    if kind == "grad":
        return _grad(None, log_int(8, 300), dend=log_int(5, 140), steps=log_int(100, 600),
                     drive=rng.choice([0, 0, 4, 9]))
    if kind == "sweep":
        if rng.random() < 0.5:
            return _net(None, "hh", log_int(1, 2000), steps=log_int(100, 800), fresh=True)
        return _net(None, "trees", log_int(2, 200), in_degree=rng.randint(1, 30), steps=log_int(100, 500),
                    max_seg=log_int(10, 300), fresh=True)
    if kind == "hh":
        return _net(None, "hh", log_int(10, 30000), steps=log_int(200, 2000), plain=rng.random() < 0.15)
    if kind == "izh":
        return _net(None, "izh", log_int(500, 80000), in_degree=rng.randint(10, 100), steps=log_int(100, 500))
    if kind == "gap":
        return _net(None, "gap", log_int(10, 2000), steps=log_int(100, 400))
    if kind == "mixed":
        return _net(None, "mixed", log_int(100, 8000), in_degree=rng.randint(10, 100), steps=log_int(200, 500),
                    pois_hz=rng.choice([0.0, 2.0, 5.0]))
    plain = rng.random() < 0.2
    dend = rng.random() < 0.4
    return _net(None, "trees", log_int(20, 1000 if plain else 1500 if dend else 8000), in_degree=rng.randint(1, 100),
                steps=log_int(100, 200 if plain else 1000), max_seg=log_int(20, 500), pois_hz=rng.choice([0.0, 5.0, 20.0]),
                dend_hh=round(rng.uniform(0.05, 0.3), 2) if dend else 0.0, dend_syn=dend, plain=plain)


# ---------------------------------------------------------------------------
# networks as plain numbers
# ---------------------------------------------------------------------------
def _random_tree(rng, n):
    """A soma and n - 1 segments, each on a uniformly chosen earlier one."""
    parent = np.concatenate([[-1], np.floor(rng.uniform(0, 1, n - 1) * np.arange(1, n)).astype(np.int64)])
    length, diam = np.round(rng.uniform(5.0, 50.0, n), 3), np.round(rng.uniform(0.5, 4.0, n), 3)
    length[0] = diam[0] = 20.0
    return parent, length, diam


def _network(case, seed):
    """The network of a case: `groups` of physical cells (parent, length,
    diameter, HH mask, axial resistivity, how many), then izhikevich cells, in
    order of their ids, and what connects and drives them."""
    rng = np.random.default_rng([int(seed), 77])
    kind, n = case["kind"], case["cells"]
    form = np.random.default_rng([n, case["max_seg"], 79])  # the cells' shapes belong to the model, not to one run of it
    net = dict(dt=25.0, groups=[], izh=0, exc=0, syn=[], pois=None, pulse=None, gap=None)
    single = (np.array([-1]), np.array([0.0]), np.array([17.8]), np.ones(1, bool), 30.0)
    if kind == "hh":
        net["groups"] = [single + (n,)]
        net["pulse"] = (np.arange(n), np.round(rng.uniform(0.0, 0.3, n), 6))
    elif kind == "trees" or kind == "mixed":
        n_izh = int(0.8 * n) if kind == "mixed" else 0
        n_tree = n - n_izh
        n_seg = (np.full(n_tree, min(100, case["max_seg"])) if kind == "mixed" else
                 np.round(np.exp(form.uniform(0.0, math.log(case["max_seg"]), n_tree))).astype(int))
        for k in n_seg:
            tree = _random_tree(form, int(k))
            hh = form.random(int(k)) < case["dend_hh"]
            hh[0] = True
            net["groups"].append(tree + (hh, 150.0, 1))
        net["izh"] = net["exc"] = n_izh
        deg = case["in_degree"]
        post = np.repeat(np.arange(n), deg)
        pre = rng.integers(0, n, post.size)
        seg = np.zeros(post.size, np.int64)
        if case["dend_syn"]:
            seg = (form.random(post.size) * np.concatenate([n_seg, np.ones(n_izh, int)])[post]).astype(np.int64)
        weight = np.round(rng.uniform(0.2, 1.0 if kind == "trees" else 0.4, post.size), 4)
        delay = np.round(rng.uniform(0.5, 5.0, post.size), 3)
        delay[0] = 0.5
        net["syn"].append((EXPTWO, pre, post, seg, weight, delay))
        if case["pois_hz"] > 0:
            net["pois"] = (case["pois_hz"], post.copy())
        driven = np.arange(0, n_tree, 10 if net["pois"] else 1)  # cells with an electrode: a tenth, or all
        net["pulse"] = (driven, np.round(rng.uniform(0.0, 0.3, len(driven)), 6))
    elif kind == "izh":
        net.update(dt=100.0, izh=n, exc=int(round(0.8 * n)))
        post = np.repeat(np.arange(n), case["in_degree"])
        pre = rng.integers(0, n, post.size)
        weight = np.round(rng.lognormal(-1.0, 0.5, post.size), 6)
        delay = rng.integers(10, 201, post.size) * 0.1
        delay[0] = 1.0
        exc = pre < net["exc"]
        zero = np.zeros(post.size, np.int64)
        for name, erev, tau, on in (("syn_exc", 0.0, 2.0, exc), ("syn_inh", -80.0, 5.0, ~exc)):
            net["syn"].append((dict(name=name, kind=SYN_EXPONE, gbase=1.0, erev=erev, tau_decay=tau), pre[on], post[on],
                               zero[on], weight[on], np.round(delay[on], 3)))
        net["pulse"] = (np.arange(n), np.round(rng.uniform(0.0, 0.5, n), 6))
    else:
        # HH somata in a ring with chords, a third of them driven, and branching
        # cells whose dendrites hang on them
        n_br = max(1, n // 4)
        n_hh = max(3, n - n_br)
        branch = (np.array([-1, 0, 1, 0]), np.array([20.0, 80.0, 60.0, 70.0]), np.array([20.0, 2.0, 1.5, 1.8]),
                  np.arange(4) == 0, 150.0)
        net["groups"] = [single + (n_hh,), branch + (n_br,)]
        hh = np.arange(n_hh)
        a = np.concatenate([hh, rng.integers(0, n_hh, n_hh // 2)])
        b = np.concatenate([np.roll(hh, -1), rng.integers(0, n_hh, n_hh // 2)])
        b = np.where(a == b, (b + 1) % n_hh, b)
        pre = np.concatenate([a, rng.integers(0, n_hh, 2 * n_br)])
        post = np.concatenate([b, np.repeat(n_hh + np.arange(n_br), 2)])
        seg = np.concatenate([np.zeros(len(a), np.int64), np.tile([2, 3], n_br)])
        net["gap"] = (1.0, pre, post, seg, np.round(rng.uniform(0.5, 1.5, len(pre)), 4))
        net["pulse"] = (hh[::3], np.round(rng.uniform(0.1, 0.3, len(hh[::3])), 4))
        target = np.concatenate([hh[1::3], n_hh + np.arange(n_br)])
        net["syn"].append((EXPTWO, rng.integers(0, n_hh, len(target)), target, np.where(target < n_hh, 0, 2),
                           np.round(rng.uniform(0.5, 1.5, len(target)), 4), np.round(rng.uniform(0.5, 3.0, len(target)), 3)))
    n_all = sum(g[5] for g in net["groups"]) + net["izh"]
    net["cells"] = n_all
    net["rec"] = np.sort(rng.choice(n_all, min(10, n_all), replace=False))
    return net


def _spec(case, seed, net):
    """The same network as the package's own description of it."""
    spec = NetworkSpec(case["kind"], net["dt"] / 1000.0, LONG_MS, int(seed) & 0x7fffffff, channels=hh_channels())
    for k, (parent, length, diam, hh, ra, count) in enumerate(net["groups"]):
        dens = [ChannelDensity(0, G_HH[0], E_HH[0], np.ones(len(parent), bool)),
                ChannelDensity(1, G_HH[1], E_HH[1], hh), ChannelDensity(2, G_HH[2], E_HH[2], hh)]
        spec.cells.append(PhysicalCell("c%d" % k, parent, length, diam, dens, cm=1.0, ra=ra, v0=-65.0, spike_thresh=-20.0))
        spec.populations.append(Population("p%d" % k, "c%d" % k, count))
    if net["izh"]:
        spec.cells.append(Izhikevich2007Cell("izRS", a=0.03, d=100.0, c=-50.0))
        spec.populations.append(Population("exc", "izRS", net["exc"]))
        if net["izh"] > net["exc"]:
            spec.cells.append(Izhikevich2007Cell("izFS", a=0.1, d=0.0, c=-55.0))
            spec.populations.append(Population("inh", "izFS", net["izh"] - net["exc"]))
    for j, (syn, pre, post, seg, weight, delay) in enumerate(net["syn"]):
        spec.synapses.append(SynapseType(**syn))
        spec.projections.append(Projection("proj%d" % j, "*", "*", syn["name"], pre, post, seg, weight, delay))
    if net["pois"]:
        rate, cell = net["pois"]
        spec.poissons.append(PoissonInputs("*", EXPTWO["name"], rate, cell, np.zeros(cell.size, np.int64)))
    if net["pulse"]:
        cell, amp = net["pulse"]
        spec.pulses.append(PulseInputs("*", cell, np.zeros(cell.size, np.int64), np.zeros(cell.size),
                                       np.full(cell.size, LONG_MS), amp))
    if net["gap"]:
        g, pre, post, seg, weight = net["gap"]
        spec.gap_types.append(GapJunctionType("gap", g))
        spec.electrical.append(ElectricalProjection("gaps", "gap", pre, np.zeros(pre.size, np.int64), post, seg, weight))
    start = np.concatenate([[0], np.cumsum([p.size for p in spec.populations])])
    where = np.searchsorted(start, net["rec"], side="right") - 1
    spec.trace_columns = [OutputColumn(spec.populations[k].name, int(g - start[k]), 0) for g, k in zip(net["rec"], where)]
    return spec


# ---------------------------------------------------------------------------
# cables to fit
# ---------------------------------------------------------------------------
def _cables(case, seed):
    """Ball-and-stick cells: a soma and `dend` segments of a 500 um cable, HH
    channels all over, seven lognormal parameters a cell, a 0.5 nA step into the
    soma; with `drive`, spike lists onto the dendrite and timed inhibition."""
    rng = np.random.default_rng([int(seed), 78])
    n, nd = case["cells"], case["dend"]
    c = dict(n=n, n_seg=nd + 1, length_ms=case["steps"] * 0.025)
    c["params"] = np.round(np.array([0.3, 120.0, 36.0, 0.3, 120.0, 36.0, 150.0]) * rng.lognormal(0.0, 0.2, (n, 7)), 6)
    c["length"], c["diam"] = np.full(nd + 1, 500.0 / nd), np.full(nd + 1, 2.0)
    c["length"][0] = c["diam"][0] = 20.0
    # the recording that the cells are fitted to: rest, an offset and a slow wave
    t = np.arange(case["steps"])[:, None] * 0.025
    c["target"] = -60.0 + rng.normal(0.0, 3.0, n) + 8.0 * np.sin(2 * np.pi * t / rng.uniform(8.0, 20.0, n))
    c["arrays"], c["syn"], c["timed"] = [], None, None
    if case["drive"]:
        def times(per_ms):  # between the grid's steps: no spike falls on a step's edge
            return np.unique(np.round(rng.uniform(0.0, c["length_ms"], max(2, int(c["length_ms"] / per_ms))), 2)) + 0.003
        c["arrays"] = [times(5.0) for _ in range(4)]
        post = np.repeat(np.arange(n), case["drive"])
        c["syn"] = (rng.integers(0, 4, post.size), post, rng.integers(1, nd + 1, post.size),
                    np.round(rng.uniform(0.5, 1.5, post.size), 4), np.round(rng.uniform(1.0, 3.0, post.size), 3))
        cells = np.repeat(np.arange(n), 2)
        c["timed"] = (cells, [times(10.0) for _ in cells], np.round(rng.uniform(0.5, 1.5, len(cells)), 4))
    return c


DRIVE = (dict(name="syn_e2", kind=SYN_EXPTWO, gbase=2.0, erev=0.0, tau_decay=5.0, tau_rise=0.5),
         dict(name="syn_i1", kind=SYN_EXPONE, gbase=3.0, erev=-80.0, tau_decay=5.0))


def _cable_spec(case, c):
    spec = NetworkSpec("cables", 0.025, c["length_ms"], 1, channels=hh_channels())
    parent = np.arange(-1, c["n_seg"] - 1)
    soma = parent < 0
    for i in range(c["n"]):
        p = c["params"][i]
        dens = [ChannelDensity(k, p[k + 3 * d], E_HH[k], m) for d, m in ((0, soma), (1, ~soma)) for k in range(3)]
        spec.cells.append(PhysicalCell("b%d" % i, parent, c["length"], c["diam"], dens, cm=1.0, ra=float(p[6]), v0=-65.0,
                                       spike_thresh=-20.0))
        spec.populations.append(Population("p%d" % i, "b%d" % i, 1))
    cells = np.arange(c["n"])
    spec.pulses.append(PulseInputs("*", cells, 0 * cells, np.zeros(c["n"]), np.full(c["n"], LONG_MS), np.full(c["n"], 0.5)))
    if c["syn"]:
        spec.synapses += [SynapseType(**s) for s in DRIVE]
        for k, t in enumerate(c["arrays"]):
            spec.cells.append(SpikeArrayCell("s%d" % k, t))
            spec.populations.append(Population("ps%d" % k, "s%d" % k, 1))
        src, post, seg, weight, delay = c["syn"]
        spec.projections.append(Projection("drive", "*", "*", "syn_e2", c["n"] + src, post, seg, weight, delay))
        cell, times, weight = c["timed"]
        spec.timed.append(TimedInputs("syn_i1", cell, 0 * cell, times, weight))
    return spec


# ---------------------------------------------------------------------------
def prepare(case, seed):
    if case["family"] == "grad":
        c = _cables(case, seed)
        low = lowering.lower(_cable_spec(case, c))
        pmap = per_cell_density_map(low, list(range(6)))
        if case["drive"]:
            pmap = with_weights(low, pmap)
        fit = CableGradient(low, pmap, rec_comp=low.phys_comp_off[:-1], n_steps=case["steps"])
        params = torch.tensor(pmap.values, device="cuda", requires_grad=True)
        return dict(case=case, fit=fit, params=params,
                    target=torch.tensor(c["target"], dtype=torch.float32, device="cuda"))
    net = _network(case, seed)
    low = lowering.lower(_spec(case, seed, net))
    options = dict(mode=MODE_PLAIN if case["plain"] else MODE_BATCHED, record_capacity_steps=case["steps"])
    # room for a spike of every cell in each 10 ms, and one more
    state = dict(case=case, low=low, options=options, room=int(net["cells"] * (2 + case["steps"] * net["dt"] / 10000.0)))
    if not case["fresh"]:
        state["sim"] = Simulation(low, **options)
        state["sim"].initialize()
    return state


def run(state):
    case = state["case"]
    if case["family"] == "grad":
        params = state["params"]
        params.grad = None
        trace = state["fit"].apply(params)
        loss = ((trace - state["target"]) ** 2).mean()
        loss.backward()
        return dict(trace=trace.detach(), loss=loss.detach(), grad=params.grad)
    if case["fresh"]:
        sim = Simulation(state["low"], **state["options"])
        rec = sim.run(case["steps"])
        v = sim.read_v()
        sim.close()
    else:
        sim = state["sim"]
        sim.run_steps(case["steps"])
        rec = sim.fetch()
        v = sim.read_v()
    src, step = np.full(state["room"], -1, np.int32), np.full(state["room"], -1, np.int32)
    src[:len(rec.spike_src)], step[:len(rec.spike_step)] = rec.spike_src, rec.spike_step
    return dict(trace=rec.trace, trace_step=rec.trace_step, spike_src=src, spike_step=step, v=v)


def _sizes(case):
    """(compartments, HH compartments, izhikevich cells, synapses, Poisson inputs) of a network, on average."""
    kind, n = case["kind"], case["cells"]
    if kind == "hh":
        return n, n, 0, 0, 0
    if kind == "izh":
        return 0, 0, n, n * case["in_degree"], 0
    if kind == "gap":
        return n - n // 4 + n // 4 * 4, n, 0, n // 2, 0
    trees, seg = n, (case["max_seg"] - 1) / max(math.log(case["max_seg"]), 1e-9)
    if kind == "mixed":
        trees, seg = n - int(0.8 * n), min(100, case["max_seg"])
    comps = trees * seg
    inputs = n * case["in_degree"]
    return comps, trees + case["dend_hh"] * (comps - trees), n - trees, inputs, inputs if case["pois_hz"] > 0 else 0


def work(case):
    """Constants and state read once, state and records written once; the
    operations of every step (a pass of the cable solve is 12 a compartment, the
    gates and currents of the HH channels 160, an izhikevich cell 20)."""
    steps = case["steps"]
    if case["family"] == "grad":
        comps = case["cells"] * (case["dend"] + 1)
        return dict(bytes=3.0 * 4.0 * steps * case["cells"] + 60.0 * comps, flops=steps * comps * (172.0 + 2 * 172.0))
    comps, hh, izh, syn, pois = _sizes(case)
    return dict(bytes=comps * 28.0 + hh * 48.0 + izh * 60.0 + syn * 40.0 + pois * 48.0 + 4.0 * steps * 10,
                flops=steps * (comps * 12.0 + hh * 160.0 + izh * 20.0))


# ---------------------------------------------------------------------------
# the same in 64 bits
# ---------------------------------------------------------------------------
def exact(case, seed):
    if case["family"] == "grad":
        if case["steps"] * case["cells"] * (case["dend"] + 1) ** 3 > 5e10:
            return None
        return _exact_grad(case, _cables(case, seed))
    comps, hh, izh, syn, pois = _sizes(case)
    if case["steps"] * (3e-3 + 4e-8 * comps + 2.5e-7 * hh + 2e-7 * izh + 3e-8 * (syn + 2 * pois)) > 18.0:
        return None
    trace, v = _exact_net(case, seed, _network(case, seed))
    return dict(trace=trace, trace_step=None, spike_src=None, spike_step=None, v=v)


def _geometry(length, diam, ra, parent):
    """(capacitance pF, area um2, axial resistance to the parent MOhm)"""
    area = np.where(length == 0, np.pi * diam ** 2, np.pi * diam * length)
    half = ra * 1e-3 * (4.0 / np.pi) * (length / 2.0) / diam ** 2 * 10.0
    return area * 1e-2, area, np.where(parent < 0, 1.0, half + half[np.maximum(parent, 0)])


def _hh_rates(v, exp, where):
    """Forward and reverse rates of m, h and n, per us."""
    def linear(r, mid, s):
        x = (v - mid) / s
        return where(x == 0, r + 0 * x, r * x / (1.0 - exp(-where(x == 0, 1.0 + 0 * x, x))))
    return ((linear(1e-3, -40.0, 10.0), 4e-3 * exp((v + 65.0) / -18.0)),
            (0.07e-3 * exp((v + 65.0) / -20.0), 1e-3 / (1.0 + exp((-35.0 - v) / 10.0))),
            (linear(0.1e-3, -55.0, 10.0), 0.125e-3 * exp((v + 65.0) / -80.0)))


class _Tree:
    """The backward-Euler cable equations of many trees, solved level by level."""

    def __init__(self, parent, c, r, dt):
        depth = np.zeros(len(parent), np.int64)
        for i in range(len(parent)):  # a parent comes before its children
            if parent[i] >= 0:
                depth[i] = depth[parent[i]] + 1
        kids = np.flatnonzero(parent >= 0)
        self.axial = np.zeros(len(parent))
        np.add.at(self.axial, kids, 1.0 / (r[kids] * c[kids]))
        np.add.at(self.axial, parent[kids], 1.0 / (r[kids] * c[parent[kids]]))
        self.u, self.l = -dt / (r * c), -dt / (r * c[np.maximum(parent, 0)])
        self.levels = []
        for d in range(int(depth.max(initial=0)), 0, -1):
            k = np.flatnonzero(depth == d)
            k = k[np.argsort(parent[k], kind="stable")]
            up, first = np.unique(parent[k], return_index=True)
            self.levels.append((k, parent[k], up, first))

    def solve(self, d, x):
        for k, p, up, first in self.levels:
            f = self.l[k] / d[k]
            d[up] -= np.add.reduceat(f * self.u[k], first)
            x[up] -= np.add.reduceat(f * x[k], first)
        x /= d  # roots; the others below replace theirs
        for k, p, up, first in reversed(self.levels):
            x[k] -= self.u[k] * x[p] / d[k]
        return x


def _uniform(item, instance, step, call):
    """The network's random numbers in [0, 1): a 64-bit hash of (cell, instance, step, call)."""
    def mix(k):
        k = ~k + (k << np.uint64(21))
        k ^= k >> np.uint64(24)
        k = (k + (k << np.uint64(3))) + (k << np.uint64(8))
        k ^= k >> np.uint64(14)
        k = (k + (k << np.uint64(2))) + (k << np.uint64(4))
        k ^= k >> np.uint64(28)
        return k + (k << np.uint64(31))
    with np.errstate(over="ignore"):
        hi = (item.astype(np.int64).view(np.uint64) << np.uint64(24)) | instance.astype(np.uint64)
        lo = np.full(1, (call << 40) | step, np.uint64)
        return (mix(mix(lo) ^ hi) & np.uint64((1 << 23) - 1)).astype(np.float64) / (1 << 23)


def _exact_net(case, seed, net):
    dt, steps = net["dt"], case["steps"]
    parent, c, area, r, hh, base = [], [], [], [], [], []
    at = 0
    for par, length, diam, mask, ra, count in net["groups"]:
        geo = _geometry(length, diam, ra, par)
        for _ in range(count):
            base.append(at)
            parent.append(np.where(par >= 0, par + at, -1)); hh.append(mask)
            c.append(geo[0]); area.append(geo[1]); r.append(geo[2])
            at += len(par)
    n_phys, n_comp = len(base), at
    base = np.concatenate([np.array(base, np.int64), n_comp + np.arange(net["izh"])])
    n = n_comp + net["izh"]
    cat = lambda parts: np.concatenate(parts) if parts else np.zeros(0)  # noqa: E731
    c, area, r = cat(c), cat(area), cat(r)
    hh = np.flatnonzero(cat(hh))
    tree = _Tree(cat(parent).astype(np.int64), c, r, dt)
    unit = 1e-5 * area  # mS/cm2 to uS
    v = np.full(n, -65.0)
    v[n_comp:] = -60.0
    u = np.zeros(net["izh"])
    fs = np.arange(net["izh"]) >= net["exc"]
    iz_a, iz_d, iz_c = np.where(fs, 0.1, 0.03), np.where(fs, 0.0, 100.0) * 1e-3, np.where(fs, -55.0, -50.0)
    gates = [a / (a + b) for a, b in _hh_rates(v[hh], np.exp, np.where)]

    def synapses(syn, target, weight):
        two = syn["kind"] == SYN_EXPTWO
        td, tr = syn["tau_decay"] * 1e3, syn.get("tau_rise", 0.0) * 1e3
        jump = syn["gbase"] * 1e-3
        if two:
            peak = math.log(td / tr) * tr * td / (td - tr)
            jump /= math.exp(-peak / td) - math.exp(-peak / tr)
        return dict(two=two, td=td, tr=tr, jump=jump, erev=syn["erev"], target=target, w=weight,
                    a=np.zeros(len(target)), b=np.zeros(len(target)))

    def conductance(s):
        return np.bincount(s["target"], s["w"] * ((s["b"] - s["a"]) if s["two"] else s["a"]), n)

    def advance(s, fire):
        if s["two"]:
            s["b"] = np.where(fire, s["b"] + s["jump"], s["b"] * (1.0 - dt / s["td"]))
            s["a"] = np.where(fire, s["a"] + s["jump"], s["a"] * (1.0 - dt / s["tr"]))
        else:
            s["a"] = np.where(fire, s["a"] + s["jump"], s["a"] * (1.0 - dt / s["td"]))

    conn = []
    for syn, pre, post, seg, weight, delay in net["syn"]:
        s = synapses(syn, base[post] + np.where(post < n_phys, seg, 0), weight)
        conn.append(dict(s, pre=pre, delay=delay * 1e3, pend=np.full(len(pre), -np.inf)))
    pois = None
    if net["pois"]:
        rate, cell = net["pois"]
        pois = synapses(EXPTWO, base[cell], np.ones(len(cell)))
        bits = int(format((int(seed) & 0x7fffffff) & 0xffffffff, "032b")[::-1], 2)
        item = (np.uint32(bits) ^ cell.astype(np.uint32)).view(np.int32).astype(np.int64)
        order = np.argsort(cell, kind="stable")
        inst = np.empty(len(cell), np.int64)
        inst[order] = np.arange(len(cell)) - np.searchsorted(cell[order], cell[order])
        mean = 1e6 / rate
        since, wait = np.zeros(len(cell)), -mean * np.log(1.0 - _uniform(item, inst, 0, 0))
    pulse = np.zeros(n)
    if net["pulse"]:
        np.add.at(pulse, base[net["pulse"][0]], net["pulse"][1])
    gap = None
    if net["gap"]:
        g, pre, post, seg, weight = net["gap"]
        ends = (base[pre], base[post] + seg)
        gap = (np.concatenate(ends), np.concatenate(ends[::-1]), np.tile(g * 1e-3 * weight, 2))
    rec = base[net["rec"]]
    trace = np.zeros((steps, len(rec)))
    spiked = np.zeros(len(base), bool)
    for k in range(1, steps + 1):
        t = (k - 1) * dt
        trace[k - 1] = v[rec]
        cur, con = pulse.copy(), np.zeros(n)
        for s in conn + ([pois] if pois else []):
            g = conductance(s)
            cur += g * (s["erev"] - v)
            con += g
        if gap:
            cur += np.bincount(gap[0], gap[2] * (v[gap[1]] - v[gap[0]]), n)
        for s in conn:  # the single pending spike, then this step's triggers
            fire = (t <= s["pend"]) & (s["pend"] < t + dt)
            trig = np.flatnonzero(spiked[s["pre"]])
            fresh = t + s["delay"][trig]
            fire[trig] |= fresh < t + dt
            late = s["pend"][trig]
            s["pend"][trig] = np.where((late < t + dt) & (late < fresh), fresh, late)
            advance(s, fire)
        if pois:
            fire = since > wait
            since = np.where(fire, 0.0, since + dt)
            if fire.any():
                wait[fire] = -mean * np.log(1.0 - _uniform(item[fire], inst[fire], k, 1))
            advance(pois, fire)
        vn = np.empty(n)
        if n_comp:
            w = v[:n_comp]
            g = unit * G_HH[0]
            cur[:n_comp] += g * (E_HH[0] - w)
            con[:n_comp] += g
            vh = w[hh]
            m, h, q = gates
            for gg, e in ((unit[hh] * G_HH[1] * m ** 3 * h, E_HH[1]), (unit[hh] * G_HH[2] * q ** 4, E_HH[2])):
                cur[hh] += gg * (e - vh)
                con[hh] += gg
            d = 1.0 + dt * (con[:n_comp] / c + tree.axial)
            vn[:n_comp] = tree.solve(d, w + dt * (cur[:n_comp] + w * con[:n_comp]) / c)
            for j, (a, b) in enumerate(_hh_rates(vh, np.exp, np.where)):
                keep = np.exp(-dt * (a + b))
                gates[j] = np.clip(keep * gates[j] + (1.0 - keep) * a / (a + b), 1e-6, 1 - 1e-6)
            soma = base[:n_phys]
            spiked[:n_phys] = (w[soma] < -20.0) & (vn[soma] > -20.0)
        if net["izh"]:
            w = v[n_comp:]
            top = w > 35.0
            vn[n_comp:] = np.where(top, iz_c, w + dt * (0.7e-3 * (w + 60.0) * (w + 40.0) + cur[n_comp:] - u) / 100.0)
            u = np.where(top, u + iz_d, u + dt * 1e-3 * iz_a * (-2e-3 * (w + 60.0) - u))
            spiked[n_phys:] = top
        v = vn
    return trace, v


def _exact_grad(case, c):
    """Trace, loss and gradient by plain automatic differentiation, a stretch of steps at a time."""
    from torch.utils.checkpoint import checkpoint
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    dt, steps, n, ns = 25.0, case["steps"], c["n"], c["n_seg"]
    f64 = lambda x: torch.tensor(np.asarray(x), dtype=torch.float64, device=dev)  # noqa: E731
    parent = np.arange(-1, ns - 1)
    cap, area, r1 = (f64(x) for x in _geometry(c["length"], c["diam"], 1.0, parent))  # r1: per ohm cm
    # axial part of the equations for 1 ohm cm: rows scale with 1 / ra
    axial = torch.zeros(ns, ns, dtype=torch.float64, device=dev)
    for i in range(1, ns):
        for a, b in ((i, i - 1), (i - 1, i)):
            axial[a, a] += 1.0 / (r1[i] * cap[a])
            axial[a, b] -= 1.0 / (r1[i] * cap[a])
    params = f64(c["params"].astype(np.float32))
    weights, unit_g = None, None
    drive = []
    if c["syn"]:
        def unit(syn, events):  # exposure of weight-1 synapses at the steps' starts, [steps, items]
            two, td = syn["kind"] == SYN_EXPTWO, syn["tau_decay"] * 1e3
            tr = syn["tau_rise"] * 1e3 if two else 1.0
            jump = syn["gbase"] * 1e-3
            if two:
                peak = math.log(td / tr) * tr * td / (td - tr)
                jump /= math.exp(-peak / td) - math.exp(-peak / tr)
            a = b = np.zeros(events.shape[1])
            out = np.zeros((steps + 1, events.shape[1]))
            for k in range(1, steps + 1):
                out[k] = b - a if two else b
                a = np.where(events[k], a + jump, a * (1.0 - dt / tr)) if two else a
                b = np.where(events[k], b + jump, b * (1.0 - dt / td))
            return f64(out)
        src, post, seg, w, delay = c["syn"]
        order = np.lexsort((np.arange(len(post)), post * ns + seg))  # by compartment, as the parameters are numbered
        src, post, seg, w, delay = src[order], post[order], seg[order], w[order], delay[order] * 1e3
        emit = [set((np.floor(t * 1e3 / dt).astype(int) + 2).tolist()) for t in c["arrays"]]
        ev = np.zeros((steps + 1, len(post)), bool)
        for i in range(len(post)):
            pend = -np.inf
            for k in range(1, steps + 1):
                t = (k - 1) * dt
                ev[k, i] = t <= pend < t + dt
                if k in emit[src[i]] and pend < t + dt and pend < t + delay[i]:
                    pend = t + delay[i]
        cell, times, tw = c["timed"]
        et = np.zeros((steps + 1, len(cell)), bool)
        for i, t in enumerate(times):
            k = np.floor(t * 1e3 / dt).astype(int) + 1
            et[k[k <= steps], i] = True
        weights = f64(np.concatenate([w, tw]).astype(np.float32))
        unit_g = torch.cat([unit(DRIVE[0], ev), unit(DRIVE[1], et)], 1)
        at = torch.tensor(np.concatenate([post * ns + seg, cell * ns]), device=dev)
        drive = f64(np.concatenate([np.full(len(post), DRIVE[0]["erev"]), np.full(len(cell), DRIVE[1]["erev"])]))
    pulse = torch.zeros(n, ns, dtype=torch.float64, device=dev)
    pulse[:, 0] = 0.5
    erev = f64(E_HH)

    def stretch(k0, k1, v, m, h, q, p, w):
        g = torch.cat([p[:, None, 0:3], p[:, None, 3:6].expand(n, ns - 1, 3)], 1) * (1e-5 * area)[None, :, None]
        ax = axial[None] * (dt / p[:, 6])[:, None, None]
        out = []
        for k in range(k0, k1):
            out.append(v[:, 0])
            cond = torch.stack([g[..., 0], g[..., 1] * m ** 3 * h, g[..., 2] * q ** 4], -1)
            cur = pulse + (cond * (erev - v[..., None])).sum(-1)
            con = cond.sum(-1)
            if w is not None:
                gd = w * unit_g[k]
                flat = torch.zeros(n * ns, dtype=torch.float64, device=dev)
                con = con + flat.index_add(0, at, gd).view(n, ns)
                cur = cur + flat.index_add(0, at, gd * (drive - v.reshape(-1)[at])).view(n, ns)
            mat = ax + torch.diag_embed(1.0 + dt * con / cap)
            vn = torch.linalg.solve(mat, v + dt * (cur + v * con) / cap)
            new = []
            for s, (a, b) in zip((m, h, q), _hh_rates(v, torch.exp, torch.where)):
                keep = torch.exp(-dt * (a + b))
                new.append((keep * s + (1.0 - keep) * a / (a + b)).clamp(1e-6, 1 - 1e-6))
            v, (m, h, q) = vn, new
        return (torch.stack(out), v, m, h, q)

    params.requires_grad_(True)
    if weights is not None:
        weights.requires_grad_(True)
    v = torch.full((n, ns), -65.0, dtype=torch.float64, device=dev)
    state = (v,) + tuple(a / (a + b) for a, b in _hh_rates(v, torch.exp, torch.where))
    rows = []
    for k0 in range(1, steps + 1, 25):
        part, *state = checkpoint(stretch, k0, min(steps + 1, k0 + 25), *state, params, weights, use_reentrant=False)
        rows.append(part)
    trace = torch.cat(rows)
    target = f64(c["target"].astype(np.float32))
    loss = ((trace - target) ** 2).mean()
    loss.backward()
    grad = params.grad.reshape(-1) if weights is None else torch.cat([params.grad.reshape(-1), weights.grad])
    return dict(trace=trace.detach(), loss=loss.detach(), grad=grad)

"""Cases for timing the framework through its public entry points.

The listed cases are the work a user of the V1 column has it do, on the synthetic networks of
``v1_glif_model_b200/synth.py`` (5,000, 66,634 and 230,924 neurons) and at the sizes of the benchmark
and the tests: one step of the cell, operator by operator; forward rollouts for evaluation (one trial of
the small net up to ten trials of the column, and from host buffers); data-parallel training steps with
the benchmark's losses and with the reference's own losses, for the one-hot basis and for a dense one
with 121 synapse types; explicit output gradients; and the LGN front end (movie -> firing rates).
``draw`` gives cases of the same kinds with sizes spread over the ranges between them.

A program keeps ONE network for its whole life and sends it ever new inputs, so networks (connectivity,
initial weights, loss tables) are a property of the case and are built once per process; ``prepare`` makes
from its seed everything a run consumes - stimulus spikes or rates, background counts, the carried state
reached by simulating 300 ms of such input, output gradients, movies - and puts the weights back to
their initial values.
"""
from __future__ import annotations

import collections
import dataclasses
import math

import numpy as np
import torch

from v1_glif_model_b200 import _lib, synth
from v1_glif_model_b200.lgn import LGN
from v1_glif_model_b200.models import V1Column
from v1_glif_model_b200.training import Trainer, WeightRegularizer

WARM_STEPS = 300          # simulated ms from the zero state to the network's working regime
# small enough that hundreds of training steps leave the network in the same activity regime
LEARNING_RATE = 1e-5
CELL = dict(dampening_factor=0.5, pseudo_width=0.5, recurrent_dampening_factor=0.5, voltage_gradient_dampening=0.5)
LOSS = dict(rate_cost=100.0, voltage_cost=1e-3, sync_cost=1.0, fano_target=1.0, sync_bin=50)
# the front end's sizes: frames of 120 x 240 pixels, 14 filter sizes, temporal kernels of 250 ms
LGN_HEIGHT, LGN_WIDTH, LGN_SIDES, LGN_TAPS = 120, 240, tuple(range(3, 31, 2)), 250

SMALL, COLUMN, STRESS = 5000, 66634, 230924


def listed():
    return [
        # a notebook or a custom-op binding stepping the small net: launches and host work count
        dict(name="call_5k_b1", kind="call", neurons=SMALL, batch=1, delay=5, basis="onehot"),
        # the gradient of one step's recurrent currents at full size, as a framework's tape asks for it
        dict(name="currents_grad_67k_b5", kind="currents", neurons=COLUMN, batch=5, delay=5, basis="onehot"),
        # forward evaluation of the small net, one trial of 200 ms, spikes and voltages written
        dict(name="eval_5k_b1_t200", kind="eval", neurons=SMALL, batch=1, steps=200, delay=5, basis="onehot", voltage=True),
        # forward evaluation of the column, spikes and voltages written: the benchmark's forward leg
        dict(name="eval_67k_b5_t2500", kind="eval", neurons=COLUMN, batch=5, steps=2500, delay=5, basis="onehot", voltage=True),
        # ten trials of one grating angle, background noise drawn on the device, spikes only
        dict(name="eval_67k_b10_t500", kind="eval", neurons=COLUMN, batch=10, steps=500, delay=5, basis="onehot", voltage=False),
        # evaluation through pinned host buffers, spikes returned as bits
        dict(name="host_67k_b5_t1000", kind="host", neurons=COLUMN, batch=5, steps=1000, delay=5, basis="onehot"),
        # training step of the small net
        dict(name="train_5k_b2_t500", kind="train", neurons=SMALL, batch=2, steps=500, delay=5, basis="onehot", losses="simple"),
        # training step of the column: the benchmark's headline
        dict(name="train_67k_b5_t500", kind="train", neurons=COLUMN, batch=5, steps=500, delay=5, basis="onehot", losses="simple"),
        # the same column with firing rates in, spikes and noise drawn on the device, the reference's
        # rate-distribution, synchrony and OSI/DSI targets and both weight regularisers
        dict(name="train_67k_b4_t300_full", kind="train", neurons=COLUMN, batch=4, steps=300, delay=5, basis="onehot", losses="full"),
        # the column with a dense basis of 121 synapse types over four channels
        dict(name="train_67k_b5_t200_dense", kind="train", neurons=COLUMN, batch=5, steps=200, delay=5, basis="dense", losses="simple"),
        # the large column in a high-activity regime
        dict(name="train_231k_b4_t100", kind="train", neurons=STRESS, batch=4, steps=100, delay=5, basis="onehot", losses="simple"),
        # one second of movie through the LGN front end
        dict(name="lgn_17400_t1000", kind="lgn", units=17400, frames=1000),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["call", "currents", "eval", "eval", "eval", "host", "train", "train", "train", "grads", "lgn"])
    if kind == "lgn":
        units, frames = _log(rng, 500, 17400), _log(rng, 50, 1000)
        return dict(kind=kind, units=units, frames=frames)
    n = _log(rng, SMALL, STRESS)
    case = dict(kind=kind, neurons=n, delay=rng.choice([5, 5, 5, 3, 8]), basis=rng.choice(["onehot", "onehot", "dense"]))
    if kind in ("call", "currents"):
        case["batch"] = rng.randint(1, 5)
        return case
    train = kind in ("train", "grads")
    # a training step holds at most 8 trials (4 on the largest networks), a host-buffer evaluation 8
    most = (4 if n > 100000 else 8) if train else 8 if kind == "host" else 10
    case["batch"] = b = rng.randint(1, most)
    t = _log(rng, 50, 500 if train else 2500)
    # no more time than the largest listed case takes: 90 M neuron-steps forth and back, 400 M forward, and
    # fewer where a neuron-step costs more (a dense basis, a state that does not fit on the chip)
    most_steps = (90e6 if train else 400e6) * (0.4 if case["basis"] == "dense" else 1.0)
    if n > 100000 and not (train and case["basis"] == "onehot"):
        most_steps *= 0.5
    case["steps"] = max(20, min(t, int(most_steps / (n * b))))
    if kind == "eval":
        case["voltage"] = rng.random() < 0.5
    if kind == "train":
        case["losses"] = rng.choice(["simple", "simple", "full"])
    return case


# ---- networks ---------------------------------------------------------------------------------------
def _config(case):
    """The synthetic configuration whose density and drive the case's size goes with."""
    n = case["neurons"]
    base = synth.CONFIGS["C2" if n < 20000 else "C4" if n <= 100000 else "C5"]
    cfg = dataclasses.replace(base, n_neurons=n, max_delay=case["delay"])
    if case["basis"] == "dense":
        # rows of the dense basis sum to about 1.5 over four channels with short time constants instead of
        # one unit entry over five: inputs rescaled so that the rate stays at about 4 Hz
        cfg = dataclasses.replace(cfg, n_receptors=4, bkg_weight_pa=base.bkg_weight_pa * 1.49, lgn_weight_pa=base.lgn_weight_pa * 1.52)
    return cfg


def _dense_basis(dicts):
    """121 synapse types over four channels, dense and partly negative, with the location and spread of a
    basis fitted to measured synapses."""
    rng = np.random.Generator(np.random.PCG64(12))
    rows = rng.normal((0.27, 0.92, 0.18, 0.17), (0.25, 0.3, 0.25, 0.2), (121, 4))
    rows *= (rng.uniform(1.2, 2.0, 121) / np.maximum(rows.sum(1), 0.6))[:, None]
    net, lgn, bkg = dicts
    net["tau_syn"] = np.array([0.99, 1.88, 3.63, 5.65])
    net["synaptic_basis_weights"] = rows.astype(np.float32)
    for d in (net["synapses"], lgn, bkg):
        d["syn_ids"] = rng.integers(0, 121, d["syn_ids"].shape[0]).astype(np.uint8)


class _Network:
    """A cell with its loss tables: what a program builds once."""

    def __init__(self, case):
        self.cfg = cfg = _config(case)
        self.dicts = dicts = synth.make_network(cfg, 0)
        if case["basis"] == "dense":
            _dense_basis(dicts)
        self.cell = cell = V1Column(*dicts, **CELL)
        self.w0 = [w.clone() for w in (cell.recurrent_weight_values, cell.input_weight_values, cell.bkg_input_weights)]
        dev = cell.device
        self.simple = dict(LOSS, rate_target=torch.from_numpy(synth.make_rate_targets(cfg)).to(dev) / 1000.0,
                           v_lo=torch.from_numpy((-20.0 / cell.voltage_scale).astype(np.float32)).to(dev))
        self._regs = None

    def reset_weights(self):
        c = self.cell
        for w, w0 in zip((c.recurrent_weight_values, c.input_weight_values, c.bkg_input_weights), self.w0):
            w.copy_(w0)
        c.refresh_weights()

    def full_losses(self, case, seed):
        """The reference's own targets; the trials' angles and the synchrony samples are the seed's."""
        cfg, net = self.cfg, self.dicts[0]
        rng = np.random.default_rng(seed)
        ids = np.asarray(net["node_type_ids"], dtype=np.int32)
        if cfg.n_classes == 0:          # the small net has a type per neuron: 17 populations as in the column
            ids = (np.arange(cfg.n_neurons) % 17).astype(np.int32)
        types = int(ids.max()) + 1
        samples, bins, targets = synth.make_sync_samples(cfg, net, case["batch"], n_samples=50, seed=seed % 1000003)
        longest = max(case["steps"] // 4, 1)
        keep = bins <= longest
        fixed = np.random.default_rng(5)
        return dict(rate_groups=synth.make_rate_groups(cfg, dict(net, node_type_ids=ids)), rate_cost=100.0,
                    voltage_cost=1e-3, v_lo=self.simple["v_lo"], sync_cost=1.0, sync_samples=samples,
                    sync_bin_sizes=bins[keep], sync_bin_targets=targets[keep], osi_cost=5.0,
                    osi_angle=rng.uniform(0, 360, case["batch"]).astype(np.float32),
                    osi_tuning_angle=fixed.uniform(0, 360, cfg.n_neurons).astype(np.float32), osi_type_ids=ids,
                    osi_targets=fixed.uniform(0.2, 0.6, types).astype(np.float32),
                    dsi_targets=fixed.uniform(0.05, 0.3, types).astype(np.float32),
                    osi_type_counts=np.bincount(ids, minlength=types).astype(np.float32))

    def regularizers(self):
        """Both weight regularisers over the recurrent edge types (target class, source class, sign of the
        weight); the initial weights differ from the current ones as after some training."""
        if self._regs is None:
            idx = self.dicts[0]["synapses"]["indices"]
            cls = np.asarray(self.dicts[0]["node_type_ids"]) % 17
            edge = (cls[idx[:, 0]] * 17 + cls[idx[:, 1]]) * 2 + (self.dicts[0]["synapses"]["weights"] > 0)
            noise = np.random.default_rng(8).normal(0.0, 0.3, edge.size).astype(np.float32)
            w0 = self.w0[0].cpu().numpy() * np.exp(noise)
            self._regs = [WeightRegularizer(self.cell, "mean_stiff", edge, w0, 5.0, relative=True, order="internal"),
                          WeightRegularizer(self.cell, "emd", edge, w0, 2.0, order="internal")]
        return self._regs


_networks = collections.OrderedDict()


def _network(case):
    key = (case["neurons"], case["delay"], case["basis"])
    if key not in _networks:
        while len(_networks) >= 2:      # a program has one; keep the last two of a process that times many
            _networks.popitem(last=False)
        _networks[key] = _Network(case)
    _networks.move_to_end(key)
    return _networks[key]


_front_ends = {}


def _front_end(units):
    if units not in _front_ends:
        _front_ends.clear()
        tables = synth.make_lgn_tables(units, LGN_HEIGHT, LGN_WIDTH, LGN_SIDES, LGN_TAPS, LGN_TAPS, seed=4)
        _front_ends[units] = LGN(**tables, row_size=LGN_HEIGHT, col_size=LGN_WIDTH)
    return _front_ends[units]


# ---- inputs -----------------------------------------------------------------------------------------
def _rates(cfg, steps, gen):
    """Firing rates of the LGN units under a drifting grating: 5 + 10 relu(sin(2 pi 2 Hz t + phi)) Hz."""
    phi = torch.rand(cfg.n_lgn, generator=gen, device="cuda") * (2 * math.pi)
    t = torch.arange(steps, device="cuda", dtype=torch.float32)[:, None] * 1e-3
    return 5.0 + 10.0 * torch.relu(torch.sin(4 * math.pi * t + phi[None, :]))


def _spikes(rates, batch, gen):
    p = 1.0 - torch.exp(-rates / 1000.0)
    return torch.stack([(torch.rand(p.shape, generator=gen, device="cuda") < p).to(torch.uint8) for _ in range(batch)])


def _counts(cfg, batch, steps, gen):
    lam = torch.full((batch, steps, cfg.n_bkg), cfg.bkg_rate_hz * 1e-3, device="cuda")
    return torch.poisson(lam, generator=gen).to(torch.int32)


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    if case["kind"] == "lgn":
        movie = torch.rand((case["frames"], LGN_HEIGHT, LGN_WIDTH), generator=gen, device="cuda") * 2 - 1
        return dict(case=case, lgn=_front_end(case["units"]), movie=movie)
    net = _network(case)
    net.reset_weights()
    cfg, cell, b = net.cfg, net.cell, case["batch"]
    s = dict(case=case, cell=cell)
    if case["kind"] == "host":
        s["x"] = _spikes(_rates(cfg, case["steps"], gen), b, gen).cpu().pin_memory()
        s["counts"] = _counts(cfg, b, case["steps"], gen).cpu().pin_memory()
        return s
    # the carried state that a run starts from
    state = cell.zero_state(b)
    cell.rollout(_spikes(_rates(cfg, WARM_STEPS, gen), b, gen), _counts(cfg, b, WARM_STEPS, gen), state=state,
                 return_z=False, return_v=False)
    cell.synchronize()
    s["warm"] = state
    if case["kind"] == "call":
        s["x"] = _spikes(_rates(cfg, 1, gen), b, gen)[:, 0].to(torch.float32)
        return s
    if case["kind"] == "currents":
        s["dy"] = torch.randn((b * cfg.n_neurons, cfg.n_receptors), generator=gen, device="cuda")
        return s
    s["state"] = tuple(t.clone() for t in state)
    t_len = case["steps"]
    rates = _rates(cfg, t_len, gen)
    full = case.get("losses") == "full"
    if full:
        s["rates"], s["lgn_seed"] = rates, int(seed) + 1
    else:
        s["x"] = _spikes(rates, b, gen)
    # the ten-trial evaluation and the full training step draw their background noise on the device
    if not full and b <= 8:
        s["counts"] = _counts(cfg, b, t_len, gen)
    s["noise_seed"] = int(seed) % 100003
    if case["kind"] == "train":
        loss = net.full_losses(case, int(seed)) if full else net.simple
        s["trainer"] = Trainer(cell, loss, learning_rate=LEARNING_RATE, train_input=True,
                               regularizers=net.regularizers() if full else ())
    if case["kind"] == "grads":
        shape = (b, t_len, cfg.n_neurons)
        s["g_z"] = torch.randn(shape, generator=gen, device="cuda") * 1e-6
        s["g_v"] = torch.randn(shape, generator=gen, device="cuda") * 1e-6
    return s


def run(s):
    kind = s["case"]["kind"]
    if kind == "lgn":
        return s["lgn"].firing_rates(s["movie"])
    cell = s["cell"]
    if kind == "call":
        (z, v), state = cell.call(s["x"], s["warm"])
        return z, v, state
    if kind == "currents":
        z_buf = s["warm"][0]
        i_rec = cell.calculate_i_rec_with_custom_grad(z_buf)
        d_x, d_w = cell.syn_currents_grad(_lib.SRC_REC, z_buf, s["dy"])
        return i_rec, d_x, d_w
    if kind == "host":
        return cell.rollout_host_pipelined(s["x"], s["counts"], z_format="bits")
    for to, frm in zip(s["state"], s["warm"]):      # every trial and every step starts from the carried state
        to.copy_(frm)
    if kind == "eval":
        if "counts" not in s:
            cell.set_noise_seed(s["noise_seed"])
        z, v = cell.rollout(s["x"], s.get("counts"), state=s["state"], return_v=s["case"]["voltage"])
        return (z, v, s["state"]) if v is not None else (z, s["state"])
    if kind == "grads":
        z, v = cell.rollout(s["x"], s["counts"], state=s["state"], save_for_bwd=True)
        dw_rec, dw_lgn, dw_bkg, _ = cell.backward(g_z=s["g_z"], g_v=s["g_v"])
        return z, v, dw_rec, dw_lgn, dw_bkg, s["state"]
    trainer = s["trainer"]
    if s["case"]["losses"] == "full":
        cell.set_noise_seed(s["noise_seed"])
        losses = trainer.step_rates(s["rates"], s["lgn_seed"], s["case"]["batch"], state=s["state"])
    else:
        losses = trainer.step(s["x"], s["counts"], state=s["state"])
    return losses, trainer.grads.flat, trainer.m, trainer.v, s["state"]


# ---- what a pass cannot do without ------------------------------------------------------------------
def work(case):
    """Inputs read once and outputs written once: a synapse is 9 bytes (4 index, 4 weight, 1 type and delay);
    the operations of the dense update and of the synaptic events at the rates the networks run at."""
    if case["kind"] == "lgn":
        u, t = case["units"], case["frames"]
        taps = 2.0 * sum((k + 1) ** 2 for k in LGN_SIDES) / len(LGN_SIDES)
        return {"bytes": 4.0 * (t * LGN_HEIGHT * LGN_WIDTH + t * u + u * (taps + 2 * LGN_TAPS)),
                "flops": 2.0 * t * u * (taps + 2 * LGN_TAPS)}
    cfg = _config(case)
    n, b, r, d = cfg.n_neurons, case["batch"], cfg.n_receptors, cfg.max_delay
    rec, lgn, bkg = n * cfg.rec_in_degree, n * cfg.lgn_in_degree, n * cfg.bkg_in_degree
    rate = 10.0 if n > 100000 else 4.0
    per_event = 2.0 * (r if case["basis"] == "dense" else 1)
    synapses = 9.0 * (rec + lgn + bkg)
    state = float(b * n * (4 * d + 4 + 1 + 8 + 8 * r))
    fwd = b * (n * (8.0 * r + 20) + per_event * (rec * rate + lgn * 8.2 + bkg * cfg.bkg_rate_hz) / 1000.0)  # per step
    if case["kind"] == "call":
        return {"bytes": 4.0 * b * cfg.n_lgn + 2 * state + 4.0 * b * n, "flops": fwd}
    if case["kind"] == "currents":
        return {"bytes": 9.0 * rec + 4.0 * rec + b * n * (4.0 * d * 2 + 8.0 * r), "flops": b * rec * 2.0 * per_event}
    t = case["steps"]
    inputs = float(t * 4 * cfg.n_lgn) if case.get("losses") == "full" else float(b * t * (cfg.n_lgn + 4 * cfg.n_bkg))
    if case["kind"] == "host":
        return {"bytes": inputs + synapses + b * t * n / 8.0, "flops": t * fwd}
    if case["kind"] == "eval":
        return {"bytes": inputs + synapses + 2 * state + b * t * n * (5.0 if case["voltage"] else 1.0), "flops": t * fwd}
    # backward: the dense adjoint, and every recurrent synapse of the rows with a gradient (0.85 of them) once
    # per step and trial
    bwd = b * (n * (10.0 * r + 30) + 0.85 * per_event * rec)
    if case["kind"] == "grads":
        return {"bytes": inputs + synapses + 2 * state + 4.0 * (rec + lgn + bkg) + b * t * n * 13.0, "flops": t * (fwd + bwd)}
    return {"bytes": inputs + synapses + 2 * state + 28.0 * (rec + lgn) + 4.0 * bkg, "flops": t * (fwd + bwd)}


def tolerance(case):
    """32-bit sums in another order for rates, currents and forward state; the parity bar of the repository's
    tests (1e-4 in relative L2) for gradients, whose adjoints are stored with 15 mantissa bits at batch 5.
    Spikes are exact but for threshold ties."""
    if case["kind"] in ("train", "grads"):
        return {"rel": 1e-4, "max": 1e-2, "differ": 1e-5}
    return {"rel": 1e-5, "max": 1e-3, "differ": 1e-5}

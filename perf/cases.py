"""The work this framework is used for, as measurable cases.

Every case is one call (or one small group of calls) a user's program makes through the public
entry points of ``engine.py``: a simulated window of one resident network in each synaptic mode,
a window of a data-assimilation ensemble advanced as one batch, the BOLD window and the ensemble
filter that follow it, and the spike-compaction operator.

* ``listed()``     the cases that are always measured;
* ``draw(rng)``    one more case of the same ranges;
* ``prepare``      what the program holds before the call (resident network, state, buffers);
* ``run``          one pass of the call, returning its outputs;
* ``work``         bytes and operations of one pass that the path cannot do without;
* ``tolerance``    how far two correct implementations may be apart;
* ``exact``        the same outputs in 64 bits, by plain numpy / torch.

Networks: the plain block (one population, fixed in-degree, uniform sources) and the regional
construction (lognormal population sizes, 70 % own-population synapses, distance-dependent rest).
In the ``saturated`` regime (the construction's own conductances) populations fire in synchronised
bursts, once per refractory period of 5 ms; in the ``quiet`` one (conductances x 0.01, OU mean 0.65)
they fire at about 8 Hz and asynchronously.  A prepared network has run past its quiet start, so the
push variant has been chosen on line as it is for any longer-running program, and then stands at a
state made by the deterministic fixed-point push, the same for every build.
"""
import importlib.util
import math
import os
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _package():
    """The package under its import name (its folder name is not an identifier)."""
    if "dtb_b200" not in sys.modules:
        folder = os.path.join(_ROOT, "digital_twin_brain-open_b200")
        spec = importlib.util.spec_from_file_location("dtb_b200", os.path.join(folder, "__init__.py"),
                                                      submodule_search_locations=[folder])
        mod = importlib.util.module_from_spec(spec)
        sys.modules["dtb_b200"] = mod
        spec.loader.exec_module(mod)
    from dtb_b200 import engine, network
    return engine, network


# simulated steps before a case's own window: past the quiet start and the push autotuner
SETTLE = 800
# the push modes by name; "pull" is the in-degree gather
SYN = {"push": 0, "exact": 1, "pull": 2, "fixed": 3}
WEIGHTS = {"f32": 0, "bf16": 1, "f16": 2, "u8": 3}
WEIGHT_BYTES = {"f32": 8, "bf16": 4, "f16": 4, "u8": 2}
# spikes per neuron and step (measured over long windows of both regimes)
RATE = {"saturated": 0.0195, "quiet": 0.0008}
SAMPLES = 200
# networks up to this size hand their whole state back after a window (28 B per neuron), larger ones V
STATE_MOST = 300000


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # the smallest network anyone steps interactively, reproducible mode, a short window:
        # the cost of a call and of its launches
        dict(name="block2k_exact", kind="run", net="block", n=2000, pops=1, degree=100, weights="f32", syn="exact",
             regime="saturated", steps=20, t_steps=1, observe=False),
        # the plain 10,000-neuron block the reference's CPU model runs, default mode
        dict(name="block10k_push", kind="run", net="block", n=10000, pops=1, degree=100, weights="f32", syn="push",
             regime="saturated", steps=100, t_steps=1, observe=False),
        # a mid-sized regional network in the default mode
        dict(name="regional200k_push", kind="run", net="regional", n=200000, pops=20, degree=1000, weights="f32",
             syn="push", regime="saturated", steps=200, t_steps=1, observe=False),
        # the largest: millions of neurons, billions of synapses, default mode
        dict(name="regional3m_push", kind="run", net="regional", n=3000000, pops=120, degree=1000, weights="f32",
             syn="push", regime="saturated", steps=100, t_steps=1, observe=False),
        # physiological rates: the membrane update carries the step, few spikes to deliver
        dict(name="quiet1m_push_bf16", kind="run", net="regional", n=1000003, pops=50, degree=200, weights="bf16",
             syn="push", regime="quiet", steps=300, t_steps=1, observe=False),
        # the served form's mode and weights on one network
        dict(name="regional250k_fixed_bf16", kind="run", net="regional", n=250000, pops=25, degree=400, weights="bf16",
             syn="fixed", regime="saturated", steps=200, t_steps=1, observe=False),
        # the deterministic in-degree gather
        dict(name="regional200k_pull_bf16", kind="run", net="regional", n=200000, pops=20, degree=500, weights="bf16",
             syn="pull", regime="saturated", steps=50, t_steps=1, observe=False),
        # a run with everything observed: substeps, sampled neurons, mean synaptic currents
        dict(name="observed100k_substeps", kind="run", net="regional", n=100000, pops=30, degree=300, weights="f32",
             syn="fixed", regime="saturated", steps=50, t_steps=4, observe=True),
        # a data-assimilation ensemble: uneven members advanced as one batch
        dict(name="ensemble12_fixed_bf16", kind="batch", members=12, n_lo=20000, n_hi=400000, weights="bf16",
             syn="fixed", regime="saturated", steps=100),
        # one assimilation window of the hemodynamic model: 100 members x 230 voxels, 800 steps
        dict(name="bold_23k_800", kind="bold", n=23000, steps=800, out=True),
        # the ensemble Kalman update that follows it
        dict(name="da_100x1000x10", kind="da", members=100, voxels=1000, states=10),
        # spike compaction of a 5M-neuron step
        dict(name="compact5m", kind="compact", n=5000000, density=0.02),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["run", "run", "run", "run", "batch", "bold", "da", "compact"])
    if kind == "bold":
        return dict(kind=kind, n=_log_int(rng, 500, 60000), steps=_log_int(rng, 100, 1000), out=rng.random() < 0.7)
    if kind == "da":
        return dict(kind=kind, members=_log_int(rng, 16, 150), voxels=_log_int(rng, 50, 3000), states=rng.randint(6, 16))
    if kind == "compact":
        return dict(kind=kind, n=_log_int(rng, 2000, 60000000), density=round(math.exp(rng.uniform(math.log(5e-4), math.log(0.45))), 5))
    if kind == "batch":
        return dict(kind=kind, members=rng.randint(2, 14), n_lo=_log_int(rng, 3000, 30000), n_hi=_log_int(rng, 50000, 400000),
                    weights=rng.choice(["bf16", "f32"]), syn="fixed", regime=rng.choice(["saturated", "quiet"]),
                    steps=rng.randint(40, 120))
    net = rng.choice(["block", "regional", "regional"])
    syn = rng.choice(["push", "push", "fixed", "exact", "pull"])
    case = dict(kind="run", net=net, weights=rng.choice(["f32", "f32", "bf16", "f16", "u8"]), syn=syn,
                regime=rng.choice(["saturated", "saturated", "quiet"]), t_steps=1, observe=False)
    if net == "block":
        case.update(n=_log_int(rng, 1000, 40000), pops=1, degree=rng.randint(30, 200), steps=rng.randint(10, 120))
    else:
        degree = _log_int(rng, 50, 1000)
        most = min(2000000, (200_000_000 if syn in ("pull", "exact") else 1_600_000_000) // degree)
        n = _log_int(rng, 20000, most)
        case.update(n=n, pops=rng.randint(4, 80), degree=degree, steps=rng.randint(30, 100) if n > 500000 else rng.randint(50, 250))
    if syn in ("push", "fixed") and rng.random() < 0.25:
        case.update(t_steps=rng.choice([1, 2, 4]), observe=True, steps=min(case["steps"], 40))
    return case


# ---------------------------------------------------------------------------
# networks
# ---------------------------------------------------------------------------
_BASE_G = (0.01, 0.002, 0.04, 0.002)


def _ou(case):
    return (0.65, 0.2, 10.0) if case["regime"] == "quiet" else (0.6, 0.2, 10.0)


def _g_scale(case, pops):
    return np.full((pops, 4), 0.01 if case["regime"] == "quiet" else 1.0, np.float32)


def _block_arrays(case, seed):
    """The plain block in the on-disk key set: `degree` uniform sources per neuron, no self-loops."""
    _, nw = _package()
    n, k = case["n"], case["degree"]
    rng = np.random.default_rng([seed, 11])
    post = np.repeat(np.arange(n, dtype=np.uint32), k)
    pre = rng.integers(0, n - 1, n * k).astype(np.uint32)
    pre[pre >= post] += 1
    g = np.tile(np.asarray(_BASE_G, np.float32), (n, 1)) * _g_scale(case, 1)
    w = rng.random((n * k, 2), dtype=np.float32)
    return dict(property=nw.lif_property(n, 0, g_ui=g.astype(np.float32)), input_block_idx=np.zeros(n * k, np.int16),
                input_neuron_idx=pre, output_neuron_idx=post,
                input_channel_offset=np.where(pre >= int(round(0.8 * n)), 2, 0).astype(np.uint8), weight=w)


def _engine(case, seed, push=None):
    E, nw = _package()
    pull = case["syn"] == "pull"
    opts = dict(weight_type=WEIGHTS[case["weights"]], seed=seed + 1, ou=_ou(case), push=(not pull) if push is None else push,
                pull=pull)
    if case["net"] == "block":
        return E.Engine.from_arrays(_block_arrays(case, seed), **opts)
    spec = nw.structured_spec(case["n"], case["pops"], case["degree"], seed % 100003 + 1, g_scale=_g_scale(case, case["pops"]))
    return E.Engine.structured(spec, **opts)


def _sampled(n):
    return np.unique(np.linspace(0, n - 1, min(SAMPLES, n)).astype(np.uint32))


def _run_args(case):
    a = dict(freq=True, vmean=True, syn_mode=SYN[case["syn"]], t_steps=case["t_steps"])
    if case["observe"]:
        a.update(sample_spike=True, sample_v=True, sample_iou=True, imean=True, receptor_imean=True, sample_isyn=True)
    return a


def _settled(case, seed):
    """An engine past its quiet start, tuned in its own mode, at a state every build reaches alike."""
    eng = _engine(case, seed)
    if case["observe"]:
        eng.set_samples(_sampled(eng.n))
    pull = case["syn"] == "pull"
    if not pull:
        eng.set_push_variant(0, 8)
    eng.run(SETTLE, syn_mode=SYN["pull" if pull else "fixed"])
    if not pull:
        blob = eng.save_state()
        eng.set_push_variant(-1)
        for _ in range(-(-SETTLE // case["steps"])):
            eng.run(case["steps"], **_run_args(case))
        eng.load_state(blob)
    return eng


def _member_specs(case, seed):
    _, nw = _package()
    rng = np.random.default_rng([seed, 23])
    sizes = np.random.default_rng([case["members"], case["n_lo"], case["n_hi"]])
    specs = []
    for m in range(case["members"]):
        n = int(sizes.integers(case["n_lo"], case["n_hi"] + 1))
        k = int(sizes.choice((100, 200, 500)))
        p = int(sizes.integers(10, 51))
        scale = rng.uniform(0.5, 1.5, (p, 4)) * (0.01 if case["regime"] == "quiet" else 1.0)
        specs.append(nw.structured_spec(n, p, k, (seed % 100003) * 1000 + m + 1, g_scale=scale))
    return specs


# ---------------------------------------------------------------------------
# prepare and run
# ---------------------------------------------------------------------------
def _gen(seed, device="cuda"):
    g = torch.Generator(device=device)
    g.manual_seed(int(seed) * 7919 + 5)
    return g


def _bold_state(n):
    s = torch.zeros(4, n, device="cuda")
    s[2:] = 1.0
    return s


def prepare(case, seed):
    E, _ = _package()
    kind = case["kind"]
    if kind == "run":
        return dict(kind=kind, eng=_settled(case, seed), steps=case["steps"], args=_run_args(case), observe=case["observe"],
                    rates=case["syn"] == "push")
    if kind == "batch":
        opts = dict(weight_type=WEIGHTS[case["weights"]], ou=_ou(case))
        engines = [E.Engine.structured(s, seed=seed + 10 + m, **opts) for m, s in enumerate(_member_specs(case, seed))]
        batch = E.Batch(engines)
        for _ in range(-(-SETTLE // case["steps"])):
            batch.run(case["steps"], syn_mode=SYN[case["syn"]])
        return dict(kind=kind, batch=batch, steps=case["steps"], syn=SYN[case["syn"]])
    g = _gen(seed)
    if kind == "bold":
        # voxel activity: a slow random walk around 0.1 spikes per neuron and step, floored as the DA driver does
        n, steps = case["n"], case["steps"]
        walk = torch.cumsum(torch.randn(steps, n, device="cuda", generator=g), 0) / 20.0
        return dict(kind=kind, u=torch.clamp(0.1 + 0.05 * walk, min=1e-5).contiguous(), state=_bold_state(n), out=case["out"])
    if kind == "da":
        e, v, s = case["members"], case["voxels"], case["states"]
        return dict(kind=kind, w=1.0 + 0.1 * torch.randn(e, v, s, device="cuda", generator=g),
                    y=1.0 + 0.05 * torch.randn(v, device="cuda", generator=g),
                    noise=torch.randn(e, v, device="cuda", generator=g))
    # compact: a step's spikes come population by population, so the density varies over blocks of neurons
    n, words = case["n"], (case["n"] + 31) // 32
    blocks = max(1, n // 20000)
    p = torch.rand(blocks, device="cuda", generator=g)
    p = (p * (2.0 * case["density"])).clamp(max=0.95).repeat_interleave(-(-words * 32 // blocks))[:words * 32]
    b = torch.rand(words * 32, device="cuda", generator=g) < p
    b[n:] = False
    shift = torch.arange(32, device="cuda", dtype=torch.int64)
    w = (b.view(words, 32).to(torch.int64) << shift).sum(1)
    return dict(kind=kind, n=n, bits=torch.where(w >= 2 ** 31, w - 2 ** 32, w).to(torch.int32),
                idx=torch.zeros(n, dtype=torch.int32, device="cuda"), count=torch.zeros(1, dtype=torch.int32, device="cuda"))


def _rates(freqs, sizes):
    """Population firing rates in Hz of each 0.1-ms step (freq_char of the reference's client)."""
    return freqs * (10000.0 / sizes)[None, :]


def run(state):
    E, _ = _package()
    kind = state["kind"]
    if kind == "run":
        eng = state["eng"]
        r = eng.run(state["steps"], **state["args"])
        out = dict(freqs=_rates(r.freqs, eng.pop_sizes) if state["rates"] else r.freqs, vmeans=r.vmeans,
                   V=eng.read_state(E.STATE_V))
        if state["observe"]:
            out.update(sample_v=r.sample_v, sample_iou=r.sample_iou, sample_isyn=r.sample_isyn, imeans=r.imeans,
                       receptor_imeans=r.receptor_imeans,
                       sample_spike=r.sample_spike.astype(np.float32) if state["rates"] else r.sample_spike)
        elif eng.n <= STATE_MOST:
            out.update(J=eng.read_state(E.STATE_J), i_ou=eng.read_state(E.STATE_I_OU), t_last=eng.read_state(E.STATE_T_LAST))
        return out
    if kind == "batch":
        rs = state["batch"].run(state["steps"], vmean=True, syn_mode=state["syn"])
        return [dict(freqs=r.freqs, vmeans=r.vmeans, V=e.read_state(E.STATE_V)) for r, e in zip(rs, state["batch"].engines)]
    if kind == "bold":
        o = E.bold_run(state["u"], state["state"], out=state["out"])
        return dict(out=o, state=state["state"]) if state["out"] else dict(state=state["state"])
    if kind == "da":
        return E.da_filter(state["w"], state["y"], state["noise"], 1e-6)
    E.compact_spikes(state["bits"].data_ptr(), state["n"], state["idx"].data_ptr(), state["count"].data_ptr())
    return dict(idx=state["idx"], count=state["count"])


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def _net_work(n, degree, wb, syn, rate, steps, t_steps, weights_all=False):
    """Bytes and operations of `steps` steps: 28 B of state read and written per neuron and substep
    (V, four receptors, OU current, last spike time), and per delivered event its target, its weight
    pair and the pair added to; the gather reads every in-edge's source instead."""
    events = n * degree * rate
    state = 56.0 * n * t_steps
    if syn == "pull":
        per = state + 4.0 * n * degree + wb * events + n / 8.0
    else:
        per = state + events * (4 + wb + 8) + 12.0 * n * rate + n / 8.0
    return steps * per, steps * (60.0 * n * t_steps + 2.0 * events)


def work(case):
    kind = case["kind"]
    if kind == "run":
        b, f = _net_work(case["n"], case["degree"], WEIGHT_BYTES[case["weights"]], case["syn"], RATE[case["regime"]],
                         case["steps"], case["t_steps"])
        return dict(bytes=b + (28.0 if case["n"] <= STATE_MOST else 4.0) * case["n"], flops=f)
    if kind == "batch":
        n = (case["n_lo"] + case["n_hi"]) / 2.0 * case["members"]
        b, f = _net_work(n, 800.0 / 3.0, WEIGHT_BYTES[case["weights"]], case["syn"], RATE[case["regime"]], case["steps"], 1)
        return dict(bytes=b + 4.0 * n, flops=f)
    if kind == "bold":
        return dict(bytes=4.0 * case["n"] * (case["steps"] * (2 if case["out"] else 1) + 8), flops=60.0 * case["n"] * case["steps"])
    if kind == "da":
        e, v, s = case["members"], case["voxels"], case["states"]
        return dict(bytes=4.0 * (2 * e * v * s + v + e * v), flops=2.0 * e * e * v * (s + 1) + 6.0 * e * v * s)
    return dict(bytes=case["n"] / 8.0 + 4.0 * case["n"] * case["density"], flops=case["n"] / 32.0)


def tolerance(case):
    kind = case["kind"]
    if kind == "run" and case["syn"] == "push":
        # float reductions land in any order: everything agrees to about 1e-7 until a neuron within
        # rounding of its threshold spikes a step later, which moves its V by a quarter of V's rms;
        # four such neurons in the network are allowed
        return dict(rel=0.25 * math.sqrt(4.0 / case["n"]), max=0.5)
    if kind in ("run", "batch", "compact"):
        return "exact"        # integer sums: the same bits in any order
    if kind == "bold":
        return dict(rel=4e-6, max=4e-5)    # powf differs by an ulp between libraries
    return dict(rel=1e-6, max=4e-6)        # sums in double, one rounding to float32


# ---------------------------------------------------------------------------
# the same in 64 bits
# ---------------------------------------------------------------------------
def _philox(c0, c1, c2, c3, k0, k1):
    """Philox4x32-10 (Salmon et al., SC'11) on numpy uint64 arrays holding 32-bit words."""
    m = np.uint64(0xFFFFFFFF)
    sh = np.uint64(32)
    for _ in range(10):
        p0, p1 = np.uint64(0xD2511F53) * c0, np.uint64(0xCD9E8D57) * c2
        c0, c1, c2, c3 = (p1 >> sh) ^ c1 ^ k0, p1 & m, (p0 >> sh) ^ c3 ^ k1, p0 & m
        k0, k1 = (k0 + np.uint64(0x9E3779B9)) & m, (k1 + np.uint64(0xBB67AE85)) & m
    return c0, c1, c2, c3


def _normals(n, step, sub, seed):
    """The OU draws of one step (or substep): slot s of a 1024-neuron tile draws for neurons s + 256 k."""
    tiles = -(-n // 1024)
    ctr = np.arange(tiles * 256, dtype=np.uint64)
    full = lambda v: np.full_like(ctr, v)  # noqa: E731
    r = _philox(ctr, full(step & 0xFFFFFFFF), full(step >> 32), full(0x0D0E0001 ^ (sub << 20)),
                full(seed & 0xFFFFFFFF), full(seed >> 32))
    z = []
    for a, b in ((r[0], r[1]), (r[2], r[3])):
        rad = np.sqrt(-2.0 * np.log(((a >> np.uint64(8)).astype(np.float64) + 1.0) / 2 ** 24))
        ang = 2.0 * np.pi * (b >> np.uint64(8)).astype(np.float64) / 2 ** 24
        z += [rad * np.cos(ang), rad * np.sin(ang)]
    return np.stack([x.reshape(tiles, 256) for x in z], 1).reshape(-1)[:n]


def _exact_run(case, seed):
    """The window in float64 from the prepared state: V, J, OU and spikes by the model's equations, on
    the network's own arrays.  The clock stays the float32 sum of dt that the model defines, since the
    refractory test compares it."""
    if case["syn"] == "push" or case["n"] * case["degree"] > 1.1e8 or case["n"] * case["steps"] * case["t_steps"] > 2.5e7:
        return None
    E, _ = _package()
    eng = _settled(case, seed)
    n, steps, ts = eng.n, case["steps"], case["t_steps"]
    dev = dict(device="cuda", dtype=torch.float64)
    V, J = (torch.tensor(eng.read_state(w).astype(np.float64), **dev) for w in (E.STATE_V, E.STATE_J))
    iou, tl = (torch.tensor(eng.read_state(w).astype(np.float64), **dev) for w in (E.STATE_I_OU, E.STATE_T_LAST))
    info = eng.info()
    t, step0 = np.float32(info.t), int(info.step)
    if case["syn"] == "pull":
        eng.close()
        eng = _engine(case, seed, push=True)
    rows, ptr, post, kind, w = eng.read_out_csr()
    sizes = np.asarray(eng.pop_sizes, np.int64)
    eng.close()
    src = torch.repeat_interleave(torch.tensor(rows.astype(np.int64), device="cuda"),
                                  torch.tensor(np.diff(ptr.astype(np.int64)), device="cuda"))
    slot = (torch.tensor(post.astype(np.int64), device="cuda") << 1) | torch.tensor(kind.astype(np.int64), device="cuda")
    w = torch.tensor(w, device="cuda")
    pop = torch.repeat_interleave(torch.arange(len(sizes), device="cuda"), torch.tensor(sizes, device="cuda"))
    f32 = lambda x: float(np.float32(x))  # noqa: E731
    scale = 0.01 if case["regime"] == "quiet" else 1.0
    g = torch.tensor([f32(np.float32(x) * np.float32(scale)) for x in _BASE_G], **dev)
    vu = torch.tensor([0.0, 0.0, -70.0, -100.0], **dev)
    dt = f32(0.1) / ts
    decay = torch.exp(-dt / torch.tensor([2.0, 40.0, 10.0, 50.0], **dev))
    mean, sigma, tau = (f32(x) for x in _ou(case))
    f1, f2 = 1.0 - math.exp(-dt / tau), math.sqrt(1.0 - math.exp(-2.0 * dt / tau)) * sigma
    dts = np.float32(np.float32(0.1) / np.float32(ts))
    count = torch.tensor(sizes, **dev)
    sel = torch.tensor(_sampled(n).astype(np.int64), device="cuda")
    res = {k: [] for k in ("vmeans", "sample_v", "sample_iou", "sample_isyn", "imeans", "receptor_imeans")}
    per_pop = lambda x: torch.zeros(len(sizes), **dev).index_add_(0, pop, x) / count  # noqa: E731
    for s in range(steps):
        fired = torch.zeros(n, dtype=torch.bool, device="cuda")
        for k in range(ts):
            t = np.float32(t + dts)
            z = torch.tensor(_normals(n, step0 + s + 1, k, seed + 1), **dev)
            isyn = ((g * (vu - V[:, None])) * J).sum(1)
            iou = iou + f1 * (mean - iou) + f2 * z
            v = V + dt * (-f32(0.03) * (V + 75.0) + isyn + iou)
            v = torch.where(float(t) >= (tl.float() + 5.0).double(), v, torch.full_like(v, -65.0))
            active = v >= -50.0
            V = torch.clamp(v, max=-50.0)
            tl = torch.where(active, torch.full_like(tl, float(t)), tl)
            fired |= active
            J = J * decay
        hit = fired[src]
        J = J + torch.zeros(2 * n, 2, **dev).index_add_(0, slot[hit], w[hit].double()).reshape(n, 4)
        res["vmeans"].append(per_pop(V))
        if case["observe"]:
            cur = g * (vu - V[:, None]) * J
            tot = cur.sum(1)
            res["sample_v"].append(V[sel]), res["sample_iou"].append(iou[sel]), res["sample_isyn"].append(tot[sel])
            res["imeans"].append(per_pop(tot))
            res["receptor_imeans"].append(torch.stack([per_pop(cur[:, c]) for c in range(4)]))
    out = {k: torch.stack(v) for k, v in res.items() if v}
    out["V"] = V
    if not case["observe"] and n <= STATE_MOST:
        out.update(J=J, i_ou=iou, t_last=tl)
    return out


def exact(case, seed):
    """None for the float push (its sums are rounded in the order the reductions land in, another one
    in every run), for batches and for networks too large to restate quickly."""
    kind = case["kind"]
    if kind == "run":
        return _exact_run(case, seed)
    if kind == "batch":
        return None
    st = prepare(case, seed)
    if kind == "bold":
        eps, ts, tf, t0, alpha, e0, v0, dt = 200.0, 0.8, 0.4, 1.0, 0.2, 0.8, 0.02, 1e-3
        s, q, v, f = st["state"].double()
        outs = []
        for u in st["u"].double():
            ds = eps * u - s / ts - (f - 1.0) / tf
            part = torch.where(f > 0, 1.0 - (1.0 - e0) ** (1.0 / f), torch.ones_like(f))
            q = q + dt * ((f * part / e0 - q * v ** (1.0 / alpha - 1.0)) / t0)
            v = v + dt * ((f - v ** (1.0 / alpha)) / t0)
            f = torch.clamp(f + s * dt, min=0.0)
            s = s + ds * dt
            if case["out"]:
                outs.append(v0 * (7.0 * e0 * (1.0 - q) + 2.0 * (1.0 - q / v) + (2.0 * e0 - 0.2) * (1.0 - v)))
        state = torch.stack([s, q, v, f])
        return dict(out=torch.stack(outs), state=state) if case["out"] else dict(state=state)
    if kind == "da":
        w, y, noise = st["w"].double(), st["y"].double(), st["noise"].double()
        d = w - w.mean(0, keepdim=True)
        m = w.shape[0] - 1
        temp = d[:, :, -1] / ((d[:, :, -1] ** 2).sum(0) / m + 1e-6) / m
        innov = y[None] + math.sqrt(1e-6) * noise - w[:, :, -1]
        gain = innov @ temp.T / w.shape[1]
        return w + 0.5 * innov[:, :, None] * (temp[:, :, None] * d).sum(0)[None] + 0.5 * torch.einsum("ef,fvs->evs", gain, d)
    return None          # compaction: whole numbers

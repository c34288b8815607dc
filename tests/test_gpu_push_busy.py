"""The population-window push decides per step: a step of few events scatters whole rows, a busy
one sums own-population spans in windows and scatters the rest, population by population.  With
the fixed-point push every route gives the same integer sums, so a run in which the tuner's
window form crosses the threshold equals the register push bit for bit; so do single steps of few
rows, whose rows are cut into parts."""
import numpy as np
import pytest

from dtb_b200 import engine as E
from dtb_b200 import network as nw

pytestmark = pytest.mark.gpu


def _run(spec, variant, steps, wt, chunk=100):
    with E.Engine.structured(spec, weight_type=wt, seed=9) as eng:
        if variant is not None:
            eng.set_push_variant(*variant)
        freqs, events = [], 0
        for _ in range(steps // chunk):
            r = eng.run(chunk, syn_mode=E.SYN_PUSH_FIXED)
            freqs.append(r.freqs)
            events += r.events
        return np.concatenate(freqs), events, eng.read_state(E.STATE_V), eng.read_state(E.STATE_J), eng.info()


@pytest.mark.parametrize("n,pops,degree,wt", [(150_011, 9, 900, E.W_F32), (120_000, 12, 900, E.W_BF16)])
def test_tuned_window_form_gives_the_register_pushs_bits(gpu, n, pops, degree, wt):
    """The tuner's window form through quiet steps, busy ones, and the populations of a busy step that
    do not pay for their windows: two populations with almost no recurrent input fire a few neurons a
    step, in bursts of the others too, and are scattered whole while those take their windows."""
    g_scale = np.ones((pops, 4), np.float32)
    g_scale[:2] = 0.01
    spec = nw.structured_spec(n, pops, degree, seed=31, g_scale=g_scale)
    f0, e0, v0, j0, inf0 = _run(spec, (E.PUSH_REG, 8), 1500, wt)
    f1, e1, v1, j1, inf = _run(spec, None, 1500, wt)              # autotuned
    f2, e2, v2, j2, _ = _run(spec, (E.PUSH_LOCAL, 2016), 1500, wt)   # windows in every step
    assert inf.push_kind == E.PUSH_LOCAL
    busy = f0.sum(1) >= 16_000_000 * n / inf0.n_edges             # the steps in which that form takes windows
    late = np.arange(len(f0)) >= 1000                             # well after it was chosen
    assert 10 <= (busy & late).sum() < late.sum() // 2
    # rows from which a window pays: (4 events a neuron + 8192) over the own-population synapses of a row
    least = (4 * spec.pop_sizes + 8192) / (0.7 * degree)
    cold = (f0[busy & late][:, :2] > 0) & (f0[busy & late][:, :2] < 0.5 * least[:2])
    hot = f0[busy & late][:, 2:] > 2 * least[2:]
    assert cold.mean() > 0.25 and hot.mean() > 0.3
    for f, e, v, j in ((f1, e1, v1, j1), (f2, e2, v2, j2)):
        assert np.array_equal(f0, f) and e0 == e
        assert np.array_equal(v0, v) and np.array_equal(j0, j)


@pytest.mark.parametrize("sizes", [(2306, 8), (2306, 6, 2), (4864, 33, 1), (1025, 1281, 9)])
def test_windows_with_a_small_last_population(gpu, sizes):
    """Populations that end inside a warp's 32-neuron word at the end of the network: the rows a
    population hands to its windows are the rows it has.  The windows of every step, with the
    fixed-point push, must leave the register push's bits; every population has windows (own-population
    spans of 36 synapses and more a neuron) and every neuron fires, so a miscounted row shows."""
    rng = np.random.default_rng(sum(sizes))
    n, off = sum(sizes), np.concatenate([[0], np.cumsum(sizes)])
    pop = np.repeat(np.arange(len(sizes)), sizes)
    own, rest = 36, 8
    post = np.repeat(np.arange(n, dtype=np.uint32), own + rest)
    lo, width = off[pop][:, None], np.asarray(sizes)[pop][:, None]
    pre = np.concatenate([lo + rng.integers(0, 2 ** 31, (n, own)) % width, rng.integers(0, n, (n, rest))], 1)
    net = dict(property=nw.lif_property(n, pop), input_neuron_idx=pre.reshape(-1).astype(np.uint32), output_neuron_idx=post,
               input_channel_offset=np.zeros(post.size, np.uint8), weight=rng.random((post.size, 2), dtype=np.float32))
    res = []
    for variant in ((E.PUSH_REG, 8), (E.PUSH_LOCAL, 8), (E.PUSH_LOCAL, 2016)):
        with E.Engine.from_arrays(net, seed=5, ou=(3.0, 0.5, 10.0)) as eng:
            assert eng.info().local_windows == len(sizes)
            eng.set_push_variant(*variant)
            r = eng.run(400, syn_mode=E.SYN_PUSH_FIXED)
            res.append((r.freqs, r.events, eng.read_state(E.STATE_V), eng.read_state(E.STATE_J)))
    assert (res[0][0].sum(0) >= np.asarray(sizes)).all()
    for other in res[1:]:
        assert all(np.array_equal(x, y) for x, y in zip(res[0], other))


@pytest.mark.parametrize("out_degree", [1, 255, 256, 257, 2047, 2049, 5000])
def test_few_long_rows_are_cut_into_parts(gpu, out_degree):
    """A step whose only spikes are three neurons of a given out-degree (a strong drive on them
    alone): J must hold every one of their synapses once."""
    n = 6000
    rng = np.random.default_rng(out_degree)
    src = np.array([5, 3001, 5999])
    pre = np.repeat(src, out_degree).astype(np.uint32)
    post = rng.integers(0, n, pre.size).astype(np.uint32)
    w = (rng.integers(0, 256, (pre.size, 2)) / 256.0).astype(np.float32)
    kind = rng.integers(0, 2, pre.size).astype(np.uint8)
    prop = nw.lif_property(n, 0)
    prop[src, 2] = 1e5                       # I_ext: over threshold in the first step
    net = dict(property=prop, input_neuron_idx=pre, output_neuron_idx=post, input_channel_offset=kind, weight=w)
    ref = np.zeros((n, 4))
    for k in (0, 1):
        np.add.at(ref, (post, 2 * kind.astype(int) + k), w[:, k].astype(np.float64))
    for syn in (E.SYN_PUSH, E.SYN_PUSH_FIXED, E.SYN_PUSH_EXACT):
        with E.Engine.from_arrays(net) as eng:
            r = eng.run(1, use_ou=False, syn_mode=syn)
            assert r.freqs.sum() == 3 and r.events == pre.size
            assert np.array_equal(eng.read_state(E.STATE_J), ref.astype(np.float32))    # dyadic weights: exact in any order


@pytest.mark.parametrize("degree,param", [(10, 1008), (23, 1008), (24, 8), (60, 8)])
def test_untuned_networks_return_to_their_default_form(gpu, degree, param):
    """A network too small to be tuned, alone and in a batch: autotuning again takes back a form chosen
    before, rows of few synapses have the quarter-warp form, and every form gives the same bits."""
    spec = nw.structured_spec(3000, 3, degree, seed=degree)
    res = []
    with E.Engine.structured(spec, seed=2, ou=(3.0, 0.5, 10.0)) as eng:
        blob = eng.save_state()
        for variant in (None, (E.PUSH_TMA, 512), (-1, 0)):
            if variant is not None:
                eng.set_push_variant(*variant)
                eng.load_state(blob)
            r = eng.run(400, syn_mode=E.SYN_PUSH_EXACT)
            inf = eng.info()
            res.append((r.freqs, r.events, eng.read_state(E.STATE_J)))
            assert (inf.push_kind, inf.push_param) == ((E.PUSH_REG, param) if variant in (None, (-1, 0)) else variant)
        with E.Batch([eng]) as b:
            b.set_push_variant(E.PUSH_TMA, 512)
            b.run(5)
            b.set_push_variant(-1)
            b.run(5)
            assert (b.info()["push_kind"], b.info()["push_param"]) == (E.PUSH_REG, param)
    assert res[0][0].sum() > 0
    for other in res[1:]:
        assert np.array_equal(res[0][0], other[0]) and res[0][1] == other[1] and np.array_equal(res[0][2], other[2])

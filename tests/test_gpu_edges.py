"""Edges of the operator kernels' tiles: compaction around its CTA and single-launch limits and on
bitmaps that start off a 16-byte boundary, the BOLD window's step remainders and both of its power
forms, the ensemble filter's ragged members, voxels and states, and the pull step with its bitmap
in shared memory and in L2."""
import numpy as np
import pytest

from dtb_b200 import engine as E
from dtb_b200 import network as nw
from oracle.bold_oracle import DA_PARAMS, BoldOracle, bold_inputs, da_filter

pytestmark = pytest.mark.gpu

CTA = 32 * 1024            # neurons per CTA of the single-launch compaction
DIRECT = 8 << 20           # its largest bitmap


@pytest.mark.parametrize("n,offset", [(CTA - 1, 0), (CTA, 0), (CTA + 1, 0), (3 * CTA + 17, 1), (40 * CTA + 5, 3),
                                      (148 * CTA, 0), (148 * CTA + 1, 0), (148 * CTA + 33, 3), (6_500_000, 0), (6_500_001, 1),
                                      (DIRECT, 0), (DIRECT + 1, 0), (DIRECT - 31, 2)])
def test_compaction_edges(gpu, n, offset):
    import torch
    g = torch.Generator(device="cuda").manual_seed(n)
    words = (n + 31) // 32
    buf = torch.randint(-2 ** 31, 2 ** 31, (words + offset,), device="cuda", generator=g).to(torch.int32)
    buf &= torch.randint(-2 ** 31, 2 ** 31, (words + offset,), device="cuda", generator=g).to(torch.int32)
    bits = buf[offset:]
    idx = torch.full((n,), -1, dtype=torch.int32, device="cuda")
    cnt = torch.zeros(1, dtype=torch.int32, device="cuda")
    E.compact_spikes(bits.data_ptr(), n, idx.data_ptr(), cnt.data_ptr(), torch.cuda.current_stream().cuda_stream)
    flags = ((bits[:, None] >> torch.arange(32, device="cuda", dtype=torch.int32)) & 1).reshape(-1)[:n]
    ref = torch.nonzero(flags).reshape(-1)
    c = int(cnt.item())
    assert c == ref.numel()
    assert torch.equal(idx[:c].long(), ref)
    assert bool((idx[c:] == -1).all())


@pytest.mark.parametrize("alpha", [0.2, 0.32, 1.0, 0.5, 1 / 8, 1 / 16, 1 / 17])
@pytest.mark.parametrize("n,steps", [(1, 1), (63, 3), (65, 4), (130, 6), (257, 203)])
def test_bold_remainders_and_powers(gpu, n, steps, alpha):
    """Whole 1/alpha up to 16 takes products, any other takes powf; both within 2e-6 of the float32 oracle,
    the difference of a few roundings per step (as in the BOLD tests)."""
    import torch
    u = bold_inputs(n, steps, steps + n)
    st = torch.tensor(np.stack([np.zeros(n), np.zeros(n), np.ones(n), np.ones(n)]), dtype=torch.float32).cuda()
    out = E.bold_run(torch.from_numpy(u).cuda(), st, params=E.bold_params(alpha=alpha)).cpu().numpy()
    o = BoldOracle(**{**DA_PARAMS, "alpha": alpha}, n=n)
    ref = np.array([o.run(x) for x in u])
    assert np.allclose(out, ref, rtol=2e-6, atol=2e-8)
    assert np.allclose(st.cpu().numpy(), o.state(), rtol=2e-6, atol=1e-7)


@pytest.mark.parametrize("members,voxels,hp", [(2, 1, 0), (3, 7, 1), (33, 65, 4), (101, 64, 10), (129, 130, 58), (16, 5, 300),
                                               (20, 1000, 4), (7, 700, 0), (151, 300, 0)])
def test_da_filter_ragged(gpu, members, voxels, hp):
    import torch
    rng = np.random.default_rng(members * 1000 + hp)
    w = (1.0 + 0.1 * rng.standard_normal((members, voxels, hp + 6))).astype(np.float32)
    y = (1.0 + 0.05 * rng.standard_normal(voxels)).astype(np.float32)
    noise = rng.standard_normal((members, voxels)).astype(np.float32)
    out = E.da_filter(torch.from_numpy(w).cuda(), torch.from_numpy(y).cuda(), torch.from_numpy(noise).cuda(), 1e-3, 0.3)
    # one float32 rounding of sums in double: half an ulp and the oracle's own rounding
    assert np.allclose(out.cpu().numpy(), da_filter(w, y, noise, hp, 1e-3, 0.3), rtol=2.5e-7, atol=1e-7)


@pytest.mark.parametrize("n,pops,degree", [(31, 1, 5), (31, 1, 300), (1025, 3, 17), (1025, 3, 257), (40_003, 9, 255), (40_003, 9, 700),
                                           (1_638_400, 5, 256), (1_700_001, 5, 20)])
def test_pull_equals_exact_push(gpu, n, pops, degree):
    """The pull's 64-bit sums equal the exact push's bit for bit, from 256 in-edges a neuron on with the
    bitmap in shared memory (1,638,400 neurons fill it), below and above that size in L2."""
    spec = nw.structured_spec(n, pops, degree, seed=n, min_pop=8)
    res = []
    for syn in (E.SYN_PUSH_EXACT, E.SYN_PULL):
        with E.Engine.structured(spec, seed=4, ou=(2.5, 0.5, 10.0), push=syn != E.SYN_PULL, pull=syn == E.SYN_PULL) as eng:
            a = eng.run(90, vmean=True, syn_mode=syn, record_spikes=n < 50_000)
            b = eng.run(37, syn_mode=syn)
            res.append((a.freqs, a.vmeans, b.freqs, a.events + b.events, eng.read_state(E.STATE_V), eng.read_state(E.STATE_J),
                        None if a.spikes is None else a.spikes))
    assert res[0][0].sum() + res[0][2].sum() >= n // 2        # most neurons fire at least once
    for x, y in zip(*res):
        assert (x is None and y is None) or np.array_equal(x, y)


def test_pulls_of_two_sizes_from_two_threads(gpu):
    """Two threads step a small network and one whose bitmap is over shared memory's default limit (both
    with their bitmaps there): each gives the bits it gives alone."""
    import threading
    specs = [nw.structured_spec(n, 3, 256, seed=n) for n in (2_000, 600_000)]

    def steps(eng, runs):
        out = [eng.run(3, syn_mode=E.SYN_PULL).freqs for _ in range(runs)]
        return np.concatenate(out), eng.read_state(E.STATE_V)

    def work(spec, runs, into, k):
        with E.Engine.structured(spec, seed=k + 1, ou=(3.0, 0.5, 10.0), push=False, pull=True) as eng:
            into[k] = steps(eng, runs)

    runs = (400, 40)
    alone, together = {}, {}
    for k in (0, 1):
        work(specs[k], runs[k], alone, k)
    threads = [threading.Thread(target=work, args=(specs[k], runs[k], together, k)) for k in (0, 1)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for k in (0, 1):
        assert alone[k][0].sum() > 0
        assert all(np.array_equal(a, b) for a, b in zip(alone[k], together[k]))


@pytest.mark.parametrize("ts", [1, 4, 255])
def test_kernel_times_with_substeps(gpu, ts):
    """Per-kernel timing of a run with substeps and synaptic-current outputs: every launch of a step
    has its pair of events."""
    with E.Engine.structured(nw.structured_spec(3000, 3, 50, seed=1)) as eng:
        r = eng.run(7, t_steps=ts, imean=True, time_kernels=True, syn_mode=E.SYN_PUSH_FIXED)
        assert all(k > 0 for k in (r.kernel_ms[0], r.kernel_ms[1], r.kernel_ms[3])) and r.imeans.shape == (7, 3)

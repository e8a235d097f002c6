"""Phasing HMM parity: GPU rephase vs the reference's
phasing_hmm::rephaseHaplotypes (phasing_hmm.cpp:247-302) on identical
haplotypes, flat flags, conditioning sets and random streams. The outputs are
discrete (sampled diplotypes and alleles) and must be identical."""
import numpy as np
import pytest

from conftest import ref_oracle_or_skip


def _noisy_haps(rng, truth, p=0.03):
    h = truth.copy()
    flip = rng.random(h.shape) < p
    h[flip] ^= 1
    return h


@pytest.mark.gpu
def test_rephase_matches_reference(small_workload):
    O = ref_oracle_or_skip()
    from glimpse_b200 import native
    w = small_workload
    P, T = w.panel, w.targets
    orc = O.RefOracle(P, T, kinit=200, kpbwt=150)
    ctx = native.Context(P)
    rng = np.random.default_rng(5)
    cases = []
    for t in range(T.n):
        for K in (6, 64, 257, 520):
            s = np.sort(rng.choice(P.n_ref_haps, size=K, replace=False)).astype(np.uint32)
            h0 = _noisy_haps(rng, T.truth[t, 0])
            h1 = _noisy_haps(rng, T.truth[t, 1])
            cases.append((s, h0, h1, T.flat[t], t))
    it = 3
    refs = [orc.rephase(s, h0, h1, fl, it, tid) for (s, h0, h1, fl, tid) in cases]
    g0, g1 = ctx.rephase_batch([c[0] for c in cases], np.stack([c[1] for c in cases]),
                               np.stack([c[2] for c in cases]), np.stack([c[3] for c in cases]), it,
                               target_ids=[c[4] for c in cases])
    bad = []
    for i, (r0, r1, dip) in enumerate(refs):
        n0 = int((g0[i] != r0).sum())
        n1 = int((g1[i] != r1).sum())
        if n0 or n1:
            bad.append((i, n0, n1, len(dip)))
    assert not bad, f"haplotype mismatches (case, #H0, #H1, nseg): {bad}"


@pytest.mark.gpu
@pytest.mark.parametrize("K", [200, 900, 1400, 1700, 2000])
def test_rephase_states_per_thread_instances(K):
    """k_phase is instantiated for the smallest J (states per thread, 256 threads)
    that holds the launch's largest K. One K per call reaches J = 1, 4, 6, 7 and 8
    (the test above runs J = 3; the iteration tests J = 2 and 5); the sampled
    haplotypes must equal rephaseHaplotypes' on identical inputs and streams."""
    O = ref_oracle_or_skip()
    from glimpse_b200 import native, synth
    w = synth.make_panel_and_targets(2048, 6000, 0.5, 0.5, 2, ("uniform", 0.5, 2.0), ("fixed", 200), seed=59,
                                     sparse_maf=0.005)
    P, T = w.panel, w.targets
    orc = O.RefOracle(P, T, kinit=200, kpbwt=150)
    ctx = native.Context(P)
    try:
        rng = np.random.default_rng(K)
        cases = []
        for t in range(T.n):
            s = np.sort(rng.choice(P.n_ref_haps, size=K, replace=False)).astype(np.uint32)
            cases.append((s, _noisy_haps(rng, T.truth[t, 0]), _noisy_haps(rng, T.truth[t, 1]), T.flat[t], t))
        it = 2
        refs = [orc.rephase(s, h0, h1, fl, it, tid) for (s, h0, h1, fl, tid) in cases]
        g0, g1 = ctx.rephase_batch([c[0] for c in cases], np.stack([c[1] for c in cases]),
                                   np.stack([c[2] for c in cases]), np.stack([c[3] for c in cases]), it,
                                   target_ids=[c[4] for c in cases])
        for i, (r0, r1, _) in enumerate(refs):
            assert np.array_equal(g0[i], r0) and np.array_equal(g1[i], r1), (K, i)
    finally:
        ctx.close()


@pytest.mark.gpu
def test_invalid_diplotype_sums_return_data_error(small_workload):
    """SAMPLE_DIP with a NaN, infinite or sub-normal sum: the reference stops on
    an assertion (phasing_hmm.cpp:175); the library finishes the call and
    returns GP_E_DATA naming the target. A NaN err_phase makes every emission,
    and so every diplotype sum, NaN. The oracle is not run here (it would abort
    the process at that assertion)."""
    from glimpse_b200 import native
    w = small_workload
    P, T = w.panel, w.targets
    rng = np.random.default_rng(8)
    good = native.Context(P)
    bad = native.Context(P, err_phase=float("nan"))
    try:
        s = np.sort(rng.choice(P.n_ref_haps, size=64, replace=False)).astype(np.uint32)
        h0 = _noisy_haps(rng, T.truth[1, 0])
        h1 = _noisy_haps(rng, T.truth[1, 1])
        good.rephase_batch([s], h0[None], h1[None], T.flat[1][None], 2, target_ids=[1])
        with pytest.raises(native.GpError, match="target 7"):
            bad.rephase_batch([s], h0[None], h1[None], T.flat[1][None], 2, target_ids=[7])
        # the context stays usable: an iteration over the targets reports the same error
        bad.set_targets(T, kpbwt=T.kpbwt)
        with pytest.raises(native.GpError, match="invalid diplotype"):
            bad.iteration(native.STAGE_INIT, 0)
    finally:
        good.close()
        bad.close()


@pytest.mark.gpu
def test_chunked_phasing_matches_single_launch(small_workload, monkeypatch):
    """When the targets' stored phasing messages do not fit the device-memory
    budget together, k_phase runs in consecutive chunks of the batch
    (GLIMPSE_B200_STORE_BUDGET_MB lowers the budget so that a small batch takes
    that path). The rephased haplotypes must be identical."""
    from glimpse_b200 import native
    w = small_workload
    P, T = w.panel, w.targets
    rng = np.random.default_rng(9)
    cases = []
    for i in range(9):
        t = i % T.n
        s = np.sort(rng.choice(P.n_ref_haps, size=int(rng.integers(50, 520)), replace=False)).astype(np.uint32)
        cases.append((s, _noisy_haps(rng, T.truth[t, 0]), _noisy_haps(rng, T.truth[t, 1]), T.flat[t], t))
    args = ([c[0] for c in cases], np.stack([c[1] for c in cases]), np.stack([c[2] for c in cases]),
            np.stack([c[3] for c in cases]), 4)
    ctx = native.Context(P)
    try:
        a0, a1 = ctx.rephase_batch(*args, target_ids=[c[4] for c in cases])
        monkeypatch.setenv("GLIMPSE_B200_STORE_BUDGET_MB", "1")
        b0, b1 = ctx.rephase_batch(*args, target_ids=[c[4] for c in cases])
        monkeypatch.delenv("GLIMPSE_B200_STORE_BUDGET_MB")
        assert np.array_equal(a0, b0) and np.array_equal(a1, b1)
    finally:
        ctx.close()


@pytest.mark.gpu
@pytest.mark.parametrize("edges", [(40, 300, 600, 900, 1100, 1500), (250, 256), (700, 760, 768, 500), (1030, 1280, 1025)])
def test_many_chains_match_single_calls(edges):
    """From about three chains per SM on, the chains of some classes run two warps
    instead of four (all classes where one holds most chains): 260 targets over
    mixed and uniform state counts must get the haplotypes they get alone."""
    from glimpse_b200 import native, synth
    w = synth.make_panel_and_targets(1600, 500, 0.2, 0.4, 2, ("uniform", 0.3, 1.5), ("fixed", 200), seed=73,
                                     sparse_maf=0.005)
    P, T = w.panel, w.targets
    rng = np.random.default_rng(edges[0])
    n = 260
    sets = [np.sort(rng.choice(P.n_ref_haps, size=edges[i % len(edges)], replace=False)).astype(np.uint32)
            for i in range(n)]
    h0 = np.stack([_noisy_haps(rng, T.truth[i % 2, 0]) for i in range(n)])
    h1 = np.stack([_noisy_haps(rng, T.truth[i % 2, 1]) for i in range(n)])
    flat = np.stack([T.flat[i % 2] for i in range(n)])
    ctx = native.Context(P)
    try:
        g0, g1 = ctx.rephase_batch(sets, h0, h1, flat, 3)
        for i in list(range(12)) + [100, 177, 259]:
            a0, a1 = ctx.rephase_batch([sets[i]], h0[i][None], h1[i][None], flat[i][None], 3, target_ids=[i])
            assert np.array_equal(a0[0], g0[i]) and np.array_equal(a1[0], g1[i]), (i, sets[i].size)
    finally:
        ctx.close()


@pytest.mark.gpu
@pytest.mark.parametrize("edges", [(1, 31, 32, 33, 64, 65), (255, 256, 257, 319, 321), (511, 512, 513, 767, 769, 1023),
                                   (1024, 1025, 1535, 1537, 1791, 1793, 2047, 2048)])
def test_state_count_edges_and_mixed_classes(edges):
    """The chain kernel has an instance per 256 states, its last two register slots
    may be partly empty, and a batch runs its instances side by side: every
    target of a mixed batch must get the haplotypes it gets alone, at state
    counts around the warp and class boundaries, and (where it is built) those
    of rephaseHaplotypes."""
    from glimpse_b200 import native, synth
    w = synth.make_panel_and_targets(2048, 1500, 0.3, 0.5, 2, ("uniform", 0.3, 1.5), ("fixed", 200), seed=61,
                                     sparse_maf=0.005)
    P, T = w.panel, w.targets
    rng = np.random.default_rng(edges[0])
    cases = []
    for i, K in enumerate(edges):
        t = i % T.n
        s = np.sort(rng.choice(P.n_ref_haps, size=K, replace=False)).astype(np.uint32)
        flat = T.flat[t].copy()
        if i % 3 == 1:
            flat[:] = 1  # flat hets only: the first VAR site starts the recursion without a sum
        if i % 3 == 2:
            flat[40:1400] = 1  # most 32-site blocks without a VAR site but flat hets
        cases.append((s, _noisy_haps(rng, T.truth[t, 0]), _noisy_haps(rng, T.truth[t, 1]), flat, i))
    ctx = native.Context(P)
    try:
        it = 3
        args = ([c[0] for c in cases], np.stack([c[1] for c in cases]), np.stack([c[2] for c in cases]),
                np.stack([c[3] for c in cases]), it)
        g0, g1 = ctx.rephase_batch(*args, target_ids=[c[4] for c in cases])
        for i, (s, h0, h1, fl, tid) in enumerate(cases):
            a0, a1 = ctx.rephase_batch([s], h0[None], h1[None], fl[None], it, target_ids=[tid])
            assert np.array_equal(a0[0], g0[i]) and np.array_equal(a1[0], g1[i]), edges[i]
        O = ref_oracle_or_skip()
        orc = O.RefOracle(P, T, kinit=200, kpbwt=150)
        for i, (s, h0, h1, fl, tid) in enumerate(cases):
            r0, r1, _ = orc.rephase(s, h0, h1, fl, it, tid)
            assert np.array_equal(g0[i], r0) and np.array_equal(g1[i], r1), edges[i]
    finally:
        ctx.close()


@pytest.mark.gpu
@pytest.mark.parametrize("K", [1, 2, 3, 40, 300])
def test_small_sets_on_long_chunks_match_restatement(K):
    """Register slots without a state must stay at 0 however long the chunk is: the
    homs that all states mismatch (here all sites where they agree on alt, the
    targets being ref) scale whatever sits there by ee / ed each, so that a small
    set overflowed it within a chunk. 20,000 sites, three targets, one of them with
    flat sites at the ends: the haplotypes of the FP32 restatement, bit for bit."""
    from oracle import oracle as O
    from glimpse_b200 import native, synth
    w = synth.make_panel_and_targets(1000, 20000, 0.5, 0.0, 3, ("uniform", 0.5, 2.0), ("fixed", 100), seed=83,
                                     sparse_maf=0.005, alt_major_frac=0.1)
    P, T = w.panel, w.targets
    rng = np.random.default_rng(K)
    cases = []
    for t in range(3):
        s = np.sort(rng.choice(P.n_ref_haps, size=K, replace=False)).astype(np.uint32)
        h0, h1, flat = _noisy_haps(rng, T.truth[t, 0]), _noisy_haps(rng, T.truth[t, 1]), T.flat[t].copy()
        alleles = (P.hvar[:, s >> 3] >> (7 - (s & 7)).astype(np.uint8)) & 1
        alt = np.flatnonzero(P.flag_common)[alleles.all(axis=1)]
        assert K == 300 or alt.size > 100
        h0[alt] = h1[alt] = 0
        if t == 1:
            flat[:500] = flat[-500:] = 1
        cases.append((s, h0, h1, flat))
    ctx = native.Context(P)
    try:
        g0, g1 = ctx.rephase_batch([c[0] for c in cases], np.stack([c[1] for c in cases]),
                                   np.stack([c[2] for c in cases]), np.stack([c[3] for c in cases]), 3)
    finally:
        ctx.close()
    for t, (s, h0, h1, flat) in enumerate(cases):
        r0, r1, invalid = O.restate_rephase(P, s, h0, h1, flat, 3, t)
        assert not invalid
        assert np.array_equal(g0[t], r0) and np.array_equal(g1[t], r1), t


@pytest.mark.gpu
def test_small_sets_in_a_large_batch_match_restatement():
    """The same for two-warp chains, whose unused slots are most of a warp: 240 targets
    with 2 states each, all of one class."""
    from oracle import oracle as O
    from glimpse_b200 import native, synth
    w = synth.make_panel_and_targets(1000, 12000, 0.3, 0.0, 3, ("uniform", 0.5, 2.0), ("fixed", 100), seed=83,
                                     sparse_maf=0.005, alt_major_frac=0.1)
    P, T = w.panel, w.targets
    rng = np.random.default_rng(2)
    n = 240
    sets = [np.sort(rng.choice(P.n_ref_haps, size=2, replace=False)).astype(np.uint32) for _ in range(n)]
    h0 = np.stack([_noisy_haps(rng, T.truth[i % 3, 0]) for i in range(n)])
    h1 = np.stack([_noisy_haps(rng, T.truth[i % 3, 1]) for i in range(n)])
    for i, s in enumerate(sets):
        alt = np.flatnonzero(P.flag_common)[((P.hvar[:, s >> 3] >> (7 - (s & 7)).astype(np.uint8)) & 1).all(axis=1)]
        h0[i, alt] = h1[i, alt] = 0
    flat = np.stack([T.flat[i % 3] for i in range(n)])
    ctx = native.Context(P)
    try:
        g0, g1 = ctx.rephase_batch(sets, h0, h1, flat, 5)
    finally:
        ctx.close()
    for i in range(0, n, 7):
        r0, r1, invalid = O.restate_rephase(P, sets[i], h0[i], h1[i], flat[i], 5, i)
        assert not invalid and np.array_equal(g0[i], r0) and np.array_equal(g1[i], r1), i

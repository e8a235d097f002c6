"""State selection parity (bit-exact):
  * init stage: haplotype_set::initRareTar + performSelection_RARE_INIT_GL
    (haplotype_set.cpp:108-169,775-833), per-target std::sample streams;
  * burn-in/main: matchHapsFromCompressedPBWTSmall (haplotype_set.cpp:317-394),
    every pbwt_states level list, and the conditioning_set::compactSelection
    union (conditioning_set.cpp:96-104)."""
import dataclasses

import numpy as np
import pytest

from conftest import ref_oracle_or_skip


def _noisy(rng, h, p):
    h = h.copy()
    h[rng.random(h.shape) < p] ^= 1
    return h


@pytest.fixture(scope="module")
def pair(small_workload):
    O = ref_oracle_or_skip()
    from glimpse_b200 import native
    w = small_workload
    kw = dict(kinit=200, kpbwt=int(w.targets.kpbwt.max()), pbwt_depth=8, pbwt_modulo_cm=0.05)
    orc = O.RefOracle(w.panel, w.targets, kpbwt_target=w.targets.kpbwt, **kw)
    ctx = native.Context(w.panel, **kw)
    ctx.set_targets(w.targets, kpbwt=w.targets.kpbwt)
    return w, orc, ctx, O


@pytest.mark.gpu
def test_init_selection_matches_reference(pair):
    w, orc, ctx, O = pair
    orc.init_select(0)
    ctx.select(O.STAGE_INIT, 0)
    for t in range(w.targets.n):
        ref = np.sort(orc.init_states(t)).astype(np.uint32)
        got = ctx.states(t)
        assert np.array_equal(ref, got), f"target {t}: {len(ref)} vs {len(got)} states"


@pytest.mark.gpu
@pytest.mark.parametrize("it,noise", [(1, 0.0), (4, 0.02), (9, 0.1)])
def test_pbwt_selection_matches_reference(pair, it, noise):
    w, orc, ctx, O = pair
    rng = np.random.default_rng(it)
    T = w.targets
    h0 = np.stack([_noisy(rng, T.truth[t, 0], noise) for t in range(T.n)])
    h1 = np.stack([_noisy(rng, T.truth[t, 1], noise) for t in range(T.n)])
    for t in range(T.n):
        orc.set_haps(t, h0[t], h1[t])
    ctx.set_haps(h0, h1)
    orc.pbwt_select(it, main_iteration=False)
    ctx.select(O.STAGE_BURN, it)
    for t in range(T.n):
        ref_lv = orc.pbwt_states(t)
        got_lv = ctx.pbwt_states(t, depth=len(ref_lv))
        for lv, (r, g) in enumerate(zip(ref_lv, got_lv)):
            assert np.array_equal(r, g), f"target {t} level {lv}: {r[:10]} vs {g[:10]} ({len(r)} vs {len(g)})"
        ref_states = orc.select(t, O.STAGE_BURN)
        assert np.array_equal(ref_states, ctx.states(t)), f"target {t} union differs"


@pytest.fixture(scope="module")
def pair_haploid(small_workload):
    """The small workload with target 1 haploid: 5 target haplotypes, an odd count,
    so the last warp of the PBWT sweep runs a partial group."""
    O = ref_oracle_or_skip()
    from glimpse_b200 import native
    w = small_workload
    T = dataclasses.replace(w.targets, ploidy=w.targets.ploidy.copy())
    T.ploidy[1] = 1
    kw = dict(kinit=200, kpbwt=int(T.kpbwt.max()), pbwt_depth=8, pbwt_modulo_cm=0.05)
    orc = O.RefOracle(w.panel, T, kpbwt_target=T.kpbwt, **kw)
    ctx = native.Context(w.panel, **kw)
    ctx.set_targets(T, kpbwt=T.kpbwt)
    return w, T, orc, ctx, O


@pytest.mark.gpu
def test_pbwt_selection_haploid_target_matches_reference(pair_haploid):
    w, T, orc, ctx, O = pair_haploid
    rng = np.random.default_rng(11)
    h0 = np.stack([_noisy(rng, T.truth[t, 0], 0.02) for t in range(T.n)])
    h1 = np.stack([_noisy(rng, T.truth[t, 1], 0.02) for t in range(T.n)])
    for t in range(T.n):
        orc.set_haps(t, h0[t], h1[t])
    ctx.set_haps(h0, h1)
    orc.pbwt_select(4, main_iteration=False)
    ctx.select(O.STAGE_BURN, 4)
    for t in range(T.n):
        ref_lv = orc.pbwt_states(t)
        got_lv = ctx.pbwt_states(t, depth=len(ref_lv))
        for lv, (r, g) in enumerate(zip(ref_lv, got_lv)):
            assert np.array_equal(r, g), f"target {t} level {lv}: {len(r)} vs {len(g)}"
        assert np.array_equal(orc.select(t, O.STAGE_BURN), ctx.states(t)), f"target {t} union differs"


@pytest.mark.gpu
def test_selection_with_capped_grid_matches_reference(small_workload, monkeypatch):
    """The event-bit and panel-transpose kernels loop over their second grid
    dimension when it would pass the hardware's 65,535 (panels with more than
    about 2M events or common sites). GLIMPSE_B200_GRID_Y_CAP=2 makes a small
    panel take those loops; selection must stay bit-exact and posteriors (which
    read the transposed panel) within 1e-5 of the reference."""
    O = ref_oracle_or_skip()
    from glimpse_b200 import native
    from conftest import init_hl
    w = small_workload
    T = w.targets
    kw = dict(kinit=200, kpbwt=int(T.kpbwt.max()), pbwt_depth=8, pbwt_modulo_cm=0.05)
    monkeypatch.setenv("GLIMPSE_B200_GRID_Y_CAP", "2")
    ctx = native.Context(w.panel, **kw)
    monkeypatch.delenv("GLIMPSE_B200_GRID_Y_CAP")
    orc = O.RefOracle(w.panel, T, kpbwt_target=T.kpbwt, **kw)
    try:
        ctx.set_targets(T, kpbwt=T.kpbwt)
        rng = np.random.default_rng(17)
        h0 = np.stack([_noisy(rng, T.truth[t, 0], 0.02) for t in range(T.n)])
        h1 = np.stack([_noisy(rng, T.truth[t, 1], 0.02) for t in range(T.n)])
        for t in range(T.n):
            orc.set_haps(t, h0[t], h1[t])
        ctx.set_haps(h0, h1)
        orc.pbwt_select(3, main_iteration=False)
        ctx.select(O.STAGE_BURN, 3)
        for t in range(T.n):
            ref_lv = orc.pbwt_states(t)
            got_lv = ctx.pbwt_states(t, depth=len(ref_lv))
            for lv, (r, g) in enumerate(zip(ref_lv, got_lv)):
                assert np.array_equal(r, g), f"target {t} level {lv}"
            assert np.array_equal(orc.select(t, O.STAGE_BURN), ctx.states(t)), f"target {t} union differs"
        s = ctx.states(0)
        hl = init_hl(T.gl[0], T.flat[0])
        got = ctx.impute_batch([s], hl[None], T.flat[0][None])[0]
        ref, _ = orc.impute(s, hl, T.flat[0])
        assert float(np.abs(got - ref).max()) <= 1e-5
    finally:
        ctx.close()


@pytest.mark.gpu
@pytest.mark.parametrize("N,L", [(1500, 900), (20000, 90), (40000, 70), (70000, 60)])
def test_sweep_shapes_and_panel_sizes_give_the_same_selection(N, L):
    """The sweep stages 4, 2 or 1 rank rows per copy, or none where a panel's rows
    do not fit shared memory (N above about 65,000), for 1, 2, 4 or 8 haplotypes
    per warp, the last warp partly idle (7 haplotypes). Every shape must select
    the same level lists and states, and (where it is built) the reference's."""
    from glimpse_b200 import native, synth
    from oracle import oracle as O
    w = synth.make_panel_and_targets(N, L, 0.2, 0.4, 4, ("uniform", 0.5, 2.0), ("fixed", 90), seed=71,
                                     sparse_maf=max(0.001, 4.5 / N))
    T = dataclasses.replace(w.targets, ploidy=w.targets.ploidy.copy())
    T.ploidy[2] = 1
    kw = dict(kinit=60, kpbwt=90, pbwt_depth=7, pbwt_modulo_cm=0.05)
    rng = np.random.default_rng(N)
    h0 = np.stack([_noisy(rng, T.truth[t, 0], 0.03) for t in range(T.n)])
    h1 = np.stack([_noisy(rng, T.truth[t, 1], 0.03) for t in range(T.n)])
    ctx = native.Context(w.panel, **kw)
    got = []
    try:
        for hpw in (1, 2, 4, 8):
            ctx.tuning_set(0, hpw, 0)
            ctx.set_targets(T, kpbwt=T.kpbwt)
            ctx.set_haps(h0, h1)
            ctx.select(O.STAGE_BURN, 3)
            got.append([([x.tolist() for x in ctx.pbwt_states(t, depth=7)], ctx.states(t).tolist()) for t in range(T.n)])
        assert got[0] == got[1] == got[2] == got[3]
        assert all(0 < len(s) <= 90 for _, s in got[0])
        orc = ref_oracle_or_skip().RefOracle(w.panel, T, kpbwt_target=T.kpbwt, **kw)
        for t in range(T.n):
            orc.set_haps(t, h0[t], h1[t])
        orc.pbwt_select(3, main_iteration=False)
        for t in range(T.n):
            assert [x.tolist() for x in orc.pbwt_states(t)] == got[0][t][0]
            assert orc.select(t, O.STAGE_BURN).tolist() == got[0][t][1]
    finally:
        ctx.close()


@pytest.mark.gpu
@pytest.mark.parametrize("kpbwt", [1, 31, 32, 33, 64, 500, 1500])
def test_union_order_and_limits(kpbwt):
    """The union takes 32 pushes at a time: limits inside, at the end of and past a
    group, and many groups, for diploid targets (two merged lists) and a haploid one,
    against the level lists walked one push at a time from the last. A limit of the
    panel's size takes the whole panel instead, without lists."""
    from glimpse_b200 import native, synth
    from oracle import oracle as O
    w = synth.make_panel_and_targets(1500, 900, 0.2, 0.4, 4, ("uniform", 0.5, 2.0), ("fixed", 90), seed=71,
                                     sparse_maf=0.003)
    T = dataclasses.replace(w.targets, ploidy=w.targets.ploidy.copy(), kpbwt=np.full(4, kpbwt, np.int32))
    T.ploidy[2] = 1
    rng = np.random.default_rng(kpbwt)
    ctx = native.Context(w.panel, kinit=60, kpbwt=kpbwt, pbwt_depth=7, pbwt_modulo_cm=0.05)
    try:
        ctx.set_targets(T, kpbwt=T.kpbwt)
        ctx.set_haps(np.stack([_noisy(rng, T.truth[t, 0], 0.03) for t in range(T.n)]),
                     np.stack([_noisy(rng, T.truth[t, 1], 0.03) for t in range(T.n)]))
        ctx.select(O.STAGE_BURN, 3)
        for t in range(T.n):
            want = set()
            for level in ctx.pbwt_states(t, depth=7):
                for h in level[::-1].tolist():
                    if len(want) < kpbwt:
                        want.add(h)
            if kpbwt >= w.panel.n_ref_haps:
                want = range(w.panel.n_ref_haps)
            assert sorted(want) == ctx.states(t).tolist()
    finally:
        ctx.close()


@pytest.mark.gpu
def test_deep_lists_on_a_panel_without_staged_rows():
    """1,450 levels: the push counts of 8 haplotypes per warp pass the default 48 KB
    of shared memory also where no rank rows are staged, and all shapes select alike.
    6,500 levels do not fit the SM for 8 haplotypes: an error, not a union of lists
    that no sweep wrote."""
    from glimpse_b200 import native, synth
    from oracle import oracle as O
    w = synth.make_panel_and_targets(70000, 60, 0.2, 0.4, 2, ("uniform", 0.5, 2.0), ("fixed", 90), seed=71,
                                     sparse_maf=0.001)
    T = w.targets
    got = []
    for depth, hpw in ((1450, 1), (1450, 8), (6500, 1), (6500, 8)):
        ctx = native.Context(w.panel, kinit=60, kpbwt=90, pbwt_depth=depth, pbwt_modulo_cm=0.05)
        try:
            ctx.tuning_set(0, hpw, 0)
            ctx.set_targets(T, kpbwt=T.kpbwt)
            ctx.set_haps(T.truth[:, 0], T.truth[:, 1])
            if (depth, hpw) == (6500, 8):
                with pytest.raises(native.GpError, match="selection launch"):
                    ctx.select(O.STAGE_BURN, 3)
                ctx.tuning_set(0, 1, 0)  # the context stays usable
            ctx.select(O.STAGE_BURN, 3)
            got.append([ctx.states(t).tolist() for t in range(T.n)])
        finally:
            ctx.close()
    assert got[0] == got[1] and got[2] == got[3] and all(0 < len(s) <= 90 for g in got for s in g)


@pytest.mark.gpu
@pytest.mark.parametrize("kinit", [1, 2, 20, 78, 93])
def test_init_selection_matches_restatement(kinit):
    """The init selection of targets that carry more rare alleles than the share of
    Kinit for them (by minor-allele count, five carriers a site), and of targets with
    fewer (all sites), against a restatement on the same streams."""
    from glimpse_b200 import native, synth
    from oracle import oracle as O
    w = synth.make_panel_and_targets(94, 8075, 0.215, 0.3, 4, ("uniform", 0.2, 12.0), ("fixed", 60), seed=1005,
                                     sparse_maf=3.5 / 94)
    ctx = native.Context(w.panel, kinit=kinit, kpbwt=11)
    try:
        ctx.set_targets(w.targets, kpbwt=w.targets.kpbwt)
        ctx.select(O.STAGE_INIT, 0)
        many = []
        for t in range(w.targets.n):
            want, sites = O.restate_init_select(w.panel, w.targets, t, kinit)
            many.append(sites > int(0.8 * kinit))
            assert want.tolist() == ctx.states(t).tolist(), t
        assert any(many)
    finally:
        ctx.close()

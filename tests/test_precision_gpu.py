"""Precision of the imputation posteriors against the FP64 restatement of the
forward-backward (oracle/restate.c, following imputation_hmm.cpp:80-429): the
GPU computes in FP32 with per-site rescaling, as the reference does. The test
prints the largest absolute HP error per panel shape (run pytest with -s to see
it) and bounds it at 1e-5, the parity tolerance against the reference."""
import numpy as np
import pytest

from conftest import init_hl

TOL = 1e-5


def _max_err_vs_fp64(w, Ks, seed):
    from glimpse_b200 import native
    from oracle import oracle as O
    P, T = w.panel, w.targets
    rng = np.random.default_rng(seed)
    ctx = native.Context(P)
    try:
        states, hls, flats = [], [], []
        for i, K in enumerate(Ks):
            t = i % T.n
            states.append(np.sort(rng.choice(P.n_ref_haps, size=K, replace=False)).astype(np.uint32))
            hls.append(init_hl(T.gl[t], T.flat[t]))
            flats.append(T.flat[t])
        hp = ctx.impute_batch(states, np.stack(hls), np.stack(flats))
    finally:
        ctx.close()
    worst = 0.0
    for i in range(len(Ks)):
        ref, _ = O.restate_impute(P, states[i], hls[i], flats[i], precision=64)
        worst = max(worst, float(np.abs(hp[i].astype(np.float64) - ref.astype(np.float64)).max()))
    return worst


@pytest.mark.gpu
def test_small_panel_posteriors_vs_fp64():
    from glimpse_b200 import synth
    # the small workload: 1,000 haplotypes x 20,000 sites, K = 500
    w = synth.workload("small", seed=3)
    err = _max_err_vs_fp64(w, [500, 500, 500, 500], seed=1)
    print(f"\nsmall panel (1,000 x 20,000, K=500): max |HP - HP_fp64| = {err:.3e}")
    assert err <= TOL


@pytest.mark.gpu
def test_batched_panel_posteriors_vs_fp64():
    from glimpse_b200 import synth
    # the batched panel (10,000 haplotypes x 150,000 sites, 80% rare), one target, K at both ends of 400-1200
    w = synth.workload("batched", seed=1, n_targets=1)
    err = _max_err_vs_fp64(w, [400, 1200], seed=2)
    print(f"\nbatched panel (10,000 x 150,000, K=400 and 1200): max |HP - HP_fp64| = {err:.3e}")
    assert err <= TOL


def _impute_modes(w, Ks, seed, modes):
    """HP (and the FP64 chunk log-likelihood of checkpointed modes) for the same
    haplotypes under each precision mode, with the FP64 restatement's."""
    from glimpse_b200 import native
    from oracle import oracle as O
    P, T = w.panel, w.targets
    rng = np.random.default_rng(seed)
    states, hls, flats = [], [], []
    for i, K in enumerate(Ks):
        t = i % T.n
        states.append(np.sort(rng.choice(P.n_ref_haps, size=K, replace=False)).astype(np.uint32))
        hls.append(init_hl(T.gl[t], T.flat[t]))
        flats.append(T.flat[t])
    ctx = native.Context(P)
    out = {}
    try:
        for m in modes:
            ctx.set_precision(m)
            hp = ctx.impute_batch(states, np.stack(hls), np.stack(flats))
            ll = ctx.loglik(len(Ks)) if m != native.PRECISION_FULL else None
            out[m] = (hp, ll)
    finally:
        ctx.close()
    ref = [O.restate_impute(P, states[i], hls[i], flats[i], precision=64) for i in range(len(Ks))]
    return out, ref


@pytest.mark.gpu
def test_checkpointed_fp32_posteriors_and_loglik():
    """FP32 checkpoints with recompute: posteriors within 1e-5 of FP64 (as the
    full store), and the FP64 chunk log-likelihood sum_l log AlphaSum_l within
    1e-6 per site of the FP64 restatement's."""
    from glimpse_b200 import native, synth
    w = synth.workload("small", seed=3)
    out, ref = _impute_modes(w, [500, 37, 256], 4, [native.PRECISION_FULL, native.PRECISION_CKPT_F32])
    hp_full, _ = out[native.PRECISION_FULL]
    hp_ck, ll = out[native.PRECISION_CKPT_F32]
    for i, (hr, llr) in enumerate(ref):
        e = float(np.abs(hp_ck[i].astype(np.float64) - hr.astype(np.float64)).max())
        assert e <= TOL, f"haplotype {i}: max |HP - HP_fp64| = {e:.3e}"
        assert float(np.abs(hp_ck[i] - hp_full[i]).max()) <= TOL
        n_poly = w.panel.n_sites
        assert abs(ll[i] - llr) <= 1e-6 * n_poly, (i, ll[i], llr)


@pytest.mark.gpu
@pytest.mark.parametrize("K", [700, 1000, 1500, 2000])
def test_checkpointed_states_per_thread_instances(K):
    """Each launch instantiates the checkpointed kernel for the smallest J (states
    per thread, 256 threads) that holds its largest K: K = 700, 1000, 1500 and 2000
    reach J = 3, 4, 6 and 8, the instances the other tests (J = 2 and 5) do not.
    FP32 checkpoints: HP within 1e-5 of the FP64 restatement and of the full
    store, the chunk log-likelihood within 1e-6 per site. The full store's own
    kernel (one warp per chain, J = K / 128 quads rounded up) runs at J = 6, 8, 12
    and 16 here, and its HP must be within 1e-5 of FP64 as well."""
    from glimpse_b200 import native, synth
    w = synth.make_panel_and_targets(2048, 6000, 0.5, 0.5, 2, ("uniform", 0.5, 2.0), ("fixed", 200), seed=53,
                                     sparse_maf=0.005)
    out, ref = _impute_modes(w, [K, K // 3], 6, [native.PRECISION_FULL, native.PRECISION_CKPT_F32])
    hp_full, _ = out[native.PRECISION_FULL]
    hp_ck, ll = out[native.PRECISION_CKPT_F32]
    for i, (hr, llr) in enumerate(ref):
        e = float(np.abs(hp_ck[i].astype(np.float64) - hr.astype(np.float64)).max())
        assert e <= TOL, f"K={K} haplotype {i}: max |HP - HP_fp64| = {e:.3e}"
        ef = float(np.abs(hp_full[i].astype(np.float64) - hr.astype(np.float64)).max())
        assert ef <= TOL, f"K={K} haplotype {i}, full store: max |HP - HP_fp64| = {ef:.3e}"
        assert float(np.abs(hp_ck[i] - hp_full[i]).max()) <= TOL
        assert abs(ll[i] - llr) <= 1e-6 * w.panel.n_sites, (i, ll[i], llr)


def _dosage(hp0, hp1):
    return hp0[1::2].astype(np.float64) + hp1[1::2].astype(np.float64)


@pytest.mark.gpu
@pytest.mark.parametrize("shape", ["small", "batched"])
def test_checkpointed_bf16_error_vs_fp64(shape):
    """BF16 checkpoints (the memory-lean variant): the largest posterior error
    and the largest error of the dosage formed from the two haplotypes'
    posteriors (DS = P(alt | hap 0) + P(alt | hap 1)), against FP64 on the same
    inputs. Printed (pytest -s) and bounded."""
    from glimpse_b200 import native, synth
    w = synth.workload("small", seed=3) if shape == "small" else synth.workload("batched", seed=1, n_targets=2)
    Ks = [500, 500, 500, 500] if shape == "small" else [400, 400, 1200, 1200]
    out, ref = _impute_modes(w, Ks, 5, [native.PRECISION_CKPT_BF16, native.PRECISION_CKPT_F32])
    hp, ll = out[native.PRECISION_CKPT_BF16]
    e_hp = max(float(np.abs(hp[i].astype(np.float64) - ref[i][0].astype(np.float64)).max()) for i in range(len(Ks)))
    e_ds = 0.0
    for i in range(0, len(Ks), 2):
        ds = _dosage(hp[i], hp[i + 1])
        ds64 = _dosage(ref[i][0], ref[i + 1][0])
        e_ds = max(e_ds, float(np.abs(ds - ds64).max()))
    e_ll = max(abs(ll[i] - ref[i][1]) / abs(ref[i][1]) for i in range(len(Ks)))
    print(f"\n{shape}: BF16 checkpoints: max |HP - HP_fp64| = {e_hp:.3e}, max |DS - DS_fp64| = {e_ds:.3e}, "
          f"max relative loglik error {e_ll:.2e}")
    assert e_hp <= 5e-3 and e_ds <= 1e-2 and e_ll <= 1e-4


@pytest.mark.gpu
def test_checkpointed_bf16_full_run_r2():
    """A complete Gibbs run on the small workload with BF16 checkpoints against
    the same run with every row kept: dosage r^2 within 0.002."""
    from glimpse_b200 import native, synth
    w = synth.make_panel_and_targets(800, 6000, 0.6, 0.6, 4, ("uniform", 0.5, 2.0), ("uniform", 150, 400), seed=21,
                                     sparse_maf=0.01)
    truth = w.targets.truth.sum(1)
    r2 = {}
    for m in (native.PRECISION_FULL, native.PRECISION_CKPT_BF16):
        ctx = native.Context(w.panel, kinit=300, kpbwt=int(w.targets.kpbwt.max()), pbwt_depth=8, pbwt_modulo_cm=0.05)
        try:
            ctx.set_precision(m)
            ctx.set_targets(w.targets, kpbwt=w.targets.kpbwt)
            ctx.run(3, 5)
            r2[m] = synth.dosage_r2(ctx.gp()[2], truth)
        finally:
            ctx.close()
    d = r2[native.PRECISION_CKPT_BF16] - r2[native.PRECISION_FULL]
    print(f"\nfull run r2: all rows {r2[native.PRECISION_FULL]:.5f}, BF16 checkpoints "
          f"{r2[native.PRECISION_CKPT_BF16]:.5f} (delta {d:+.5f})")
    assert abs(d) <= 0.002


@pytest.mark.gpu
@pytest.mark.parametrize("sites", [1, 16, 17, 32, 33, 63, 64, 65, 97, 200])
def test_checkpointed_block_and_state_count_edges(sites):
    """Site counts around the kept rows (16 sites), the blocks (32) and the split of
    the BF16 rows (np / 2 rounded down to a block: none below 64 sites), and state
    counts around the rows of 128 and 256, in one batch. FP32: HP within 1e-5 of
    FP64, the log-likelihood within 1e-6 per site. BF16: rows rounded to 8 bits, a
    relative error of 2^-9, at most two in a posterior and one in the likelihood: HP
    within 5e-3, the log-likelihood within 2^-8 more."""
    import dataclasses
    from glimpse_b200 import native, synth
    w = synth.make_panel_and_targets(2050, 260, 0.2, 0.0, 2, ("uniform", 0.4, 2.0), ("fixed", 200), seed=67,
                                     sparse_maf=0.005)
    P, T = w.panel, w.targets
    keep = slice(0, sites)
    P = dataclasses.replace(P, n_sites=sites, bp=P.bp[keep], cm=P.cm[keep], cref=P.cref[keep], calt=P.calt[keep],
                            lq=P.lq[keep], flag_common=P.flag_common[keep], major=P.major[keep],
                            hvar=np.ascontiguousarray(P.hvar[keep]))
    T = dataclasses.replace(T, gl=np.ascontiguousarray(T.gl[:, keep]), flat=np.ascontiguousarray(T.flat[:, keep]))
    Ks = [1, 31, 32, 33, 127, 128, 129, 255, 256, 257, 511, 513, 769, 1025, 1537, 2047, 2048]
    out, ref = _impute_modes(dataclasses.replace(w, panel=P, targets=T), Ks, sites,
                             [native.PRECISION_CKPT_F32, native.PRECISION_CKPT_BF16])
    for m, tol, ll_tol in ((native.PRECISION_CKPT_F32, TOL, 0.0), (native.PRECISION_CKPT_BF16, 5e-3, 2.0 ** -8)):
        hp, ll = out[m]
        for i, (hr, llr) in enumerate(ref):
            e = float(np.abs(hp[i].astype(np.float64) - hr.astype(np.float64)).max())
            assert e <= tol, f"mode {m}, K={Ks[i]}: max |HP - HP_fp64| = {e:.3e}"
            assert abs(ll[i] - llr) <= 1e-6 * sites + ll_tol, (m, Ks[i])


@pytest.mark.gpu
def test_confident_likelihoods_against_all_states():
    """Forty sites where every panel haplotype carries alt and the target is ref for
    certain (likelihoods 1 and 1e-10, the clamp): each scales by up to 1e10 what is
    not a state, so that four of a block's 16 sites would overflow an unused slot.
    State counts with unused slots in either kernel, all precision modes: finite HP
    within 1e-5 of FP64 (BF16 rows: 5e-3), the log-likelihood within 1e-6 per site
    (BF16: 2^-8 more)."""
    from glimpse_b200 import native, synth
    from oracle import oracle as O
    L, run = 260, slice(90, 130)
    w = synth.make_panel_and_targets(1000, L, 0.2, 0.0, 2, ("uniform", 0.4, 2.0), ("fixed", 200), seed=67,
                                     sparse_maf=0.005)
    P, T = w.panel, w.targets
    P.hvar[run], P.calt[run], P.cref[run], P.major[run] = 255, 1000, 0, 1
    rng = np.random.default_rng(3)
    Ks = [1, 2, 3, 127, 130, 255, 257, 520]
    states = [np.sort(rng.choice(1000, size=K, replace=False)).astype(np.uint32) for K in Ks]
    flats = np.stack([T.flat[i % 2] for i in range(len(Ks))])
    flats[:, run] = 0
    hls = np.stack([init_hl(T.gl[i % 2], flats[i]) for i in range(len(Ks))])
    hls[:, 2 * run.start:2 * run.stop:2], hls[:, 2 * run.start + 1:2 * run.stop:2] = 1.0, 1e-10
    ref = [O.restate_impute(P, s, hl, fl, precision=64) for s, hl, fl in zip(states, hls, flats)]
    ctx = native.Context(P)
    try:
        for m, tol, ll_tol in ((native.PRECISION_FULL, TOL, None), (native.PRECISION_CKPT_F32, TOL, 0.0),
                               (native.PRECISION_CKPT_BF16, 5e-3, 2.0 ** -8)):
            ctx.set_precision(m)
            hp = ctx.impute_batch(states, hls, flats)
            assert np.isfinite(hp).all(), m
            for i, (hr, llr) in enumerate(ref):
                e = float(np.abs(hp[i].astype(np.float64) - hr.astype(np.float64)).max())
                assert e <= tol, f"mode {m}, K={Ks[i]}: max |HP - HP_fp64| = {e:.3e}"
                if ll_tol is not None:
                    assert abs(ctx.loglik(len(Ks))[i] - llr) <= 1e-6 * L + ll_tol, (m, Ks[i])
    finally:
        ctx.close()


@pytest.mark.gpu
def test_checkpointed_modes_need_less_memory():
    """Device memory of a context after one call of 12 sets of 2,000 states (rows of
    2,048) over 40,000 sites, all polymorphic. Full precision keeps half a byte per cell
    (site, state), in a buffer with 1/8 to spare; the modes share all else but 4 bytes
    per site. FP32 checkpoints: 1/4 byte and windows of 1/32; BF16: 1/16 and windows of
    1/16; each with 1/8 to spare and 1/100 for what is not per cell."""
    import torch
    from glimpse_b200 import native, synth
    L, n = 40000, 12
    w = synth.make_panel_and_targets(2048, L, 1.3, 0.0, 2, ("uniform", 0.5, 2.0), ("fixed", 200), seed=53)
    P, T = w.panel, w.targets
    rng = np.random.default_rng(1)
    states = [np.sort(rng.choice(2048, size=2000, replace=False)).astype(np.uint32) for _ in range(n)]
    hls = np.stack([init_hl(T.gl[i % 2], T.flat[i % 2]) for i in range(n)])
    flats = np.stack([T.flat[i % 2] for i in range(n)])
    modes = (native.PRECISION_FULL, native.PRECISION_CKPT_F32, native.PRECISION_CKPT_BF16)
    taken = {}
    for _ in range(2):  # the first pass loads the kernels
        for m in modes:
            before = torch.cuda.mem_get_info()[0]
            ctx = native.Context(P)
            try:
                ctx.set_precision(m)
                ctx.impute_batch(states, hls, flats)
                taken[m] = before - torch.cuda.mem_get_info()[0]
            finally:
                ctx.close()
    cells = n * L * 2048
    shared = taken[modes[0]] - 0.5 * 9 / 8 * cells
    assert taken[modes[1]] - shared <= ((1 / 4 + 1 / 32) * 9 / 8 + 1 / 100) * cells
    assert taken[modes[2]] - shared <= ((1 / 16 + 1 / 16) * 9 / 8 + 1 / 100) * cells


@pytest.mark.gpu
@pytest.mark.parametrize("mode", [1, 2])
def test_windows_chunks_and_classes_give_the_same_bits(mode, monkeypatch):
    """The number of windows follows the batch, and with more than four classes of 256
    states some run their blocks behind their chains on one stream: eight classes in
    one call, four, each set alone, and in chunks under a budget of 4 MB must give the
    same posteriors and log-likelihoods, bit for bit."""
    from glimpse_b200 import native, synth
    w = synth.make_panel_and_targets(2100, 9000, 0.3, 0.3, 2, ("uniform", 0.5, 2.0), ("fixed", 200), seed=57,
                                     sparse_maf=0.005)
    P, T = w.panel, w.targets
    rng = np.random.default_rng(mode)
    Ks = [2, 300, 600, 900, 1100, 1400, 1700, 2048]
    states = [np.sort(rng.choice(2100, size=K, replace=False)).astype(np.uint32) for K in Ks]
    hls = np.stack([init_hl(T.gl[i % 2], T.flat[i % 2]) for i in range(len(Ks))])
    flats = np.stack([T.flat[i % 2] for i in range(len(Ks))])
    ctx = native.Context(P)

    def run(idx):
        hp = ctx.impute_batch([states[i] for i in idx], hls[idx], flats[idx])
        return hp, np.asarray(ctx.loglik(len(idx)))

    try:
        ctx.set_precision(mode)
        hp, ll = run(list(range(8)))
        monkeypatch.setenv("GLIMPSE_B200_STORE_BUDGET_MB", "4")
        parts = [(list(range(8)), run(list(range(8))))]
        monkeypatch.delenv("GLIMPSE_B200_STORE_BUDGET_MB")
        parts += [(idx, run(idx)) for idx in [[0, 1, 2, 3], [4, 5, 6, 7]] + [[i] for i in range(8)]]
        for idx, (h, l) in parts:
            assert np.array_equal(h, hp[idx]) and np.array_equal(l, ll[idx]), idx
    finally:
        ctx.close()

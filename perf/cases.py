"""The work that a user of the library has it do, as timed cases.

A case is a call sequence through glimpse_b200.native on a seeded synthetic
panel (glimpse_b200.synth) with targets drawn from the seed. Its "op" is one of

  impute   one call of impute_batch (imputation_hmm::computePosteriors) for n
           haplotypes with conditioning sets of kmin..kmax states; precision 0
           keeps every forward row, 1 / 2 the checkpointed FP32 / BF16 variant
  rephase  one call of rephase_batch (phasing_hmm::rephaseHaplotypes) for n
           diploid targets
  run      a Gibbs run over n targets (the last `haploid` of them haploid):
           targets in, 1 init + burnin + main iterations, results out; learned
           1 selects states with the learned proposal's network
  train    one training step of the learned proposal's network on n rows
  gl       FORMAT/PL or FORMAT/GL values of n targets turned into phred bytes

The panel (reference haplotypes x sites over mb megabases, a share `rare` of
the sites rare) stays on the GPU in one context, as a program keeps it while
batches of targets come and go; only one panel's context is held at a time.
"""
import collections
import math

import numpy as np
import torch

from glimpse_b200 import native, synth

_POOL = 16        # held-out diploid targets per panel, from which a seed's targets are recombined
_KCAND = 1024     # candidates of the learned proposal (its default)
_panels = collections.OrderedDict()
_held = {}        # the one context in use: {key: context}


def listed():
    small = dict(N=1000, L=20000, mb=2.0, rare=0.0)
    mid = dict(N=2503, L=30011, mb=1.3, rare=0.6)
    large = dict(N=10000, L=150000, mb=4.0, rare=0.8)
    return [
        # one haplotype against a small panel: the smallest call, a single chain's latency
        dict(name="impute-1-small", op="impute", precision=0, n=1, kmin=500, kmax=500, **small),
        # a complete run (5 burn-in + 15 main) for a single sample, as the reference is run per sample
        dict(name="run-1-small", op="run", learned=0, n=1, haploid=0, burnin=5, main=15, kmin=500, kmax=500,
             kinit=500, **small),
        # a few dozen haplotypes on a panel of odd sizes with uneven sets
        dict(name="impute-37-mid", op="impute", precision=0, n=37, kmin=130, kmax=900, **mid),
        # an ordinary run with some haploid targets (chromosome X) and the writer's record fields
        dict(name="run-24-mid", op="run", learned=0, n=24, haploid=5, burnin=2, main=3, kmin=150, kmax=700, kinit=600,
             **mid),
        # the phasing method on its own, small batch
        dict(name="rephase-11-mid", op="rephase", n=11, kmin=130, kmax=900, **mid),
        # many haplotypes on a whole 4 Mb chunk
        dict(name="impute-64-large", op="impute", precision=0, n=64, kmin=400, kmax=1200, **large),
        # the memory-saving variant on the same chunk
        dict(name="impute-32-large-bf16", op="impute", precision=2, n=32, kmin=400, kmax=1200, **large),
        # the batched workload: 256 targets on the chunk, every stage once
        dict(name="run-256-large", op="run", learned=0, n=256, haploid=0, burnin=1, main=1, kmin=400, kmax=1200,
             kinit=1000, **large),
        # a smaller batch on the chunk: the last batch of a cohort, low K
        dict(name="run-40-large", op="run", learned=0, n=40, haploid=0, burnin=1, main=1, kmin=160, kmax=480,
             kinit=1000, **large),
        # the learned proposal picks small sets from many candidates
        dict(name="run-64-learned", op="run", learned=1, n=64, haploid=0, burnin=1, main=1, kmin=160, kmax=480,
             kinit=1000, **large),
        # a training step of the proposal's network
        dict(name="train-16384", op="train", n=16384),
        # a chunk's genotype likelihoods as the VCF reader hands them over
        dict(name="gl-64-large", op="gl", n=64, L=150000, fmt="PL", haploid=0),
    ]


def draw(rng):
    def log(a, b):
        return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))

    op = rng.choice(["impute", "impute", "impute", "rephase", "rephase", "run", "run", "run", "learned", "train", "gl"])
    if op == "train":
        return dict(op=op, n=log(500, 60000))
    if op == "gl":
        n = log(2, 64)
        return dict(op=op, n=n, L=log(2000, 150000), fmt=rng.choice(["PL", "GL"]), haploid=rng.choice([0, n // 3]))
    L = log(3000, 150000)
    N = log(3000, 10000) if op == "learned" else log(400, 10000)
    rare = rng.choice([0.0, 0.6, 0.8]) if L < 40000 else 0.8
    panel = dict(N=N, L=L, mb=round(max(0.3, L * 4.0 / 150000), 3), rare=rare)
    cap = min(1200, N // 2)
    kmin = log(40, cap // 2)
    kmax = rng.randint(kmin, min(cap, 3 * kmin))
    if op == "impute":
        return dict(op=op, precision=rng.choice([0, 0, 0, 1, 2]), n=log(1, 64), kmin=kmin, kmax=kmax, **panel)
    if op == "rephase":
        return dict(op=op, n=log(1, 64), kmin=kmin, kmax=kmax, **panel)
    # runs: many iterations on short chunks, few on long ones
    total = min(21, 450000 // L)
    burnin = rng.randint(1, max(1, min(5, total - 2)))
    main = max(1, min(15, total - 1 - burnin))
    n = log(1, 200)
    return dict(op="run", learned=int(op == "learned"), n=n, haploid=rng.choice([0, 0, n // 4]), burnin=burnin,
                main=main, kmin=kmin, kmax=kmax, kinit=min(1000, N // 2), **panel)


# ---- panels, targets and genotype likelihoods ----

def _panel(case):
    """The synthetic panel of these sizes, its sparse PBWT and the pool of held-out haplotypes."""
    key = (case["N"], case["L"], case["mb"], case["rare"])
    if key not in _panels:
        while len(_panels) >= 3:
            _panels.popitem(last=False)
        N, L, mb, rare = key
        w = synth.make_panel_and_targets(N, L, mb, rare, _POOL, ("fixed", 0.01), ("fixed", 1), seed=N + L,
                                         sparse_maf=max(0.001, 3.5 / N))
        _panels[key] = (w.panel, native.build_sparse_pbwt(w.panel), w.targets.truth.reshape(2 * _POOL, L))
    return _panels[key]


def _context(case):
    """The context of the case's panel; another panel's context is closed first."""
    opts = (case.get("kinit", 1000), case.get("learned", 0))
    key = (case["N"], case["L"], case["mb"], case["rare"]) + opts
    if key not in _held:
        for old in _held.values():
            old.close()
        _held.clear()
        panel, (ypacked, asmall_off, asmall), _ = _panel(case)
        ctx = native.Context(panel, kinit=opts[0], kpbwt=min(2000, case["N"] - 1), ypacked=ypacked,
                             asmall=(asmall_off, asmall))
        if opts[1]:
            ctx.mlp_set_params(_weights(17))
        _held[key] = ctx
    return _held[key]


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) * 7919 + 11)


def _haplotypes(case, n, g):
    """n target haplotypes: recombinants of the panel's held-out pool, [n, L] on the GPU."""
    pool = torch.from_numpy(_panel(case)[2]).cuda()
    L = pool.shape[1]
    cuts = 24
    place = torch.sort(torch.randint(0, L, (n, cuts), generator=g, device="cuda"), dim=1).values
    which = torch.randint(0, pool.shape[0], (n, cuts + 1), generator=g, device="cuda")
    out = torch.empty((n, L), dtype=torch.uint8, device="cuda")
    site = torch.arange(L, device="cuda")
    for i in range(n):
        piece = torch.searchsorted(place[i], site, right=True)
        out[i] = pool[which[i][piece], site]
    return out


def _likelihoods(truth, coverage, g):
    """Poisson read counts over diploid truth [n, 2, L] as phred bytes [n, L, 3] and flat flags [n, L]."""
    n, _, L = truth.shape
    e = 0.01
    p = torch.tensor([e, 0.5, 1 - e], dtype=torch.float64, device="cuda")
    gl = torch.empty((n, L, 3), dtype=torch.uint8, device="cuda")
    flat = torch.empty((n, L), dtype=torch.uint8, device="cuda")
    for i in range(n):
        depth = torch.poisson(coverage[i].expand(L), generator=g)
        dose = truth[i].sum(0, dtype=torch.long)
        alt = torch.binomial(depth, p[dose].float(), generator=g).double()
        ref = depth.double() - alt
        ll = alt[:, None] * torch.log10(p) + ref[:, None] * torch.log10(1 - p)
        ll = ll - ll.max(1, keepdim=True).values
        gl[i] = torch.clamp(torch.round(-10 * ll), max=255).to(torch.uint8)
        flat[i] = ((gl[i, :, 0] == gl[i, :, 1]) & (gl[i, :, 0] == gl[i, :, 2])).to(torch.uint8)
    return gl, flat


def _hap_likelihoods(gl, flat):
    """A haplotype's likelihood pairs [n, 2L] from diploid phred bytes, as the init iteration has them."""
    x = torch.pow(10.0, gl.double() / -10.0)
    x = x / x.sum(2, keepdim=True)
    hl = torch.stack([x[..., 0] + 0.5 * x[..., 1], x[..., 2] + 0.5 * x[..., 1]], dim=2)
    hl[flat != 0] = 0.5
    return hl.clamp(min=1e-10).float().reshape(gl.shape[0], -1).cpu().numpy()


def _state_sets(case, n, g):
    ks = torch.randint(case["kmin"], case["kmax"] + 1, (n,), generator=g, device="cuda").tolist()
    return [torch.sort(torch.randperm(case["N"], generator=g, device="cuda")[:k]).values.cpu().numpy().astype(np.uint32)
            for k in ks]


def _weights(seed):
    """He-uniform parameters of the proposal's network in its packed order (W1 256x64 with 48 used columns, b1,
    W2 256x256, b2, w3, b3)."""
    r = np.random.default_rng(seed)
    w1 = np.zeros((256, 64))
    w1[:, :48] = r.uniform(-1, 1, (256, 48)) * math.sqrt(6 / 48)
    return np.concatenate([w1.ravel(), 0.1 * r.uniform(-1, 1, 256), (r.uniform(-1, 1, 65536) * math.sqrt(6 / 256)),
                           0.1 * r.uniform(-1, 1, 256), r.uniform(-1, 1, 256) * math.sqrt(3 / 256),
                           [0.1]]).astype(np.float32)


def _pinned(a):
    return a.cpu().pin_memory()


def prepare(case, seed):
    op = case["op"]
    g = _generator(seed)
    s = dict(op=op, case=case)
    if op == "train":
        n = case["n"]
        p = dict(N=400, L=3000, mb=0.3, rare=0.0)
        panel, (ypacked, off, idx), _ = _panel(p)
        s["ctx"] = native.Context(panel, kinit=150, kpbwt=200, ypacked=ypacked, asmall=(off, idx))
        s["ctx"].mlp_set_params(_weights(seed))
        s["x"], s["y"], s["wt"] = _rows(n, g)
        return s
    if op == "gl":
        n, L = case["n"], case["L"]
        p = dict(N=400, L=3000, mb=0.3, rare=0.0)
        panel, (ypacked, off, idx), _ = _panel(p)
        s["ctx"] = native.Context(panel, kinit=150, kpbwt=200, ypacked=ypacked, asmall=(off, idx))
        dose = torch.randint(0, 2, (n, 2, L), generator=g, device="cuda").to(torch.uint8)
        gl, _ = _likelihoods(dose, torch.full((n,), 1.0, device="cuda"), g)
        v = gl.transpose(0, 1).contiguous()
        absent = torch.rand((L, n), generator=g, device="cuda") < 0.02
        if case["fmt"] == "PL":
            src = v.to(torch.int32)
            src[absent] = -(1 << 31)  # htslib's bcf_int32_missing
        else:
            src = (v.to(torch.float32) / -10.0).view(torch.int32)
            src[absent] = 0x7F800001  # htslib's bcf_float_missing
            src = src.view(torch.float32)
        s["src"] = src.cpu().numpy()
        s["ploidy"] = np.full(n, 2, np.int32)
        s["ploidy"][n - case["haploid"]:] = 1
        return s
    n = case["n"]
    s["ctx"] = _context(case)
    truth = _haplotypes(case, 2 * n, g).reshape(n, 2, -1)
    coverage = 0.5 + 1.5 * torch.rand(n, generator=g, device="cuda")
    gl, flat = _likelihoods(truth, coverage, g)
    if op == "impute":
        s["states"] = _state_sets(case, n, g)
        s["hl"] = _hap_likelihoods(gl, flat)
        s["flat"] = flat.cpu().numpy()
    elif op == "rephase":
        s["states"] = _state_sets(case, n, g)
        swap = torch.rand(truth.shape, generator=g, device="cuda") < 0.02
        h = (truth ^ swap.to(torch.uint8)).cpu().numpy()
        s["h0"], s["h1"], s["flat"] = np.ascontiguousarray(h[:, 0]), np.ascontiguousarray(h[:, 1]), flat.cpu().numpy()
    else:
        L = case["L"]
        s["gl"], s["flat"] = _pinned(gl), _pinned(flat)
        ploidy = torch.full((n,), 2, dtype=torch.int32)
        ploidy[n - case["haploid"]:] = 1
        s["ploidy"] = ploidy.pin_memory()
        s["k"] = _pinned(torch.randint(case["kmin"], case["kmax"] + 1, (n,), generator=g, device="cuda").int())
        s["ds"] = torch.empty((n, L), dtype=torch.float32).pin_memory()
        s["gt0"], s["gt1"] = (torch.empty((n, L), dtype=torch.uint8).pin_memory() for _ in range(2))
    del truth, gl, flat
    torch.cuda.empty_cache()
    return s


def _rows(n, g):
    """Feature rows, labels and weights of a learnable problem."""
    x = torch.randn((n, 48), generator=g, device="cuda")
    w = torch.randn(48, generator=g, device="cuda")
    y = (torch.rand(n, generator=g, device="cuda") < torch.sigmoid(x @ w / 48 ** 0.5 * 3)).float()
    wt = 0.5 + 1.5 * torch.rand(n, generator=g, device="cuda")
    return x.cpu().numpy(), y.cpu().numpy(), wt.cpu().numpy()


def run(s):
    op, ctx, case = s["op"], s["ctx"], s["case"]
    if op == "impute":
        ctx.set_precision(case["precision"])
        hp = ctx.impute_batch(s["states"], s["hl"], s["flat"])
        if case["precision"] == 0:
            return {"hp": hp}
        return {"hp": hp, "loglik": ctx.loglik(case["n"])}
    if op == "rephase":
        h0, h1 = ctx.rephase_batch(s["states"], s["h0"], s["h1"], s["flat"], 3)
        return {"h0": h0, "h1": h1}
    if op == "train":
        loss, grad = ctx.mlp_train_step(s["x"], s["y"], s["wt"], lr=1e-3, grad=True)
        return {"loss": loss, "grad": grad, "params": ctx.mlp_params()}
    if op == "gl":
        gl, flat = ctx.gl_from_format(case["fmt"], s["src"], s["ploidy"])
        return {"gl": gl, "flat": flat}
    ctx.set_precision(0)
    ctx.set_targets_raw(case["n"], s["gl"].data_ptr(), s["flat"].data_ptr(), s["ploidy"].data_ptr(), s["k"].data_ptr())
    if case["learned"]:
        ctx.learned_enable(True, kcand=_KCAND)
    ctx.run(case["burnin"], case["main"])
    ctx.gp_raw(s["ds"].data_ptr(), s["gt0"].data_ptr(), s["gt1"].data_ptr())
    out = {"ds": s["ds"], "gt0": s["gt0"], "gt1": s["gt1"]}
    if case["haploid"]:
        gp, raf, af, info = ctx.output_records()
        # a haploid target's third value is a marker, not a number
        out.update(gp=gp[..., :2], raf=raf, af=af, info=info)
    return out


# ---- what a pass cannot do without ----

def _poly(case, k):
    """Expected polymorphic sites of a set of k states: the common sites and the rare sites that a state carries."""
    carriers = 2.5
    return case["L"] * ((1 - case["rare"]) + case["rare"] * (1 - (1 - min(1.0, k / case["N"])) ** carriers))


def work(case):
    n, op = case["n"], case["op"]
    if op == "train":
        mac = n * (64 * 256 + 256 * 256 + 256)
        return {"bytes": 4.0 * n * 50 + 4.0 * 83000 * 3, "flops": 6.0 * mac}
    L = case["L"]
    if op == "gl":
        return {"bytes": n * L * (16.0 if case["haploid"] < n else 12.0), "flops": 0.0}
    k = (case["kmin"] + case["kmax"]) / 2
    cells = _poly(case, k) * k  # per haplotype and pass over the set
    if op == "impute":
        # likelihoods and flags in, posteriors out, the set's alleles; two recursions and the posterior sums
        return {"bytes": n * (17.0 * L + cells / 8), "flops": n * cells * 10.0}
    if op == "rephase":
        return {"bytes": n * (5.0 * L + cells / 8), "flops": n * cells * 2 * 8 * 4.0}
    iters = case["burnin"] + case["main"]
    k0 = case["kinit"]
    cells = iters * cells + _poly(case, k0) * k0
    haps, dips = 2 * n - case["haploid"], n - case["haploid"]
    return {"bytes": n * 10.0 * L + n * cells / 8, "flops": haps * cells * 10.0 + dips * cells * 2 * 8 * 4.0}


# ---- 64-bit values ----

def _exact_impute(case, seed):
    """The Li-Stephens forward-backward over explicit conditioning sets in 64 bits, all haplotypes side by side."""
    n, N, L = case["n"], case["N"], case["L"]
    g = _generator(seed)
    panel = _panel(case)[0]
    truth = _haplotypes(case, 2 * n, g).reshape(n, 2, -1)
    coverage = 0.5 + 1.5 * torch.rand(n, generator=g, device="cuda")
    gl, flat_d = _likelihoods(truth, coverage, g)
    sets = _state_sets(case, n, g)
    hl = _hap_likelihoods(gl, flat_d).astype(np.float64).reshape(n, L, 2)
    flat = flat_d.cpu().numpy().astype(bool)
    del truth, gl, flat_d
    ed = float(np.float32(1e-12))
    ee = float(np.float32(1.0 - ed))
    common = panel.flag_common != 0
    rows = np.cumsum(common) - 1
    kmax = max(len(x) for x in sets)
    hvar = torch.from_numpy(panel.hvar).cuda()
    polys, bits = [], []
    for x in sets:
        carried = [panel.shap_sites[panel.shap_off[h]:panel.shap_off[h + 1]] for h in x]
        poly = common.copy()
        poly[np.concatenate(carried)] = True
        sites = np.flatnonzero(poly)
        where = np.full(L, -1, np.int64)
        where[sites] = np.arange(sites.size)
        b = torch.from_numpy(panel.major[sites]).cuda()[:, None].repeat(1, len(x))
        c = common[sites]
        ids = torch.from_numpy(x.astype(np.int64)).cuda()
        words = hvar[torch.from_numpy(rows[sites[c]]).cuda()][:, ids >> 3]
        b[torch.from_numpy(c).cuda()] = (words >> (7 - (ids & 7)).to(torch.uint8)) & 1
        at = np.concatenate(carried)
        col = np.repeat(np.arange(len(x)), [v.size for v in carried])
        b[torch.from_numpy(where[at]).cuda(), torch.from_numpy(col).cuda()] = torch.from_numpy(1 - panel.major[at]).cuda()
        polys.append(sites)
        bits.append(b)
    most = max(x.size for x in polys)
    B = torch.zeros((most, n, kmax), dtype=torch.bool, device="cuda")
    E = np.ones((most, n, 2))
    T = np.zeros((most, n))
    last = np.zeros((most, n), bool)
    for i, (sites, b) in enumerate(zip(polys, bits)):
        m = sites.size
        B[:m, i, :b.shape[1]] = b != 0
        h = hl[i, sites]
        p = np.stack([h[:, 0] * ee + h[:, 1] * ed, h[:, 0] * ed + h[:, 1] * ee], 1)
        e = p / p.sum(1, keepdims=True)
        e[flat[i, sites] | (panel.lq[sites] != 0)] = 1.0
        E[:m, i] = e
        d = -np.expm1(-0.04 * 100000 / N * np.diff(panel.cm[sites]))
        T[:m - 1, i] = np.clip(d, 1e-7, 1 - 1e-7).astype(np.float32)
        last[m - 1, i] = True
    K = torch.tensor([float(len(x)) for x in sets], dtype=torch.float64, device="cuda")
    valid = (torch.arange(kmax, device="cuda")[None, :] < K[:, None]).double()
    E, T, last = (torch.from_numpy(v).cuda() for v in (E, T, last))
    alpha = torch.empty((most, n, kmax), dtype=torch.float64, device="cuda")
    ll = torch.zeros((most, n), dtype=torch.float64, device="cuda")
    pre = valid / K[:, None]
    for l in range(most):
        a = pre * torch.where(B[l], E[l, :, 1:], E[l, :, :1])
        alpha[l] = a
        tot = a.sum(1, keepdim=True)
        ll[l] = tot[:, 0].log()
        pre = (a * ((1 - T[l])[:, None] / tot) + (T[l] / K)[:, None]) * valid
    ph = torch.zeros((most, n, 2), dtype=torch.float64, device="cuda")
    beta = torch.zeros((n, kmax), dtype=torch.float64, device="cuda")
    for l in range(most - 1, -1, -1):
        tot = beta.sum(1, keepdim=True)
        pc = torch.where(tot > 0, beta * ((1 - T[l])[:, None] / tot) + (T[l] / K)[:, None], valid)
        pc = torch.where(last[l][:, None], valid, pc) * valid
        d = alpha[l] * pc
        one = (d * B[l]).sum(1)
        ph[l, :, 1] = one
        ph[l, :, 0] = (d * ~B[l]).sum(1)
        scale = torch.where(last[l][:, None], 1 / K[:, None], torch.ones_like(tot))
        beta = pc * scale * torch.where(B[l], E[l, :, 1:], E[l, :, :1])
    ph, E, ll = ph.cpu().numpy(), E.cpu().numpy(), ll.cpu().numpy()
    hp = np.empty((n, L, 2))
    logs = np.empty(n)
    base = np.where(panel.major[:, None] != 0, [[ed, ee]], [[ee, ed]])
    for i, sites in enumerate(polys):
        m = sites.size
        logs[i] = ll[:m, i].sum()
        out = base.copy()
        out[~flat[i]] *= hl[i][~flat[i]]
        q = ph[:m, i] / E[:m, i]
        q = np.stack([q[:, 0] * ee + q[:, 1] * ed, q[:, 0] * ed + q[:, 1] * ee], 1)
        f = flat[i, sites]
        q[~f] *= hl[i, sites][~f]
        out[sites] = q
        hp[i] = out / out.sum(1, keepdims=True)
    return hp.reshape(n, 2 * L), logs


def _exact_train(case, seed):
    """Loss and packed gradient of the network in 64 bits without any rounding."""
    x, y, wt = (torch.from_numpy(v).cuda().double() for v in _rows(case["n"], _generator(seed)))
    p = torch.from_numpy(_weights(seed)).cuda().double().requires_grad_()
    o = np.cumsum([0, 256 * 64, 256, 65536, 256, 256, 1])
    w1, b1, w2, b2, w3, b3 = (p[o[i]:o[i + 1]] for i in range(6))
    h = torch.relu(x @ w1.reshape(256, 64)[:, :48].T + b1)
    z = torch.relu(h @ w2.reshape(256, 256).T + b2) @ w3 + b3
    loss = torch.nn.functional.binary_cross_entropy_with_logits(z, y, wt, reduction="sum") / case["n"]
    loss.backward()
    return float(loss), p.grad.cpu().numpy()


def exact(case, seed):
    if case["op"] == "impute":
        if _poly(case, case["kmax"]) * case["n"] * case["kmax"] > 6e9:
            return None  # 8 bytes a cell would not fit the card comfortably
        v = _exact_impute(case, seed)
        return {"hp": v[0]} if case["precision"] == 0 else {"hp": v[0], "loglik": v[1]}
    if case["op"] == "train":
        loss, grad = _exact_train(case, seed)
        return {"loss": loss, "grad": grad, "params": None}
    return None

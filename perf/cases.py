"""Workloads of the GSEA pipeline for timing and comparing builds.

A case names how the pipeline is called (`call`), the problem's size (genes,
samples, sets, permutations), the ranking metric, the precision and the form.
`prepare` makes what a user's program holds before the call, `run` is one
call, `exact` the same result in 64-bit arithmetic with plain torch.

Data: log2-like expression ~ N(8, sd_g^2), sd_g ~ U[0.3, 3], clamped at 1e-3,
2.5 % of the genes shifted by +-U[0.5, 2] in class B, gene sets of 15 to 500
members of which 20 % are enriched for shifted genes -- the distributions of
the benchmark's synthetic workloads (cudagsea_gb300/synthetic.py).
"""
import math

import numpy as np
import torch

from cudagsea_gb300 import _native as N
from cudagsea_gb300 import allocator, api
from cudagsea_gb300.synthetic import GseaInput

FORMS = {"plain": N.FORM_PLAIN, "chosen": N.FORM_CHOSEN, "chosen_fp64": N.FORM_CHOSEN_FP64}
SET_MIN, SET_MAX = 15, 500


def _case(call, genes, samples, sets, perms, metric="twopass_signal2noise", precision=32, form="plain",
          ascending=False, **more):
    c = dict(call=call, genes=genes, samples=samples, sets=sets, perms=perms, metric=metric, precision=precision,
             form=form, ascending=ascending)
    c.update(more)
    return c


def listed():
    return [
        # the repository's small workload: a hallmark-sized collection on a
        # filtered table, where launches and latency count
        dict(_case("execute", 2000, 40, 50, 1024), name="small_plain"),
        # the benchmark's headline problem, in the reference's arithmetic ...
        dict(_case("execute", 20000, 200, 1000, 1000), name="full_plain"),
        # ... with the tensor-core class statistics ...
        dict(_case("execute", 20000, 200, 1000, 1000, form="chosen"), name="full_chosen"),
        # ... and with doublePrecision = TRUE
        dict(_case("execute", 20000, 200, 1000, 1000, precision=64), name="full_double"),
        # one of the accurate accumulators, a mid-sized study, odd sizes
        dict(_case("execute", 15013, 121, 403, 500, metric="overkill_t_test"), name="accurate_ttest"),
        # a small study with many permutations, ranked in ascending order
        dict(_case("execute", 7411, 57, 257, 2000, metric="onepass_t_test", ascending=True), name="ascending_ttest"),
        # a large cohort (600 samples) with a large collection
        dict(_case("execute", 20000, 600, 2000, 1000, metric="twopass_t_test", form="chosen"), name="cohort_chosen"),
        # transcript-level tables: more genes than one SM's registers sort
        dict(_case("execute", 60000, 100, 500, 300, metric="naive_diff_of_classes"), name="transcripts"),
        # the headline problem from the host: tables in pinned memory, scores
        # and statistics back, a plan kept for one table after the other
        dict(_case("run_host", 20000, 200, 1000, 1000, form="chosen"), name="host_tables"),
        # the R / C one-shot call on ordinary host arrays
        dict(_case("one_shot", 10007, 60, 200, 1000, metric="onepass_signal2noise"), name="one_shot"),
        # several uneven studies in one call (batched instances)
        dict(_case("batch", 30000, 300, 1500, 300, form="chosen", instances=12), name="batch_uneven"),
        # a large collection with many permutations through the adaptive
        # permutation allocator
        dict(_case("adaptive", 20000, 200, 5000, 20000, form="chosen"), name="allocator"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    call = rng.choice(["execute"] * 7 + ["run_host", "one_shot", "batch"])
    precision = 64 if call != "batch" and rng.random() < 0.2 else 32
    form = "plain" if precision == 64 or call == "one_shot" else rng.choice(["plain", "chosen", "plain", "chosen",
                                                                              "chosen_fp64"])
    metric = rng.choice(api.METRICS)
    genes, samples = _log_int(rng, 2000, 60000), _log_int(rng, 20, 600)
    sets, perms = _log_int(rng, 50, 5000), _log_int(rng, 64, 2000)
    ascending = call != "batch" and rng.random() < 0.25
    # no more than the listed cases ask for: table x permutations (a quarter
    # of it in 64 bits and with the accurate accumulators) and scores
    slow = precision == 64 or metric.startswith(("stable", "overkill"))
    table = 2.0e9 if slow else 1.0e10
    scores = 5.0e5 if precision == 64 else 1.5e6
    more = {}
    if call == "batch":
        genes, sets, more = min(genes, 30000), min(sets, 1500), {"instances": rng.randint(2, 12)}
        table, scores = table / more["instances"], scores / more["instances"]
    perms = max(16, min(perms, int(table / (genes * samples)), int(scores / sets)))
    return _case(call, genes, samples, sets, perms, metric, precision, form, ascending, **more)


# ---------------------------------------------------------------- inputs
def _problem(genes, samples, sets, perms, rng):
    """One study: table [samples][genes] float32, labels, gene sets (CSR)."""
    n_b = int(np.clip(round(samples * rng.uniform(0.4, 0.6)), 1, samples - 1))
    labels = np.zeros(samples, np.uint8)
    labels[rng.permutation(samples)[:n_b]] = 1
    sd = rng.uniform(0.3, 3.0, genes).astype(np.float32)
    x = rng.standard_normal((samples, genes), dtype=np.float32)
    x *= sd
    x += np.float32(8.0)
    shifted = rng.choice(genes, size=max(1, genes // 40), replace=False)
    amount = (rng.uniform(0.5, 2.0, shifted.size) * rng.choice([-1.0, 1.0], shifted.size)).astype(np.float32)
    x[np.ix_(labels == 1, shifted)] += amount
    np.maximum(x, np.float32(1e-3), out=x)
    hi = min(SET_MAX, genes)
    members = []
    for n in rng.integers(SET_MIN, hi + 1, sets):
        if rng.random() < 0.2:
            own = rng.choice(shifted, size=min(int(n) // 2, shifted.size), replace=False)
            rest = rng.choice(genes, size=int(n) - own.size, replace=False)
            m = np.union1d(own, rest)
        else:
            m = np.sort(rng.choice(genes, size=int(n), replace=False))
        members.append(m.astype(np.int32))
    off = np.zeros(sets + 1, np.int64)
    off[1:] = np.cumsum([m.size for m in members])
    return GseaInput(x, labels, off, np.concatenate(members), perms)


def _problems(case, seed):
    rng = np.random.default_rng([seed, 103])
    if case["call"] != "batch":
        d = _problem(case["genes"], case["samples"], case["sets"], case["perms"], rng)
        if case["precision"] == 64:  # values with all their 53 bits, as R's numerics have
            d.exprs = d.exprs.astype(np.float64)
            d.exprs *= 1.0 + 2.0 ** -26 * rng.standard_normal(d.exprs.shape)
        return [d]
    out = []
    sizes = np.random.default_rng(17)  # the case's own, whatever the seed
    for _ in range(case["instances"]):  # uneven: up to the case's sizes, down to a sixth of them
        g, s, k = (max(20, int(case[n] * sizes.uniform(1 / 6, 1))) for n in ("genes", "samples", "sets"))
        out.append(_problem(g, s, k, case["perms"], rng))
    return out


class _Device:
    """A device buffer of the library as an array torch can view; keeps its
    owner (a plan, a batch) alive as long as a view of it exists."""

    def __init__(self, owner, which, shape):
        self.owner = owner
        self.__cuda_array_interface__ = {"data": (owner.buffer(which)[0], False), "shape": tuple(shape), "version": 2,
                                         "typestr": np.dtype(owner.dtype).str}


def _results(plan):
    """The plan's scores [sets][permutations] and statistics [5 * sets], in place."""
    k, p = plan.cfg.num_sets, plan.cfg.num_perms
    return {"es": torch.as_tensor(_Device(plan, N.BUF_ES, (k, p)), device="cuda"),
            "stats": torch.as_tensor(_Device(plan, N.BUF_STATS, (5 * k,)), device="cuda")}


def _plan(case, d):
    return api.Plan(d.num_genes, d.num_samples, d.num_sets, d.num_perms, case["metric"], precision=case["precision"],
                    ascending=case["ascending"], form=FORMS[case["form"]])


class _InstancePlan:
    """The buffers of one instance of a batch (gsea_batch_plan in the C ABI)."""

    def __init__(self, batch, i):
        self.batch, self.cfg, self.dtype = batch, batch.cfgs[i], batch.dtype
        self._h = N._p()
        N.check(N.lib().gsea_batch_plan(batch._h, i, self._h))

    buffer = api.Plan.buffer


def _pinned(a):
    t = torch.empty(a.shape, dtype=torch.from_numpy(a).dtype, pin_memory=True)
    t.numpy()[...] = a
    return t.numpy()


def prepare(case, seed):
    torch.cuda.init()
    ds = _problems(case, seed)
    d = ds[0]
    if case["call"] == "batch":
        b = api.Batch(ds, case["metric"], precision=case["precision"], form=FORMS[case["form"]])
        return {"call": "batch", "batch": b, "out": [_results(_InstancePlan(b, i)) for i in range(len(ds))]}
    if case["call"] == "one_shot":
        return {"call": "one_shot", "d": d, "case": dict(case)}
    plan = _plan(case, d)
    if case["call"] == "run_host":
        es = _pinned(np.zeros((d.num_sets, d.num_perms), plan.dtype))
        stats = _pinned(np.zeros(5 * d.num_sets, plan.dtype))
        return {"call": "run_host", "plan": plan, "out": (es, stats),
                "in": [_pinned(a) for a in (d.exprs, d.labels, d.set_offsets, d.set_genes)]}
    plan.set_inputs(d.exprs, d.labels, d.set_offsets, d.set_genes)
    return {"call": case["call"], "plan": plan, "out": _results(plan) if case["call"] == "execute" else None}


def run(state):
    call = state["call"]
    if call == "execute":
        state["plan"].execute()
        return state["out"]
    if call == "batch":
        state["batch"].execute()
        return state["out"]
    if call == "run_host":
        es, stats = state["plan"].run_host(*state["in"], es_out=state["out"][0], stats_out=state["out"][1])
        return {"es": es, "stats": stats}
    if call == "one_shot":
        c, d = state["case"], state["d"]
        es, stats = api.gsea(d.exprs, d.labels, d.set_offsets, d.set_genes, d.num_perms, c["metric"], c["precision"],
                             c["ascending"])
        return {"es": es, "stats": stats}
    # the adaptive test: how many permutations every set received, and the
    # statistics of those
    r = allocator.execute_adaptive(state["plan"])
    return {"counts": r.counts, "stats": state["plan"].read(es=False)[1]}


def work(case):
    """Inputs read once, scores and statistics written once; the class sums (and
    sums of squares) of every permutation and six operations per member and
    permutation.  Uneven instances count as their average size; the adaptive
    test as a twentieth of its scores after a pilot of 1,000 permutations."""
    e = case["precision"] // 8
    n, g, s, k = case.get("instances", 1), case["genes"], case["samples"], case["sets"]
    if n > 1:
        g, s, k = 7 * g // 12, 7 * s // 12, 7 * k // 12
    p = scores = case["perms"]
    if case["call"] == "adaptive":
        scores = min(p, 1000) + max(0, p - 1000) // 20
    members = k * (SET_MIN + SET_MAX) / 2
    moments = 2 if "signal2noise" in case["metric"] or "t_test" in case["metric"] else 1
    return {"bytes": n * (e * g * s + s + 4 * members + 8 * k + e * k * (scores + 5)),
            "flops": n * (2.0 * moments * g * s * p + 6.0 * members * scores)}


# ---------------------------------------------------------------- 64 bits
def _shuffled(labels, perms, seed=42):
    """Class-A indicators [perms][samples]: Fisher-Yates driven by one KISS
    generator per permutation, seeded by its index; permutation 0 as given."""
    m32 = np.uint64(0xFFFFFFFF)

    def hashed(x):
        def shl(v, n):
            return (v << np.uint64(n)) & m32
        x = (x + np.uint64(0x7ed55d16) + shl(x, 12)) & m32
        x = (x ^ np.uint64(0xc761c23c)) ^ (x >> np.uint64(19))
        x = (x + np.uint64(0x165667b1) + shl(x, 5)) & m32
        x = ((x + np.uint64(0xd3a2646c)) & m32) ^ shl(x, 9)
        x = (x + np.uint64(0xfd7046c5) + shl(x, 3)) & m32
        return (x ^ np.uint64(0xb55a4f09)) ^ (x >> np.uint64(16))

    w = (np.arange(perms, dtype=np.uint64) + np.uint64(seed)) & m32
    for _ in range(8):
        x = hashed(w)
        y = hashed(x)
        z = hashed(y)
        w = hashed(z)
    c = np.zeros(perms, np.uint64)
    lab = np.repeat(labels[None, :], perms, 0)
    rows = np.arange(1, perms)
    for i in range(labels.size - 1, 0, -1):
        y = y ^ ((y << np.uint64(5)) & m32)
        y = y ^ (y >> np.uint64(7))
        y = y ^ ((y << np.uint64(22)) & m32)
        t = (z + w + c) & m32
        z, c, w = w, t >> np.uint64(31), t & np.uint64(0x7FFFFFFF)
        x = (x + np.uint64(1411392427)) & m32
        r = ((((x + y + w) & m32) * np.uint64(i + 1)) >> np.uint64(32)).astype(np.int64)[1:]
        a = lab[rows, i].copy()
        lab[rows, i] = lab[rows, r]
        lab[rows, r] = a
    return lab == 0


def _keys(metric, x, in_a):
    """Ranking metric [perms][genes] of table x [samples][genes], float64."""
    la = in_a.to(torch.float64)
    na, nb = la.sum(1, keepdim=True), (1 - la).sum(1, keepdim=True)
    mu = x.mean(0)
    xc = x - mu
    ca, cb = la @ xc / na, (1 - la) @ xc / nb
    ma, mb = ca + mu, cb + mu
    if "log2" in metric:
        return torch.log(ma / mb) * 1.44269504089
    if "ratio" in metric:
        return ma / mb
    if "diff" in metric:
        return ca - cb
    va = (la @ (xc * xc) / na - ca * ca).clamp_min(0)
    vb = ((1 - la) @ (xc * xc) / nb - cb * cb).clamp_min(0)
    if "signal2noise" in metric:
        return (ca - cb) / (torch.maximum(va.sqrt(), 0.2 * ma.abs()) + torch.maximum(vb.sqrt(), 0.2 * mb.abs()))
    return (ca - cb) / (torch.maximum(va, 0.04 * ma.abs()) / na + torch.maximum(vb, 0.04 * mb.abs()) / nb).sqrt()


def _scores(keys, off, genes, ascending):
    """Enrichment scores [sets][perms] of keys [perms][genes]."""
    p, g = keys.shape
    order = torch.sort(keys, dim=1, descending=not ascending, stable=True).indices
    ranks = torch.empty_like(order)
    ranks.scatter_(1, order, torch.arange(g, device=keys.device).expand(p, g))
    genes = torch.as_tensor(genes.astype(np.int64), device=keys.device)
    out = torch.empty((len(off) - 1, p), dtype=torch.float64, device=keys.device)
    for k in range(len(off) - 1):
        m = genes[int(off[k]):int(off[k + 1])]
        n = m.numel()
        r, at = torch.sort(ranks[:, m], dim=1)
        w = torch.gather(keys[:, m].abs(), 1, at)
        total = w.sum(1, keepdim=True)
        miss = (r - torch.arange(n, device=r.device)).to(torch.float64) / max(1, g - n)
        up = torch.cumsum(w, 1) / total - miss
        down = (torch.cumsum(w, 1) - w) / total - miss
        hi, lo = up.max(1).values.clamp_min(0), down.min(1).values.clamp_max(0)
        out[k] = torch.where(hi >= -lo, hi, lo)
    return out


def _statistics(es):
    """ES, NES, NP, FWER and FDR, one after the other, of scores [sets][perms]."""
    k, p = es.shape
    nes = es * (p / es.abs().sum(1, keepdim=True))
    obs, es0 = nes[:, 0].contiguous(), es[:, 0]
    np_ = (es.abs() >= es0.abs()[:, None]).double().mean(1)
    hi, lo = nes.max(0).values.sort().values, nes.min(0).values.sort().values
    fwer = torch.where(obs > 0, p - torch.searchsorted(hi, obs), torch.searchsorted(lo, obs, right=True)) / p

    def at_least(values, x):
        v = values.sort().values
        return (v.numel() - torch.searchsorted(v, x)).double()

    null = nes[:, 1:].reshape(-1)
    q = torch.zeros_like(obs)
    for side in (1.0, -1.0):
        nl, ob = side * null, side * obs
        nl, ob_side = nl[nl >= 0], ob[ob >= 0]
        mine = ob > 0 if side > 0 else ob >= 0
        top = at_least(nl, ob.contiguous()) / max(1, nl.numel())
        bottom = at_least(ob_side, ob.contiguous()) / max(1, ob_side.numel())
        q = torch.where(mine, (top / bottom).clamp_max(1.0), q)
    return torch.cat([es0, obs, np_, fwer, q])


def exact(case, seed):
    if case["call"] == "adaptive":  # its stopping decisions have no other form
        return None
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    out = []
    for d in _problems(case, seed):
        in_a = torch.as_tensor(_shuffled(d.labels, d.num_perms), device=dev)
        x = torch.as_tensor(d.exprs, device=dev).to(torch.float64)
        es = _scores(_keys(case["metric"], x, in_a), d.set_offsets, d.set_genes, case["ascending"])
        out.append({"es": es, "stats": _statistics(es)})
    return out if case["call"] == "batch" else out[0]

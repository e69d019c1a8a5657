"""The work that performance is judged on: calls of the public Python API over the C ABI.

A case is one call on data of the stated shape: a score of one parameter
vector (one step of a search), a batch of candidate vectors scored together,
a whole likelihood search, an ancestral reconstruction, or the p-values. The
species tree belongs to the case; the gene families and the parameters come
from the seed, simulated under the model they are then scored with
(`cafe5_gb300.synth`).

Every evaluation of a search is at new parameters and builds its own
transition matrices (the reference's matrix cache lives for one evaluation).
The contexts here bound their matrix cache below one evaluation's matrices, so
a repeated pass does that work too instead of finding the matrices of the pass
before.
"""
import math

import numpy as np
import torch

from cafe5_gb300 import synth
from cafe5_gb300.engine import BaseModel, Context, GammaModel, LambdaOptimizerScorer, MultipleLambda, Optimizer, SingleLambda
from cafe5_gb300.families import FamilySet, bin_families, global_bounds
from cafe5_gb300.inputs import ErrorModel, RootPrior, discrete_gamma
from cafe5_gb300.tree import parse_newick


def _case(name, op, precision="fp64_ref", taxa=24, age=150.0, families=10000, root=8.0, lam=0.002, K=1, alpha=0.5,
          candidates=1, clade=False, eps=0.0, heavy=0.0, sims=0, tree=0):
    c = dict(op=op, precision=precision, taxa=taxa, age=age, families=families, root=root, lam=lam, K=K, alpha=alpha,
             candidates=candidates, clade=clade, eps=eps, heavy=heavy, sims=sims, tree=tree)
    return dict(c, name=name) if name else c


def listed():
    return [
        # the smallest calls: one search step on a hundred families of a small clade
        _case("score_8taxa_100", "score", "mixed_tf32x3", taxa=8, age=60.0, families=100, root=3.0, lam=0.004, tree=1),
        # the plain base model at the reference's global bounds (the default precision)
        _case("score_12taxa_1k_ref", "score", "fp64_ref", taxa=12, age=100.0, families=1000, root=5.0, lam=0.0025),
        # a whole search for lambda on that data: what a user runs first
        _case("fit_12taxa_1k_ref", "fit", "fp64_ref", taxa=12, age=100.0, families=1000, root=5.0, lam=0.0025),
        # odd sizes: 17 taxa, 2,777 families, five rate categories, an error model
        _case("score_gamma5_17taxa_2777_err", "score", "fp64_binned", taxa=17, age=120.0, families=2777, root=6.0,
              lam=0.0025, K=5, alpha=0.8, eps=0.04, tree=3),
        # the gamma workload of the headline benchmark: one step, a batch of 16, and the default precision
        _case("score_gamma4_24taxa_10k", "score", "mixed_tf32x3", K=4),
        _case("batch16_gamma4_24taxa_10k", "batch", "mixed_tf32x3", K=4, candidates=16),
        _case("score_gamma4_24taxa_10k_ref", "score", "fp64_ref", K=4),
        # two rates, an error model and a heavy tail of large families: widths from 32 to 512 states and more
        _case("batch4_twolambda_32taxa_50k", "batch", "mixed_tf32x3", taxa=32, families=50000, root=4.0, lam=0.0012,
              candidates=4, clade=True, eps=0.05, heavy=0.05),
        _case("score_twolambda_32taxa_50k_binned", "score", "fp64_binned", taxa=32, families=50000, root=4.0, lam=0.0012,
              clade=True, eps=0.05, heavy=0.05),
        # one round of many optimizers on a large gamma problem
        _case("batch64_gamma8_48taxa_20k", "batch", "mixed_tf32x3", taxa=48, families=20000, root=5.0, lam=0.001,
              K=8, candidates=64),
        # the analyses that follow a search
        _case("reconstruct_gamma4_24taxa_10k", "reconstruct", K=4),
        _case("pvalues_12taxa_1k", "pvalues", taxa=12, age=100.0, families=1000, root=5.0, lam=0.0025, sims=1000),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["score", "score", "score", "score", "batch", "batch", "batch", "reconstruct", "pvalues", "fit"])
    precision = "fp64_ref"
    if op in ("score", "batch"):
        precision = rng.choice(["mixed_tf32x3", "mixed_tf32x3", "fp64_ref", "fp64_binned"])
    taxa = _log_int(rng, 8, 64)
    families = _log_int(rng, 100, 50000)
    K = rng.choice([1, 1, 2, 3, 4, 5, 8]) if op in ("score", "batch", "reconstruct") else 1
    candidates = _log_int(rng, 2, 64) if op == "batch" else 1
    sims = rng.choice([200, 500, 1000]) if op == "pvalues" else 0
    clade = rng.random() < 0.3
    # a rate model with categories has one lambda here; error models apply to scores
    clade = clade and K == 1 and op in ("score", "batch")
    eps = round(rng.uniform(0.01, 0.08), 3) if op in ("score", "batch") and rng.random() < 0.3 else 0.0
    heavy = round(rng.uniform(0.005, 0.05), 4) if K == 1 and op in ("score", "batch") and rng.random() < 0.3 else 0.0
    if heavy and precision == "fp64_ref":
        precision = "fp64_binned"
    if op == "fit":
        taxa, families = min(taxa, 20), min(families, 2000)
    if op == "pvalues":
        taxa, families = min(taxa, 16), min(families, 4000)
    # no more than the listed cases' work: family-category-node contractions at the widths in use
    limit = {"fp64_ref": 8.0e5, "fp64_binned": 1.5e6, "mixed_tf32x3": 4.0e8}[precision]
    while families * K * candidates * taxa > limit and candidates > 2:
        candidates //= 2
    families = max(100, min(families, int(limit / (K * candidates * taxa))))
    age, tree, alpha = float(rng.randint(60, 200)), rng.randint(0, 9999), round(rng.uniform(0.45, 1.5), 3)
    # a rate whose longest branch stays below saturation (lambda t < 1) in the fastest category
    fastest = max(discrete_gamma(0.9 * alpha, K)[1]) if K > 1 else 1.0
    longest = max(synth.yule_tree(taxa, age, tree).branch_length)
    lam = min(rng.uniform(0.001, 0.0025), 0.7 / (longest * fastest * (4.0 if clade else 1.0)))
    return _case(None, op, precision, taxa=taxa, age=age, families=families, root=round(rng.uniform(2.0, 9.0), 2),
                 lam=round(lam, 7), K=K, alpha=alpha, candidates=candidates, clade=clade, eps=eps, heavy=heavy,
                 sims=sims, tree=tree)


# ---------------------------------------------------------------- inputs

class _Data:
    """Tree, counts and parameter vectors of a case."""

    def __init__(self, case, seed):
        self.case = case
        self.tree = tree = synth.yule_tree(case["taxa"], case["age"], case["tree"])
        n = tree.n_nodes
        self.lam_idx = [0] * n
        if case["clade"]:      # a clade of about a third of the taxa evolves at its own rate
            size = [0] * n
            for v in tree.reverse_level_order():
                size[v] = 1 if tree.is_leaf(v) else sum(size[c] for c in tree.children[v])
            inner = [v for v in range(n) if not tree.is_leaf(v) and v != tree.root]
            stack = [min(inner, key=lambda v: abs(size[v] - case["taxa"] / 3.0))]
            while stack:
                v = stack.pop()
                self.lam_idx[v] = 1
                stack.extend(tree.children[v])
        rng = np.random.default_rng([int(seed), 17])
        F, K = case["families"], case["K"]
        mult = np.asarray(discrete_gamma(case["alpha"], K)[1] if K > 1 else [1.0])
        lam = case["lam"] * mult[rng.integers(0, K, F)]
        root = rng.poisson(case["root"], F)
        if case["heavy"] > 0:
            root = np.where(rng.random(F) < case["heavy"], rng.geometric(0.02, F), root)
        factor = [4.0 if i else 1.0 for i in self.lam_idx]
        c = synth.simulate_families(tree, F, lam, np.maximum(root, 1), int(rng.integers(1 << 31)), lambda_of_node=factor)
        if case["eps"] > 0:    # counting errors of -1 and +1
            u = rng.random(c.shape)
            c = np.where(u < case["eps"], c - 1, np.where(u > 1 - case["eps"], c + 1, c))
        c = np.maximum(c, 0).astype(np.int32)
        c[c.max(axis=1) == 0, 0] = 1        # a family has a gene in some species
        self.families = FamilySet([f"F{i:06d}" for i in range(F)], np.ascontiguousarray(c))
        self.S, self.R = global_bounds(self.families)
        self.prior = RootPrior.uniform(self.R)
        self.error = ErrorModel.symmetric(case["eps"], int(c.max())) if case["eps"] > 0 else None
        base = case["lam"] * math.exp(rng.uniform(-0.1, 0.1))
        self.candidates = []
        for _ in range(case["candidates"]):
            l = base * math.exp(rng.uniform(-0.08, 0.08))
            cand = {"lambdas": [l, 4.0 * l * math.exp(rng.uniform(-0.05, 0.05))] if case["clade"] else [l]}
            if K > 1:
                probs, m = discrete_gamma(case["alpha"] * math.exp(rng.uniform(-0.1, 0.1)), K)
                cand.update(cat_probs=probs, multipliers=m)
            self.candidates.append(cand)

    def lambda_tree(self):
        t = parse_newick(self.tree.to_newick())
        t.lambda_index = [i + 1 for i in self.lam_idx]
        return t


class _State:
    pass


def prepare(case, seed):
    d = _Data(case, seed)
    s = _State()
    s.case, s.data = case, d
    s.ctx = Context(n_streams=1, matrix_cache_bytes=1 << 20)
    cand = d.candidates[0]
    if case["op"] in ("batch", "pvalues"):
        s.tree_id = s.ctx.upload_tree(d.tree, d.lam_idx)
        s.set_id = s.ctx.upload_families(s.tree_id, d.families.counts)
        s.ctx.set_prior(d.prior.vector())
        if d.error is not None:
            s.ctx.set_error_model(d.error.table())
        n = len(d.candidates)
        s.lnl = torch.zeros((n, case["families"]), dtype=torch.float64, device="cuda")
        s.total = torch.zeros(n, dtype=torch.float64, device="cuda")
        s.kw = dict(model=1 if case["K"] > 1 else 0, lambda_kind=1 if case["clade"] else 0,
                    use_error_model=d.error is not None, precision=case["precision"])
        if case["precision"] == "fp64_ref":
            s.kw.update(S=d.S, R=d.R)
        return s
    lam = MultipleLambda(d.lambda_tree(), cand["lambdas"]) if case["clade"] else SingleLambda(cand["lambdas"][0])
    kw = dict(precision=case["precision"], ctx=s.ctx)
    if case["K"] > 1:
        s.model = GammaModel(lam, d.tree, d.families, d.S, d.R, error_model=d.error, cat_probs=cand["cat_probs"],
                             multipliers=cand["multipliers"], **kw)
    else:
        s.model = BaseModel(lam, d.tree, d.families, d.S, d.R, error_model=d.error, **kw)
    if case["op"] == "fit":
        s.scorer = LambdaOptimizerScorer(lam, s.model, d.prior, max(d.tree.branch_length))
        s.guess = [cand["lambdas"][0]]
    return s


def run(state):
    op, d = state.case["op"], state.data
    if op == "score":
        total = state.model.infer_family_likelihoods(d.prior)
        out = {"total": total, "family_lnl": state.model.results}
        if state.case["K"] > 1:
            out["category_lnl"] = state.model.category_results
        return out
    if op == "batch":
        state.ctx.score_batch_device(state.tree_id, state.set_id, d.candidates, d_family_lnl=state.lnl.data_ptr(),
                                     d_total=state.total.data_ptr(), **state.kw)
        return {"total": state.total, "family_lnl": state.lnl}
    if op == "fit":
        r = Optimizer(state.scorer).optimize(initial=state.guess)
        return {"lambda": r.values[0], "score": r.score}
    if op == "reconstruct":
        r = state.model.reconstruct_ancestral_states(d.prior)
        return {"node_count": r.node_count, "node_mean": r.node_mean, "category_state": r.category_state,
                "root_max": r.root_max}
    r = state.ctx.pvalues(state.tree_id, state.set_id, d.candidates[0]["lambdas"], S=d.S, R=d.R,
                          n_simulations=state.case["sims"], seed=10)
    return {k: r[k] for k in ("pvalues", "conditional", "root_likelihood")}


# ---------------------------------------------------------------- work

def _groups(case, d):
    """(families, states) of each group that shares a state bound."""
    c = d.families.counts
    if case["precision"] == "fp64_ref":
        return [(np.arange(len(c)), d.S + 1, np.full(len(c), d.R))]
    W, _, R = bin_families(d.families)
    return [(np.nonzero(W == w)[0], int(w), R) for w in np.unique(W)]


def work(case):
    """Multiply-adds of the contractions over distinct rows: families of a
    group with the same counts below a node share that node's vector."""
    d = _Data(case, 1)
    t, K, n = d.tree, case["K"], case["candidates"]
    flops = 0.0
    inner = [v for v in t.reverse_level_order() if not t.is_leaf(v) and v != t.root]
    for fam, W, _ in _groups(case, d):
        key = {v: d.families.counts[fam, i].astype(np.int64) for i, v in enumerate(t.leaves)}
        for v in inner:
            x = key[t.children[v][0]]
            for u in t.children[v][1:]:
                x = np.unique(x * (int(key[u].max()) + 1) + key[u], return_inverse=True)[1].reshape(-1)
            key[v] = x
            flops += 2.0 * W * W * (int(x.max()) + 1) * K * n
    F, L = d.families.counts.shape
    out = F * n * 8.0
    if case["op"] == "score" and K > 1:
        out += F * K * 8.0
    if case["op"] == "fit":
        flops *= 30             # evaluations of a one-parameter search
        out = 16.0
    if case["op"] == "reconstruct":
        out = F * t.n_nodes * (4.0 + 8.0 + 4.0 * K) + F * K * 8.0
    if case["op"] == "pvalues":  # simulated families of root size r have about r + 50 states
        flops += sum(2.0 * min(d.S, r + 50) ** 2 for r in range(1, d.R + 1)) * case["sims"] * len(inner)
        out = (F + F * d.R + d.R * case["sims"]) * 8.0
    return {"bytes": F * L * 4.0 + out, "flops": flops}


# ---------------------------------------------------------------- 64-bit values

def _matrix(lam, t, n, dev):
    """Birth-death transition probabilities of side n at the cache key's
    values: row s is the distribution of s independent copies of row 1."""
    lq, tq = int(lam * 1000000000) / 1000000000.0, int(t * 1000) / 1000.0
    a = lq * tq / (1 + lq * tq)
    M = torch.zeros((n, n), dtype=torch.float64, device=dev)
    M[0, 0] = 1.0
    if not 0 < 1 - 2 * a < 1:
        return M
    c = torch.arange(n, dtype=torch.float64, device=dev)
    one = (1 - a) ** 2 * a ** (c - 1)
    one[0] = a
    i = torch.arange(n, device=dev)
    shift = i[None, :] - i[:, None]
    toep = torch.where(shift >= 0, one[shift.clamp(min=0)], torch.zeros((), dtype=torch.float64, device=dev))
    # doubling: rows h .. 2h - 1 are rows 0 .. h - 1 with h more copies
    M[1] = one
    step, h = toep, 2
    step = step @ toep
    while h < n:
        m = min(h, n - h)
        M[h:h + m] = M[:m] @ step
        step = step @ step
        h *= 2
    return M


def _leaf(M, n, S, err):
    """Columns of M at the counts n (rows: families), with the error model's weights."""
    if err is None:
        return M[:, n].T
    rows = torch.as_tensor(err, dtype=torch.float64, device=M.device)
    pr = rows[n.clamp(max=len(rows) - 1)]
    out = torch.zeros((len(n), len(M)), dtype=torch.float64, device=M.device)
    for k in range(3):
        c = n + k - 1
        ok = (c >= 0) & (c <= S)
        out += torch.where(ok, pr[:, k], torch.zeros_like(pr[:, k]))[:, None] * M[:, c.clamp(0, len(M) - 1)].T
    return out


def _walk(d, case, mats, counts, W, scaled):
    """Root product over states 0 .. W - 1 for every family, and its exponents (natural log)."""
    t = d.tree
    col = {v: i for i, v in enumerate(t.leaves)}
    dev = counts.device
    err = d.error.table() if d.error is not None else None
    shift = torch.zeros(len(counts), dtype=torch.float64, device=dev)
    vec = {}
    for v in t.reverse_level_order():
        if t.is_leaf(v):
            continue
        x = torch.ones((len(counts), W), dtype=torch.float64, device=dev)
        for u in t.children[v]:
            M = mats[u][:W, :W]
            x = x * (_leaf(M, counts[:, col[u]], W - 1, err) if u in col else vec.pop(u) @ M.T)
        if scaled:
            e = torch.frexp(x.max(dim=1).values)[1].to(torch.float64)
            x = x * torch.exp2(-e)[:, None]
            shift = shift + e * math.log(2.0)
        vec[v] = x
    return vec[t.root], shift


def _mats(d, cand, k, n, dev):
    m = cand["multipliers"][k] if "multipliers" in cand else 1.0
    return {v: _matrix(cand["lambdas"][d.lam_idx[v]] * m, d.tree.branch_length[v], n, dev)
            for v in range(d.tree.n_nodes) if v != d.tree.root}


def _exact_score(d, case, cand, dev):
    F, K = case["families"], case["K"]
    ref = case["precision"] == "fp64_ref"
    prior = torch.as_tensor(d.prior.vector(), dtype=torch.float64, device=dev)
    counts = torch.as_tensor(d.families.counts.astype(np.int64), device=dev)
    lnl = torch.zeros(F, dtype=torch.float64, device=dev)
    cats = torch.zeros((F, K), dtype=torch.float64, device=dev)
    groups = _groups(case, d)
    n = max(W for _, W, _ in groups)
    if ref:
        n = max(n, d.R + 1)
    for k in range(K):
        mats = _mats(d, cand, k, n, dev)
        for fam, W, R in groups:
            for lo in range(0, len(fam), 20000):
                f = torch.as_tensor(fam[lo:lo + 20000], device=dev)
                x, shift = _walk(d, case, mats, counts[f], W, not ref)
                j = torch.arange(1, W, device=dev)
                p = torch.zeros(W - 1, dtype=torch.float64, device=dev)
                m = min(len(prior), W - 1)
                p[:m] = prior[:m]
                rows = torch.as_tensor(np.asarray(R)[fam[lo:lo + 20000]].astype(np.int64), device=dev)
                v = torch.where(j[None, :] <= rows[:, None], x[:, 1:] * p, torch.zeros((), dtype=torch.float64, device=dev))
                best = torch.log(v.max(dim=1).values) + shift
                cats[f, k] = best + (math.log(cand["cat_probs"][k]) if K > 1 else 0.0)
    lnl = torch.logsumexp(cats, dim=1) if K > 1 else cats[:, 0]
    return -lnl.sum(), lnl, cats


def _exact_root_max(d, case, cand, dev):
    """Largest root value of the max-product recursion, per category and family."""
    t, F, K, n = d.tree, case["families"], case["K"], d.S + 1
    col = {v: i for i, v in enumerate(t.leaves)}
    counts = torch.as_tensor(d.families.counts.astype(np.int64), device=dev)
    prior = torch.zeros(n, dtype=torch.float64, device=dev)
    p = torch.as_tensor(d.prior.vector(), dtype=torch.float64, device=dev)
    prior[:min(n, len(p))] = p[:n]
    out = torch.zeros((K, F), dtype=torch.float64, device=dev)
    for k in range(K):
        mats = _mats(d, cand, k, max(d.S, d.R) + 1, dev)
        best = {}
        for v in t.reverse_level_order():
            if t.is_leaf(v):
                continue
            u = torch.ones((F, n), dtype=torch.float64, device=dev)
            for c in t.children[v]:
                u = u * (mats[c][:n, :][:, counts[:, col[c]]].T if c in col else best.pop(c))
            if v == t.root:
                r = min(d.S, d.R) + 1
                out[k] = (u[:, 1:r] * prior[1:r]).max(dim=1).values
                break
            M = mats[v][:n, :n]
            best[v] = torch.cat([(x[:, None, :] * M[None]).amax(dim=2) for x in torch.split(u, 256)])
    return out


def exact(case, seed):
    d = _Data(case, seed)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    op, K = case["op"], case["K"]
    rows = case["families"] * K * case["candidates"]
    if op in ("score", "batch"):
        # about 20 seconds of 64-bit products at most
        side = (d.S + 1) if case["precision"] == "fp64_ref" else 60
        if rows * case["taxa"] * 2.0 * side * side > 8e12:
            return None
        got = [_exact_score(d, case, cand, dev) for cand in d.candidates]
        if op == "batch":
            return {"total": torch.stack([g[0] for g in got]), "family_lnl": torch.stack([g[1] for g in got])}
        out = {"total": float(got[0][0]), "family_lnl": got[0][1]}
        if K > 1:
            out["category_lnl"] = got[0][2]
        return out
    if op == "reconstruct":
        return {"node_count": None, "node_mean": None, "category_state": None,
                "root_max": _exact_root_max(d, case, d.candidates[0], dev)}
    if op == "pvalues":      # the observed root vectors; the rest hangs on a random stream
        counts = torch.as_tensor(d.families.counts.astype(np.int64), device=dev)
        mats = _mats(d, d.candidates[0], 0, max(d.S, d.R) + 1, dev)
        x, _ = _walk(d, case, mats, counts, d.S + 1, False)
        return {"pvalues": None, "conditional": None, "root_likelihood": x[:, 1:d.R + 1]}
    return None

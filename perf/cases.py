"""The work that a user of this library has it do, as cases that can be timed.

The cases cover the path from a character matrix to a supported tree: the
greedy joins (indel and bit-coded, unit and fractional weights, from a call of
a few milliseconds to the largest), the two radius searches, the transfer
distance, the batched bootstrap, and the likelihood with its adjoint gradient
and branch-length optimisation.  Each goes through the entry point that a
program calls: `casphy_b200.lib` on host arrays, or the `_dev` function of the
C ABI where the matrix is already on the GPU.

Inputs are simulated on the GPU from the seed alone, with the distributions of
`casphy_b200.synth` (lineages with irreversible Zipf edits and dropout, HKY85
alignments on Yule trees), and are handed over as the entry point takes them.
"""
import ctypes as C
import math
import random

import numpy as np
import torch

from casphy_b200 import lib

PI = (0.3, 0.2, 0.2, 0.3)  # A, T, C, G
KAPPA = 4.0


def listed():
    return [
        # a clone or a partition of a larger tree: the whole join takes a few
        # milliseconds, the small configuration of the benchmark
        {"name": "indel_small", "kind": "indel", "ncell": 1024, "nsite": 256, "nallele": 64, "weights": "unit",
         "entry": "host"},
        # an ordinary experiment with the information-weighted score (-log of
        # the allele frequency): the binary16 sums of the reference, odd sizes
        {"name": "indel_logfreq", "kind": "indel", "ncell": 4001, "nsite": 499, "nallele": 64, "weights": "logfreq",
         "entry": "host"},
        # one chip of cells with many sites, unit weights
        {"name": "indel_chip", "kind": "indel", "ncell": 12345, "nsite": 777, "nallele": 256, "weights": "unit",
         "entry": "host"},
        # a pooled atlas, codes already on the GPU: the benchmark's headline
        # workload at a third of its cells
        {"name": "indel_large", "kind": "indel", "ncell": 65000, "nsite": 1024, "nallele": 256, "weights": "unit",
         "entry": "dev"},
        # the base-editor matrix of the benchmark
        {"name": "bit_unit", "kind": "bit", "ncell": 10000, "nsite": 512, "weights": "unit", "anc": 1},
        # the same data with fractional site weights: binary32 sums in order
        {"name": "bit_logfreq", "kind": "bit", "ncell": 2999, "nsite": 352, "weights": "logfreq", "anc": 0},
        # near-duplicate cells of the base-editor matrix
        {"name": "radius_bit", "kind": "radius_bit", "ncell": 20000, "nsite": 512},
        # near-duplicate sequences of an alignment, the benchmark's size
        {"name": "radius_dna", "kind": "radius_dna", "ntip": 20000, "nsite": 2000},
        # clades of a reference tree against those of an estimated one
        {"name": "transfer", "kind": "transfer", "ntip": 10000},
        # support of a tree's clades from resampled replicates
        {"name": "bootstrap", "kind": "bootstrap", "ncell": 5000, "nsite": 512, "nrep": 64},
        # log L and gradient of the edit model on a lineage tree
        {"name": "loglik_edit", "kind": "loglik", "model": "irreversible", "ntip": 4099, "nsite": 500},
        # branch lengths of a gene tree, a bounded number of L-BFGS steps
        {"name": "optimize_dna", "kind": "optimize", "model": "hky85", "ntip": 2000, "nsite": 1500, "iters": 40},
    ]


def draw(rng: random.Random):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["indel", "indel", "indel", "bit", "bit", "radius_bit", "radius_dna", "transfer", "bootstrap",
                       "loglik", "optimize"])
    if kind == "indel":
        return {"kind": kind, "ncell": size(500, 40000), "nsite": size(60, 1024), "nallele": rng.choice([32, 64, 256]),
                "weights": "unit", "entry": rng.choice(["host", "dev"])} if rng.random() < 0.7 else \
            {"kind": kind, "ncell": size(500, 8000), "nsite": size(60, 800), "nallele": rng.choice([32, 64]),
             "weights": "logfreq", "entry": rng.choice(["host", "dev"])}
    if kind == "bit":
        w = rng.choice(["unit", "unit", "counts", "logfreq"])
        return {"kind": kind, "ncell": size(500, 10000 if w != "logfreq" else 4000), "nsite": size(64, 1024),
                "weights": w, "anc": rng.choice([0, 1])}
    if kind == "radius_bit":
        return {"kind": kind, "ncell": size(1000, 20000), "nsite": size(128, 1024)}
    if kind == "radius_dna":
        return {"kind": kind, "ntip": size(1000, 20000), "nsite": size(200, 2000)}
    if kind == "transfer":
        return {"kind": kind, "ntip": size(500, 10000)}
    if kind == "bootstrap":
        return {"kind": kind, "ncell": size(1000, 5000), "nsite": size(128, 512), "nrep": size(16, 100)}
    model = rng.choice(["hky85", "irreversible"])
    if kind == "loglik":
        return {"kind": kind, "model": model, "ntip": size(100, 5000), "nsite": size(100, 1500)}
    return {"kind": kind, "model": model, "ntip": size(100, 2000), "nsite": size(100, 1500), "iters": rng.randint(10, 40)}


# --------------------------------------------------------------------------
# simulated inputs (torch on the GPU, numpy for the trees)

def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _lineage(ncell, nsite, depth, p_edit, nallele, zipf_s, p_missing, g):
    """int16 states (ncell, nsite): -1 missing, 0 unedited, 1.. allele."""
    dev = torch.device("cuda")
    leaves = torch.randperm(1 << depth, device=dev, generator=g)[:ncell]
    cum = None
    if nallele > 1:
        p = torch.arange(1, nallele + 1, device=dev, dtype=torch.float64) ** -zipf_s
        cum = torch.cumsum(p / p.sum(), 0).float()
    prev = torch.zeros(1, dtype=torch.int64, device=dev)
    state = torch.zeros((1, nsite), dtype=torch.int16, device=dev)
    for level in range(1, depth + 1):
        cur = torch.unique(leaves >> (depth - level))
        state = state[torch.searchsorted(prev, cur >> 1)]
        hit = (torch.rand(state.shape, device=dev, generator=g) < p_edit) & (state == 0)
        if cum is None:
            state[hit] = 1
        else:
            u = torch.rand(int(hit.sum()), device=dev, generator=g)
            state[hit] = (torch.searchsorted(cum, u).clamp_(max=nallele - 1) + 1).to(torch.int16)
        prev = cur
    state = state[torch.searchsorted(prev, leaves)]
    if p_missing > 0:
        state[torch.rand(state.shape, device=dev, generator=g) < p_missing] = -1
    return state


def _indel_codes(state, nallele):
    """.tbmat codes (0 missing, 1 unedited, 2.. the column's alleles), nState."""
    nsite = state.shape[1]
    seen = torch.zeros((nsite, nallele + 2), dtype=torch.int32, device=state.device)
    col = torch.arange(nsite, device=state.device).expand_as(state)
    seen[col, state.long() + 1] = 1
    seen[:, :2] = 1  # missing and unedited are always ranked
    rank = torch.cumsum(seen, 1, dtype=torch.int32) - 1
    codes = torch.gather(rank.t().contiguous(), 0, state.long() + 1)
    return codes, max(int(rank[:, -1].max()) - 1, 1)


def _indel_weights(codes, nstate, how):
    if how == "unit":
        return np.ones((nstate, codes.shape[1]))
    count = torch.zeros((nstate + 2, codes.shape[1]), dtype=torch.float64, device=codes.device)
    count.scatter_add_(0, codes.long(), torch.ones(codes.shape, dtype=torch.float64, device=codes.device))
    return (-torch.log(count[2:].clamp(min=1) / codes.shape[0])).cpu().numpy()


def _pack(bits):
    """bool (rows, n) -> u32 words (rows, ceil(n/32)), bit j of word k = 32k+j."""
    rows, n = bits.shape
    nw = (n + 31) // 32
    full = torch.zeros((rows, nw * 32), dtype=torch.uint8, device=bits.device)
    full[:, :n] = bits
    by = (full.view(rows, nw * 4, 8) << torch.arange(8, device=bits.device, dtype=torch.uint8)).sum(2, dtype=torch.uint8)
    return by.contiguous().cpu().numpy().view(np.uint32)


def _bit_weights(state, how, g):
    n = state.shape[1]
    w = np.zeros((n + 31) // 32 * 32)
    if how == "unit":
        w[:] = 1.0
    elif how == "counts":  # multiplicities of resampled columns
        w[:n] = torch.bincount(torch.randint(0, n, (n,), device="cuda", generator=g), minlength=n).cpu().numpy()
    else:
        f = (state == 1).double().mean(0).clamp(min=1.0 / state.shape[0])
        w[:n] = (-torch.log(f)).cpu().numpy()
    return w


def _yule(ntip, rng):
    """Random Yule topology as (edge (2n-2, 2), pre-order lo, hi of every node):
    uniform splits of intervals of a random tip order; tips 0..n-1, root n."""
    perm = rng.permutation(ntip)
    u = rng.random(2 * ntip)
    edge = np.empty((2 * ntip - 2, 2), np.uint32)
    lo, hi = np.zeros(2 * ntip - 1, np.int64), np.zeros(2 * ntip - 1, np.int64)
    hi[ntip] = ntip
    stack, nxt, ne = [ntip], ntip + 1, 0
    while stack:
        v = stack.pop()
        a, b = int(lo[v]), int(hi[v])
        m = a + 1 + min(int(u[v] * (b - a - 1)), b - a - 2)
        for x, y in ((a, m), (m, b)):
            if y - x == 1:
                c = int(perm[x])
            else:
                c, nxt = nxt, nxt + 1
                stack.append(c)
            lo[c], hi[c] = x, y
            edge[ne] = v, c
            ne += 1
    return edge, lo, hi, perm


def _clades(ntip, lo, hi, perm):
    """Tip bitsets of the internal nodes except the root."""
    l = torch.from_numpy(lo[ntip + 1:]).cuda()[:, None]
    h = torch.from_numpy(hi[ntip + 1:]).cuda()[:, None]
    rank = torch.empty(ntip, dtype=torch.int64, device="cuda")
    rank[torch.from_numpy(perm).cuda()] = torch.arange(ntip, device="cuda")
    return _pack((rank >= l) & (rank < h))


def _levels(edge, ntip):
    """Per internal node: children and their edges, and the nodes by depth and by height."""
    nn = len(edge) + 1
    kid = np.full((nn, 2), -1, np.int64)
    ked = np.full((nn, 2), -1, np.int64)
    order = np.argsort(edge[:, 0], kind="stable")
    kid[edge[order[0::2], 0]] = edge[np.stack([order[0::2], order[1::2]], 1), 1]
    ked[edge[order[0::2], 0]] = np.stack([order[0::2], order[1::2]], 1)
    depths, cur = [], np.array([ntip])
    while len(cur):
        depths.append(cur)
        k = kid[cur].reshape(-1)
        cur = k[k >= ntip]
    height = np.zeros(nn, np.int64)
    for nodes in reversed(depths):
        height[nodes] = 1 + height[kid[nodes]].max(1)
    internal = np.arange(ntip, nn)
    heights = [internal[height[internal] == h] for h in range(1, int(height.max()) + 1)]
    return kid, ked, depths, heights


def _hky(t):
    """P(t) and dP/dt (edges, 4, 4) of HKY85, states A, T, C, G, in 64 bits."""
    pi = np.array(PI)
    q = np.tile(pi, (4, 1))
    for i, j in ((0, 3), (3, 0), (1, 2), (2, 1)):  # transitions A<->G, T<->C
        q[i, j] *= KAPPA
    np.fill_diagonal(q, 0.0)
    np.fill_diagonal(q, -q.sum(1))
    q /= -(pi * np.diag(q)).sum()
    r = np.sqrt(pi)
    lam, w = np.linalg.eigh((q * r[:, None] / r[None, :] + (q * r[:, None] / r[None, :]).T) / 2)
    v, vi = w / r[:, None], w.T * r[None, :]
    e = np.exp(lam[None, :] * np.asarray(t)[:, None])
    return np.einsum("ik,ek,kj->eij", v, e, vi), np.einsum("ik,ek,kj->eij", v, e * lam, vi)


def _likelihood_inputs(case, seed):
    ntip, nsite, g = case["ntip"], case["nsite"], _generator(seed)
    rng = np.random.default_rng(seed)
    edge, _, _, _ = _yule(ntip, rng)
    true_t = rng.exponential(0.02, len(edge))
    kid, ked, depths, _ = _levels(edge, ntip)
    nn = 2 * ntip - 1
    state = torch.zeros((nn, nsite), dtype=torch.int64, device="cuda")
    hky = case["model"] == "hky85"
    if hky:
        cum = torch.from_numpy(np.cumsum(_hky(true_t)[0], 2)).float().cuda()
        state[ntip] = torch.multinomial(torch.tensor(PI, device="cuda"), nsite, replacement=True, generator=g)
    else:
        zipf = 1.0 / torch.arange(1, 33, device="cuda", dtype=torch.float32) ** 1.3
        zc = torch.cumsum(zipf / zipf.sum(), 0)
        stay = torch.from_numpy(np.exp(-true_t)).float().cuda()
    for nodes in depths:
        p = torch.from_numpy(nodes).cuda()
        for side in (0, 1):
            c, e = torch.from_numpy(kid[nodes, side]).cuda(), torch.from_numpy(ked[nodes, side]).cuda()
            u = torch.rand((len(nodes), nsite), device="cuda", generator=g)
            if hky:
                row = torch.gather(cum[e], 1, state[p][:, :, None].expand(-1, -1, 4))
                state[c] = (u[:, :, None] > row).sum(2).clamp_(max=3)
            else:
                al = torch.searchsorted(zc, torch.rand(u.shape, device="cuda", generator=g)).clamp_(max=31) + 1
                state[c] = torch.where((state[p] == 0) & (u > stay[e][:, None]), al, state[p])
    tips = state[:ntip]
    miss = torch.rand(tips.shape, device="cuda", generator=g) < (0.02 if hky else 0.1)
    codes = torch.where(miss, 0, (1 << tips) if hky else tips + 1)
    start = np.clip(true_t * rng.uniform(0.5, 2.0, len(edge)), 1e-4, None)
    args = {"edge": edge, "codes": codes.to(torch.int32).cpu().numpy().view(np.uint32), "brlen": start}
    args["model"] = {"model": "hky85", "kappa": KAPPA, "pi": PI} if hky else \
        {"model": "irreversible", "rate": 1.0, "nallele": 32}
    return args


# --------------------------------------------------------------------------

def prepare(case, seed):
    kind, s = case["kind"], {"case": case}
    if kind in ("loglik", "optimize"):
        s.update(_likelihood_inputs(case, seed))
        return s
    g = _generator(seed)
    if kind == "indel":
        state = _lineage(case["ncell"], case["nsite"], 20, 0.02, case["nallele"], 1.3, 0.15, g)
        codes, s["nstate"] = _indel_codes(state, case["nallele"])
        s["weights"] = _indel_weights(codes, s["nstate"], case["weights"])
        if case["entry"] == "host":
            s["codes"] = codes.cpu().numpy().view(np.uint32)
        else:
            n = case["ncell"]
            s["codes"] = codes.contiguous()
            s["state"] = torch.empty((n - 1, case["nsite"]), dtype=torch.int32, device="cuda")
            s["edge"] = np.empty((2 * n - 2, 2), np.uint32)
            s["weights"] = np.ascontiguousarray(s["weights"]).reshape(-1)
            s["tip_size"] = np.ones(n, np.uint32)
    elif kind in ("bit", "radius_bit", "bootstrap"):
        state = _lineage(case["ncell"], case["nsite"], 16, 0.03, 1, 1.0, 0.05, g)
        words = _pack(state == 1)
        if kind == "bit":
            s["words"], s["weights"] = words, _bit_weights(state, case["weights"], g)
        elif kind == "radius_bit":
            # about a handful of neighbours per cell: pairs that share nearly
            # all edits of a typical cell
            s["bmat"], s["weights"] = np.ascontiguousarray(words.T), _bit_weights(state, "unit", g)
            s["radius"] = int(0.78 * float((state == 1).sum(1).double().mean()))
        else:
            rng = np.random.default_rng(seed)
            n = rng.integers(case["ncell"] // 3, case["ncell"] + 1, case["nrep"])
            s["words"] = words
            s["offsets"] = np.concatenate([[0], np.cumsum(n)]).astype(np.uint32)
            s["cells"] = np.concatenate([np.sort(rng.permutation(case["ncell"])[:k]) for k in n]).astype(np.uint32)
            nb, ns = words.shape[1] * 32, case["nsite"]
            s["weights"] = np.stack([np.bincount(rng.integers(0, ns, ns), minlength=nb) for _ in n]).astype(np.float64)
            s["full_edge"] = lib.join_bit(words, None, 1)[0]
    elif kind == "radius_dna":
        a = _likelihood_inputs({"ntip": case["ntip"], "nsite": case["nsite"], "model": "hky85"}, seed)
        codes = torch.from_numpy(a["codes"].view(np.int32)).cuda()
        by = torch.zeros((case["ntip"], (case["nsite"] + 3) // 4 * 4), dtype=torch.uint8, device="cuda")
        by[:, :case["nsite"]] = torch.where(codes == 0, 0x10, codes)  # fasta2bin writes a gap as 0x10
        s["raw"] = by.cpu().numpy().view(np.uint32)
        s["radius"] = int(0.925 * case["nsite"])
    else:
        rng = np.random.default_rng(seed)
        n = case["ntip"]
        _, lo, hi, perm = _yule(n, rng)
        s["y"] = _clades(n, lo, hi, perm)
        # the estimate: the same splits with a tenth of the tips misplaced
        moved = np.sort(rng.permutation(n)[:max(n // 10, 2)])
        perm = perm.copy()
        perm[moved] = perm[np.roll(moved, 1)]
        s["x"] = _clades(n, lo, hi, perm)
    if kind in ("radius_bit", "radius_dna"):
        # a program that searches again and again keeps room for the lists
        n = case["ncell" if kind == "radius_bit" else "ntip"]
        s["counts"], s["idx"] = np.zeros(n, np.uint32), np.zeros(128 * n, np.uint32)
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "indel":
        if case["entry"] == "host":
            edge, state, _ = lib.join_indel(s["codes"], s["nstate"], s["weights"])
            return {"edge": edge, "state": state}
        rc = lib.lib().casphy_join_indel_dev(case["ncell"], case["nsite"], C.c_void_p(s["codes"].data_ptr()),
                                             s["nstate"], s["weights"], s["tip_size"], 0, 2.0, s["edge"].reshape(-1),
                                             C.c_void_p(s["state"].data_ptr()), None,
                                             C.c_void_p(torch.cuda.current_stream().cuda_stream))
        if rc != 0:
            raise lib.CasphyError(rc, "casphy_join_indel_dev")
        return {"edge": s["edge"], "state": s["state"]}
    if kind == "bit":
        edge, state, _ = lib.join_bit(s["words"], s["weights"], case["anc"])
        return {"edge": edge, "state": state}
    if kind in ("radius_bit", "radius_dna"):
        total, idx = C.c_uint64(0), s["idx"]
        rest = (s["radius"], s["counts"], idx.ctypes.data_as(C.c_void_p), idx.size, C.byref(total))
        if kind == "radius_bit":
            rc = lib.lib().casphy_radius_bit(*s["bmat"].shape, s["bmat"], s["weights"], *rest)
        else:
            rc = lib.lib().casphy_radius_dna(*s["raw"].shape, s["raw"], *rest)
        if rc != 0:
            raise lib.CasphyError(rc, "casphy_" + kind)
        return {"counts": s["counts"], "idx": idx, "total": total.value}
    if kind == "transfer":
        return lib.transfer_dis(s["y"], s["x"], case["ntip"])
    if kind == "bootstrap":
        got = lib.bootstrap_bit(s["words"], s["full_edge"], s["offsets"], s["cells"], s["weights"], threshold=0.2)
        return {"support": got["support"], "ymin": got["ymin"], "ysize": got["ysize"]}
    if kind == "loglik":
        ll, grad = lib.felsenstein_loglik(s["edge"], s["brlen"], s["codes"], grad=True, **s["model"])
        return {"loglik": ll, "grad": grad}
    t, stats = lib.felsenstein_optimize(s["edge"], s["brlen"], s["codes"], max_iter=case["iters"], rel_tol=1e-9,
                                        **s["model"])
    return {"brlen": t, "loglik": stats["loglik_end"]}


def work(case):
    """Bytes: each input read once and each output written once.  Operations:
    one per (pair, character) that has to be scored, two per multiply-add."""
    kind = case["kind"]
    if kind == "indel":
        n, m = case["ncell"], case["nsite"]
        # all pairs once, and every join's new node against the remaining ones;
        # about a third of a cell's sites carry an allele that can match
        return {"bytes": 4.0 * (2 * n - 1) * m + 16.0 * n, "flops": n * (n - 1.0) * m / 3}
    if kind == "bit":
        n, w = case["ncell"], (case["nsite"] + 31) // 32
        return {"bytes": 4.0 * (2 * n - 1) * w + 16.0 * n, "flops": n * (n - 1.0) * case["nsite"] / 3}
    if kind == "radius_bit":
        n, w = case["ncell"], (case["nsite"] + 31) // 32
        return {"bytes": 4.0 * n * w + 4.0 * n, "flops": n * (n - 1.0) / 2 * case["nsite"]}
    if kind == "radius_dna":
        n, m = case["ntip"], case["nsite"]
        return {"bytes": 1.0 * n * m + 4.0 * n, "flops": n * (n - 1.0) / 2 * m}
    if kind == "transfer":
        n = case["ntip"]
        return {"bytes": 2.0 * (n - 2) * 4 * ((n + 31) // 32) + 16.0 * n, "flops": 2.0 * (n - 2.0) ** 2 * n}
    if kind == "bootstrap":
        n, r, w = 2 * case["ncell"] / 3, case["nrep"], (case["nsite"] + 31) // 32
        return {"bytes": 4.0 * case["ncell"] * w + r * (4.0 * n + 256.0 * w + 8.0 * case["ncell"]),
                "flops": r * n * (n - 1.0) * case["nsite"] / 3}
    n, m = case["ntip"], case["nsite"]
    # two 4x4 products and their combination per internal node and site inward,
    # four outward; the edit model's partial is a pair
    per = (70.0 + 180.0) if case["model"] == "hky85" else 40.0
    passes = 1 if kind == "loglik" else case["iters"] + 1
    return {"bytes": 4.0 * n * m + 40.0 * n, "flops": passes * per * (n - 1.0) * m}


# --------------------------------------------------------------------------
# 64-bit values of the likelihood cases

def exact(case, seed):
    if case["kind"] != "loglik":
        return None  # integers and bytes, or an iteration that its own rounding steers
    a = _likelihood_inputs(case, seed)
    f = _exact_hky if case["model"] == "hky85" else _exact_edit
    return dict(zip(("loglik", "grad"), f(a, case["ntip"])))


def _scale(top):
    """Power of two that brings positive values to [1, 2), and its exponent."""
    e = torch.floor(torch.log2(torch.where(top > 0, top, torch.ones_like(top))))
    return torch.exp2(-e), e


def _exact_hky(a, ntip):
    kid, ked, depths, heights = _levels(a["edge"], ntip)
    P, dP = (torch.from_numpy(x).cuda() for x in _hky(a["brlen"]))
    codes = torch.from_numpy(a["codes"].view(np.int32)).cuda()
    nn, nsite = 2 * ntip - 1, codes.shape[1]
    L = torch.empty((nn, nsite, 4), dtype=torch.float64, device="cuda")
    n = torch.where(codes == 0, 15, codes)
    for k in range(4):
        L[:ntip, :, k] = ((n >> k) & 1).double()
    logs = torch.zeros(nsite, dtype=torch.float64, device="cuda")
    idx = lambda x: torch.from_numpy(x).cuda()  # noqa: E731
    for v in heights:
        m = [L[idx(kid[v, s])] @ P[idx(ked[v, s])].transpose(1, 2) for s in (0, 1)]
        x = m[0] * m[1]
        sc, e = _scale(x.amax(2))
        L[idx(v)] = x * sc[:, :, None]
        logs += e.sum(0) * math.log(2.0)
    pi = torch.tensor(PI, dtype=torch.float64, device="cuda")
    ll = float((torch.log(L[ntip] @ pi) + logs).sum())
    U = torch.empty_like(L)
    U[ntip] = pi
    grad = torch.zeros(nn - 1, dtype=torch.float64, device="cuda")
    for v in depths:
        m = [L[idx(kid[v, s])] @ P[idx(ked[v, s])].transpose(1, 2) for s in (0, 1)]
        for s in (0, 1):
            c, e = idx(kid[v, s]), idx(ked[v, s])
            r = U[idx(v)] * m[1 - s]
            dm = L[c] @ dP[e].transpose(1, 2)
            grad[e] = ((r * dm).sum(2) / (r * m[s]).sum(2)).sum(1)
            u = r @ P[e]
            U[c] = u * _scale(u.amax(2))[0][:, :, None]
    return ll, grad.cpu().numpy()


def _exact_edit(a, ntip):
    """A subtree's partial: L0 (unedited), LA (its one possible allele, or any
    when the subtree is missing), and which: -1 none, -2 any."""
    kid, ked, depths, heights = _levels(a["edge"], ntip)
    codes = torch.from_numpy(a["codes"].view(np.int32)).cuda().long()
    nn, nsite = 2 * ntip - 1, codes.shape[1]
    nallele = a["model"]["nallele"]
    t = torch.from_numpy(a["brlen"]).cuda()
    count = torch.zeros((nallele + 2, nsite), dtype=torch.float64, device="cuda")
    count.scatter_add_(0, codes, torch.ones_like(codes, dtype=torch.float64))
    tot = count[2:].sum(0)
    q = torch.where(tot > 0, count[2:] / tot.clamp(min=1), torch.full_like(count[2:], 1.0 / nallele))
    f64 = lambda *shape: torch.zeros(shape, dtype=torch.float64, device="cuda")  # noqa: E731
    L0, LA, sc = f64(nn, nsite), f64(nn, nsite), f64(nn, nsite)
    al = torch.full((nn, nsite), -1, dtype=torch.int64, device="cuda")
    L0[:ntip] = (codes < 2).double()
    LA[:ntip] = (codes != 1).double()
    al[:ntip] = torch.where(codes == 0, -2, torch.where(codes == 1, -1, codes - 2))
    logs = f64(nsite)
    idx = lambda x: torch.from_numpy(x).cuda()  # noqa: E731

    def message(c, e):
        coef = torch.gather(q, 0, al[c].clamp(min=0))
        coef = torch.where(al[c] == -2, torch.ones_like(coef), torch.where(al[c] == -1, torch.zeros_like(coef), coef))
        stay, edit = torch.exp(-t[e])[:, None], -torch.expm1(-t[e])[:, None]
        diff = coef * LA[c] - L0[c]
        return L0[c] + edit * diff, stay * diff, coef, stay, edit

    for v in heights:
        iv, ca, cb = idx(v), idx(kid[v, 0]), idx(kid[v, 1])
        ma, mb = message(ca, idx(ked[v, 0]))[0], message(cb, idx(ked[v, 1]))[0]
        x, y = al[ca], al[cb]
        which = torch.where(x == -2, y, torch.where((y == -2) | (x == y), x, torch.full_like(x, -1)))
        l0 = ma * mb
        la = torch.where(which == -1, torch.zeros_like(l0), LA[ca] * LA[cb])
        s, e = _scale(torch.maximum(l0, la))
        L0[iv], LA[iv], sc[iv], al[iv] = l0 * s, la * s, s, torch.where(la > 0, which, torch.full_like(which, -1))
        logs += e.sum(0) * math.log(2.0)
    ll = float((torch.log(L0[ntip]) + logs).sum())
    g0, ga = f64(nn, nsite), f64(nn, nsite)
    g0[ntip] = 1.0 / L0[ntip]
    grad = f64(nn - 1)
    for v in depths:
        iv = idx(v)
        cs, es = [idx(kid[v, s]) for s in (0, 1)], [idx(ked[v, s]) for s in (0, 1)]
        m = [message(c, e) for c, e in zip(cs, es)]
        h0 = g0[iv] * sc[iv]
        hA = torch.where(al[iv] == -1, torch.zeros_like(h0), ga[iv] * sc[iv])
        for s in (0, 1):
            _, dm, coef, stay, edit = m[s]
            gm = h0 * m[1 - s][0]
            grad[es[s]] = (gm * dm).sum(1)
            g0[cs[s]] = gm * stay
            ga[cs[s]] = gm * edit * coef + hA * LA[cs[1 - s]]
    return ll, grad.cpu().numpy()

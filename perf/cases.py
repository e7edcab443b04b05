"""The calls a program makes into this framework, as cases to be timed.

A case names one public entry point of the package, the sizes and options of
the call, and the distribution its tensor is drawn from:

  s3ttmc   SpSymtensor.s3ttmc_device: Y = X_(1) (U x ... x U), U and Y on the
           device, packed or full rows, FP64 or FP32 (the kernel every solver
           iteration spends most of its time in)
  host     SpSymtensor.S3TTMc: the same with NumPy arrays in and out (the call
           that replaces the reference's SpSymtensor::S3TTMc)
  gram     gram_device: the m x m Gram matrix of the scaled packed rows, HOOI's
           dense step (FP64 for the drop-in, FP32 input for mixed precision)
  hooi     SpSymtensor.TuckerHOOI: whole iterations, FP64

Tensors are seeded synthetic ones of the families the package is used on:
ids ~ Zipf(s) over a random ranking of the nodes, or power-law, Zipf or equal
degrees with a fraction of the tuples inside one of k planted communities.
"""
import itertools
import math

import numpy as np
import torch

import symprop_b200 as sp

DEV = "cuda"


def listed():
    return [
        # Warm-start training tensors (orders 3 to 6, rank 8): order 3, full (unpacked) FP32 rows.
        {"name": "s3ttmc_o3_planted_f32_full", "kind": "s3ttmc", "order": 3, "n": 12007, "nnz": 240011, "R": 8,
         "prec": "f32", "packed": False, "family": "planted_zipf", "communities": 10, "s": 1.2},
        # The S3TTMc-alone workload: order 4, 5M Zipf tuples, rank 16.
        {"name": "s3ttmc_o4_zipf_f64", "kind": "s3ttmc", "order": 4, "n": 100000, "nnz": 5000000, "R": 16,
         "prec": "f64", "packed": True, "family": "zipf", "communities": 0, "s": 1.1},
        # An ordinary order-4 tensor in FP32 with sizes that divide nothing and an odd rank.
        {"name": "s3ttmc_o4_ragged_f32", "kind": "s3ttmc", "order": 4, "n": 30011, "nnz": 900001, "R": 13,
         "prec": "f32", "packed": True, "family": "zipf", "communities": 0, "s": 1.1},
        # The reference's plain HOOI tensor (order 5, 250 nodes, 10k tuples, rank 8): the smallest call.
        {"name": "s3ttmc_o5_small_f64", "kind": "s3ttmc", "order": 5, "n": 250, "nnz": 10000, "R": 8,
         "prec": "f64", "packed": True, "family": "zipf", "communities": 0, "s": 1.2},
        # The learned-start HOOI workload at full size, FP64: the largest call.
        {"name": "s3ttmc_o5_powerlaw_f64", "kind": "s3ttmc", "order": 5, "n": 200000, "nnz": 20000000, "R": 16,
         "prec": "f64", "packed": True, "family": "powerlaw", "communities": 16, "s": 0.0},
        # A tenth of it in FP32: the S3TTMc of mixed-precision HOOI.
        {"name": "s3ttmc_o5_powerlaw_f32", "kind": "s3ttmc", "order": 5, "n": 20000, "nnz": 2000000, "R": 16,
         "prec": "f32", "packed": True, "family": "powerlaw", "communities": 16, "s": 0.0},
        # The mixed-precision order-6 workload, rank 10.
        {"name": "s3ttmc_o6_planted_f32", "kind": "s3ttmc", "order": 6, "n": 50000, "nnz": 2000000, "R": 10,
         "prec": "f32", "packed": True, "family": "planted", "communities": 8, "s": 0.0},
        # The drop-in call with host arrays on an ordinary tensor.
        {"name": "host_o4_zipf_f64", "kind": "host", "order": 4, "n": 5000, "nnz": 200000, "R": 8,
         "prec": "f64", "packed": True, "family": "zipf", "communities": 0, "s": 1.1},
        # HOOI's FP64 Gram on the learned-start workload (packed rows of order 5, rank 16).
        {"name": "gram_f64", "kind": "gram", "n": 200000, "m": 3876, "prec": "f64"},
        # HOOI's mixed-precision Gram on the order-6 workload (packed rows of order 6, rank 10).
        {"name": "gram_f32", "kind": "gram", "n": 50000, "m": 2002, "prec": "f32"},
        # The reference's HOOI configuration: 250 nodes, rank 8, delta 0.1 (n <= m: the n x n Gram).
        {"name": "hooi_o5_small", "kind": "hooi", "order": 5, "n": 250, "nnz": 10000, "R": 8, "iters": 6,
         "delta": 0.1, "family": "zipf", "communities": 0, "s": 1.2},
        # FP64 HOOI on a tenth of the learned-start workload (n > m: the m x m Gram).
        {"name": "hooi_o5_powerlaw", "kind": "hooi", "order": 5, "n": 20000, "nnz": 2000000, "R": 16, "iters": 2,
         "delta": 1.0, "family": "powerlaw", "communities": 16, "s": 0.0},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _tensor(rng, order):
    """Sizes of one tensor of this order: the ranges of the listed ones."""
    lo_n, hi_n, lo_z, hi_z = {3: (1000, 20000, 10000, 500000), 4: (1000, 100000, 10000, 5000000),
                              5: (250, 200000, 10000, 10000000), 6: (1000, 50000, 10000, 2000000)}[order]
    n = _log(rng, lo_n, hi_n)
    nnz = max(2000, min(_log(rng, lo_z, hi_z), (20 if order == 3 else 100) * n))
    family = rng.choice({3: ["planted_zipf", "zipf"], 4: ["zipf", "planted_zipf"], 5: ["powerlaw", "zipf"],
                         6: ["planted", "planted_zipf"]}[order])
    communities = 0 if family == "zipf" else rng.randint(4, 16)
    s = rng.choice([1.1, 1.2]) if "zipf" in family else 0.0
    return {"order": order, "n": n, "nnz": nnz, "family": family, "communities": communities, "s": s}


def draw(rng):
    kind = rng.choice(["s3ttmc", "s3ttmc", "s3ttmc", "host", "gram", "hooi"])
    if kind == "gram":
        m = rng.choice([120, 330, 816, 1365, 2002, 3060, 3876])  # packed widths of orders 4 to 6, ranks 8 to 16
        return {"kind": "gram", "n": _log(rng, 1000, 150000), "m": m, "prec": rng.choice(["f64", "f32"])}
    if kind == "hooi":
        case = _tensor(rng, rng.choice([4, 5]))
        case["nnz"] = min(case["nnz"], 2000000)
        case["n"] = min(case["n"], 40000)
        return {"kind": "hooi", "R": rng.randint(4, 12), "iters": rng.randint(2, 4), "delta": 1.0, **case}
    if kind == "host":
        case = _tensor(rng, rng.choice([3, 4]))
        case["n"] = min(case["n"], 20000)
        case["nnz"] = min(case["nnz"], 500000, (20 if case["order"] == 3 else 100) * case["n"])
        return {"kind": "host", "R": rng.randint(4, 12), "prec": rng.choice(["f64", "f32"]), "packed": True, **case}
    order = rng.choice([3, 4, 5, 6])
    case = _tensor(rng, order)
    R = rng.choice([rng.randint(4, 10 if order == 6 else 16), 8, 10 if order == 6 else 16])
    packed = True if order > 4 else rng.choice([True, True, False])
    return {"kind": "s3ttmc", "R": R, "prec": rng.choice(["f64", "f32"]), "packed": packed, **case}


# ------------------------------------------------------------------ inputs

def _zipf(n, s):
    return np.arange(1, n + 1, dtype=np.float64) ** (-s)


def _tuples(case, seed):
    """nnz unique sorted tuples (device, 0-based) of the case's family."""
    order, n, nnz, k = case["order"], case["n"], case["nnz"], case["communities"]
    g = torch.Generator(device=DEV).manual_seed(seed)
    w = {"zipf": lambda: _zipf(n, case["s"]), "planted_zipf": lambda: _zipf(n, case["s"]),
         "powerlaw": lambda: _zipf(n, 1.0 / 1.1), "planted": lambda: np.ones(n)}[case["family"]]()
    node = torch.randperm(n, generator=g, device=DEV)  # node of every weight rank
    cdf = torch.from_numpy(np.cumsum(w) / w.sum()).to(DEV)
    if k:
        # ranks c, c + k, c + 2k, ... are community c: one increasing table c + cdf_c over all communities
        parts = [np.arange(c, n, k) for c in range(k)]
        table = torch.from_numpy(np.concatenate([c + np.cumsum(w[p]) / w[p].sum() for c, p in enumerate(parts)])).to(DEV)
        ranks = torch.from_numpy(np.concatenate(parts)).to(DEV)
        last = torch.tensor(np.cumsum([len(p) for p in parts]) - 1, device=DEV)
    frac_in = {"powerlaw": 0.8, "planted": 0.8, "planted_zipf": 0.9}.get(case["family"], 0.0)
    bits = max(1, (n - 1).bit_length())
    per = 63 // bits

    def some(count):
        u = torch.rand((count, order), generator=g, device=DEV, dtype=torch.float64)
        t = torch.searchsorted(cdf, u, right=True).clamp_(max=n - 1)
        if k:
            inside = torch.rand((count, 1), generator=g, device=DEV) < frac_in
            c = torch.randint(0, k, (count, 1), generator=g, device=DEV)
            at = torch.minimum(torch.searchsorted(table, u + c, right=True), last[c])
            t = torch.where(inside, ranks[at], t)
        return node[t].sort(dim=1).values

    def unique(t):
        keys = []
        for a in range(0, order, per):
            key = torch.zeros(t.shape[0], dtype=torch.int64, device=DEV)
            for j in range(a, min(order, a + per)):
                key = (key << bits) | t[:, j]
            keys.append(key)
        p = torch.arange(t.shape[0], device=DEV)
        for key in reversed(keys):
            p = p[torch.sort(key[p], stable=True).indices]
        new = torch.ones(t.shape[0], dtype=torch.bool, device=DEV)
        new[1:] = False
        for key in keys:
            new[1:] |= key[p][1:] != key[p][:-1]
        return t[p[new]]

    have = unique(some(int(nnz * 1.3) + 1024))
    for _ in range(60):
        if have.shape[0] >= nnz:
            break
        have = unique(torch.cat([have, some(int(nnz * 0.7) + 1024)]))
    if have.shape[0] < nnz:
        raise ValueError("could not draw %d unique tuples" % nnz)
    return have[torch.randperm(have.shape[0], generator=g, device=DEV)[:nnz]]


def _values(case, seed):
    """Order 4: uniform (0, 1]; the other workloads count occurrences (1.0)."""
    if case["order"] != 4:
        return np.ones(case["nnz"])
    return (1.0 - np.random.default_rng(seed + 7919).random(case["nnz"], dtype=np.float32)).astype(np.float64)


def _factor(case, seed):
    """Orthonormal n x R, FP64."""
    g = torch.Generator(device=DEV).manual_seed(seed + 104729)
    return torch.linalg.qr(torch.randn((case["n"], case["R"]), generator=g, device=DEV, dtype=torch.float64)).Q.contiguous()


def _rows(case, seed):
    """Packed rows as S3TTMc leaves them (row scales of a power-law degree
    sequence, most rows light, a common part in all of them) and the square
    roots of the packed columns' multiplicities."""
    n, m = case["n"], case["m"]
    g = torch.Generator(device=DEV).manual_seed(seed)
    f64 = case["prec"] == "f64"
    dt = torch.float64 if f64 else torch.float32
    Y = torch.randn((n, m), generator=g, device=DEV, dtype=dt)
    Y += torch.randn((n, 1), generator=g, device=DEV, dtype=dt) * torch.randn((1, m), generator=g, device=DEV, dtype=dt)
    rank = torch.randperm(n, generator=g, device=DEV) + 1
    Y *= (rank.to(torch.float64) / n).pow(-1.0 / 2.2).to(dt)[:, None] * 1e-3
    D = torch.tensor([1.0, 4.0, 6.0, 12.0, 24.0], dtype=torch.float64, device=DEV)
    sd = D[torch.randint(0, 5, (m,), generator=g, device=DEV)].sqrt().to(dt)
    return Y, sd


def prepare(case, seed):
    kind = case["kind"]
    if kind == "gram":
        Y, sd = _rows(case, seed)
        return {"case": case, "Y": Y, "sd": sd, "G": torch.empty((case["m"], case["m"]), dtype=torch.float64, device=DEV)}
    inds = (_tuples(case, seed) + 1).to(torch.int32).cpu().numpy().view(np.uint32)
    U = _factor(case, seed)
    state = {"case": case, "X": sp.SpSymtensor(case["n"], case["order"], inds, _values(case, seed))}
    if kind == "hooi":
        state["U"] = U.cpu().numpy()
        return state
    dt = torch.float64 if case["prec"] == "f64" else torch.float32
    U = U.to(dt)
    if kind == "host":
        state["U"] = U.cpu().numpy()
    else:
        state["U"] = U
        state["Y"] = torch.empty((case["n"], state["X"].ncols(case["R"], case["packed"])), dtype=dt, device=DEV)
    return state


def run(state):
    case = state["case"]
    kind = case["kind"]
    prec = sp.FP64 if case.get("prec", "f64") == "f64" else sp.FP32
    stream = torch.cuda.current_stream().cuda_stream
    if kind == "gram":
        sp.gram_device(state["Y"].data_ptr(), case["n"], case["m"], state["sd"].data_ptr(), state["G"].data_ptr(), prec, stream)
        return state["G"]
    if kind == "s3ttmc":
        state["X"].s3ttmc_device(state["U"].data_ptr(), case["R"], state["Y"].data_ptr(), case["packed"], prec, stream)
        return state["Y"]
    if kind == "host":
        return state["X"].S3TTMc(state["U"], case["R"], case["packed"], prec)
    d = state["X"].TuckerHOOI(rank=case["R"], max_iter=case["iters"], rel_tol=0.0, delta=case["delta"], init="user",
                              init_factor=state["U"])
    return {"core": d.core, "factor": d.factor, "error_trace": d.error_trace}


def work(case):
    if case["kind"] == "gram":
        n, m, s = case["n"], case["m"], 8 if case["prec"] == "f64" else 4
        return {"bytes": s * (n * m + m) + 8 * m * m, "flops": n * m * (m + 1)}
    N, n, nnz, R = case["order"], case["n"], case["nnz"], case["R"]
    s = 4 if case.get("prec") == "f32" else 8
    m = math.comb(R + N - 2, N - 1)
    cols = m if case.get("packed", True) else R ** (N - 1)
    # tuples, values and U read, Y written; every tuple meets each of its N
    # rows with at least one order-2 product, and every row is symmetrised
    one = {"bytes": nnz * (4 * N + 8) + s * n * (R + cols), "flops": N * nnz * R * (R + 1) + 2 * n * (N - 1) * m}
    if case["kind"] != "hooi":
        return one
    small, long = min(n, m), max(n, m)  # the Gram of the smaller side, U and the core
    flops = one["flops"] + long * small * (small + 1) + 4 * n * m * R
    return {"bytes": case["iters"] * one["bytes"], "flops": case["iters"] * flops}


# ------------------------------------------------- 64-bit values, plain torch

def _multisets(R, d):
    return torch.tensor(list(itertools.combinations_with_replacement(range(R), d)), device=DEV)


def _at(R, d):
    """(R,)*d table: the packed (lexicographic) place of a sorted index tuple."""
    table = torch.zeros((R,) * d, dtype=torch.int64, device=DEV)
    q = _multisets(R, d)
    table[tuple(q.T)] = torch.arange(q.shape[0], device=DEV)
    return table


def _sym(U, ids):
    """rows x packed(d): the sum over all orderings of the ids' rows, P[q] = sum_perm prod_k U[id_perm(k)][q_k]."""
    R = U.shape[1]
    P = U[ids[:, 0]]
    for d in range(2, ids.shape[1] + 1):
        q, u, old = _multisets(R, d), U[ids[:, d - 1]], _at(R, d - 1)
        out = torch.zeros((ids.shape[0], q.shape[0]), dtype=U.dtype, device=DEV)
        for t in range(d):
            rest = [q[:, j] for j in range(d) if j != t]
            out += u[:, q[:, t]] * P[:, old[tuple(rest)]]
        P = out
    return P


def _s3ttmc(case, inds, vals, U):
    """Packed Y in 64 bits: for a leaf split into parts A and B,
    K(S)[q] = sum over the places I of A of P_A[q_I] P_B[q without I], so a
    row needs M = sum_o c_o P_A (x) P_B once (rows of like length together)."""
    N, n, R = case["order"], case["n"], case["R"]
    L, a = N - 1, N // 2
    same = torch.ones(inds.shape[0], dtype=torch.float64, device=DEV)
    run = torch.ones_like(same)
    for j in range(1, N):  # product of the factorials of the ids' multiplicities
        run = torch.where(inds[:, j] == inds[:, j - 1], run + 1, torch.ones_like(run))
        same *= run
    coef = vals / same
    rows = torch.cat([inds[:, j] for j in range(N)])
    by_row = torch.sort(rows, stable=True).indices
    count = torch.bincount(rows, minlength=n)
    start = torch.cumsum(count, 0) - count
    z = inds.shape[0]
    others = torch.tensor([[k for k in range(N) if k != j] for j in range(N)], device=DEV)
    q = _multisets(R, L)
    pa, pb = _at(R, a), _at(R, L - a)
    places = []
    for I in itertools.combinations(range(L), a):
        J = [j for j in range(L) if j not in I]
        places.append(pa[tuple(q[:, i] for i in I)] * math.comb(R + L - a - 1, L - a) + pb[tuple(q[:, j] for j in J)])
    ma, mb = math.comb(R + a - 1, a), math.comb(R + L - a - 1, L - a)
    Y = torch.zeros((n, q.shape[0]), dtype=torch.float64, device=DEV)

    def block(owner, ok):  # (rows, K) places in by_row and which of them count
        o = by_row[owner.reshape(-1)]
        t, j = o % z, torch.div(o, z, rounding_mode="floor")
        S = inds[t].gather(1, others[j])
        c = coef[t] * ok.reshape(-1)
        A = _sym(U, S[:, :a]) * c[:, None]
        B = _sym(U, S[:, a:])
        k = min(owner.shape[1], 256)  # short sums, added pairwise: little rounding of its own
        M = torch.bmm(A.view(-1, k, ma).transpose(1, 2), B.view(-1, k, mb))
        return M.view(owner.shape[0], -1, ma, mb).sum(dim=1)

    most = 1 << int(math.log2(2e8 / (ma + mb)))  # owners at a time
    longest = int(count.max())
    width = 1
    while width < 2 * longest:
        sel = torch.nonzero((count <= width) & (count > width // 2)).reshape(-1)
        step = max(1, min(most // width, int(4e8) // (ma * mb)))
        for b in range(0, sel.shape[0], step):
            r = sel[b:b + step]
            M = torch.zeros((r.shape[0], ma, mb), dtype=torch.float64, device=DEV)
            for x in range(0, width, most):
                at = torch.arange(x, min(width, x + most), device=DEV)[None, :]
                ok = at < count[r][:, None]
                M += block((start[r][:, None] + at).clamp(max=rows.shape[0] - 1), ok)
            M = M.view(r.shape[0], -1)
            y = torch.zeros((r.shape[0], q.shape[0]), dtype=torch.float64, device=DEV)
            for p in places:
                y += M[:, p]
            Y[r] = y
        width *= 2
    return Y


def _hooi_errors(case, inds, vals, U):
    N, n, R = case["order"], case["n"], case["R"]
    q = _multisets(R, N - 1)
    D = torch.tensor([math.factorial(N - 1) / math.prod(math.factorial(c) for c in np.unique(x, return_counts=True)[1])
                      for x in q.cpu().numpy()], dtype=torch.float64, device=DEV)
    same, run = torch.ones_like(vals), torch.ones_like(vals)
    for j in range(1, N):
        run = torch.where(inds[:, j] == inds[:, j - 1], run + 1, torch.ones_like(run))
        same *= run
    x2 = (vals * vals * math.factorial(N) / same).sum()
    errors = []
    for _ in range(case["iters"]):
        norm = U.norm(dim=1, keepdim=True)
        U = torch.where(norm > case["delta"], U * (case["delta"] / norm), U)
        U = torch.linalg.qr(U).Q
        Z = _s3ttmc(case, inds, vals, U) * D.sqrt()
        if n <= q.shape[0]:
            U = torch.linalg.eigh(Z @ Z.T).eigenvectors[:, -R:].contiguous()
        else:
            U = torch.linalg.qr(Z @ torch.linalg.eigh(Z.T @ Z).eigenvectors[:, -R:]).Q
        errors.append(((x2 - (U.T @ Z).square().sum()) / x2).sqrt())
    return torch.stack(errors)


def exact(case, seed):
    if case["kind"] == "gram":
        Y, sd = _rows(case, seed)
        Y, sd = Y.double(), sd.double()
        G = torch.zeros((case["m"], case["m"]), dtype=torch.float64, device=DEV)
        low = torch.zeros_like(G)
        for b in range(0, case["n"], 256):  # short sums, added with their rounding errors (Knuth's two-sum)
            P = Y[b:b + 256].T @ Y[b:b + 256]
            S = G + P
            z = S - G
            low += (G - (S - z)) + (P - z)
            G = S
        return (G + low) * (sd[:, None] * sd[None, :])
    inds = _tuples(case, seed)
    vals = torch.from_numpy(_values(case, seed)).to(DEV)
    U = _factor(case, seed)
    if case["kind"] == "hooi":  # the basis of the factor and the core is the solver's own
        return {"core": None, "factor": None, "error_trace": _hooi_errors(case, inds, vals, U)}
    if case["prec"] == "f32":
        U = U.float().double()
    Y = _s3ttmc(case, inds, vals, U)
    if not case["packed"]:
        R, L = case["R"], case["order"] - 1
        full = torch.tensor(list(itertools.product(range(R), repeat=L)), device=DEV).sort(dim=1).values
        Y = Y[:, _at(R, L)[tuple(full.T)]]
    return Y

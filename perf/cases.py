"""The workloads whose speed this framework is judged by: exact KRP draws,
partition-tree rebuilds and the steps of randomized CP-ALS, each through the
calls a user's program makes.

Kinds of a case:
  draw     one draw of J samples from the KRP of N factors (Sampler)
  tree     the rebuild of one factor's partition tree (Sampler.update_sampler)
  als      one sampled update of mode j against a sparse tensor (ALS)
  exact    one exact least-squares update of mode j against a sparse tensor
  rrf      range-finder initialisation of all factors from a sparse tensor
  fit      the residual of a model against a sparse tensor
  lowrank  one sampled update of mode j against an implicit low-rank tensor
"""
import math

import numpy as np
import torch

DEV = "cuda"


# ------------------------------------------------------------------ cases

def listed():
    return [
        # The documented first example: a 10^12-row KRP drawn from with the
        # default precision into numpy arrays.  Launches, host calls and
        # copies back count most here.
        {"name": "readme draw, numpy", "kind": "draw", "dims": "1000,1000,1000,1000", "R": 8, "J": 10000, "j": 5,
         "precision": "fp64", "host": True},
        # The headline: 50,000 samples from a 6e20-row KRP, no mode excluded,
        # mixed precision, results left on the device.
        {"name": "large draw, mixed", "kind": "draw", "dims": "8388608,8388608,8388608", "R": 32, "J": 50000, "j": 4,
         "precision": "fp32", "host": False},
        # The same kind of draw at the default precision with one mode
        # excluded, as every least-squares solve of ALS asks for it.
        {"name": "large draw, fp64, one excluded", "kind": "draw", "dims": "4194304,4194304,4194304", "R": 32,
         "J": 50000, "j": 0, "precision": "fp64", "host": False},
        # A request of the serving mix: ragged modes, rank 64.
        {"name": "rank-64 draw, mixed", "kind": "draw", "dims": "1000003,300007,100003,1000003", "R": 64, "J": 32768,
         "j": 5, "precision": "fp32", "host": False},
        # Rebuild of a headline factor's tree through the tensor cores.
        {"name": "tree rebuild, tf32x3", "kind": "tree", "I": 8388608, "R": 32, "precision": "tf32x3"},
        # Rebuild after an update of a 1.8e6-row factor at rank 25, default precision.
        {"name": "tree rebuild, fp64", "kind": "tree", "I": 1800000, "R": 25, "precision": "fp64"},
        # Randomized CP-ALS on the power-law tensor at 1/6 of its full size:
        # one sampled update of its longest mode, mixed-precision sampling.
        {"name": "sparse ALS update, mixed", "kind": "als", "dims": "801600,300600,300600", "nnz": 25050000, "R": 25,
         "J": 65536, "j": 0, "precision": "fp32"},
        # The same at rank 100 (a rank the method is published at) and the
        # default precision, on a smaller tensor.
        {"name": "sparse ALS update, fp64, rank 100", "kind": "als", "dims": "200400,75150,75150", "nnz": 6262500,
         "R": 100, "J": 65536, "j": 1, "precision": "fp64"},
        # The baseline method against the same kind of tensor.
        {"name": "exact ALS update", "kind": "exact", "dims": "200400,75150,75150", "nnz": 6262500, "R": 25, "j": 0},
        # Initialisation of a run.
        {"name": "range finder", "kind": "rrf", "dims": "200400,75150,75150", "nnz": 6262500, "R": 25},
        # The fit that is taken every few sweeps.
        {"name": "fit", "kind": "fit", "dims": "801600,300600,300600", "nnz": 25050000, "R": 25},
        # The dense low-rank study: 65,536^4 entries of true rank 16,
        # decomposed at rank 64 with 2^17 samples.
        {"name": "low-rank ALS update, mixed", "kind": "lowrank", "dims": "65536,65536,65536,65536", "R": 64, "rank": 16,
         "J": 131072, "j": 1, "precision": "fp32", "snr_db": 0.0},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _odd(rng, v):
    """Half of the sizes as they fall, the others moved to a ragged one."""
    return v if rng.random() < 0.5 else v | 1


def draw(rng):
    """One more case: the kinds above over ranks 8..128, 3..6 modes, mode
    sizes 10^3..8*10^6, 2^10..2^17 samples, every tree precision."""
    kind = rng.choice(["draw"] * 5 + ["tree"] * 2 + ["als"] * 2 + ["exact", "rrf", "fit", "lowrank"])
    if kind == "draw":
        R = rng.choice([8, 16, 20, 25, 32, 32, 64, 100, 128])
        N = rng.randint(3, 6 if R <= 32 else 4)
        precision = rng.choice(["fp64", "fp64", "fp32", "fp32", "tf32x3", "bf16"])
        top = 8e6 * min(1.0, (32 / R) ** 2) * (0.5 if precision == "fp64" else 1.0)
        dims = [_odd(rng, _log(rng, 1e3, top)) for _ in range(N)]
        J = _log(rng, 1 << 10, (1 << 17) * min(1.0, (32 / R) ** 2))
        return {"kind": "draw", "dims": ",".join(map(str, dims)), "R": R, "J": _odd(rng, J),
                "j": rng.choice([0, N - 1, N + 1, N + 1]), "precision": precision, "host": rng.random() < 0.3}
    if kind == "tree":
        R = rng.choice([8, 16, 25, 32, 32, 64, 100])
        precision = rng.choice(["fp64", "fp32", "tf32x3", "bf16"])
        top = 8e6 * min(1.0, 32 / R) * (0.4 if precision == "fp64" else 1.0)
        return {"kind": "tree", "I": _odd(rng, _log(rng, 1e4, top)), "R": R, "precision": precision}
    if kind == "lowrank":
        R = rng.choice([16, 25, 64])
        N = rng.choice([3, 4])
        I = _odd(rng, _log(rng, 4096, 65536))
        snr = rng.choice([0.0, 0.0, 0.0, 20.0])
        return {"kind": "lowrank", "dims": ",".join([str(I)] * N), "R": R, "rank": rng.choice([8, 16]),
                "J": _odd(rng, _log(rng, 1 << 12, 1 << (17 if snr == 0.0 else 14))), "j": rng.randrange(N),
                "precision": rng.choice(["fp64", "fp32", "tf32x3"]) if R <= 25 else "fp32", "snr_db": snr}
    N = rng.choice([3, 3, 4])
    scale = math.exp(rng.uniform(math.log(0.005), math.log(0.12)))
    dims = [_odd(rng, max(500, int(d * scale))) for d in (4.8e6, 1.8e6, 1.8e6, 2e4)[:N]]
    c = {"kind": kind, "dims": ",".join(map(str, dims)), "nnz": int(1.5e8 * scale), "R": rng.choice([8, 16, 25, 25, 40])}
    if kind == "als":
        c["J"] = _odd(rng, _log(rng, 1 << 12, 1 << 16))
        c["precision"] = rng.choice(["fp64", "fp32", "tf32x3"])
    if kind in ("als", "exact"):
        c["j"] = rng.randrange(N)
    return c


def _dims(case):
    return [int(d) for d in case["dims"].split(",")]


# ----------------------------------------------------------------- inputs

def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return g


def _gaussian_factor(I, R, g):
    """N(0, 1) entries, 1% of the rows (at random) times 100: non-uniform leverage."""
    u = torch.randn((I, R), generator=g, device=DEV, dtype=torch.float64)
    u *= torch.where(torch.rand((I, 1), generator=g, device=DEV) < 0.01, 100.0, 1.0).to(torch.float64)
    return u


def _factors(case, seed):
    g = _gen(seed)
    dims = _dims(case) if "dims" in case else [case["I"]]
    return [_gaussian_factor(I, case["R"], g) for I in dims]


def _tensor(case, seed):
    from fast_tensor_leverage_gb300.synthetic import sparse_powerlaw_tensor
    return sparse_powerlaw_tensor(_dims(case), case["nnz"], 1.1, seed=seed, device=DEV)


def _energy_factors(case, seed, idx):
    """Factors as a range finder leaves them: a row's energy follows the
    number of its nonzeros, rows without any are zero, columns are unit."""
    g = _gen(seed + 77)
    out = []
    for k, I in enumerate(_dims(case)):
        deg = torch.bincount(idx[:, k].to(torch.int64), minlength=I).to(torch.float64)
        u = torch.randn((I, case["R"]), generator=g, device=DEV, dtype=torch.float64) * deg.sqrt().unsqueeze(1)
        out.append(u / u.square().sum(dim=0).sqrt())
    return out


def _model(case, seed):
    """The implicit low-rank tensor's factors and the decomposition's."""
    g = _gen(seed)
    dims = _dims(case)
    V = [torch.randn((I, case["rank"]), generator=g, device=DEV, dtype=torch.float64) for I in dims]
    U = [torch.randn((I, case["R"]), generator=g, device=DEV, dtype=torch.float64) for I in dims]
    return V, U


def prepare(case, seed):
    import fast_tensor_leverage_gb300 as ftl
    kind, R = case["kind"], case["R"]
    s = {"case": case}
    if kind in ("draw", "tree"):
        U = _factors(case, seed)
        s["sampler"] = ftl.Sampler(U, case.get("J", 1), R, "efficient", precision=case["precision"], seed=seed)
        if case.get("host"):
            N, J = len(U), case["J"]
            s["out"] = (np.zeros((N, J), dtype=np.uint64), np.zeros((J, R)), np.zeros(J))
        return s
    if kind == "lowrank":
        V, U = _model(case, seed)
        rhs = ftl.LowRankTensor(case["rank"], 10000, V, sync_host=False)
        if case["snr_db"]:
            rhs.set_noise_snr(case["snr_db"], seed=seed)
        lr = ftl.LowRankTensor(R, U, sync_host=False)
        s["als"] = ftl.ALS(lr, rhs)
        s["als"].initialize_ds_als(case["J"], "efficient", precision=case["precision"], seed=seed)
        return s
    idx, vals = _tensor(case, seed)
    sp = s["tensor"] = ftl.SparseTensor(idx, vals, "sort", dims=_dims(case))
    if kind == "rrf":
        s["seed"] = seed
        s["lr"] = ftl.PyLowRank(_dims(case), R, seed=1, sync_host=False).ten
        return s
    lr = s["lr"] = ftl.LowRankTensor(R, _energy_factors(case, seed, idx), sync_host=False)
    if kind in ("als", "exact"):
        s["als"] = ftl.ALS(lr, sp)
    if kind == "als":
        s["als"].initialize_ds_als(case["J"], "efficient", precision=case["precision"], seed=seed)
    return s


# -------------------------------------------------------------------- run

def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "draw":
        sampler = state["sampler"]
        if case["host"]:
            samples, h, w = state["out"]
            sampler.KRPDrawSamples_materialize(case["j"], samples, h, w)
            return {"samples": samples.view(np.int64), "h": h, "weights": w}
        samples, h, w = sampler.draw(case["j"])
        return {"samples": samples, "h": h, "weights": w}
    if kind == "tree":
        sampler = state["sampler"]
        sampler.update_sampler(0)
        out = {"tree": sampler.trees[0]}
        if sampler.U32 is not None:
            out["copy"] = sampler.U32[0]
        return out
    if kind in ("als", "lowrank"):
        als, j = state["als"], case["j"]
        als.execute_ds_als_update(j, True, True)
        return {"factor": als.cp_decomp.U_dev[j], "sigma": als.cp_decomp.sigma_dev}
    if kind == "exact":
        als, j = state["als"], case["j"]
        als.execute_exact_als_update(j, True, True)
        return {"factor": als.cp_decomp.U_dev[j], "sigma": als.cp_decomp.sigma_dev}
    if kind == "rrf":
        lr = state["lr"]
        state["tensor"].execute_rrf(lr, seed=state["seed"])
        return {"factors": list(lr.U_dev), "sigma": lr.sigma_dev}
    if kind == "fit":
        lr = state["lr"]
        return {"terms": state["tensor"].residual_terms_async(lr.sigma_dev, lr.U_dev)}
    raise ValueError(kind)


# ------------------------------------------------------------------- work

def _tree_levels(n, F):
    leaves = -(-n // F)
    return max(0, (leaves - 1).bit_length()), leaves


def _draw_work(dims, R, J, j, precision):
    """One node read per level of a sampled path (each distinct node once),
    the leaf blocks, the outputs; two operations per entry of a node's
    triangle, of a leaf block and of the row table."""
    P = R * (R + 1) // 2
    es = 8 if precision == "fp64" else 4
    nbytes = nflops = 0.0
    for k, n in enumerate(dims):
        if k == j:
            continue
        F = min(R, n)
        levels, leaves = _tree_levels(n, F)
        el = max(1, (R - 1).bit_length())
        nodes = 1 + sum(min(J, 2 ** d) for d in range(levels))
        enodes = min(R, 1 + sum(2 ** d for d in range(el)))
        nbytes += (nodes + enodes) * P * es + min(J, leaves) * F * R * es + R * R * 8
        nflops += J * (2.0 * P * (levels + el + 2) + 2.0 * F * R)
    nbytes += J * (8.0 * (len(dims) - (1 if j < len(dims) else 0)) + 8.0 * R + 8.0)
    nflops += J * 2.0 * P
    return nbytes, nflops


def _tree_work(I, R, precision):
    P = R * (R + 1) // 2
    es = 8 if precision == "fp64" else 4
    leaves = -(-I // min(R, I))
    nbytes = I * R * (8 if es == 8 else 12) + (2 * leaves - 1) * P * es
    return nbytes, 2.0 * I * P + leaves * P


def work(case):
    kind, R = case["kind"], case["R"]
    P = R * (R + 1) // 2
    if kind == "draw":
        b, f = _draw_work(_dims(case), R, case["J"], case["j"], case["precision"])
        return {"bytes": b, "flops": f}
    if kind == "tree":
        b, f = _tree_work(case["I"], R, case["precision"])
        return {"bytes": b, "flops": f}
    dims = _dims(case)
    if kind in ("als", "lowrank"):
        J, j = case["J"], case["j"]
        b, f = _draw_work(dims, R, J, j, case["precision"])
        tb, tf = _tree_work(dims[j], R, case["precision"])
        f += tf + J * (2.0 * P + 2.0 * R * R)
        b += tb - (dims[j] * R * 4 if case["precision"] != "fp64" else 0)  # no FP32 copy is kept here
        if kind == "als":
            b += case["nnz"] * 20.0 + dims[j] * R * 16.0
        else:
            b += sum(8.0 * n * case["rank"] for n in dims) + dims[j] * R * 16.0
            f += 2.0 * J * case["rank"] * R + 2.0 * dims[j] * case["rank"] * R
        return {"bytes": b, "flops": f}
    nnz, N = float(case["nnz"]), len(dims)
    if kind == "exact":
        others = sum(dims) - dims[case["j"]]
        return {"bytes": nnz * (4 * N + 8) + others * R * 8.0 + dims[case["j"]] * R * 8.0,
                "flops": nnz * R * N + others * 2.0 * P + dims[case["j"]] * 2.0 * R * R}
    if kind == "rrf":
        return {"bytes": N * nnz * 20.0 + sum(dims) * R * 8.0, "flops": N * nnz * R * 2.0}
    return {"bytes": nnz * (4 * N + 8) + sum(dims) * R * 8.0, "flops": nnz * R * (N + 1) + sum(dims) * 2.0 * P}


# ------------------------------------------------------------------ exact
# What run() returns, in plain torch in 64 bits.

def _philox(c0, c1, c2, c3, seed):
    """Philox4x32-10 on int64 tensors holding 32-bit words."""
    mask = 0xFFFFFFFF
    k0, k1 = seed & mask, (seed >> 32) & mask
    for _ in range(10):
        p0, p1 = c0 * 0xD2511F53, c2 * 0xCD9E8D57
        c0, c1, c2, c3 = (((p1 >> 32) & mask) ^ c1 ^ k0, p1 & mask, ((p0 >> 32) & mask) ^ c3 ^ k1, p0 & mask)
        k0, k1 = (k0 + 0x9E3779B9) & mask, (k1 + 0xBB67AE85) & mask
    return c0, c1


def _uniforms(n, seed):
    i = torch.arange(n, device=DEV, dtype=torch.int64)
    z = torch.zeros_like(i)
    a, b = _philox(i & 0xFFFFFFFF, i >> 32, z, z, seed)
    return (((a >> 5) << 26) | (b >> 6)).to(torch.float64) * 2.0 ** -53


def _pick(mass, u):
    """First index whose running share of the row's mass reaches u, and
    where in that share u falls."""
    c = torch.cumsum(mass, dim=1)
    t = u.unsqueeze(1) * c[:, -1:]
    i = torch.searchsorted(c, t).clamp_(max=mass.shape[1] - 1)
    lo = torch.where(i > 0, c.gather(1, (i - 1).clamp_(min=0)), torch.zeros_like(t))
    m = mass.gather(1, i)
    return i.squeeze(1), ((t - lo) / m).squeeze(1).clamp_(0.0, 1.0)


def _exact_draw(U, J, j, seed):
    """J samples of the KRP of U without mode j: samples (N x J), rows h, weights."""
    N, R = len(U), U[0].shape[1]
    modes = [k for k in range(N) if k != j]
    uni = _uniforms(2 * N * J, seed).reshape(2 * N, J)
    G = [u.T @ u for u in U]
    M = torch.ones((R, R), device=DEV, dtype=torch.float64)
    suffix = {}
    for k in reversed(modes):
        M = M * G[k]
        suffix[k] = M
    lam, Q = torch.linalg.eigh(suffix[modes[0]])
    inv = torch.where(lam > 1e-8, 1.0 / lam, torch.zeros_like(lam))
    pinv = (Q * inv) @ Q.T
    h = torch.ones((J, R), device=DEV, dtype=torch.float64)
    samples = torch.zeros((N, J), device=DEV, dtype=torch.int64)
    for at, k in enumerate(modes):
        if at + 1 < len(modes):
            lk, Qk = torch.linalg.eigh(suffix[modes[at + 1]] * pinv)
            W = (Qk * lk.clamp(min=0.0).sqrt()).T.contiguous()
        else:
            W = (Q * inv.sqrt()).T.flip(0).contiguous()
        B = 2048                                   # rows per block of the two-stage pick
        I = U[k].shape[0]
        nb = -(-I // B)
        pad = torch.zeros((nb * B, R), device=DEV, dtype=torch.float64)
        pad[:I] = U[k]
        blocks = pad.reshape(nb, B, R)
        bg = torch.cat([torch.bmm(b.transpose(1, 2), b) for b in blocks.split(64)]).reshape(nb, R * R)
        step = max(1, min(1 << 14, (1 << 27) // (R * R)))
        small = max(1, (1 << 27) // (B * R))
        for a in range(0, J, step):
            hh = h[a:a + step]
            S = hh.shape[0]
            V = (hh.unsqueeze(1) * W).reshape(S * R, R)
            e, _ = _pick(((V @ G[k]) * V).sum(dim=1).reshape(S, R).clamp_(min=0.0), uni[k, a:a + S])
            x = hh * W[e]
            xx = (x.unsqueeze(2) * x.unsqueeze(1)).reshape(S, R * R)
            b, f = _pick((xx @ bg.T).clamp_(min=0.0), uni[N + k, a:a + S])
            for c in range(0, S, small):
                q = torch.bmm(blocks[b[c:c + small]], x[c:c + small].unsqueeze(2)).squeeze(2).square()
                r, _ = _pick(q, f[c:c + small])
                row = (b[c:c + small] * B + r).clamp_(max=I - 1)
                samples[k, a + c:a + c + row.shape[0]] = row
            h[a:a + S] = hh * U[k][samples[k, a:a + S]]
        del pad, blocks, bg
    w = R / (J * ((h @ pinv) * h).sum(dim=1))
    return samples, h, w


def _pinv(G, tol):
    lam, Q = torch.linalg.eigh(G)
    inv = torch.where(lam > tol, 1.0 / lam, torch.zeros_like(lam))
    return (Q * inv) @ Q.T


def _normalised(u):
    n = u.square().sum(dim=0).sqrt()
    n = torch.where(n <= 1e-7, torch.ones_like(n), n)
    return u / n, n


def _node_of(n, F):
    """Heap positions of the leaves and the number of nodes of a tree over n rows."""
    leaves = -(-n // F)
    full = 1 << (leaves.bit_length() - 1)
    upto = 2 * full - 1
    nodes = 2 * leaves - 1
    deep = nodes - upto
    leaf = torch.arange(leaves, device=DEV)
    return torch.where(leaf < deep, upto + leaf, leaf + (full - 1) - deep // 2), nodes


def _exact_tree(U, R, precision):
    """Node Grams in the layout that ftl.h documents."""
    n = U.shape[0]
    F = min(R, n)
    node, count = _node_of(n, F)
    leaves = node.shape[0]
    if precision != "fp64" and 16 < R <= 32:       # wrapped diagonals of the padded 32 x 32 Gram
        e = torch.arange(544, device=DEV)
        a = torch.where(e < 512, (e >> 2) & 31, e - 512)
        d = torch.where(e < 512, ((e >> 7) << 2) + (e & 3), 16)
        b = (a + d) & 31
        keep = (a < R) & (b < R)
        a, b = a.clamp(max=R - 1), b.clamp(max=R - 1)
    else:
        a, b = torch.triu_indices(R, R, device=DEV)
        w = 2 if precision == "fp64" else 4
        padding = -a.numel() % w
        keep = torch.cat([torch.ones_like(a), torch.zeros(padding, device=DEV, dtype=a.dtype)]).bool()
        a, b = (torch.cat([t, torch.zeros(padding, device=DEV, dtype=t.dtype)]) for t in (a, b))
    T = torch.zeros((count, a.numel()), device=DEV, dtype=torch.float64)
    pos = a * R + b
    for l0 in range(0, leaves, 1 << 14):
        l1 = min(leaves, l0 + (1 << 14))
        rows = torch.zeros(((l1 - l0) * F, R), device=DEV, dtype=torch.float64)
        rows[:min(n, l1 * F) - l0 * F] = U[l0 * F:l1 * F]
        blk = rows.reshape(l1 - l0, F, R)
        T[node[l0:l1]] = torch.bmm(blk.transpose(1, 2), blk).reshape(l1 - l0, R * R)[:, pos] * keep
    hi = count - leaves                            # nodes below hi are internal
    while hi > 0:
        lo = (1 << (hi.bit_length() - 1)) - 1      # the deepest level with an internal node
        T[lo:hi] = T[2 * lo + 1:2 * hi + 1:2] + T[2 * lo + 2:2 * hi + 2:2]
        hi = lo
    return T.reshape(-1)


def _keys(cols, dims, j):
    key = torch.zeros_like(cols[0], dtype=torch.int64)
    for k, d in enumerate(dims):
        if k != j:
            key = key * d + cols[k].to(torch.int64)
    return key


def _exact_als(case, seed):
    dims, R, J, j = _dims(case), case["R"], case["J"], case["j"]
    idx, vals = _tensor(case, seed)
    U = _energy_factors(case, seed, idx)
    samples, h, w = _exact_draw(U, J, j, seed)
    gram = (h * w.unsqueeze(1)).T @ h
    cols = [idx[:, k] for k in range(len(dims))]
    sk, inverse = torch.unique(_keys(samples, dims, j), return_inverse=True)
    rows = torch.zeros((sk.shape[0], R), device=DEV, dtype=torch.float64)
    rows.index_add_(0, inverse, h * w.unsqueeze(1))
    zk = _keys(cols, dims, j)
    at = torch.searchsorted(sk, zk).clamp_(max=sk.shape[0] - 1)
    hit = torch.nonzero(sk[at] == zk).squeeze(1)
    out = torch.zeros((dims[j], R), device=DEV, dtype=torch.float64)
    for part in hit.split(1 << 22):
        out.index_add_(0, cols[j][part].to(torch.int64), vals[part].unsqueeze(1) * rows[at[part]])
    f, sigma = _normalised(out @ _pinv(gram, 1e-11))
    return {"factor": f, "sigma": sigma}


def _exact_update(case, seed):
    dims, R, j = _dims(case), case["R"], case["j"]
    idx, vals = _tensor(case, seed)
    U = _energy_factors(case, seed, idx)
    M = torch.ones((R, R), device=DEV, dtype=torch.float64)
    for k, u in enumerate(U):
        if k != j:
            M = M * (u.T @ u)
    out = torch.zeros((dims[j], R), device=DEV, dtype=torch.float64)
    for z in torch.arange(idx.shape[0], device=DEV).split(1 << 21):
        p = vals[z].unsqueeze(1).expand(-1, R)
        for k, u in enumerate(U):
            if k != j:
                p = p * u[idx[z, k].to(torch.int64)]
        out.index_add_(0, idx[z, j].to(torch.int64), p)
    f, sigma = _normalised(out @ _pinv(M, 1e-11))
    return {"factor": f, "sigma": sigma}


def _exact_rrf(case, seed):
    dims, R = _dims(case), case["R"]
    idx, vals = _tensor(case, seed)
    cols = [idx[:, k] for k in range(len(dims))]
    factors, sigma = [], torch.ones(R, device=DEV, dtype=torch.float64)
    for j in range(len(dims)):
        keys = _keys(cols, dims, j)
        out = torch.zeros((dims[j], R), device=DEV, dtype=torch.float64)
        for z in torch.arange(idx.shape[0], device=DEV).split(1 << 20):
            k = keys[z].unsqueeze(1)
            p = torch.arange((R + 1) // 2, device=DEV, dtype=torch.int64).unsqueeze(0).expand(k.shape[0], -1)
            a, b = _philox((k & 0xFFFFFFFF).expand_as(p), ((k >> 32) & 0xFFFFFFFF).expand_as(p), p,
                           torch.full_like(p, j), seed)
            u1 = ((a >> 8) + 1).to(torch.float64) * 2.0 ** -24
            u2 = (b >> 8).to(torch.float64) * 2.0 ** -24
            r, t = (-2.0 * u1.log()).sqrt(), 2.0 * math.pi * u2
            g = torch.stack([r * t.cos(), r * t.sin()], dim=2).reshape(k.shape[0], -1)[:, :R]
            out.index_add_(0, cols[j][z].to(torch.int64), vals[z].unsqueeze(1) * g)
        f, n = _normalised(out)
        factors.append(f)
        sigma = sigma * n
    return {"factors": factors, "sigma": sigma}


def _exact_fit(case, seed):
    idx, vals = _tensor(case, seed)
    U = _energy_factors(case, seed, idx)
    R = case["R"]
    first = torch.zeros((), device=DEV, dtype=torch.float64)
    for z in torch.arange(idx.shape[0], device=DEV).split(1 << 21):
        p = torch.ones((z.shape[0], R), device=DEV, dtype=torch.float64)
        for k, u in enumerate(U):
            p = p * u[idx[z, k].to(torch.int64)]
        first = first + (vals[z].square() - 2.0 * vals[z] * p.sum(dim=1)).sum()
    M = torch.ones((R, R), device=DEV, dtype=torch.float64)
    for u in U:
        M = M * (u.T @ u)
    return {"terms": torch.stack([first, M.sum()])}


def _exact_lowrank(case, seed):
    V, U = _model(case, seed)
    j, J = case["j"], case["J"]
    samples, h, w = _exact_draw(U, J, j, seed)
    gram = (h * w.unsqueeze(1)).T @ h
    P = torch.ones((J, case["rank"]), device=DEV, dtype=torch.float64)
    for k, v in enumerate(V):
        if k != j:
            P = P * v[samples[k]]
    f, sigma = _normalised(V[j] @ (P.T @ (h * w.unsqueeze(1))) @ _pinv(gram, 1e-11))
    return {"factor": f, "sigma": sigma}


def exact(case, seed):
    """None where the result follows FP32 decisions (mixed-precision draws
    pick other rows of the same law) or hashed noise."""
    kind = case["kind"]
    if kind == "tree":
        U = _factors(case, seed)[0]
        out = {"tree": _exact_tree(U, case["R"], case["precision"])}
        if case["precision"] != "fp64":
            out["copy"] = U
        return out
    if kind == "exact":
        return _exact_update(case, seed)
    if kind == "rrf":
        return _exact_rrf(case, seed)
    if kind == "fit":
        return _exact_fit(case, seed)
    if case["precision"] != "fp64" or case.get("snr_db"):
        return None
    if kind == "draw":
        samples, h, w = _exact_draw(_factors(case, seed), case["J"], case["j"], seed)
        return {"samples": samples, "h": h, "weights": w}
    if kind == "als":
        return _exact_als(case, seed)
    return _exact_lowrank(case, seed)

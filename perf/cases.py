"""The work that a user of this framework has it do, as timed cases.

A case is one call (or the two calls of the solver interface, or of the column-split interface) through the public
Python API: sparsify a graph, sparsify several at once, sparsify again after inserting edges, or solve a Laplacian
system and take the edges' norms.  Graph families, sizes, weights and parameters are those of this repository's
benchmark, tests and serving mix: random geometric graphs (the serving mix), 2-D grids, 3-D grids with weights over
six decades, Erdos-Renyi graphs (average degree 20, and dense ones that the sampler thins), R-MAT graphs.

Parameters: "cli" are the reference command line's (k = 4 log2 n columns, absolute stopping rule), "baseline" the
benchmark configurations' (k = 24 ln n / eps^2 columns, relative residual 1e-8).
"""
import functools
import math

import numpy as np
import torch

import spec_spars_b200 as ssp


def listed():
    return [
        # the smallest request of the serving mix with the command line's parameters: launches and host latency
        {"name": "rgg_1k_cli", "do": "sparsify", "family": "rgg", "n": 1009, "degree": 12.0, "params": "cli",
         "eps": 0.5, "precision": 0, "device": False, "uniform": False},
        # the small benchmark configuration: 2-D grid, about 900 columns
        {"name": "grid2d_100", "do": "sparsify", "family": "grid2d", "nx": 100, "ny": 100, "params": "baseline",
         "eps": 0.5, "precision": 0, "device": False, "uniform": False},
        # a large request of the serving mix at the tighter accuracy (about 2600 columns)
        {"name": "rgg_20k_eps03", "do": "sparsify", "family": "rgg", "n": 20011, "degree": 16.0, "params": "baseline",
         "eps": 0.3, "precision": 0, "device": False, "uniform": False},
        # continuous batching: the serving mix's small requests as one disjoint union
        {"name": "batch_20", "do": "batch", "count": 20, "n_lo": 1000, "n_hi": 2000, "eps": 0.5},
        # the ill-conditioned mesh configuration at a size whose pass stays within a second; odd sides
        {"name": "mesh_47x40x43", "do": "sparsify", "family": "grid3d", "nx": 47, "ny": 40, "nz": 43,
         "decades": 3.0, "params": "baseline", "eps": 0.5, "precision": 0, "device": True, "uniform": False},
        # power-law graph with hubs at the R-MAT configuration's accuracy
        {"name": "rmat_s15", "do": "sparsify", "family": "rmat", "scale": 15, "params": "baseline", "eps": 0.3,
         "precision": 0, "device": True, "uniform": False},
        # a dense graph: the sampler drops a good part of its edges
        {"name": "er_20k_deg200", "do": "sparsify", "family": "er", "n": 20000, "degree": 200.0, "params": "baseline",
         "eps": 0.5, "precision": 0, "device": True, "uniform": False},
        # the headline family at a size that is held several times: the column-split entry points with one rank
        {"name": "er_250k_split", "do": "split", "family": "er", "n": 250000, "degree": 20.0, "eps": 0.5},
        # the same family in mixed precision, an odd size
        {"name": "er_229k_mixed", "do": "sparsify", "family": "er", "n": 229373, "degree": 20.0, "params": "baseline",
         "eps": 0.5, "precision": 1, "device": True, "uniform": False},
        # the headline graph (1M vertices, 10M edges) with the command line's parameters (80 columns)
        {"name": "er_1m_cli", "do": "sparsify", "family": "er", "n": 1000000, "degree": 20.0, "params": "cli",
         "eps": 0.5, "precision": 0, "device": True, "uniform": False},
        # the solver interface on its own: host right-hand sides in, host solution out, then the edges' norms
        {"name": "solve_grid3d_40", "do": "solve", "nx": 40, "ny": 40, "nz": 40, "decades": 0.0, "k": 64},
        # streaming: a current Laplacian plus a batch of inserted edges, uniform sketch entries
        {"name": "update_30k", "do": "update", "n": 30011, "degree": 16.0, "new_degree": 3.0, "eps": 0.5,
         "uniform": True},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["rgg", "rgg", "grid2d", "grid3d", "er", "er_dense", "er_mixed", "er_cli", "rmat", "batch", "split",
                       "solve", "update"])
    base = {"do": "sparsify", "params": "baseline", "eps": 0.5, "precision": 0, "device": rng.random() < 0.5,
            "uniform": rng.random() < 0.1}
    if kind == "rgg":
        cli = rng.random() < 0.4
        return dict(base, family="rgg", n=_log(rng, 1000, 20000), degree=round(rng.uniform(8, 32), 2),
                    eps=rng.choice([0.3, 0.5]), params="cli" if cli else "baseline")
    if kind == "grid2d":
        return dict(base, family="grid2d", nx=_log(rng, 30, 140), ny=_log(rng, 30, 140))
    if kind == "grid3d":
        return dict(base, family="grid3d", nx=_log(rng, 10, 44), ny=_log(rng, 10, 44), nz=_log(rng, 10, 40),
                    decades=rng.choice([0.0, 1.0, 3.0]))
    if kind == "er":
        return dict(base, family="er", n=_log(rng, 3000, 250000), degree=20.0)
    if kind == "er_dense":
        return dict(base, family="er", n=_log(rng, 2000, 20000), degree=round(rng.uniform(100, 200), 1))
    if kind == "er_mixed":
        return dict(base, family="er", n=_log(rng, 20000, 230000), degree=20.0, precision=1, uniform=False)
    if kind == "er_cli":
        return dict(base, family="er", n=_log(rng, 50000, 1000000), degree=20.0, params="cli")
    if kind == "rmat":
        return dict(base, family="rmat", scale=rng.randint(11, 15), eps=rng.choice([0.3, 0.5]))
    if kind == "batch":
        return {"do": "batch", "count": rng.randint(3, 20), "n_lo": 1000, "n_hi": rng.choice([1500, 2000]), "eps": 0.5}
    if kind == "split":
        return {"do": "split", "family": "er", "n": _log(rng, 20000, 250000), "degree": 20.0, "eps": 0.5}
    if kind == "solve":
        return {"do": "solve", "nx": _log(rng, 12, 40), "ny": _log(rng, 12, 40), "nz": _log(rng, 12, 40),
                "decades": rng.choice([0.0, 1.0]), "k": rng.randint(5, 64)}
    return {"do": "update", "n": _log(rng, 3000, 30000), "degree": 16.0, "new_degree": round(rng.uniform(1, 4), 1),
            "eps": 0.5, "uniform": rng.random() < 0.5}


# ------------------------------------------------------------------------------------------------ inputs
# A case's sizes fix the graph's structure; the seed draws its weights, signs and coins.
@functools.lru_cache(maxsize=4)
def _structure(family, *size):
    if family == "rgg":
        g = ssp.gen_rgg(*size)
    elif family == "er":
        g = ssp.gen_er(size[0], size[1], 0.5, 2.0, size[2])
    elif family == "rmat":
        g = ssp.gen_rmat(size[0], 16, seed=3)
    else:
        g = ssp.gen_grid3d(*size, 0.0, 0.0, 2) if family == "grid3d" else ssp.gen_grid2d(*size)
    return g.n, g.colptr, g.rowidx


def _uniform(key, seed):
    """One number in (0, 1) for each key: the finaliser of SplitMix64 over (key, seed)."""
    x = key + _s64(seed * 0x9E3779B97F4A7C15 & (1 << 64) - 1)
    for shift, mult in ((30, -0x40A7B892E31B1A47), (27, -0x6B2FB644ECCEEE15)):
        x = (x ^ ((x >> shift) & ((1 << (64 - shift)) - 1))) * mult
    x = x ^ ((x >> 31) & ((1 << 33) - 1))
    return (((x >> 11) & ((1 << 53) - 1)).double() + 0.5) * 2.0 ** -53


def _weighted(family, size, seed, decades=3.0):
    """The graph of this structure with weights of its family: symmetric, one draw for each edge."""
    n, colptr, rowidx = _structure(family, *size)
    cols = torch.from_numpy(np.repeat(np.arange(n, dtype=np.int64), np.diff(colptr))).cuda()
    rows = torch.from_numpy(rowidx).cuda().long()
    key = torch.minimum(rows, cols) * n + torch.maximum(rows, cols)
    u = _uniform(key, 2 * seed)
    if family == "rgg":
        w = 0.1 + 9.9 * u
    elif family == "grid3d":
        w = 10.0 ** (decades * (2 * u - 1))
    elif family == "rmat":  # log-normal
        w = torch.exp((-2 * torch.log(u)).sqrt() * torch.cos(2 * math.pi * _uniform(key, 2 * seed + 1)))
    else:
        w = 0.5 + 1.5 * u
    return ssp.CSC(n, colptr, rowidx, w.cpu().numpy())


def _graph(case, seed):
    f = case["family"]
    size = {"rgg": lambda: (case["n"], case["degree"], 0.1, 10.0, 1), "er": lambda: (case["n"], case["degree"], 1),
            "rmat": lambda: (case["scale"],), "grid2d": lambda: (case["nx"], case["ny"]),
            "grid3d": lambda: (case["nx"], case["ny"], case["nz"])}[f]()
    return _weighted(f, size, seed, case.get("decades", 3.0))


def _params(case, seed):
    if case.get("params") == "cli":
        p = ssp.SparsifierParameters.cli(case["eps"], sketch_seed=seed, sampling_seed=seed + 1)
    else:
        p = ssp.SparsifierParameters.baseline(case["eps"], sketch_seed=seed, sampling_seed=seed + 1)
    p.precision = case.get("precision", 0)
    p.sketch_uniform = int(case.get("uniform", False))
    return p


def _on_device(g):
    return [torch.from_numpy(a).cuda() for a in (g.colptr, g.rowidx, g.values)]


def _batch_graphs(case, seed):
    r = np.random.default_rng(case["count"])
    out = []
    for i in range(case["count"]):
        n = int(round(math.exp(r.uniform(math.log(case["n_lo"]), math.log(case["n_hi"])))))
        d = float(r.uniform(8, 32))
        size = (n, d, 0.1, 10.0, i) if r.random() < 0.5 else (n, d, i)
        out.append(_weighted("rgg" if len(size) == 5 else "er", size, 1000 * seed + i))
    return out


def _edges(g):
    """Upper-triangle entries (row < column) in column order, on the GPU: v1, v2, w."""
    cols = torch.from_numpy(np.repeat(np.arange(g.n, dtype=np.int64), np.diff(g.colptr))).cuda()
    rows = torch.from_numpy(g.rowidx.astype(np.int64)).cuda()
    up = rows < cols
    return rows[up], cols[up], torch.from_numpy(g.values).cuda()[up]


def _laplacian(n, v1, v2, w):
    """The Laplacian of an edge list as a host CSC."""
    r = torch.cat([v1, v2, v1, v2])
    c = torch.cat([v2, v1, v1, v2])
    a = torch.sparse_coo_tensor(torch.stack([c, r]), torch.cat([-w, -w, w, w]), (n, n)).coalesce()
    ptr = torch.zeros(n + 1, dtype=torch.int64)
    ptr[1:] = torch.bincount(a.indices()[0], minlength=n).cumsum(0).cpu()
    return ssp.CSC(n, ptr.numpy(), a.indices()[1].to(torch.int32).cpu().numpy(), a.values().cpu().numpy())


def _right_hand_sides(case, seed, v1, v2, w, n):
    """Random signs through the weighted incidence matrix, as the solver interface is given them: n x k."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    q = torch.randint(0, 2, (v1.numel(), case["k"]), generator=gen, device="cuda").double().mul_(2).sub_(1)
    q *= w.sqrt()[:, None] * math.sqrt(3.0)
    y = torch.zeros(n, case["k"], dtype=torch.float64, device="cuda")
    y.index_add_(0, v2, q)
    y.index_add_(0, v1, q, alpha=-1.0)
    return y


def _update_inputs(case, seed):
    g = _weighted("rgg", (case["n"], case["degree"], 0.1, 10.0, 1), seed)
    return _laplacian(g.n, *_edges(g)), _weighted("er", (g.n, case["new_degree"], 8), seed + 7)


def _grid(case, seed):
    return _weighted("grid3d", (case["nx"], case["ny"], case["nz"]), seed, case["decades"])


def prepare(case, seed):
    do = case["do"]
    s = {"do": do, "ctx": ssp.Context(0)}
    if do == "batch":
        s["graphs"] = _batch_graphs(case, seed)
        s["params"] = []
        for i in range(case["count"]):
            p = ssp.SparsifierParameters.baseline(case["eps"], sampling_seed=seed + i)
            p.dense_threshold = 0
            s["params"].append(p)
    elif do == "solve":
        g = _grid(case, seed)
        v1, v2, w = _edges(g)
        s["lap"] = _laplacian(g.n, v1, v2, w)
        s["Y"] = _right_hand_sides(case, seed, v1, v2, w, g.n).cpu().numpy()
        s["v1"], s["v2"] = (t.to(torch.int32).cpu().numpy() for t in (v1, v2))
    elif do == "update":
        s["lap"], s["new"] = _update_inputs(case, seed)
        s["params"] = _params(dict(case, params="cli"), seed)
    else:
        g = _graph(case, seed)
        s["params"] = _params(case, seed)
        s["graph"], s["device"] = g, case.get("device", True)
        if s["device"]:
            s["arrays"] = _on_device(g)
            s["graph"] = ssp.DeviceCSC(g.n, g.nnz, *(t.data_ptr() for t in s["arrays"]))
        if do == "split":
            s["sq"] = torch.empty(g.num_edges(), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    return s


class _View:
    def __init__(self, ptr, count, typestr):
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": (count,), "typestr": typestr, "version": 3}


def _device_csc(n, cap, out):
    """The context's L_H in tensors of the caller's own (the context reuses its buffers and frees them when it closes),
    with room for every entry of L_G."""
    nnz, ptr, idx, val = out
    res = [torch.empty(n + 1, dtype=torch.int64, device="cuda"), torch.zeros(cap, dtype=torch.int32, device="cuda"),
           torch.zeros(cap, dtype=torch.float64, device="cuda")]
    for r, p, c, t in zip(res, (ptr, idx, val), (n + 1, nnz, nnz), ("<i8", "<i4", "<f8")):
        r[:c] = torch.as_tensor(_View(p, c, t), device="cuda")
    return res


def _host_csc(cap, h):
    """L_H in arrays with room for every entry of L_G."""
    idx, val = np.zeros(cap, np.int32), np.zeros(cap)
    idx[:h.nnz], val[:h.nnz] = h.rowidx, h.values
    return [h.colptr, idx, val]


def run(s):
    do, ctx = s["do"], s["ctx"]
    if do == "batch":
        return [_host_csc(g.nnz + g.n, h) for g, (h, _) in zip(s["graphs"], ctx.sparsify_batch(s["graphs"], s["params"]))]
    if do == "solve":
        z, _ = ctx.solve_lap(s["lap"], s["Y"])
        return [z, ssp.stage_diff_norms(ctx, s["v1"], s["v2"], z)]
    if do == "update":
        h, _ = ctx.sparsify_update(s["lap"], s["new"], s["params"])
        return _host_csc(s["lap"].nnz + s["new"].nnz, h)
    g, p = s["graph"], s["params"]
    if do == "split":
        ctx.shard_leverage(g, p, 0, p.jl_dim(g.n), s["sq"].data_ptr())
        out, _ = ctx.shard_finish(g, p, s["sq"].data_ptr(), device_out=True)
        return _device_csc(g.n, g.nnz + g.n, out) + [s["sq"]]
    if s["device"]:
        out, _ = ctx.sparsify_device(g.n, g.nnz, *g._p, p)
        return _device_csc(g.n, g.nnz + g.n, out)
    h, _ = ctx.sparsify(g, p)
    return _host_csc(g.nnz + g.n, h)


# ------------------------------------------------------------------------------------------------ work
def _sizes(case):
    """(vertices, edges, columns), estimated from the case alone."""
    if case["do"] == "batch":
        n = case["count"] * (case["n_lo"] + case["n_hi"]) / 2
        return n, n * 10, math.ceil(24 * math.log((case["n_lo"] + case["n_hi"]) / 2) / case["eps"] ** 2)
    if "nx" in case:
        dim = 3 if "nz" in case else 2
        n = case["nx"] * case["ny"] * case.get("nz", 1)
        m = dim * n
    elif "scale" in case:
        n, m = 0.75 * 2 ** case["scale"], 13.5 * 2 ** case["scale"]
    else:
        n = case["n"]
        m = n * (case["degree"] + case.get("new_degree", 0.0)) / 2
    if case["do"] == "solve":
        return n, m, case["k"]
    cli = case.get("params") == "cli" or case["do"] == "update"
    return n, m, math.ceil(4 * math.log2(n)) if cli else math.ceil(24 * math.log(n) / case["eps"] ** 2)


def work(case):
    """One pass cannot do without: the graph read and L_H written; the n x k right-hand sides written once and the
    solution's rows read for the edges' norms; and for a solve, at least one product with the Laplacian and one
    application of a preconditioner with as many entries as the graph has edges (an iteration reads and writes its
    five n x k blocks)."""
    n, m, k = _sizes(case)
    b = 4.0 if case.get("precision") == 1 else 8.0
    io = 2 * (2 * m * 12 + n * 8)
    block = n * k * b
    return {"bytes": io + 7 * block, "flops": k * (2 * (2 * m + n) + 4 * m + 10 * n + 3 * m)}


# ------------------------------------------------------------------------------------------------ 64-bit values
_M32 = 0xFFFFFFFF


def _s64(x):
    return x - (1 << 64) if x >= 1 << 63 else x


def _mulhi(a, b):
    """High 64 bits of the unsigned product of an int64 tensor and an integer."""
    al, ah, bl, bh = a & _M32, (a >> 32) & _M32, b & _M32, b >> 32
    lo, m1, m2 = al * bl, ah * bl, al * bh
    mid = ((lo >> 32) & _M32) + (m1 & _M32) + (m2 & _M32)
    return ah * bh + ((m1 >> 32) & _M32) + ((m2 >> 32) & _M32) + ((mid >> 32) & _M32)


def _philox(c0, c1, k0, k1):
    """Philox4x64-10 (Salmon et al., 2011) of the counters (c0, c1, 0, 0): four int64 tensors."""
    c2, c3 = torch.zeros_like(c0), torch.zeros_like(c0)
    c1 = torch.zeros_like(c0) + c1
    M0, M1 = 0xD2E7470EE14C6C93, 0xCA5A826395121157
    for r in range(10):
        a, b = _mulhi(c0, M0), _mulhi(c2, M1)
        c0, c1, c2, c3 = b ^ c1 ^ _s64(k0), c2 * _s64(M1), a ^ c3 ^ _s64(k1), c0 * _s64(M0)
        k0 = (k0 + 0x9E3779B97F4A7C15) & (1 << 64) - 1
        k1 = (k1 + 0xBB67AE8584CAA73B) & (1 << 64) - 1
    return c0, c1, c2, c3


def _sketch(n, v1, v2, w, k, scale, seed, uniform):
    """Y = B^T Q: Philox signs (one bit per column, 256 to a call) or uniform (-1, 1) entries (32 bits, 8 to a call)."""
    y = torch.zeros(n, k, dtype=torch.float64, device="cuda")
    m = v1.numel()
    step = max(1, int(2e8) // (k + 256))
    col = torch.arange(256, device="cuda")
    for e0 in range(0, m, step):
        e = torch.arange(e0, min(m, e0 + step), device="cuda")
        q = []
        for t in range((k + 255) // 256):
            if uniform:
                call = torch.arange(32, device="cuda")[None, :] + 32 * t
                r = torch.stack(_philox(e[:, None].expand(-1, 32).contiguous(), call, seed, 0x554E4946), -1)
                x = torch.stack([r & _M32, (r >> 32) & _M32], -1).reshape(e.numel(), 256)
                q.append(2.0 * ((x.double() + 0.5) / 4294967296.0) - 1.0)
            else:
                r = torch.stack(_philox(e, t, seed, 0x5349474E), -1)
                q.append(1.0 - 2.0 * ((r[:, col // 64] >> (col % 64)) & 1).double())
        q = torch.cat(q, 1)[:, :k] * (scale * w[e].sqrt())[:, None]
        y.index_add_(0, v2[e], q)
        y.index_add_(0, v1[e], q, alpha=-1.0)
    return y


def _components(n, v1, v2):
    lab = torch.arange(n, device="cuda")
    while True:
        new = lab.clone()
        new.scatter_reduce_(0, v1, lab[v2], "amin")
        new.scatter_reduce_(0, v2, lab[v1], "amin")
        new = new[new]
        if torch.equal(new, lab):
            return lab
        lab = new


def _solve(n, v1, v2, w, y, dense):
    """A solution of L x = y (consistent on every component) to 64-bit accuracy: Cholesky, or conjugate gradients."""
    if dense:
        a = torch.zeros(n, n, dtype=torch.float64, device="cuda")
        a.index_put_((torch.cat([v1, v2, v1, v2]), torch.cat([v2, v1, v1, v2])), torch.cat([-w, -w, w, w]), accumulate=True)
        lab = _components(n, v1, v2)
        size = torch.bincount(lab, minlength=n).double()[lab]
        scale = float(w.mean())
        a += (lab[:, None] == lab[None, :]).double() * (scale / size)[:, None]
        return torch.cholesky_solve(y, torch.linalg.cholesky(a))
    r = torch.cat([v1, v2, v1, v2])
    c = torch.cat([v2, v1, v1, v2])
    a = torch.sparse_coo_tensor(torch.stack([r, c]), torch.cat([-w, -w, w, w]), (n, n)).coalesce().to_sparse_csr()
    d = torch.zeros(n, dtype=torch.float64, device="cuda").index_add_(0, v1, w).index_add_(0, v2, w).clamp_min(1e-300)
    x = torch.zeros_like(y)
    r = y.clone()
    z = r / d[:, None]
    p = z.clone()
    rz = (r * z).sum(0)
    goal = 1e-13 * y.norm(dim=0)
    for _ in range(400):
        q = a @ p
        al = rz / (p * q).sum(0).clamp_min(1e-300)
        x += al * p
        r -= al * q
        if bool((r.norm(dim=0) <= goal).all()):
            break
        z = r / d[:, None]
        rn = (r * z).sum(0)
        p = z + (rn / rz.clamp_min(1e-300)) * p
        rz = rn
    return x


def _edge_squares(x, v1, v2):
    sq = torch.zeros(v1.numel(), dtype=torch.float64, device="cuda")
    step = max(1, int(2e8) // x.shape[1])
    for e0 in range(0, v1.numel(), step):
        sq[e0:e0 + step] = (x[v1[e0:e0 + step]] - x[v2[e0:e0 + step]]).square_().sum(1)
    return sq


def _sampled(n, v1, v2, w, sq, eps, k, scale, cli, seed):
    """L_H of the coins for these leverage estimates, entries in column order, and nothing for the whole numbers."""
    m = v1.numel()
    beta = eps ** -2.0 * 4 * math.log(n)
    p = (beta * w * sq / (k if cli else k * scale * scale)).clamp_max(1.0)
    r = torch.stack(_philox(torch.arange((m + 3) // 4, device="cuda"), 0, seed, 0x434F494E), -1).reshape(-1)[:m]
    coin = ((r >> 11) & ((1 << 53) - 1)).double() * 2.0 ** -53
    kept = coin < p
    h = torch.where(kept, w / (p.sqrt() if cli else p), torch.zeros_like(w))
    # L_H = L_G + change, entry by entry: a kept edge's change is h - w
    rows, cols = torch.cat([v1, v2, v1, v2]), torch.cat([v2, v1, v1, v2])
    a = torch.sparse_coo_tensor(torch.stack([cols, rows]), torch.cat([-h, -h, h, h]), (n, n)).coalesce().values()
    out = torch.zeros(2 * m + n, dtype=torch.float64)
    a = a[a != 0].cpu()
    out[:a.numel()] = a
    return [None, None, out.numpy()]


def _exact_graph(g, eps, params, sketch_seed, sampling_seed, uniform, dense):
    v1, v2, w = _edges(g)
    cli = params == "cli"
    k = math.ceil(4 * math.log2(g.n)) if cli else math.ceil(24 * math.log(g.n) / eps ** 2)
    scale = math.sqrt(3.0) if cli else 1 / math.sqrt(k)
    y = _sketch(g.n, v1, v2, w, k, scale, sketch_seed, uniform)
    sq = _edge_squares(_solve(g.n, v1, v2, w, y, dense), v1, v2)
    return _sampled(g.n, v1, v2, w, sq, eps, k, scale, cli, sampling_seed) + [sq.cpu().numpy()]


def exact(case, seed):
    do = case["do"]
    n, m, k = _sizes(case)
    if do == "batch":
        return [_exact_graph(g, case["eps"], "baseline", 0, seed + i, False, True)[:3]
                for i, g in enumerate(_batch_graphs(case, seed))]
    if do == "solve":  # the solution is unique up to a constant in each column; its differences along edges are unique
        g = _grid(case, seed)
        v1, v2, w = _edges(g)
        x = _solve(g.n, v1, v2, w, _right_hand_sides(case, seed, v1, v2, w, g.n), g.n <= 12000)
        return [None, _edge_squares(x, v1, v2).sqrt().cpu().numpy()]
    if do == "update" or n * k > 3.1e8 or m * k > 3.2e9:
        return None
    dense = n <= 12000
    if not dense and case["family"] != "er":
        return None
    out = _exact_graph(_graph(case, seed), case["eps"], case.get("params", "baseline"), seed, seed + 1,
                       case.get("uniform", False), dense)
    return out if do == "split" else out[:3]

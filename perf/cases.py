"""Timed cases of the PCA -> exact-kNN path: the calls a user of kyto_b200 makes, at the
sizes they are made at, with plain 64-bit restatements of what each returns.

A case is a dict of plain values: ``kind`` names the call, the rest its sizes and options.
Inputs are made on the GPU from the seed alone; device arrays go in and come out (the C
ABI takes either kind of pointer), except where a caller has host arrays by nature (a
reader's tile offsets, the graph of a small interactive search).
"""

from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

import kyto_b200 as K

DEV = "cuda"
TARGET_SUM = 1e4
TILE_CELLS, TILE_GENES = 4096, 1024  # the store's default tile
PUSH_CELLS = 8192                    # cells of a pushed block


def listed() -> list[dict]:
    return [
        # normalize_total + log1p of one store block of a whole-transcriptome layer: the
        # smallest call of the path, made once per block of a stream.
        {"name": "normalize_block", "kind": "normalize", "cells": 8192, "genes": 20000,
         "nnz": 2000, "dtype": "u32"},
        # The seurat moments pass over a dataset's raw counts (gene selection before the
        # PCA): 20,000 genes, ~2,000 stored a cell.
        {"name": "hvg_50k", "kind": "hvg", "cells": 50000, "genes": 20000, "nnz": 2000},
        # One cell block of a tiled layer joined into rows, as a store reader streams it.
        {"name": "tile_block", "kind": "tiles", "cells": 4096, "genes": 2000, "nnz": 660},
        # A pbmc3k-sized dataset: latency counts (eleven passes over a few MB).
        {"name": "pca_pbmc3k", "kind": "pca", "cells": 2700, "genes": 2000, "nnz": 600,
         "k": 50, "types": 8, "counts": True, "stream_genes": 2000},
        # Raw counts of 20,000 genes pushed in blocks, normalized and cut to 2,000 highly
        # variable genes on the way: the ordinary whole analysis of one study.
        {"name": "pca_hvg_50k", "kind": "pca", "cells": 50000, "genes": 2000, "nnz": 2000,
         "k": 50, "types": 20, "counts": True, "stream_genes": 20000},
        # The benchmark's matrix: 1M cells x 2,000 genes of log1p values.
        {"name": "pca_1m", "kind": "pca", "cells": 1000000, "genes": 2000, "nnz": 600,
         "k": 50, "types": 50, "counts": False, "stream_genes": 2000},
        # The graph of a pbmc3k-sized embedding, read back to the host at once.
        {"name": "knn_pbmc3k", "kind": "knn", "cells": 2700, "width": 50, "neighbors": 15,
         "data": "scores", "host": True},
        # An ordinary study's graph with fewer components and more neighbours.
        {"name": "knn_60k", "kind": "knn", "cells": 60013, "width": 30, "neighbors": 30,
         "data": "scores", "host": False},
        # The benchmark's search: every row of 1M against 1M.
        {"name": "knn_1m", "kind": "knn", "cells": 1000000, "width": 50, "neighbors": 15,
         "data": "scores", "host": False},
        # A batch of samples of uneven sizes searched in one call.
        {"name": "knn_batch_16", "kind": "knn_batch", "samples": 16, "least": 500,
         "most": 20000, "width": 30, "neighbors": 15},
        # The step after the search: UMAP connectivities of the graph.
        {"name": "connect_200k", "kind": "connect", "cells": 200000, "neighbors": 15},
        # The learned-partition search on well-separated components.
        {"name": "learned_500k", "kind": "learned", "cells": 500000, "width": 50,
         "neighbors": 15},
    ]


def draw(rng) -> dict:
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["normalize", "hvg", "tiles", "pca", "pca", "pca", "knn", "knn", "knn",
                       "knn_batch", "connect", "learned"])
    if kind == "normalize":
        return {"kind": kind, "cells": size(500, 20000), "genes": 20000,
                "nnz": size(300, 2500), "dtype": rng.choice(["u32", "f32"])}
    if kind == "hvg":
        return {"kind": kind, "cells": size(2000, 60000), "genes": rng.choice([2000, 20000]),
                "nnz": size(300, 1200)}
    if kind == "tiles":
        return {"kind": kind, "cells": rng.choice([4096, 4096, rng.randint(100, 4096)]),
                "genes": rng.randint(1500, 20000), "nnz": size(200, 1200)}
    if kind == "pca":
        counts = rng.random() < 0.5
        genes = rng.randint(800, 3000)
        return {"kind": kind, "cells": size(2000, 60000 if counts else 400000),
                "genes": genes, "nnz": size(150, 700), "k": rng.choice([20, 30, 50]),
                "types": rng.choice([12, 20, 50]), "counts": counts,
                "stream_genes": genes if rng.random() < 0.5 or not counts else 8 * genes}
    if kind == "knn":
        return {"kind": kind, "cells": size(2000, 400000), "width": rng.randint(20, 50),
                "neighbors": rng.choice([10, 15, 15, 30]),
                "data": rng.choice(["scores", "scores", "mixture"]),
                "host": False}
    if kind == "knn_batch":
        return {"kind": kind, "samples": rng.randint(4, 32), "least": 500,
                "most": size(4000, 20000), "width": rng.choice([30, 50]), "neighbors": 15}
    if kind == "connect":
        return {"kind": kind, "cells": size(2000, 300000), "neighbors": rng.choice([10, 15, 30])}
    return {"kind": kind, "cells": size(150000, 500000), "width": rng.randint(30, 50),
            "neighbors": rng.choice([10, 15])}


# ------------------------------------------------------------------ inputs -----------
def _gen(seed: int) -> torch.Generator:
    g = torch.Generator(device=DEV)
    g.manual_seed(1_000_003 * seed + 12345)
    return g


def _scaled(mean: np.ndarray, per_cell: float, dispersion: float) -> float:
    """The factor at which a cell stores about ``per_cell`` nonzero counts."""
    lo, hi = 1e-6, 1e6
    for _ in range(60):
        mid = math.sqrt(lo * hi)
        stored = np.sum(1.0 - (1.0 + mean * mid * dispersion) ** (-1.0 / dispersion))
        lo, hi = (mid, hi) if stored < per_cell else (lo, mid)
    return math.sqrt(lo * hi)


def _counts(cells: int, genes: int, per_cell: float, types: int, seed: int):
    """Raw counts as a CSR on the device (int64 indptr, int32 genes, int32 counts):
    log-normal gene means, a tenth of the genes shifted in each cell type, log-normal
    cell sizes, negative-binomial counts; thinned evenly to the case's stored values."""
    want = _stored(cells, genes, per_cell)
    aim = 1.0
    while True:
        indptr, idx, val = _draw_counts(cells, genes, aim * per_cell, types, seed)
        if idx.numel() >= want:
            break
        aim *= 1.1
    excess = idx.numel() - want
    if excess:
        keep = torch.ones(idx.numel(), dtype=torch.bool, device=DEV)
        keep[torch.arange(excess, device=DEV) * idx.numel() // excess] = False
        before = torch.zeros(idx.numel() + 1, dtype=torch.int64, device=DEV)
        torch.cumsum(keep, 0, out=before[1:])
        indptr, idx, val = before[indptr], idx[keep], val[keep]
    return indptr, idx, val


def _stored(cells: int, genes: int, per_cell: float) -> int:
    """Stored values of a case, whatever its seed."""
    return int(0.95 * cells * min(per_cell, 0.8 * genes))


def _draw_counts(cells: int, genes: int, per_cell: float, types: int, seed: int):
    rng = np.random.default_rng(seed)
    mean = np.exp(rng.normal(0.0, 1.5, genes))
    shift = np.ones((types, genes))
    for t in range(types):
        at = rng.choice(genes, size=max(1, genes // 10), replace=False)
        shift[t, at] = rng.uniform(2.0, 8.0, at.size)
    dispersion = 0.3
    mean *= _scaled(mean, min(per_cell, 0.9 * genes), dispersion)
    gen = _gen(seed)
    mean_d = torch.tensor(mean, dtype=torch.float32, device=DEV)
    shift_d = torch.tensor(shift, dtype=torch.float32, device=DEV)
    shape = torch.tensor(1.0 / dispersion, device=DEV)
    step = max(1, 100_000_000 // genes)
    rows, idx, val = [], [], []
    for a in range(0, cells, step):
        m = min(cells, a + step) - a
        kind = torch.randint(types, (m,), generator=gen, device=DEV)
        mu = shift_d[kind] * mean_d
        mu *= torch.exp(0.3 * torch.randn((m, 1), generator=gen, device=DEV))
        mu *= torch._standard_gamma(shape.expand(mu.shape).contiguous(), generator=gen) / shape
        c = torch.poisson(mu, generator=gen).to(torch.int32)
        del mu
        rows.append((c != 0).sum(1))
        at = c.nonzero()
        idx.append(at[:, 1].to(torch.int32))
        val.append(c[at[:, 0], at[:, 1]])
        del c, at
    indptr = torch.zeros(cells + 1, dtype=torch.int64, device=DEV)
    torch.cumsum(torch.cat(rows), 0, out=indptr[1:])
    return indptr, torch.cat(idx), torch.cat(val)


def _rows(indptr):
    return torch.repeat_interleave(torch.arange(indptr.numel() - 1, device=DEV),
                                   indptr[1:] - indptr[:-1])


def _log1p(indptr, counts, dtype=torch.float32):
    """normalize_total + log1p by torch: f32 divisor and quotient then log1p in f64 as the
    path's maps define it (float32), or all of it in 64 bits (float64)."""
    n = indptr.numel() - 1
    out = torch.empty(counts.numel(), dtype=dtype, device=DEV)
    step = max(1, int(50_000_000 * n // max(counts.numel(), 1)))
    for a in range(0, n, step):
        b = min(n, a + step)
        s, e = int(indptr[a]), int(indptr[b])
        part = counts[s:e].double()
        total = torch.segment_reduce(part, "sum", lengths=(indptr[a + 1:b + 1] - indptr[a:b]))
        if dtype == torch.float32:
            div = total.float() / TARGET_SUM
        else:
            div = total / TARGET_SUM
        div = torch.where(div == 0, torch.ones_like(div), div)
        v = part.to(dtype) / div[_rows(indptr[a:b + 1])]
        out[s:e] = torch.log1p(v.double()).to(dtype)
    return out


def _scores(n: int, width: int, seed: int) -> torch.Tensor:
    """Rows like a PCA's embedding of cell types: type centres whose spread falls with the
    component, unequal type sizes, noise that falls more slowly; columns centred."""
    rng = np.random.default_rng(seed)
    types = 40
    fall = 12.0 / (1.0 + np.arange(width)) ** 0.55
    centre = torch.tensor(rng.normal(size=(types, width)) * fall, dtype=torch.float32, device=DEV)
    noise = torch.tensor(1.0 + 1.5 / np.sqrt(1.0 + np.arange(width)), dtype=torch.float32,
                         device=DEV)
    weight = torch.tensor(rng.dirichlet(np.full(types, 2.0)), device=DEV)
    gen = _gen(seed)
    kind = torch.multinomial(weight, n, replacement=True, generator=gen)
    x = centre[kind] + noise * torch.randn((n, width), generator=gen, device=DEV)
    return (x - x.mean(0)).contiguous()


def _mixture(n: int, width: int, seed: int) -> torch.Tensor:
    """An isotropic Gaussian mixture: 200 components, Dirichlet(1) weights, means of spread
    3, sigma log-uniform in [0.2, 2]."""
    rng = np.random.default_rng(seed)
    mean = torch.tensor(rng.normal(0.0, 3.0, (200, width)), dtype=torch.float32, device=DEV)
    sigma = torch.tensor(np.exp(rng.uniform(math.log(0.2), math.log(2.0), 200)),
                         dtype=torch.float32, device=DEV)
    weight = torch.tensor(rng.dirichlet(np.ones(200)), device=DEV)
    gen = _gen(seed)
    kind = torch.multinomial(weight, n, replacement=True, generator=gen)
    x = torch.randn((n, width), generator=gen, device=DEV) * sigma[kind, None]
    return (x + mean[kind]).contiguous()


def _tiles(indptr, idx, val, genes: int):
    """One cell block's tiles as the store's writer lays them out: tile-major entries with
    local gene indices, an indptr shard (gene blocks x (C + 1)), tile offsets (host)."""
    n = indptr.numel() - 1
    n_gb = -(-genes // TILE_GENES)
    gb = idx.long() // TILE_GENES
    key = gb * TILE_CELLS + _rows(indptr)
    key, order = torch.sort(key, stable=True)
    local = (idx.long()[order] - gb[order] * TILE_GENES).to(torch.int32)
    per_row = torch.bincount(key, minlength=n_gb * TILE_CELLS).view(n_gb, TILE_CELLS)
    shard = torch.zeros(n_gb, TILE_CELLS + 1, dtype=torch.int32, device=DEV)
    shard[:, 1:] = torch.cumsum(per_row, 1).to(torch.int32)
    offsets = np.zeros(n_gb + 1, dtype=np.uint64)
    offsets[1:] = np.cumsum(per_row.sum(1).cpu().numpy())
    assert n <= TILE_CELLS
    return shard, offsets, local, val[order].contiguous()


def _sizes(case: dict) -> np.ndarray:
    rng = np.random.default_rng([case["samples"], case["most"]])
    return np.exp(rng.uniform(math.log(case["least"]), math.log(case["most"]),
                              case["samples"])).astype(np.int64)


def _neighbor_lists(n: int, k: int, seed: int):
    """A kNN-like graph: each row's k distinct columns increasing, most of them mutual,
    distances as of rows in 30 dimensions."""
    gen = _gen(seed)
    reach = max(2 * k, 40)
    step = torch.rand((n, reach), generator=gen, device=DEV).argsort(1)[:, :k]
    offset = torch.where(step % 2 == 0, step // 2 + 1, -(step // 2 + 1))
    cols = torch.sort((torch.arange(n, device=DEV)[:, None] + offset) % n, 1).values
    near = 4.0 + 2.0 * torch.rand((n, 1), generator=gen, device=DEV)
    dist = near * (1.0 + 0.5 * torch.rand((n, k), generator=gen, device=DEV))
    indptr = torch.arange(n + 1, dtype=torch.int64, device=DEV) * k
    return indptr, cols.to(torch.int32).contiguous(), dist.float().contiguous()


def _hvg_flags(indptr, idx, counts, genes: int, keep: int) -> np.ndarray:
    """A gene set as an analysis has it in hand: the ``keep`` genes of the largest log
    dispersion of the normalized counts."""
    v = torch.expm1(_log1p(indptr, counts).double())
    s = torch.zeros(genes, dtype=torch.float64, device=DEV).index_add_(0, idx.long(), v)
    q = torch.zeros(genes, dtype=torch.float64, device=DEV).index_add_(0, idx.long(), v * v)
    n = indptr.numel() - 1
    mean = s / n
    ratio = (q / n - mean * mean) / mean.clamp_min(1e-12)
    flags = torch.zeros(genes, dtype=torch.bool, device=DEV)
    flags[torch.sort(ratio, descending=True, stable=True).indices[:keep]] = True
    return flags.cpu().numpy()


def _graph_out(rows: int, k: int, extra: int = 1) -> dict:
    return {"indptr": torch.empty(rows + extra, dtype=torch.int64, device=DEV),
            "indices": torch.empty(rows * k, dtype=torch.int32, device=DEV),
            "distances": torch.empty(rows * k, dtype=torch.float32, device=DEV)}


def _pca_input(case: dict, seed: int):
    """(blocks, gene flags or None, whole CSR) of a PCA case."""
    sg = case["stream_genes"]
    indptr, idx, val = _counts(case["cells"], sg, case["nnz"], case["types"], seed)
    if not case["counts"]:
        return [(indptr, idx, _log1p(indptr, val))], None
    flags = None
    if sg > case["genes"]:
        flags = _hvg_flags(indptr, idx, val, sg, case["genes"])
    blocks = []
    for a in range(0, case["cells"], PUSH_CELLS):
        b = min(case["cells"], a + PUSH_CELLS)
        s, e = int(indptr[a]), int(indptr[b])
        blocks.append(((indptr[a:b + 1] - s).clone(), idx[s:e].clone(), val[s:e].clone()))
    return blocks, flags


def prepare(case: dict, seed: int) -> dict:
    K.default_context()
    kind = case["kind"]
    st = {"case": case}
    if kind in ("normalize", "hvg"):
        indptr, idx, val = _counts(case["cells"], case["genes"], case["nnz"], 8, seed)
        if case.get("dtype") == "f32":
            val = val.float()
        st |= {"indptr": indptr, "idx": idx, "val": val}
        if kind == "normalize":
            st["out"] = torch.empty(val.numel(), dtype=torch.float32, device=DEV)
        else:
            g = case["genes"]
            st["out"] = {"sums": torch.empty(g, dtype=torch.float64, device=DEV),
                         "squares": torch.empty(g, dtype=torch.float64, device=DEV),
                         "positives": torch.empty(g, dtype=torch.int64, device=DEV)}
    elif kind == "tiles":
        indptr, idx, val = _counts(case["cells"], case["genes"], case["nnz"], 8, seed)
        shard, offsets, local, data = _tiles(indptr, idx, val, case["genes"])
        st |= {"shard": shard, "offsets": offsets, "local": local, "data": data}
        st["out"] = {"indptr": torch.empty(case["cells"] + 1, dtype=torch.int64, device=DEV),
                     "indices": torch.empty_like(local), "values": torch.empty_like(data)}
    elif kind == "pca":
        st["blocks"], st["flags"] = _pca_input(case, seed)
        n, k, sg = case["cells"], case["k"], case["stream_genes"]
        st["out"] = {"embedding": torch.empty((n, k), dtype=torch.float32, device=DEV),
                     "loadings": torch.empty((sg, k), dtype=torch.float32, device=DEV)}
    elif kind == "knn":
        make = _scores if case["data"] == "scores" else _mixture
        st["x"] = make(case["cells"], case["width"], seed)
        if not case["host"]:
            st["out"] = _graph_out(case["cells"], case["neighbors"] - 1)
    elif kind == "knn_batch":
        sizes = _sizes(case)
        st["x"] = torch.cat([_scores(int(m), case["width"], seed * 100 + i)
                             for i, m in enumerate(sizes)])
        st["first"] = np.concatenate([[0], np.cumsum(sizes)]).astype(np.uint64)
        st["out"] = _graph_out(int(sizes.sum()), case["neighbors"] - 1, case["samples"])
    elif kind == "connect":
        n, k = case["cells"], case["neighbors"] - 1
        st["graph"] = _neighbor_lists(n, k, seed)
        st["out"] = (torch.empty(n + 1, dtype=torch.int64, device=DEV),
                     torch.zeros(2 * n * k, dtype=torch.int32, device=DEV),
                     torch.zeros(2 * n * k, dtype=torch.float32, device=DEV))
    else:
        st["x"] = _mixture(case["cells"], case["width"], seed)
        st["out"] = _graph_out(case["cells"], case["neighbors"] - 1)
    return st


# ------------------------------------------------------------------ the calls --------
def _call(name: str, *args) -> None:
    status = getattr(K.library(), name)(*args)
    if status != K.KG_OK:
        buf = ctypes.create_string_buffer(4096)
        K.library().kg_last_error(None, buf, len(buf))
        raise K.KytoError(status, buf.value.decode(errors="replace"))


def _p(a):
    return a.ctypes.data if isinstance(a, np.ndarray) else a.data_ptr()


def run(st: dict):
    case = st["case"]
    kind = case["kind"]
    ctx = K.default_context().handle
    out = st.get("out")
    if kind == "normalize":
        dtype = K.KG_F32 if case["dtype"] == "f32" else K.KG_U32
        _call("kg_normalize_log1p", ctx, _p(st["indptr"]), _p(st["val"]), dtype, case["cells"],
              TARGET_SUM, 1, _p(out))
        return out
    if kind == "hvg":
        _call("kg_hvg_moments", ctx, _p(st["indptr"]), _p(st["idx"]), _p(st["val"]), K.KG_U32,
              case["cells"], case["genes"], TARGET_SUM, 1, _p(out["sums"]), _p(out["squares"]),
              _p(out["positives"]))
        return out
    if kind == "tiles":
        tb = K.TileBlock(0, case["cells"], TILE_CELLS, TILE_GENES, case["genes"],
                         _p(st["shard"]), _p(st["offsets"]), _p(st["local"]), _p(st["data"]),
                         K.KG_U32, 0)
        _call("kg_tiles_to_csr", ctx, ctypes.byref(tb), _p(out["indptr"]), _p(out["indices"]),
              _p(out["values"]))
        return out
    if kind == "pca":
        sess = K.PcaSession(case["k"], case["stream_genes"], seed=0, gene_set=st["flags"],
                            target_sum=TARGET_SUM if case["counts"] else None,
                            log1p=case["counts"])
        for indptr, idx, val in st["blocks"]:
            sess.push(indptr, idx, val)
        sess.run()
        k = case["k"]
        variance, ratio, means = np.empty(k), np.empty(k), np.empty(case["genes"])
        _call("kg_pca_results", sess._h, _p(out["embedding"]), _p(out["loadings"]),
              _p(variance), _p(ratio), _p(means))
        sess.close()
        return {**out, "variance": variance, "variance_ratio": ratio, "means": means}
    if kind == "knn":
        if case["host"]:
            g = K.neighbors(st["x"], case["neighbors"])
            return {"indptr": g.indptr, "indices": g.indices, "distances": g.distances}
        _call("kg_knn_exact", ctx, _p(st["x"]), case["cells"], case["width"], 0,
              case["neighbors"], _p(out["indptr"]), _p(out["indices"]), _p(out["distances"]),
              None)
        return out
    if kind == "knn_batch":
        _call("kg_knn_batch", ctx, _p(st["x"]), st["x"].shape[0], case["width"], 0,
              case["neighbors"], _p(st["first"]), case["samples"], _p(out["indptr"]),
              _p(out["indices"]), _p(out["distances"]), None)
        return out
    if kind == "connect":
        indptr, cols, dist = st["graph"]
        nnz = ctypes.c_uint64()
        _call("kg_connectivities", ctx, _p(indptr), _p(cols), _p(dist), case["cells"],
              case["neighbors"], _p(out[0]), _p(out[1]), _p(out[2]), ctypes.byref(nnz))
        return {"indptr": out[0], "indices": out[1], "weights": out[2], "nnz": nnz.value}
    params = K.LearnedParams()
    _call("kg_knn_learned", ctx, _p(st["x"]), case["cells"], case["width"], 0,
          case["neighbors"], ctypes.byref(params), _p(out["indptr"]), _p(out["indices"]),
          _p(out["distances"]), None)
    return out


# ------------------------------------------------------------------ work -------------
def work(case: dict) -> dict:
    """Bytes and operations a pass cannot do without: inputs read once, outputs written
    once, and the path's own arithmetic."""
    kind = case["kind"]
    if kind in ("normalize", "hvg", "tiles"):
        nnz = _stored(case["cells"], case["genes"], case["nnz"])
        if kind == "normalize":
            return {"bytes": 8 * nnz + 8 * case["cells"], "flops": 0}
        if kind == "hvg":
            return {"bytes": 8 * nnz + 8 * case["cells"] + 24 * case["genes"], "flops": 0}
        shard = 4 * (TILE_CELLS + 1) * -(-case["genes"] // TILE_GENES)
        return {"bytes": 16 * nnz + 8 * case["cells"] + shard, "flops": 0}
    if kind == "pca":
        # 21 sparse x dense products (the sketch, two in each of nine passes, the
        # embedding, the gene sums), each of which meets every stored value; one read of
        # the input and one write of the results.
        nnz = _stored(case["cells"], case["stream_genes"], case["nnz"])
        kept = nnz * case["genes"] / case["stream_genes"]
        w = min(case["k"] + 10, case["genes"])
        dense = 2.0 * case["genes"] * (9 * w) ** 2
        return {"bytes": 8 * nnz + 4 * case["k"] * (case["cells"] + case["stream_genes"]),
                "flops": 21 * 2.0 * kept * w + dense}
    if kind == "connect":
        e = case["cells"] * (case["neighbors"] - 1)
        return {"bytes": 8 * e + 8 * 1.2 * e + 16 * case["cells"], "flops": 0}
    k = case["neighbors"] - 1
    if kind == "knn_batch":
        sizes = _sizes(case).astype(np.float64)
        n, pairs = float(sizes.sum()), float((sizes * sizes).sum())
    else:
        n = case["cells"]
        # The learned form looks at about a hundredth of the pairs.
        pairs = n * float(n) * (0.01 if kind == "learned" else 1.0)
    return {"bytes": 4 * n * case["width"] + 8 * n * k + 8 * n,
            "flops": 2.0 * pairs * case["width"]}


# ------------------------------------------------------------------ 64-bit values ----
def _exact_hvg(st: dict) -> dict:
    case, g = st["case"], st["case"]["genes"]
    s = torch.zeros(g, dtype=torch.float64, device=DEV)
    q = torch.zeros(g, dtype=torch.float64, device=DEV)
    v = torch.expm1(_log1p(st["indptr"], st["val"], torch.float64))
    at = st["idx"].long()
    s.index_add_(0, at, v)
    q.index_add_(0, at, v * v)
    assert case["kind"] == "hvg"
    return {"sums": s, "squares": q, "positives": None}


def _wrap(v: int) -> int:
    return v - (1 << 64) if v >= 1 << 63 else v


def _shr(v: torch.Tensor, by: int) -> torch.Tensor:
    return (v >> by) & ((1 << (64 - by)) - 1)


def _mix(v: torch.Tensor) -> torch.Tensor:
    v = (v ^ _shr(v, 30)) * _wrap(0xBF58476D1CE4E5B9)
    v = (v ^ _shr(v, 27)) * _wrap(0x94D049BB133111EB)
    return v ^ _shr(v, 31)


def _omega(cells: int, width: int, seed: int = 0) -> torch.Tensor:
    """The sketch's random rows: SplitMix64 seeded from (seed, cell), in [-1, 1)."""
    golden = _wrap(0x9E3779B97F4A7C15)
    c = torch.arange(cells, dtype=torch.int64, device=DEV)
    state = _mix(_mix(c + golden) ^ seed)
    out = torch.empty((cells, width), dtype=torch.float64, device=DEV)
    for j in range(width):
        state = state + golden
        out[:, j] = _shr(_mix(state), 11).double() * 2.0 ** -52 - 1.0
    return out


def _extend(basis: torch.Tensor, block: torch.Tensor) -> torch.Tensor:
    scale = float(torch.linalg.norm(block))
    rest = block.clone()
    if basis.shape[1]:
        for _ in range(2):
            rest -= basis @ (basis.T @ rest)
    u, s, _ = torch.linalg.svd(rest, full_matrices=False)
    keep = int((s > 1e-10 * scale).sum()) if scale > 0 else 0
    return u[:, :keep].contiguous()


def _exact_pca(case: dict, seed: int) -> dict:
    """The block Krylov PCA on the dense matrix in 64 bits: the sketch, nine products, the
    Rayleigh-Ritz step over the whole basis, each loading's largest entry positive."""
    blocks, flags = _pca_input(case, seed)
    n, g, k, sg = case["cells"], case["genes"], case["k"], case["stream_genes"]
    x = torch.zeros((n, g), dtype=torch.float64, device=DEV)
    at = 0
    place = None
    if flags is not None:
        place = torch.full((sg,), -1, dtype=torch.int64, device=DEV)
        place[torch.from_numpy(flags).to(DEV)] = torch.arange(g, device=DEV)
    for indptr, idx, val in blocks:
        if case["counts"]:
            val = _log1p(indptr, val, torch.float64)
        m = indptr.numel() - 1
        for a in range(0, m, 65536):
            b = min(m, a + 65536)
            s, e = int(indptr[a]), int(indptr[b])
            r, c = _rows(indptr[a:b + 1]) + at + a, idx[s:e].long()
            v = val[s:e].double()
            if place is not None:
                c = place[c]
                keep = c >= 0
                r, c, v = r[keep], c[keep], v[keep]
            x[r, c] = v
        at += m
    means = x.mean(0)
    width = min(k + 10, g)
    omega = _omega(n, width)
    block = _extend(torch.zeros((g, 0), dtype=torch.float64, device=DEV),
                    x.T @ omega - torch.outer(means, omega.sum(0)))
    del omega
    basis = torch.zeros((g, 0), dtype=torch.float64, device=DEV)
    prod = torch.zeros((g, 0), dtype=torch.float64, device=DEV)
    for p in range(9):
        w = x @ block - means @ block
        c = x.T @ w - torch.outer(means, w.sum(0))
        basis, prod = torch.cat([basis, block], 1), torch.cat([prod, c], 1)
        if p < 8:
            block = _extend(basis, c)
            if block.shape[1] == 0:
                break
    t = basis.T @ prod
    values, vectors = torch.linalg.eigh(0.5 * (t + t.T))
    load = basis @ vectors.flip(1)[:, :k]
    eig = values.flip(0)[:k].clamp_min(0)
    top = load.gather(0, load.abs().argmax(0)[None, :])
    load = load * torch.where(top < 0, -1.0, 1.0)
    emb = torch.empty((n, k), dtype=torch.float64, device=DEV)
    torch.matmul(x, load, out=emb)
    emb -= means @ load
    x -= means
    total = sum(float(x[a:a + 65536].square().sum()) for a in range(0, n, 65536)) / (n - 1.0)
    full = torch.zeros((sg, k), dtype=torch.float64, device=DEV)
    if flags is None:
        full[:] = load
    else:
        full[torch.from_numpy(flags).to(DEV)] = load
    variance = eig / (n - 1.0)
    return {"embedding": emb, "loadings": full, "variance": variance,
            "variance_ratio": variance / total, "means": means}


def _exact_search(x: torch.Tensor, k: int) -> torch.Tensor:
    """Distances of each row's k nearest other rows, in the order of their columns."""
    n = x.shape[0]
    x = x.double()
    x = x - x.mean(0)
    norm = x.square().sum(1)
    out = torch.empty((n, k), dtype=torch.float64, device=DEV)
    step = max(1, min(n, 400_000_000 // n))
    more = min(n, k + 8)
    for a in range(0, n, step):
        b = min(n, a + step)
        d = norm[None, :] - 2.0 * (x[a:b] @ x.T)
        d[torch.arange(b - a, device=DEV), torch.arange(a, b, device=DEV)] = math.inf
        near = torch.topk(d, min(more, n - 1), dim=1, largest=False).indices
        del d
        near = near.sort(1).values
        key = (x[a:b, None, :] - x[near]).square().sum(2)
        pick = torch.sort(key, dim=1, stable=True).indices[:, :k].sort(1).values
        out[a:b] = torch.gather(key, 1, pick).sqrt()
    return out.reshape(-1)


def _exact_connect(st: dict) -> dict:
    """The UMAP weights in 64 bits: rho, the 64-step bisection for sigma, memberships,
    fuzzy union; rows then columns increasing."""
    n, nn = st["case"]["cells"], st["case"]["neighbors"]
    k = nn - 1
    cols, dist = st["graph"][1].view(n, k).long(), st["graph"][2].view(n, k).double()
    rho = dist.min(1).values
    gap = (dist - rho[:, None]).clamp_min(0)
    lo = torch.zeros(n, dtype=torch.float64, device=DEV)
    hi = torch.full((n,), math.inf, dtype=torch.float64, device=DEV)
    mid = torch.ones(n, dtype=torch.float64, device=DEV)
    live = torch.ones(n, dtype=torch.bool, device=DEV)
    for _ in range(64):
        total = torch.exp(-gap / mid[:, None]).sum(1)
        live &= (total - math.log2(nn)).abs() >= 1e-5
        up, down = live & (total > math.log2(nn)), live & (total <= math.log2(nn))
        hi = torch.where(up, mid, hi)
        lo = torch.where(down, mid, lo)
        step = torch.where(torch.isinf(hi), mid * 2.0, 0.5 * (lo + hi))
        mid = torch.where(live, step, mid)
    sigma = torch.maximum(mid, 1e-3 * dist.sum(1) / nn)
    w = torch.exp(-gap / sigma[:, None])
    row = torch.arange(n, device=DEV)[:, None].expand(n, k)
    keys = torch.cat([(row * n + cols).reshape(-1), (cols * n + row).reshape(-1)])
    keys, at = torch.unique(keys, return_inverse=True)
    a = torch.zeros(keys.numel(), dtype=torch.float64, device=DEV)
    b = torch.zeros(keys.numel(), dtype=torch.float64, device=DEV)
    a[at[:n * k]] = w.reshape(-1)
    b[at[n * k:]] = w.reshape(-1)
    weights = torch.zeros(2 * n * k, dtype=torch.float64, device=DEV)
    weights[:keys.numel()] = a + b - a * b
    return {"indptr": None, "indices": None, "weights": weights, "nnz": None}


def exact(case: dict, seed: int):
    kind = case["kind"]
    if kind == "pca":
        return _exact_pca(case, seed)
    if kind in ("tiles", "learned"):
        # Whole numbers moved; and a search inside parts that a trained network proposes.
        return None
    if kind == "knn" and case["cells"] > 250_000:
        return None  # tens of seconds
    st = prepare(case, seed)
    if kind == "normalize":
        return _log1p(st["indptr"], st["val"], torch.float64)
    if kind == "hvg":
        return _exact_hvg(st)
    if kind == "connect":
        return _exact_connect(st)
    k = case["neighbors"] - 1
    if kind == "knn":
        return {"indptr": None, "indices": None, "distances": _exact_search(st["x"], k)}
    first = st["first"].astype(np.int64)
    parts = [_exact_search(st["x"][a:b], k) for a, b in zip(first[:-1], first[1:])]
    return {"indptr": None, "indices": None, "distances": torch.cat(parts)}

"""Performance cases of the all-pairs library: what its users have it do.

Three containers make up the interface: StormContig (dense rows of one length),
Storm (sparse and mixed rows split into 65536-bit chunks) and StormRows (the
kernel layer, one representation per row).  A program fills a container once
and asks for the counts of all pairs: into device memory, into host memory, as
one sum, or only the pairs above a Jaccard threshold.  Row counts, row lengths
and value distributions are those of tests/gen.py and bench.py (dense Bernoulli
rows, haplotype-like rows, Bernoulli sets, Zipf cardinalities, unions of runs).
"""
import ctypes
import importlib
import math

import numpy as np
import torch

sb = importlib.import_module("stormbitmaps-internal_b200")

DEV = "cuda:0"
JACCARD = 0.8


def listed():
    return [
        # A handful of short rows: a call's fixed cost.
        {"name": "contig_tiny", "kind": "contig", "rows": 100, "bits": 1000, "dist": "half", "call": "host"},
        # The plain dense matrix every bitmap x bitmap path is quoted on, counts left on the device.
        {"name": "contig_4096x65536", "kind": "contig", "rows": 4096, "bits": 65536, "dist": "half", "call": "device"},
        # Variant sites x haplotypes: many short rows, output-heavy.
        {"name": "contig_haplotypes", "kind": "contig", "rows": 50000, "bits": 20000, "dist": "haplotypes", "call": "device"},
        # The largest dense matrix of one call: 2 GiB of rows, 8.6 GB of counts.
        {"name": "contig_65536x262144", "kind": "contig", "rows": 65536, "bits": 262144, "dist": "mixed", "call": "device"},
        # storm.h's own result, the sum over all pairs, of rows whose sizes are no round numbers.
        {"name": "contig_sum", "kind": "contig", "rows": 10007, "bits": 100003, "dist": "mixed", "call": "sum"},
        # Rows and counts both in host memory, in one call.
        {"name": "contig_from_host", "kind": "contig", "rows": 8192, "bits": 65536, "dist": "mixed", "call": "from_host"},
        # Only similar pairs are wanted.
        {"name": "contig_threshold", "kind": "contig", "rows": 12000, "bits": 20000, "dist": "haplotypes", "call": "threshold"},
        # A few mixed rows, counts in host memory.
        {"name": "storm_small", "kind": "storm", "rows": 200, "universe": 1 << 20, "dist": "zipf", "arg": 1.1, "call": "host"},
        # Very sparse sets over a large universe (the middle of the density sweep).
        {"name": "storm_bernoulli", "kind": "storm", "rows": 20000, "universe": 1 << 24, "dist": "bernoulli", "arg": 1e-4,
         "call": "device"},
        # Rows of 16 values beside rows of millions.
        {"name": "storm_zipf", "kind": "storm", "rows": 4096, "universe": 1 << 24, "dist": "zipf", "arg": 1.1, "call": "device"},
        # Rows made of long runs.
        {"name": "storm_runs", "kind": "storm", "rows": 4000, "universe": 1 << 26, "dist": "runs", "arg": 200.0, "call": "device"},
        # The kernel layer: mixed densities, one cell per tile by the cost model, one batched launch.
        {"name": "rows_zipf", "kind": "rows", "rows": 2048, "universe": 1 << 20, "dist": "zipf", "arg": 1.1, "call": "host"},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["contig"] * 6 + ["storm"] * 5 + ["rows"])
    if kind == "contig":
        call = rng.choice(["device", "device", "host", "sum", "from_host", "threshold"])
        bits = _log(rng, 5000 if call == "threshold" else 500, 500000)
        rows = _log(rng, 50, 40000 if call in ("device", "sum") else 12000)
        rows = min(rows, int((1 << 50) / bits) and int(math.sqrt((1 << 50) / bits)))
        dist = "haplotypes" if call == "threshold" or bits < 30000 and rng.random() < 0.5 else rng.choice(["half", "mixed"])
        return {"kind": kind, "rows": rows, "bits": bits, "dist": dist, "call": call}
    if kind == "rows":
        return {"kind": kind, "rows": _log(rng, 100, 2048), "universe": _log(rng, 1 << 16, 1 << 20), "dist": "zipf",
                "arg": 1.1, "call": "host"}
    call = rng.choice(["device", "device", "host", "sum"])
    dist = rng.choice(["bernoulli", "bernoulli", "zipf", "runs"])
    universe = _log(rng, 1 << 20, 1 << 26 if dist == "runs" else 1 << 24)
    if dist == "bernoulli":
        arg = float("%.3g" % math.exp(rng.uniform(math.log(1e-6), math.log(1e-2))))
        mean = arg * universe
    elif dist == "zipf":
        arg, mean = 1.1, universe / 250.0
    else:
        arg = float(_log(rng, 20, 200))
        mean = arg * 256
    rows = _log(rng, 100, max(200, min(20000, 8e7 / max(mean, 1.0))))
    return {"kind": "storm", "rows": rows, "universe": universe, "dist": dist, "arg": arg, "call": call}


# ------------------------------------------------------------------ inputs
def _generator(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return g


def _words(g, rows, words):
    """Uniform random 64-bit words."""
    return torch.randint(-(1 << 63), (1 << 63) - 1, (rows, words), generator=g, device=DEV, dtype=torch.int64)


def _dense_rows(case, seed):
    """[rows, ceil(bits / 64)] int64 on the GPU, bits past the row's end zero."""
    n, bits = case["rows"], case["bits"]
    w = (bits + 63) // 64
    g = _generator(seed)
    if case["dist"] == "haplotypes":
        return _haplotypes(g, n, bits, w)
    out = torch.empty((n, w), dtype=torch.int64, device=DEV)
    step = max(1, (1 << 26) // w)
    for r0 in range(0, n, step):
        k = min(n, r0 + step) - r0
        if case["dist"] == "half":
            out[r0:r0 + k] = _words(g, k, w)
            continue
        # density m / 64, m uniform over 3 .. 32 per row: one random word per
        # binary digit of the density, from the last digit up
        m = torch.randint(3, 33, (k, 1), generator=g, device=DEV)
        acc = torch.zeros((k, w), dtype=torch.int64, device=DEV)
        for digit in range(6):
            r = _words(g, k, w)
            acc = torch.where((m >> digit) & 1 == 1, acc | r, acc & r)
        out[r0:r0 + k] = acc
    if bits % 64:
        out[:, -1] &= (1 << (bits % 64)) - 1
    return out


def _haplotypes(g, n, bits, w, block=32):
    """Sites x haplotypes: k carriers, P(k) ~ 1/k on [1, bits), in whole blocks of
    `block` haplotypes, the last block taken only in part."""
    out = torch.empty((n, w), dtype=torch.int64, device=DEV)
    shifts = torch.arange(64, device=DEV, dtype=torch.int64)
    hap = torch.arange(w * 64, device=DEV)
    blocks = (bits + block - 1) // block
    of = (hap // block).clamp(max=blocks - 1)
    step = max(1, (1 << 27) // (w * 64))
    for r0 in range(0, n, step):
        m = min(n, r0 + step) - r0
        k = torch.exp(torch.rand((m, 1), generator=g, device=DEV) * math.log(bits)).long().clamp(1, bits - 1)
        nb = ((k + block - 1) // block).clamp(max=blocks)
        keys = torch.rand((m, blocks), generator=g, device=DEV)
        chosen = keys <= torch.gather(keys.sort(dim=1).values, 1, nb - 1)
        order = torch.cumsum(chosen.to(torch.int32), dim=1)
        b = chosen[:, of] & ((order[:, of] < nb) | (hap % block < k - block * (nb - 1))) & (hap < bits)
        out[r0:r0 + m] = (b.view(m, w, 64).long() << shifts).sum(dim=-1)
    return out


def _sets(case, seed):
    """Sorted positions of all rows and the rows' offsets, on the GPU (int64)."""
    n, u = case["rows"], case["universe"]
    g = _generator(seed)
    if case["dist"] == "runs":
        runs = torch.poisson(torch.full((n,), float(case["arg"]), device=DEV), generator=g).long()
        row = torch.repeat_interleave(torch.arange(n, device=DEV), runs)
        start = torch.randint(0, u, (row.numel(),), generator=g, device=DEV)
        length = torch.empty(row.numel(), device=DEV).geometric_(1.0 / 256, generator=g).long()
        length = torch.minimum(length, u - start)
        first = torch.cumsum(length, 0) - length
        key = torch.repeat_interleave(row * u + start - first, length)
        key += torch.arange(key.numel(), device=DEV)
    else:
        if case["dist"] == "zipf":
            lo, hi, a = 16.0, u / 4.0, 1.0 - case["arg"]
            x = torch.rand(n, generator=g, device=DEV, dtype=torch.float64)
            card = (lo ** a + x * (hi ** a - lo ** a)) ** (1.0 / a)
            card = -u * torch.log1p(-card / u)          # draws that leave about `card` distinct values
        else:
            p = u * case["arg"]
            card = p + math.sqrt(p) * torch.randn(n, generator=g, device=DEV, dtype=torch.float64)
        card = card.round().long().clamp(min=1)
        row = torch.repeat_interleave(torch.arange(n, device=DEV), card)
        key = row * u + torch.randint(0, u, (row.numel(),), generator=g, device=DEV)
    key = torch.unique(key)
    offs = torch.searchsorted(key, torch.arange(n + 1, device=DEV) * u)
    return key % u, offs


def _host_sets(case, seed):
    vals, offs = _sets(case, seed)
    return vals.to(torch.int32).cpu().numpy().view(np.uint32), offs.cpu().numpy().astype(np.uint64)


def _pairs(n):
    return n * (n + 1) // 2


def prepare(case, seed):
    n, kind, call = case["rows"], case["kind"], case["call"]
    st = {"call": call, "kind": kind, "cap": 8 * n}   # cap: the thresholded call's room for pairs
    if call == "device":
        st["out"] = torch.empty(_pairs(n), dtype=torch.int32, device=DEV)
    elif call in ("host", "from_host") and kind != "rows":
        st["pinned"] = torch.empty(_pairs(n), dtype=torch.int32).pin_memory()
        st["out"] = st["pinned"].numpy().view(np.uint32)
    if kind == "contig":
        rows = _dense_rows(case, seed)
        c = st["c"] = sb.StormContig(case["bits"])
        if call == "from_host":
            st["pinned_rows"] = rows.cpu().pin_memory()
            st["rows"] = st["pinned_rows"].numpy().view(np.uint64)
        else:
            ptr = ctypes.cast(rows.data_ptr(), sb.u64p)
            if sb.lib().STORM_contig_add_bitmaps(c.h, ptr, n, rows.shape[1]) != n:
                raise RuntimeError("STORM_contig_add_bitmaps")
            c.upload()
    else:
        vals, offs = _host_sets(case, seed)
        if kind == "rows":
            c = st["c"] = sb.StormRows(case["universe"])
            for r in range(n):
                c.add(vals[int(offs[r]):int(offs[r + 1])])
        else:
            c = st["c"] = sb.Storm()
            c.add_rows(vals, offs)
        c.upload()
    return st


def _padded(a, length):
    """The pairs found in arrays of one length, as a program with fixed buffers keeps them."""
    out = np.zeros(length, np.uint32)
    out[:len(a)] = a
    return out


def run(state):
    c, call = state["c"], state["call"]
    if state["kind"] == "rows":
        tri, stats = c.allpairs_matrix(sb.POLICY_PERTILE)
        return {"counts": tri, "sum": int(stats["sum"])}
    if call == "device":
        total = c.matrix_device(state["out"].data_ptr(), state["out"].numel())
        return {"counts": state["out"], "sum": total}
    if call == "host":
        tri, total = c.matrix(state["out"])
        return {"counts": tri, "sum": total}
    if call == "from_host":
        tri, total = c.matrix_from_host(state["rows"], state["out"])
        return {"counts": tri, "sum": total}
    if call == "threshold":
        i, j, counts, found = c.threshold(JACCARD, state["cap"])
        return {"i": _padded(i, state["cap"]), "j": _padded(j, state["cap"]), "counts": _padded(counts, state["cap"]),
                "found": found}
    return {"sum": c.pairw_intersect_cardinality()}


def work(case):
    """Rows in once, counts out once; dense rows as one multiply and one add per
    bit of every pair, sets as the values they hold.  A sum alone needs the rows
    and one count per column."""
    n = case["rows"]
    out = 4 * _pairs(n) if case["call"] in ("device", "host", "from_host") else 8
    if case["kind"] == "contig":
        bits = case["bits"]
        flops = 2 * n * bits if case["call"] == "sum" else 2 * _pairs(n) * bits
        return {"bytes": n * ((bits + 63) // 64) * 8 + out, "flops": flops}
    u = case["universe"]
    if case["dist"] == "bernoulli":
        mean = u * case["arg"]
    elif case["dist"] == "runs":
        mean = case["arg"] * 256
    else:
        lo, hi, s = 16.0, u / 4.0, case["arg"]
        mean = (hi ** (2 - s) - lo ** (2 - s)) / (2 - s) * (1 - s) / (hi ** (1 - s) - lo ** (1 - s))
    values = n * mean
    return {"bytes": min(4 * values, n * u / 8) + out, "flops": 2 * values}


# ------------------------------------------------------------------- exact
def _counts(case, seed):
    """All pairs' counts as a dense float64 matrix on the GPU (whole numbers)."""
    n = case["rows"]
    full = torch.zeros((n, n), dtype=torch.float64, device=DEV)
    if case["kind"] == "contig":
        rows = _dense_rows(case, seed)
        shifts = torch.arange(64, device=DEV, dtype=torch.int64)
        step = max(1, (1 << 28) // (64 * n))
        for w0 in range(0, rows.shape[1], step):
            b = ((rows[:, w0:w0 + step, None] >> shifts) & 1).reshape(n, -1).double()
            full += b @ b.T
        return full
    vals, offs = _sets(case, seed)
    row = torch.repeat_interleave(torch.arange(n, device=DEV), offs[1:] - offs[:-1])
    order = torch.argsort(vals)
    vals, row = vals[order], row[order]
    step = max(64, (1 << 28) // n)
    edges = torch.searchsorted(vals, torch.arange(0, case["universe"] + step, step, device=DEV)).tolist()
    for k in range(len(edges) - 1):
        lo, hi = edges[k], edges[k + 1]
        if lo == hi:
            continue
        b = torch.zeros((n, step), dtype=torch.float64, device=DEV)
        b[row[lo:hi], vals[lo:hi] - k * step] = 1.0
        full += b @ b.T
    return full


def exact(case, seed):
    n = case["rows"]
    if case["call"] == "sum":
        if case["kind"] == "contig":
            rows = _dense_rows(case, seed)
            cols = torch.stack([((rows >> b) & 1).sum(dim=0) for b in range(64)])
        else:
            cols = torch.bincount(_sets(case, seed)[0], minlength=case["universe"])
        return {"sum": int((cols * (cols - 1) // 2).sum())}
    length = case["bits"] if case["kind"] == "contig" else case["universe"]
    if n > 16384 or 2.0 * n * n * length > 1e14:
        return None
    full = _counts(case, seed)
    if case["call"] == "threshold":
        card = full.diagonal()
        ok = torch.triu((full > 0) & (full / (card[:, None] + card[None, :] - full) >= JACCARD), 1)
        i, j = torch.nonzero(ok, as_tuple=True)
        cols = {"i": i, "j": j, "counts": full[i, j].long()}
        cols = {k: torch.nn.functional.pad(v, (0, 8 * n - v.numel())) for k, v in cols.items()}
        return {**cols, "found": int(i.numel())}
    i, j = torch.triu_indices(n, n, device=DEV)
    return {"counts": full[i, j].long(), "sum": int(torch.triu(full, 1).sum().item())}

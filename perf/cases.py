"""The calls that users of this package make, for timing them.

Seven kinds of call on ``turboquant.TurboQuantSpace`` and ``turboquant.Index``:

  encode      encode_batch of device rows (indexing new vectors)
  scan        distance_1_to_n of one query over a corpus (brute-force search,
              re-ranking a candidate list), on device arrays or, as the
              reference's numpy users call it, on host arrays
  batch       distance_m_to_n of a query batch over a corpus
  sym         distance_m_to_n_symmetric of codes against codes (deduplication,
              clustering)
  sym_qjl     distance_m_to_n_symmetric_light / _full: the same with the QJL
              correction terms
  search      Index.search, the exact top-k of a resident corpus for host queries

Vectors are L2-normalised rows, as embedding models give them: i.i.d. normal
ones, or (``mixture``) a 1024-centre Gaussian mixture, where queries have near
neighbours.  Codes are drawn without the package: the rows go through the
quantizer's own definition in torch, which is what encode_batch would give but
for a few rounding ties.  ``exact`` decodes them and evaluates each distance's
formula in FP64.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "turboquant-space_b200", "python"))
import turboquant  # noqa: E402

ROT_SEED, QJL_SEED = 42, 137
DIMS = (64, 96, 100, 128, 200, 256, 300, 384, 512, 768, 1000, 1024, 1536)


# ---------------------------------------------------------------------------
# cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # A few documents' embeddings added to an index: launch latency.
        {"name": "encode_page", "kind": "encode", "n": 64, "dim": 384, "bits": 4},
        # Bulk indexing at the byte-code setting of the encode + scan workload.
        {"name": "encode_bulk", "kind": "encode", "n": 2_000_000, "dim": 768, "bits": 8},
        # A drop-in caller re-ranks 1,000 candidates on numpy arrays: the smallest call.
        {"name": "scan_host_rerank", "kind": "scan", "n": 1000, "dim": 128, "bits": 4, "host": True},
        # One query over a ragged million-code corpus of narrow 3-bit codes (padded dim 256).
        {"name": "scan_ragged", "kind": "scan", "n": 1_000_003, "dim": 200, "bits": 3, "host": False},
        # One query over the 10M x 768-d byte-code corpus, the HBM-bound headline scan.
        {"name": "scan_corpus", "kind": "scan", "n": 10_000_000, "dim": 768, "bits": 8, "host": False},
        # A handful of queries together (one user request with several passages).
        {"name": "batch_few", "kind": "batch", "m": 8, "n": 200_000, "dim": 384, "bits": 4,
         "precision": "fp32"},
        # An evaluation batch in the default precision, ragged on both sides.
        {"name": "batch_default", "kind": "batch", "m": 2000, "n": 250_007, "dim": 768, "bits": 4,
         "precision": "fp32"},
        # The dense batch of the split-BF16 workload, over half its corpus.
        {"name": "batch_bf16", "kind": "batch", "m": 4096, "n": 500_000, "dim": 768, "bits": 4,
         "precision": "split_bf16"},
        # Deduplicating new codes against a stored set, non-power-of-two dim.
        {"name": "sym_default", "kind": "sym", "m": 500, "n": 50_021, "dim": 1536, "bits": 4,
         "precision": "fp32"},
        # The same with the QJL correction (the light variant) on a smaller set.
        {"name": "sym_light", "kind": "sym_qjl", "m": 300, "n": 20_000, "dim": 384, "bits": 4,
         "precision": "fp32", "variant": "light"},
        # Interactive search: one request of a few queries over a modest corpus.
        {"name": "search_few", "kind": "search", "m": 5, "n": 300_000, "dim": 384, "bits": 4, "k": 10},
        # A full serving batch over a resident corpus.
        {"name": "search_batch", "kind": "search", "m": 1024, "n": 2_000_000, "dim": 384, "bits": 4,
         "k": 10},
    ]


def _log(rng, lo, hi):
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return max(lo, min(hi, int(round(v)) | rng.randint(0, 1)))


def draw(rng):
    """One more case: a kind, then sizes over the whole range of that kind, held
    to the work of the largest listed case."""
    kind = rng.choice(["encode", "scan", "batch", "batch", "sym", "sym_qjl", "search"])
    dim = rng.choice(DIMS) if rng.random() < 0.7 else rng.randint(64, 1536)
    bits = rng.choice([3, 4, 4, 4, 6, 8, 8])
    D = _padded(dim)
    cs = _code_size(D, bits)
    if kind == "encode":
        hi = min(2_000_000, 8_000_000_000 // (4 * dim + cs))
        return {"kind": kind, "n": _log(rng, 1, hi), "dim": dim, "bits": bits}
    if kind == "scan":
        host = rng.random() < 0.25
        hi = 100_000 if host else min(10_000_000, 10_000_000_000 // cs)
        return {"kind": kind, "n": _log(rng, 500, hi), "dim": dim, "bits": bits, "host": host}
    if kind == "search":
        n = _log(rng, 20_000, min(2_000_000, 2_000_000 * 512 // D))
        return {"kind": kind, "m": _log(rng, 1, 1024), "n": n, "dim": dim, "bits": bits,
                "k": rng.choice([1, 10, 16])}
    # Dense m x n: at most the listed cases' pairs x padded dim for the precision.
    if kind == "batch":
        precision = rng.choice(["fp32", "split_bf16"])
        m, pairs = _log(rng, 2, 4096), 4096 * 500_000 * 1024
        if precision == "fp32":
            pairs //= 4
    elif kind == "sym":
        precision = rng.choice(["fp32", "split_bf16"])
        m, pairs = _log(rng, 2, 2048), 500 * 50_021 * 2048
    else:
        precision = rng.choice(["fp32", "split_tf32"])
        m, pairs = _log(rng, 2, 1024), 500 * 50_021 * 1024
    n = _log(rng, 1000, max(1001, min(1_000_000, pairs // (m * D))))
    case = {"kind": kind, "m": m, "n": n, "dim": dim, "bits": bits, "precision": precision}
    if kind == "sym_qjl":
        case["variant"] = rng.choice(["light", "full"])
    return case


# ---------------------------------------------------------------------------
# the quantizer's definition, in torch (no package code)
# ---------------------------------------------------------------------------
def _padded(dim):
    return 1 << max(2, (dim - 1).bit_length())


def _code_size(D, bits):
    return (D // 2 if bits <= 4 else D) + 12


def _signs(D, seed):
    """splitmix64 stream, lowest bit 1 -> +1."""
    mask, state, out = (1 << 64) - 1, seed, []
    for _ in range(D):
        state = (state + 0x9E3779B97F4A7C15) & mask
        z = ((state ^ (state >> 30)) * 0xBF58476D1CE4E5B9) & mask
        z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & mask
        out.append(1.0 if (z ^ (z >> 31)) & 1 else -1.0)
    return out


_CENTROIDS = {}


def _centroids(bits):
    """Lloyd-Max levels of N(0,1) for bits - 1 index bits, rounded to float32."""
    if bits not in _CENTROIDS:
        half = 1 << (bits - 2)
        pdf = lambda x: math.exp(-0.5 * x * x) / math.sqrt(2 * math.pi)  # noqa: E731
        cdf = lambda x: 0.5 * math.erfc(-x * math.sqrt(0.5))  # noqa: E731
        c = [(i + 0.5) * 3.5 / half for i in range(half)]
        for _ in range(1000):
            edge = [0.0] + [0.5 * (c[i] + c[i + 1]) for i in range(half - 1)] + [1e10]
            nxt = []
            for a, b in zip(edge, edge[1:]):
                mass = cdf(b) - cdf(a)
                nxt.append((pdf(a) - pdf(b)) / mass if mass >= 1e-15 else 0.5 * (a + b))
            worst = max(abs(x - y) for x, y in zip(nxt, c))
            c = nxt
            if worst < 1e-12:
                break
        pos = np.array(c, dtype=np.float32)
        _CENTROIDS[bits] = np.concatenate([-pos[::-1], pos])
    return _CENTROIDS[bits]


def _rht(x, signs):
    """Randomized Hadamard transform of each row: signs, FWHT, 1/sqrt(D)."""
    n, D = x.shape
    x = x * signs
    h = 1
    while h < D:
        v = x.view(n, D // (2 * h), 2, h)
        x = torch.stack((v[:, :, 0] + v[:, :, 1], v[:, :, 0] - v[:, :, 1]), 2).view(n, D)
        h *= 2
    return x * (1.0 / math.sqrt(D))


def _sign_rows(D, device, dtype):
    return (torch.tensor(_signs(D, ROT_SEED), device=device, dtype=dtype),
            torch.tensor(_signs(D, QJL_SEED), device=device, dtype=dtype))


def _rows(gen, n, dim, centres, device):
    x = torch.randn(n, dim, generator=gen, device=device)
    if centres is not None:
        pick = torch.randint(0, centres.shape[0], (n,), generator=gen, device=device)
        x = x.mul_(0.3).add_(centres[pick])
    return x / x.norm(dim=1, keepdim=True)


def _draw_codes(gen, n, dim, bits, centres, device):
    D, pb = _padded(dim), _code_size(_padded(dim), bits) - 12
    cent = torch.from_numpy(_centroids(bits)).to(device)
    bound = (cent[1:] + cent[:-1]) * 0.5
    rot, qjl = _sign_rows(D, device, torch.float32)
    codes = torch.empty(n, pb + 12, dtype=torch.uint8, device=device)
    step = max(1, (1 << 28) // D)
    for a in range(0, n, step):
        b = min(n, a + step)
        x = _rows(gen, b - a, dim, centres, device)
        norm = x.norm(dim=1, keepdim=True)
        z = _rht(torch.nn.functional.pad(x / norm, (0, D - dim)), rot)
        sigma = z.square().mean(dim=1, keepdim=True).sqrt()
        idx = torch.bucketize(z / sigma, bound)
        res = z - cent[idx] * sigma
        gamma = res.norm(dim=1, keepdim=True)
        unit = (idx * 2).to(torch.uint8) + (_rht(res, qjl) >= 0)
        codes[a:b, :pb] = unit[:, ::2] + unit[:, 1::2] * 16 if bits <= 4 else unit
        codes[a:b, pb:] = torch.cat((norm, gamma, sigma), 1).contiguous().view(torch.uint8)
    return codes


def _inputs(case, seed, device="cuda"):
    """The case's rows, queries and codes, from the seed alone."""
    gen = torch.Generator(device=device)
    gen.manual_seed(1_000_003 * seed + 17)
    kind, dim, bits = case["kind"], case["dim"], case["bits"]
    centres = torch.randn(1024, dim, generator=gen, device=device) \
        if kind in ("sym", "sym_qjl", "search") else None
    if kind == "encode":
        return {"X": _rows(gen, case["n"], dim, centres, device)}
    d = {"codes": _draw_codes(gen, case["n"], dim, bits, centres, device)}
    if kind in ("sym", "sym_qjl"):
        d["codes_a"] = _draw_codes(gen, case["m"], dim, bits, centres, device)
    else:
        d["queries"] = _rows(gen, case.get("m", 1), dim, centres, device)
    return d


# ---------------------------------------------------------------------------
# what a program has in hand, and the call
# ---------------------------------------------------------------------------
def prepare(case, seed):
    d = _inputs(case, seed)
    s = {"case": case, "space": turboquant.TurboQuantSpace(case["dim"], case["bits"])}
    if case["kind"] == "scan":
        q, c = d["queries"][0].contiguous(), d["codes"]
        s["queries"], s["codes"] = (q.cpu().numpy(), c.cpu().numpy()) if case["host"] else (q, c)
    elif case["kind"] == "search":
        s["queries"] = d["queries"].cpu().numpy()
        torch.cuda.synchronize()
        s["index"] = s["space"].index(d["codes"])
        # a serving program starts its search server before the first request
        s["index"].search(s["queries"][::-1][:1] * np.float32(0.5), k=case["k"])
    else:
        s.update(d)
    return s


def run(state):
    case, space = state["case"], state["space"]
    kind = case["kind"]
    if kind == "encode":
        return space.encode_batch(state["X"])
    if kind == "scan":
        return space.distance_1_to_n(state["queries"], state["codes"])
    if kind == "batch":
        return space.distance_m_to_n(state["queries"], state["codes"], precision=case["precision"])
    if kind == "sym":
        return space.distance_m_to_n_symmetric(state["codes_a"], state["codes"],
                                               precision=case["precision"])
    if kind == "sym_qjl":
        call = space.distance_m_to_n_symmetric_light if case["variant"] == "light" \
            else space.distance_m_to_n_symmetric_full
        return call(state["codes_a"], state["codes"], precision=case["precision"])
    return state["index"].search(state["queries"], k=case["k"])


def work(case):
    kind, dim, n = case["kind"], case["dim"], case["n"]
    D = _padded(dim)
    cs = _code_size(D, case["bits"])
    if kind == "encode":  # two FWHTs, three reductions, quantize + residual
        return {"bytes": n * (4 * dim + cs), "flops": n * D * (2 * int(math.log2(D)) + 12)}
    if kind == "scan":
        return {"bytes": n * (cs + 4) + 4 * dim, "flops": 4 * D * n}
    m = case["m"]
    if kind == "batch":
        return {"bytes": n * cs + 4 * m * dim + 4 * m * n, "flops": 4 * D * m * n}
    if kind == "search":
        return {"bytes": n * cs + m * (4 * dim + 12 * case["k"]), "flops": 4 * D * m * n}
    per = 2 if kind == "sym" else 4 if case["variant"] == "light" else 8
    return {"bytes": (n + m) * cs + 4 * m * n, "flops": per * D * m * n}


# ---------------------------------------------------------------------------
# FP64
# ---------------------------------------------------------------------------
def _decode64(codes, D, bits):
    """Centroid values, +-1 signs [rows, D] and the trailer [rows, 3], FP64."""
    pb = codes.shape[1] - 12
    unit = codes[:, :pb]
    if bits <= 4:
        unit = torch.stack((unit & 15, unit >> 4), 2).reshape(codes.shape[0], D)
    cent = torch.from_numpy(_centroids(bits)).to(codes.device).double()
    meta = codes[:, pb:].contiguous().view(torch.float32).double()
    return cent[(unit >> 1).long()], (unit & 1).double() * 2 - 1, meta


def _query64(q, D):
    """q_rot and s_q of the normalised queries, and |q|, FP64."""
    rot, qjl = _sign_rows(D, q.device, torch.float64)
    q = q.double()
    norm = q.norm(dim=1, keepdim=True)
    q_rot = _rht(torch.nn.functional.pad(q / norm, (0, D - q.shape[1])), rot)
    return q_rot, _rht(q_rot, qjl), norm


def _chunks(n, rows, D):
    step = max(1, (1 << 27) // max(D, rows))
    return [(a, min(n, a + step)) for a in range(0, n, step)]


def _asym64(d, D, bits):
    """[(first code, distances [m, codes])] over chunks of the codes."""
    q_rot, s_q, qn = _query64(d["queries"], D)
    for a, b in _chunks(d["codes"].shape[0], q_rot.shape[0], D):
        c, sgn, meta = _decode64(d["codes"][a:b], D, bits)
        norm, gamma, sigma = meta.unbind(1)
        ip = (q_rot @ c.T) * sigma + (s_q @ sgn.T) * (math.sqrt(math.pi / 2 / D) * gamma)
        yield a, (qn * qn + norm * norm - 2 * ip * norm * qn).clamp_(min=0)


def _sym64(d, D, bits, variant):
    ca, sa, ma = _decode64(d["codes_a"], D, bits)
    na, ga, siga = (t[:, None] for t in ma.unbind(1))
    qjl = _sign_rows(D, ca.device, torch.float64)[1]
    scale = math.sqrt(math.pi / 2 / D)
    for a, b in _chunks(d["codes"].shape[0], ca.shape[0], D):
        c, sgn, meta = _decode64(d["codes"][a:b], D, bits)
        norm, gamma, sigma = meta.unbind(1)
        ip = (ca @ c.T) * siga * sigma
        if variant:
            corr = (sa @ sgn.T) * ga * gamma * (math.pi / (2 * D))
            if variant == "full":
                ra, rb = _rht(ca * siga, qjl), _rht(c * sigma[:, None], qjl)
                corr = corr + (ra @ sgn.T) * (scale * gamma) + (sa @ rb.T) * (scale * ga)
            ip = ip + torch.minimum(torch.maximum(corr, -ip.abs()), ip.abs())
        yield a, (na * na + norm * norm - 2 * ip * na * norm).clamp_(min=0)


def exact(case, seed):
    kind, bits = case["kind"], case["bits"]
    if kind == "encode":  # bytes: held equal as they are
        return None
    d, D = _inputs(case, seed), _padded(case["dim"])
    if kind in ("sym", "sym_qjl"):
        parts = _sym64(d, D, bits, case.get("variant"))
    else:
        parts = _asym64(d, D, bits)
    if kind != "search":
        out = torch.cat([p for _, p in parts], 1)
        return out[0] if kind == "scan" else out
    best = None
    for _, p in parts:
        best = p if best is None else torch.cat((best, p), 1)
        best = best.topk(case["k"], dim=1, largest=False, sorted=True).values
    return best, None

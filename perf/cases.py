"""Timed cases of the GF(2^16) erasure-coding library.

Each case is one call (or one batch) that a program using the library makes:
recovery-slice creation, repair, per-slice hashing, the decode matrix, the
strategy's region multiply-accumulate and a batch of mixed jobs, over the
sizes that PAR2 sets have in practice: from a handful of small slices to the
format's tens of thousands, even slice lengths that are no multiple of any
tile, redundancies of 1 to 20 %.  Slices are uniform random bytes, which is
what compressed archives (the usual content of a PAR2 set) look like.

listed() gives the fixed cases, draw(rng) one more of the same ranges,
prepare(case, seed) the buffers, run(state) one pass, work(case) the bytes and
operations that the pass cannot do without, exact(case, seed) the outputs from
the definitions (logarithm tables, hashlib, zlib) where that is quick.
"""
import hashlib
import os
import sys
import zlib

import numpy as np
import torch

_PKG = os.path.join(os.getcwd(), "par2-rs_b200")
if _PKG not in sys.path:
    sys.path.insert(1, _PKG)

import par2gpu  # noqa: E402

KIB = 1024
MIB = 1024 * KIB
# the most one drawn case may cost: source bytes, symbol multiply-accumulates
MAX_BYTES = 1 << 30
MAX_MACS = 2.5e11


def listed():
    return [
        # a small document set: QuickPar-sized slices, two recovery slices;
        # the call's latency and launches are all there is
        {"name": "encode_tiny", "kind": "encode", "k": 20, "slice_bytes": 4 * KIB, "r": 2},
        # one 16 MiB file in 64 KiB slices at 5 %
        {"name": "encode_plain", "kind": "encode", "k": 256, "slice_bytes": 64 * KIB, "r": 13},
        # a set whose slice size was derived from a block count: even, but a
        # multiple of nothing; 8 %
        {"name": "encode_ragged", "kind": "encode", "k": 777, "slice_bytes": 150002, "r": 61},
        # 4 files x 512 MiB in 1 MiB slices at 10 %: the headline encode
        {"name": "encode_large", "kind": "encode", "k": 2048, "slice_bytes": MIB, "r": 205},
        # 512 MiB encoded from pinned host buffers, copies included: what a
        # program pays whose files are in host memory
        {"name": "encode_host", "kind": "encode_host", "k": 1024, "slice_bytes": 512 * KIB,
         "r": 102},
        # the plain set with all its redundancy used up by scattered damage
        {"name": "repair_plain", "kind": "repair", "k": 256, "slice_bytes": 64 * KIB, "m": 13,
         "lost": 0},
        # the high-slice-count set: 1600 of 32000 slices rebuilt
        {"name": "repair_many", "kind": "repair", "k": 32000, "slice_bytes": 64 * KIB, "m": 1600,
         "lost": 0},
        # its decode matrix alone, three of the recovery slices lost as well
        {"name": "decode_matrix", "kind": "matrix", "k": 32000, "m": 1600, "lost": 3},
        # verification of the high-slice-count set
        {"name": "verify_many", "kind": "verify", "n": 32000, "slice_bytes": 64 * KIB},
        # checksums of few large slices
        {"name": "hash_large_slices", "kind": "hash", "n": 300, "slice_bytes": MIB},
        # the strategy's region call as a chunked reconstruction makes it:
        # every present slice's chunk into the accumulators of the missing
        {"name": "region_chunk", "kind": "region", "nsrc": 400, "ndst": 32, "n": 32768},
        # uneven sets of a service: creates, repairs and verifications in one
        # batch
        {"name": "batch_mixed", "kind": "batch", "jobs": 48, "mean_bytes": 8 * MIB,
         "mix": 1},
    ]


def _log_uniform(rng, lo, hi):
    return lo * (hi / lo) ** rng.random()


def _slices(rng, macs_of):
    """k, S and r within the cost limits; macs_of(k, r, S)."""
    while True:
        k = int(_log_uniform(rng, 12, 32000))
        S = int(_log_uniform(rng, 1 * KIB, 4 * MIB))
        # half of the sets use whole KiB, the others any even length
        S = max(KIB, S // KIB * KIB) if rng.random() < 0.5 else S & ~1
        r = max(1, int(k * rng.uniform(0.01, 0.2)))
        if k * S <= MAX_BYTES and macs_of(k, r, S) <= MAX_MACS and r <= 2000:
            return k, S, r


def draw(rng):
    x = rng.random()
    macs = lambda k, r, S: k * r * S / 2  # noqa: E731
    if x < 0.40:
        k, S, r = _slices(rng, macs)
        return {"kind": "encode", "k": k, "slice_bytes": S, "r": r}
    if x < 0.60:
        k, S, r = _slices(rng, macs)
        return {"kind": "repair", "k": k, "slice_bytes": S, "m": r, "lost": rng.choice([0, 0, 1, 5])}
    if x < 0.68:
        k, S, r = _slices(rng, lambda k, r, S: macs(k, r, S) * 2)
        return {"kind": "encode_host", "k": k, "slice_bytes": S, "r": r}
    if x < 0.75:
        m = int(_log_uniform(rng, 5, 2000))
        return {"kind": "matrix", "k": min(32000, m * rng.randint(5, 40)), "m": m,
                "lost": rng.choice([0, 1, 5, 20])}
    if x < 0.83:
        n = int(_log_uniform(rng, 20, 32000))
        S = int(_log_uniform(rng, 1 * KIB, min(MIB, MAX_BYTES // n))) & ~1
        return {"kind": rng.choice(["verify", "hash"]), "n": n, "slice_bytes": S}
    if x < 0.92:
        return {"kind": "region", "nsrc": int(_log_uniform(rng, 1, 1000)),
                "ndst": int(_log_uniform(rng, 1, 128)), "n": int(_log_uniform(rng, 500, 100000))}
    return {"kind": "batch", "jobs": rng.randint(4, 64),
            "mean_bytes": int(_log_uniform(rng, 256 * KIB, 12 * MIB)),
            "mix": rng.randint(0, 1 << 30)}


# --- inputs ---------------------------------------------------------------

_ctx = None


def _context():
    """The one context a program keeps, ordered with torch's stream."""
    global _ctx
    if _ctx is None:
        _ctx = par2gpu.Context(0)
        _ctx.set_stream(torch.cuda.current_stream().cuda_stream)
    return _ctx


def _rows(n, S, gen, fill=True):
    """n slices of S bytes, each starting on a 16-byte boundary, as an [n, S]
    view of one allocation."""
    pitch = (S + 15) // 16 * 16
    if fill:
        t = torch.randint(0, 256, (n, pitch), dtype=torch.uint8, device="cuda", generator=gen)
    else:
        t = torch.zeros((n, pitch), dtype=torch.uint8, device="cuda")
    return t[:, :S]


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _addr(t):
    return (np.uint64(t.data_ptr()) +
            np.arange(t.shape[0], dtype=np.uint64) * np.uint64(t.stride(0)))


def _choice(n, m, seed):
    """m ascending indices below n."""
    return np.sort(np.random.default_rng(seed).choice(n, m, replace=False)).astype(np.uint64)


def _exponents(m, lost, seed):
    """The m lowest exponents left when `lost` of the first m + lost are gone."""
    gone = set(int(e) for e in _choice(m + lost, lost, seed + 77)) if lost else set()
    return np.array([e for e in range(m + lost) if e not in gone], np.uint32)


def _repair_inputs(k, S, m, lost, seed):
    """A set with m slices erased: the slices and the recovery slices that a
    set on disk would hold (made by the library's encode)."""
    data = _rows(k, S, _gen(seed))
    exps = _exponents(m, lost, seed)
    rec = _rows(m, S, None, fill=False)
    _context().encode(_addr(data), S, exps, _addr(rec), device=True)
    missing = _choice(k, m, seed)
    present = _addr(data)[np.setdiff1d(np.arange(k), missing.astype(np.int64))]
    return {"data": data, "exps": exps, "rec": rec, "missing": missing, "present": present,
            "out": _rows(m, S, None, fill=False)}


def _batch_specs(case):
    """Job descriptions of the batch: uneven sets, 40 % creates, 40 % repairs,
    20 % verifications; sizes log-uniform over a factor of 64."""
    rng = np.random.default_rng(case["mix"])
    specs = []
    mean = case["mean_bytes"]
    for _ in range(case["jobs"]):
        total = mean / 16 * 64 ** rng.random()
        S = int(min(max(1024, 4096 * 64 ** rng.random()), total / 8)) & ~1
        S = max(S, 512)
        k = int(min(4000, max(8, total // S)))
        r = max(1, int(k * rng.uniform(0.01, 0.2)))
        specs.append((("create", "repair", "verify")[int(rng.choice(3, p=[0.4, 0.4, 0.2]))],
                      k, S, r))
    return specs


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case, "ctx": _context()}
    if kind == "encode":
        s["src"] = _rows(case["k"], case["slice_bytes"], _gen(seed))
        s["out"] = _rows(case["r"], case["slice_bytes"], None, fill=False)
        s["exps"] = np.arange(case["r"], dtype=np.uint32)
        s["src_addr"], s["out_addr"] = _addr(s["src"]), _addr(s["out"])
    elif kind == "encode_host":
        k, S, r = case["k"], case["slice_bytes"], case["r"]
        src = torch.empty((k, S), dtype=torch.uint8, pin_memory=True)
        src.copy_(torch.randint(0, 256, (k, S), dtype=torch.uint8, device="cuda",
                                generator=_gen(seed)))
        s["src"] = src.numpy()
        s["out"] = torch.zeros((r, S), dtype=torch.uint8, pin_memory=True).numpy()
        s["exps"] = np.arange(r, dtype=np.uint32)
    elif kind == "repair":
        s.update(_repair_inputs(case["k"], case["slice_bytes"], case["m"], case["lost"], seed))
        s["rec_addr"], s["out_addr"] = _addr(s["rec"]), _addr(s["out"])
    elif kind == "matrix":
        s["missing"] = _choice(case["k"], case["m"], seed)
        s["exps"] = _exponents(case["m"], case["lost"], seed)
    elif kind in ("hash", "verify"):
        n, S = case["n"], case["slice_bytes"]
        s["src"] = _rows(n, S, _gen(seed))
        s["src_addr"] = _addr(s["src"])
        if kind == "verify":
            # the set's checksums, then one slice in twenty damaged
            s["md5"], s["crc"] = s["ctx"].hash_slices(s["src_addr"], S, device=True)
            bad = _choice(n, max(1, n // 20), seed)
            s["src"][torch.from_numpy(bad.astype(np.int64)).cuda(), S // 2] ^= 0x5A
    elif kind == "region":
        rng = np.random.default_rng(seed)
        s["src"] = _rows(case["nsrc"], 2 * case["n"], _gen(seed))
        s["dst"] = _rows(case["ndst"], 2 * case["n"], None, fill=False)
        s["coeff"] = rng.integers(0, 65536, (case["ndst"], case["nsrc"])).astype(np.uint16)
        s["src_addr"], s["dst_addr"] = _addr(s["src"]), _addr(s["dst"])
    elif kind == "batch":
        s.update(_prepare_batch(case, seed))
    return s


def _prepare_batch(case, seed):
    specs = _batch_specs(case)
    pitches = [(S + 15) // 16 * 16 for _, _, S, _ in specs]
    total = sum(r * p for (what, _, _, r), p in zip(specs, pitches) if what != "verify")
    out = torch.zeros(max(16, total), dtype=torch.uint8, device="cuda")
    jobs, keep, at = [], [], 0
    for j, (what, k, S, r) in enumerate(specs):
        if what == "verify":
            src = _rows(k, S, _gen(seed * 1000 + j))
            keep.append(src)
            jobs.append({"kind": par2gpu.JOB_VERIFY, "k": k, "slice_bytes": S, "src": _addr(src)})
            continue
        dst = out[at:at + r * pitches[j]].view(r, pitches[j])[:, :S]
        at += r * pitches[j]
        if what == "create":
            src = _rows(k, S, _gen(seed * 1000 + j))
            keep.append(src)
            jobs.append({"kind": par2gpu.JOB_CREATE, "k": k, "slice_bytes": S, "src": _addr(src),
                         "exps": np.arange(r, dtype=np.uint32), "out": _addr(dst)})
        else:
            p = _repair_inputs(k, S, r, 0, seed * 1000 + j)
            keep.append(p)
            jobs.append({"kind": par2gpu.JOB_REPAIR, "k": k, "slice_bytes": S,
                         "src": p["present"], "missing": p["missing"], "exps": p["exps"],
                         "recovery": _addr(p["rec"]), "out": _addr(dst)})
    return {"jobs": jobs, "out": out, "keep": keep}


# --- one pass -------------------------------------------------------------

def run(s):
    case, ctx = s["case"], s["ctx"]
    kind = case["kind"]
    if kind == "encode":
        ctx.encode(s["src_addr"], case["slice_bytes"], s["exps"], s["out_addr"], device=True)
        return s["out"]
    if kind == "encode_host":
        ctx.encode(s["src"], case["slice_bytes"], s["exps"], s["out"])
        return s["out"]
    if kind == "repair":
        ctx.repair(case["k"], case["slice_bytes"], s["missing"], s["present"], s["exps"],
                   s["rec_addr"], s["out_addr"], device=True)
        return s["out"]
    if kind == "matrix":
        return ctx.reconstruction_matrix(case["k"], s["missing"], s["exps"])
    if kind == "hash":
        return list(ctx.hash_slices(s["src_addr"], case["slice_bytes"], device=True))
    if kind == "verify":
        return ctx.verify_slices(s["src_addr"], case["slice_bytes"], s["md5"], s["crc"],
                                 device=True)
    if kind == "region":
        # a chunk's accumulators start at zero
        s["dst"].zero_()
        ctx.muladd_region(s["dst_addr"], s["src_addr"], s["coeff"], 0, case["n"], device=True)
        return s["dst"]
    batch = par2gpu.Batch(ctx, s["jobs"])
    status = batch.run()
    sums = [(res["md5"], res["crc"]) for res in batch.results if res]
    batch.close()
    none = (np.zeros((0, 16), np.uint8), np.zeros(0, np.uint32))
    return {"out": s["out"], "status": np.array(status, np.int32),
            "md5": np.concatenate([a for a, _ in sums] or [none[0]]),
            "crc": np.concatenate([b for _, b in sums] or [none[1]])}


# --- what a pass cannot do without ----------------------------------------

def _muladd_work(k, r, S):
    """Every source read once, every output written once; a multiplication and
    an addition per symbol of each (source, output) pair."""
    return {"bytes": (k + r) * S, "flops": k * r * S}


def _md5_work(n, S):
    # 64 steps of 5 additions and logic operations and one rotation per 64 bytes
    return {"bytes": n * S + 20 * n, "flops": n * (S // 64 + 1) * 64 * 6}


def work(case):
    kind = case["kind"]
    if kind in ("encode", "encode_host"):
        return _muladd_work(case["k"], case["r"], case["slice_bytes"])
    if kind == "repair":
        return _muladd_work(case["k"], case["m"], case["slice_bytes"])
    if kind == "matrix":
        # the inverse of a Vandermonde matrix takes a few operations an entry
        return {"bytes": 2 * case["m"] ** 2, "flops": 4 * case["m"] ** 2}
    if kind in ("hash", "verify"):
        return _md5_work(case["n"], case["slice_bytes"])
    if kind == "region":
        w = _muladd_work(case["nsrc"], case["ndst"], 2 * case["n"])
        return w
    total = {"bytes": 0, "flops": 0}
    for what, k, S, r in _batch_specs(case):
        w = _md5_work(k, S) if what == "verify" else _muladd_work(k, r, S)
        total = {q: total[q] + w[q] for q in total}
    return total


# --- outputs from the definitions -----------------------------------------

def _tables():
    """Antilogarithms and logarithms of GF(2^16), polynomial 0x1100B."""
    exp = np.zeros(131070, np.uint16)
    log = np.zeros(65536, np.int64)
    b = 1
    for i in range(65535):
        exp[i] = exp[i + 65535] = b
        log[b] = i
        b <<= 1
        if b & 0x10000:
            b ^= 0x1100B
    return exp, log


def _constants(k, exp):
    n, out = 1, []
    while len(out) < k:
        if n % 3 and n % 5 and n % 17 and n % 257:
            out.append(int(exp[n % 65535]))
        n += 1
    return out


def _products(coeff, src, exp, log):
    """coeff [r][k] times src [k][n] over GF(2^16)."""
    out = np.zeros((coeff.shape[0], src.shape[1]), np.uint16)
    for i in range(src.shape[0]):
        row, lg = src[i], log[src[i]]
        nz = row != 0
        for o in range(coeff.shape[0]):
            if coeff[o, i]:
                out[o] ^= np.where(nz, exp[lg + log[coeff[o, i]]], 0).astype(np.uint16)
    return out


def _symbols(rows):
    return np.ascontiguousarray(rows).view("<u2")


def exact(case, seed):
    kind = case["kind"]
    if kind == "encode" and case["k"] * case["r"] * case["slice_bytes"] <= 5e8:
        exp, log = _tables()
        src = _rows(case["k"], case["slice_bytes"], _gen(seed)).cpu().numpy()
        cs = _constants(case["k"], exp)
        coeff = np.array([[exp[log[c] * e % 65535] for c in cs] for e in range(case["r"])],
                         np.uint16)
        return _products(coeff, _symbols(src), exp, log).view(np.uint8)
    if kind == "region" and case["nsrc"] * case["ndst"] * case["n"] <= 2.5e8:
        exp, log = _tables()
        src = _rows(case["nsrc"], 2 * case["n"], _gen(seed)).cpu().numpy()
        rng = np.random.default_rng(seed)
        coeff = rng.integers(0, 65536, (case["ndst"], case["nsrc"])).astype(np.uint16)
        return _products(coeff, _symbols(src), exp, log).view(np.uint8)
    if kind == "repair" and case["k"] * case["slice_bytes"] <= MAX_BYTES:
        # what was erased
        data = _rows(case["k"], case["slice_bytes"], _gen(seed))
        miss = _choice(case["k"], case["m"], seed).astype(np.int64)
        return data[torch.from_numpy(miss).cuda()].cpu().numpy()
    if kind == "hash" and case["n"] * case["slice_bytes"] <= MAX_BYTES:
        src = _rows(case["n"], case["slice_bytes"], _gen(seed)).cpu().numpy()
        md5 = [np.frombuffer(hashlib.md5(row.tobytes()).digest(), np.uint8) for row in src]
        return [np.stack(md5), np.array([zlib.crc32(row.tobytes()) for row in src], np.uint32)]
    if kind == "verify":
        ok = np.ones(case["n"], bool)
        ok[_choice(case["n"], max(1, case["n"] // 20), seed).astype(np.int64)] = False
        return ok
    return None

"""The work that a user of turbovec_b200 has it do, as cases that can be timed and compared.

A case is a plain dict.  `kind`:
  search  an index that has been built, and one batch of queries against it (the serving path);
  build   rows into a fresh index and a first batch of queries against the result (the loading path);
  upsert  rows of a serving index replaced under their ids, and the next batch of queries (the updating path).
`api` is "host" (numpy arrays, as the reference's binding takes them) or "device" (rows, queries and results in
device memory).  `filter` is "none", "mask" (a slot mask) or "allow" (an id allowlist); `allowed` is the share of the
rows that pass it.  Bits 4 runs the permute-dot score family, bits 2 and 3 the u8-table families (dimension 200 at
2 bits the flush form).
"""
import math

import numpy as np
import torch

import turbovec_b200 as tv

CHUNK_ROWS = 250_000          # rows generated and added at a time
DIMS = [64, 96, 128, 200, 256, 384, 512, 768, 1000, 1024, 1152, 1536, 2048, 3072]


def _search(name, n, dim, bits, nq, k, api, filter="none", allowed=1.0):
    return {"name": name, "kind": "search", "n": n, "dim": dim, "bits": bits, "nq": nq, "k": k, "api": api,
            "filter": filter, "allowed": allowed}


def listed():
    return [
        # one user's question against a small collection: latency and launches are all there is
        _search("single_100k", 100_000, 1536, 4, 1, 10, "host"),
        # one question against the largest collection of one GPU, caller and results on the device: streams the codes
        _search("single_10m", 10_000_000, 1536, 4, 1, 10, "device"),
        # the offline or heavily loaded end: a full batch against the largest collection, a dense int8 contraction
        _search("batch1024_10m", 10_000_000, 1536, 4, 1024, 10, "device"),
        # a server that gathers a few dozen requests at a time, numpy in and numpy out
        _search("batch32_1m", 1_000_000, 1536, 4, 32, 10, "host"),
        # word vectors: short rows, ragged sizes, long result lists (candidates for a later re-ranking)
        _search("words_4bit", 1_193_517, 200, 4, 100, 100, "host"),
        # the same rows at two bits in a full batch: the flush form of the u8-table family
        _search("words_2bit", 1_193_517, 200, 2, 1024, 10, "device"),
        # long embeddings at two bits, one question
        _search("long_2bit_single", 1_000_000, 3072, 2, 1, 10, "device"),
        # long embeddings at two bits, a gathered batch
        _search("long_2bit_batch", 1_000_000, 3072, 2, 64, 10, "host"),
        # one tenant of many: an id allowlist of a hundredth of the rows, resolved on each call
        dict(_search("tenant", 1_000_000, 768, 4, 16, 10, "host", "allow", 0.01)),
        # bulk load of embeddings that a model has left in device memory, the scales for the caller's records, the first questions
        {"name": "build_2m", "kind": "build", "n": 2_000_000, "dim": 1536, "bits": 4, "nq": 16, "k": 100, "api": "device"},
        # a small collection from numpy rows, ragged, three bits, its parts exported
        {"name": "build_host", "kind": "build", "n": 20_011, "dim": 384, "bits": 3, "nq": 3, "k": 10, "api": "host"},
        # a serving index under change: 64 documents replaced, then the next eight questions
        {"name": "upsert", "kind": "upsert", "n": 200_000, "dim": 768, "bits": 4, "nq": 8, "k": 10, "api": "host", "rows": 64},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choices(["search", "build", "upsert"], [12, 2, 1])[0]
    dim = rng.choice(DIMS)
    bits = rng.choices([4, 2, 3], [3, 1, 1])[0]
    k = rng.choice([1, 10, 10, 100, _log_int(rng, 1, 200)])
    api = rng.choice(["host", "device"])
    if kind == "build":
        n = min(_log_int(rng, 1_000, 2_000_000), 2_000_000 * 1536 // dim)
        if api == "host":
            n = min(n, 20_000)
        return {"kind": kind, "n": n, "dim": dim, "bits": bits, "nq": _log_int(rng, 1, 64), "k": k, "api": api}
    if kind == "upsert":
        return {"kind": kind, "n": _log_int(rng, 5_000, 500_000), "dim": dim, "bits": bits, "nq": _log_int(rng, 1, 64), "k": k,
                "api": "host", "rows": _log_int(rng, 1, 256)}
    nq = _log_int(rng, 1, 1024)
    n = _log_int(rng, 2_000, 4_000_000)
    # no drawn batch costs more than the largest listed one: the u8-table families take about eight times the int8 form's
    # operations, and an id-mapped index is filled through host tables
    n = min(n, int(1e7 * 1024 * 1536 / (nq * dim * (1 if bits == 4 else 8))), int(6e9 / dim))
    filter = rng.choices(["none", "mask", "allow"], [4, 1, 1])[0]
    if filter == "allow":
        n, api = min(n, 1_000_000), "host"
    n = max(n, 1_000)
    allowed = 1.0 if filter == "none" else math.exp(rng.uniform(math.log(0.001), math.log(0.9)))
    c = _search("", n, dim, bits, nq, k, api, filter, round(allowed, 4))
    del c["name"]
    return c


# ---- inputs -------------------------------------------------------------------------------------------------------

def _rows(case, n, gen, scale):
    """L2-normalised rows with one spread per dimension, the distribution that embeddings have here."""
    x = torch.randn((n, case["dim"]), generator=gen, device="cuda") * scale
    x /= torch.linalg.vector_norm(x, dim=1, keepdim=True)
    return x


def _generator(seed, stream):
    g = torch.Generator(device="cuda")
    g.manual_seed((seed * 1_000_003 + stream * 7919) % (1 << 62))
    return g


def _filled(case, seed, scale, ids=None):
    """An index of case["n"] rows; `ids` makes it an id-mapped one."""
    idx = (tv.TurboQuantIndex if ids is None else tv.IdMapIndex)(case["dim"], case["bits"])
    gen = _generator(seed, 1)
    for lo in range(0, case["n"], CHUNK_ROWS):
        x = _rows(case, min(CHUNK_ROWS, case["n"] - lo), gen, scale)
        torch.cuda.current_stream().synchronize()              # the library works on streams of its own
        if ids is None:
            idx.add_device(x.data_ptr(), x.shape[0], x.shape[1])
        else:
            idx.add_with_ids_device(x.data_ptr(), x.shape[0], x.shape[1], ids[lo:lo + x.shape[0]])
    idx.prepare()
    return idx


def _ids(n, seed):
    """Distinct 64-bit ids in no order."""
    return (np.random.default_rng(seed).permutation(n).astype(np.uint64) + np.uint64(1)) * np.uint64(0x9E3779B97F4A7C15)


def _results(nq, width):
    return torch.empty((nq, width), dtype=torch.float32, device="cuda"), torch.empty((nq, width), dtype=torch.int64, device="cuda")


def prepare(case, seed):
    scale = torch.exp(0.5 * torch.randn(case["dim"], generator=_generator(seed, 0), device="cuda"))
    queries = _rows(case, case["nq"], _generator(seed, 2), scale)
    state = {"case": case, "queries": queries if case["api"] == "device" else queries.cpu().numpy()}
    rng = np.random.default_rng(seed)
    if case["kind"] == "build":
        rows = _rows(case, case["n"], _generator(seed, 1), scale)
        state["rows"] = rows if case["api"] == "device" else rows.cpu().numpy()
        if case["api"] == "device":
            state["out"] = _results(case["nq"], min(case["k"], case["n"]))
    elif case["kind"] == "upsert":
        ids = _ids(case["n"], seed)
        state["index"] = _filled(case, seed, scale, ids)
        state["ids"] = np.ascontiguousarray(rng.choice(ids, case["rows"], replace=False))
        state["rows"] = _rows(case, case["rows"], _generator(seed, 3), scale).cpu().numpy()
    elif case["filter"] == "allow":
        ids = _ids(case["n"], seed)
        state["index"] = _filled(case, seed, scale, ids)
        state["allow"] = np.ascontiguousarray(rng.choice(ids, _allowed(case), replace=False))
    else:
        state["index"] = _filled(case, seed, scale)
        width = min(case["k"], _allowed(case))
        if case["filter"] == "mask":
            mask = np.zeros(case["n"], np.bool_)
            mask[rng.choice(case["n"], _allowed(case), replace=False)] = True
            if case["api"] == "device":
                padded = np.zeros((case["n"] + 63) // 64 * 64, np.bool_)
                padded[:case["n"]] = mask
                state["mask"] = torch.from_numpy(np.packbits(padded, bitorder="little").view(np.int64).copy()).cuda()
            else:
                state["mask"] = mask
        if case["api"] == "device":
            state["out"] = _results(case["nq"], width)
    torch.cuda.current_stream().synchronize()
    return state


# ---- the path -----------------------------------------------------------------------------------------------------

def _search_device(index, state):
    q, (scores, slots), mask = state["queries"], state["out"], state.get("mask")
    index.search_device(q.data_ptr(), q.shape[0], state["case"]["k"], scores.data_ptr(), slots.data_ptr(),
                        0 if mask is None else mask.data_ptr())
    return scores, slots


def run(state):
    case = state["case"]
    if case["kind"] == "build":
        index = tv.TurboQuantIndex(case["dim"], case["bits"])
        if case["api"] == "device":
            rows = state["rows"]
            index.add_device(rows.data_ptr(), rows.shape[0], rows.shape[1])
            # a row's scale depends on its norm and on every one of its codes
            return _search_device(index, state), index.scales()
        index.add(state["rows"])
        # a small collection is kept as its parts as well
        return index.search(state["queries"], case["k"]), index.codes_blocked_seq(), index.scales()
    if case["kind"] == "upsert":
        index = state["index"]
        for i in state["ids"]:
            index.remove(i)
        index.add_with_ids(state["rows"], state["ids"])
        return index.search(state["queries"], case["k"])
    if case["filter"] == "allow":
        return state["index"].search(state["queries"], case["k"], allowlist=state["allow"])
    if case["api"] == "device":
        return _search_device(state["index"], state)
    return state["index"].search(state["queries"], case["k"], mask=state.get("mask"))


# ---- what it takes ------------------------------------------------------------------------------------------------

def _allowed(case):
    return max(1, int(round(case["n"] * case.get("allowed", 1.0))))


def _code_bytes(case):
    return case["dim"] // (8 // case["bits"])


def _live_rows(case):
    """Rows whose codes have to be read: those in 32-row blocks that hold an allowed row (expected number)."""
    a = case.get("allowed", 1.0)
    return case["n"] * (1.0 - (1.0 - a) ** 32) if a < 1.0 else float(case["n"])


def work(case):
    n, dim, nq, cb = case["n"], case["dim"], case["nq"], _code_bytes(case)
    b = _live_rows(case) * (cb + 4) + nq * (dim * 4 + min(case["k"], n) * 12)
    # one multiply-add for each coordinate, or two table values for each byte of the code
    f = 2.0 * _allowed(case) * nq * (dim if case["bits"] == 4 else cb)
    rows = n if case["kind"] == "build" else case.get("rows", 0)
    b += rows * (dim * 4 + cb + 4)
    if case["kind"] == "build":                                # what is exported
        b += 2 * rows * 4 if case["api"] == "device" else 2 * rows * (cb + 4)
    f += rows * 2.0 * dim * (math.log2(dim & -dim) + 4)        # two rounds of butterflies; norm, quantisation, inner product
    if case.get("filter") == "mask":
        b += n if case["api"] == "host" else n / 8
    elif case.get("filter") == "allow":
        b += _allowed(case) * 8
    return {"bytes": b, "flops": f}


def tolerance(case):
    # integer sums are exact and the few float operations are done in a stated order: scores and ids are the same bit for bit
    return "exact"

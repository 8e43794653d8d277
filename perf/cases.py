"""What the performance of this library is measured on.

The work is the Goldilocks polynomial commitment as a prover calls it: single
commits (small, ordinary, large), a batch of uneven commits, Merkle trees of
given leaves under the supported hashers, batched transforms in both
directions, the row LDE with its transpose, the drop-in C ABI with host
buffers, and the FRI commit phase.  Every value is a 64-bit field element,
digest word or permutation of such words, so results have to be equal bit for
bit; outputs are returned as int64 views of the uint64 buffers.
"""

import torch

import zeknox_b200 as zk
from zeknox_b200 import capi

P = 0xFFFFFFFF00000001
HASHES = {"poseidon": 0, "keccak": 1, "bn128": 2, "poseidon2": 3, "monolith": 4}


def listed():
    return [
        # The smallest commit: a short trace of a recursive proof.  Launches and latency count.
        {"name": "commit_small", "kind": "commit", "lg": 9, "polys": 12, "rate": 3, "cap": 4, "hash": "poseidon"},
        # The benchmark's commit: 135 wires of a 2^15-row circuit, rate 3.
        {"name": "commit_plain", "kind": "commit", "lg": 15, "polys": 135, "rate": 3, "cap": 4, "hash": "poseidon"},
        # A width that is no multiple of the sponge's rate, low blow-up, the other common hasher.
        {"name": "commit_poseidon2", "kind": "commit", "lg": 16, "polys": 77, "rate": 1, "cap": 4, "hash": "poseidon2"},
        # A long trace with few columns: three-pass transforms, wide trees, short leaves.
        {"name": "commit_large", "kind": "commit", "lg": 19, "polys": 40, "rate": 3, "cap": 4, "hash": "poseidon"},
        # Uneven jobs handed over together, as a proving service does.
        {"name": "commit_batch", "kind": "batch", "jobs": 12, "lg_lo": 12, "lg_hi": 15, "polys_hi": 200, "mix": 3},
        # The hash-only benchmark: a Poseidon tree of 8192 leaves of 135 words.
        {"name": "tree_small", "kind": "tree", "lg": 13, "width": 135, "cap": 4, "hash": "poseidon"},
        # The sweep over hashers on wide leaves, Keccak's part.
        {"name": "tree_keccak", "kind": "tree", "lg": 18, "width": 135, "cap": 4, "hash": "keccak"},
        # Leaves hashed for a BN254 verifier.
        {"name": "tree_bn128", "kind": "tree", "lg": 13, "width": 135, "cap": 4, "hash": "bn128"},
        # Witness values back to coefficients: the inverse transform in place, device buffers.
        {"name": "intt", "kind": "ntt", "lg": 15, "polys": 135, "inverse": True, "coset": False},
        # The LDE as rows and its transpose as two calls, for callers that keep both.
        {"name": "lde_transpose", "kind": "lde", "lg": 17, "polys": 64, "rate": 2},
        # The drop-in C ABI end to end: pinned host coefficients in, digests and cap back on the host.
        {"name": "dropin_host", "kind": "dropin", "lg": 15, "polys": 135, "rate": 3, "cap": 4, "hash": "poseidon"},
        # The FRI commit phase and its query openings: short dependent steps with a host round trip each.
        {"name": "fri", "kind": "fri", "lg": 15, "rate": 3, "arity": "4,4,4", "cap": 4, "queries": 28},
    ]


def _perms(width, hash_name):
    """Permutations of one leaf."""
    if hash_name == "keccak":
        return width // 17 + 1
    return 0 if width <= 4 else -(-width // 8)


# 32-bit multiply-adds (x 2 operations) of the products that a permutation cannot
# do without (S-boxes, diagonal layers); for Keccak its 32-bit logic operations.
_OPS = {"poseidon": 472 * 8, "poseidon2": 736 * 8, "monolith": 66 * 8, "bn128": 840 * 256, "keccak": 24 * 2 * 76}
# Seconds per permutation, roughly, to keep drawn cases no larger than the listed ones.
_COST = {"poseidon": 1e-9, "poseidon2": 1e-9, "monolith": 0.25e-9, "bn128": 42e-9, "keccak": 0.32e-9}


def _tree_work(n, width, cap, hash_name):
    perms = n * _perms(width, hash_name) + max(0, n - (1 << cap)) + (1 << cap)
    return {"bytes": 8 * n * width + 32 * (2 * n - (1 << cap)), "flops": perms * _OPS[hash_name], "perms": perms}


def _ntt_flops(lg, polys):
    return polys * (lg << (lg - 1)) * 8  # one 64 x 64 product per butterfly


def _batch_jobs(case):
    """(lg_n, rate, polys) of each job; the same for every seed."""
    x, jobs = case["mix"] * 2654435761 % 2**32, []
    for _ in range(case["jobs"]):
        v = []
        for _ in range(3):
            x = (1664525 * x + 1013904223) % 2**32
            v.append(x >> 8)
        jobs.append((case["lg_lo"] + v[0] % (case["lg_hi"] - case["lg_lo"] + 1), 1 + v[1] % 3, 4 + v[2] % (case["polys_hi"] - 3)))
    return jobs


def work(case):
    k = case["kind"]
    if k in ("commit", "dropin"):
        lg = case["lg"] + case["rate"]
        t = _tree_work(1 << lg, case["polys"], case["cap"], case["hash"])
        inputs = 8 * case["polys"] << case["lg"]
        return {"bytes": inputs + t["bytes"], "flops": t["flops"] + _ntt_flops(lg, case["polys"])}
    if k == "batch":
        b = f = 0
        for lg, rate, polys in _batch_jobs(case):
            t = _tree_work(1 << (lg + rate), polys, 4, "poseidon")
            b += (8 * polys << lg) + t["bytes"]
            f += t["flops"] + _ntt_flops(lg + rate, polys)
        return {"bytes": b, "flops": f}
    if k == "tree":
        t = _tree_work(1 << case["lg"], case["width"], case["cap"], case["hash"])
        return {"bytes": t["bytes"], "flops": t["flops"]}
    if k == "ntt":
        return {"bytes": 16 * case["polys"] << case["lg"], "flops": _ntt_flops(case["lg"], case["polys"])}
    if k == "lde":
        n, big = case["polys"] << case["lg"], case["polys"] << (case["lg"] + case["rate"])
        return {"bytes": 8 * (n + 2 * big), "flops": _ntt_flops(case["lg"] + case["rate"], case["polys"])}
    b = f = 0
    lg = case["lg"]
    for a in _arity(case):
        t = _tree_work(1 << (lg + case["rate"] - a), 2 << a, case["cap"], "poseidon")
        b += (16 << lg) + t["bytes"] + (16 << (lg - a))
        f += t["flops"] + _ntt_flops(lg + case["rate"], 2) + (32 << lg)
        lg -= a
    return {"bytes": b, "flops": f}


def _seconds(case):
    """A rough cost, only to bound the drawn cases."""
    k = case["kind"]
    if k == "batch":
        return sum((n := 1 << (lg + r)) * (_perms(p, "poseidon") + 1) * 1e-9 + n * p * 1.5e-11 for lg, r, p in _batch_jobs(case))
    if k in ("commit", "dropin"):
        n = 1 << (case["lg"] + case["rate"])
        return n * (_perms(case["polys"], case["hash"]) + 1) * _COST[case["hash"]] + n * case["polys"] * 2e-11
    if k == "tree":
        return (1 << case["lg"]) * (_perms(case["width"], case["hash"]) + 1) * _COST[case["hash"]]
    if k in ("ntt", "lde"):
        return (case["polys"] << (case["lg"] + case.get("rate", 0))) * 3e-11
    return 1e-3


def _log(rng, lo, hi):
    """A whole number in lo..hi, uniform in its logarithm."""
    return max(lo, min(hi, round(lo * (hi / lo) ** rng.random())))


def draw(rng):
    most = max(_seconds(c) for c in listed())
    while True:
        kind = rng.choice(["commit", "commit", "commit", "tree", "tree", "batch", "ntt", "lde", "dropin", "fri"])
        if kind in ("commit", "dropin"):
            # a dropped-in host buffer is not as large as a resident one
            case = {"kind": kind, "lg": rng.randint(6, 19 if kind == "commit" else 16), "polys": _log(rng, 2, 300), "rate": rng.randint(1, 3),
                    "cap": rng.randint(0, 5), "hash": rng.choice(["poseidon", "poseidon", "poseidon2", "keccak", "monolith"])}
        elif kind == "batch":
            lo = rng.randint(8, 13)
            case = {"kind": kind, "jobs": rng.randint(3, 20), "lg_lo": lo, "lg_hi": rng.randint(lo, 16), "polys_hi": rng.randint(20, 200),
                    "mix": rng.randint(1, 10**6)}
        elif kind == "tree":
            case = {"kind": kind, "lg": rng.randint(8, 20), "width": _log(rng, 3, 300), "cap": rng.randint(0, 5), "hash": rng.choice(sorted(HASHES))}
        elif kind == "ntt":
            case = {"kind": kind, "lg": rng.randint(6, 23), "polys": _log(rng, 1, 200), "inverse": rng.random() < 0.5, "coset": rng.random() < 0.5}
        elif kind == "lde":
            case = {"kind": kind, "lg": rng.randint(6, 20), "polys": _log(rng, 1, 200), "rate": rng.randint(1, 3)}
        else:
            arity = [rng.randint(1, 5) for _ in range(rng.randint(1, 3))]
            case = {"kind": kind, "lg": rng.randint(sum(arity) + 3, 18), "rate": rng.randint(1, 3), "arity": ",".join(map(str, arity)), "cap": rng.randint(0, 4),
                    "queries": rng.randint(1, 100)}
        if _seconds(case) <= most:
            return case


def _arity(case):
    return [int(a) for a in case["arity"].split(",")]


def _field(shape, seed):
    """Field elements uniform in [0, p)."""
    return zk.fill_field(torch.empty(shape, dtype=torch.uint64, device="cuda"), seed * 0x9E3779B97F4A7C15 + 1)


def prepare(case, seed):
    k = case["kind"]
    s = {"case": case}
    if k in ("commit", "dropin"):
        lg, n = case["lg"], case["polys"]
        s["coeffs"] = _field((n, 1 << lg), seed)
        if k == "commit":
            s["out"] = zk.CommitBuffers(1 << (lg + case["rate"]), n, case["cap"])
            for t in (s["out"].digests, s["out"].cap):  # a Keccak digest of fewer than 4 words keeps what was there
                t.view(torch.int64).zero_()
        else:
            big = 1 << (lg + case["rate"])
            nd, nc = zk.merkle_sizes(big, case["cap"])
            dev = lambda *shape: torch.empty(shape, dtype=torch.uint64, device="cuda")  # noqa: E731
            s["host_in"] = torch.empty((n, 1 << lg), dtype=torch.int64, pin_memory=True)
            s["host_in"].copy_(s.pop("coeffs").view(torch.int64))
            s["lde"], s["leaves"], s["digests"], s["cap"] = dev(n, big), dev(big, n), dev(max(nd, 1), 4), dev(nc, 4)
            s["host_digests"] = torch.empty((max(nd, 1), 4), dtype=torch.int64, pin_memory=True)
            s["host_cap"] = torch.empty((nc, 4), dtype=torch.int64, pin_memory=True)
            for t in (s["digests"], s["cap"]):
                t.view(torch.int64).zero_()
    elif k == "batch":
        s["items"] = []
        for j, (lg, rate, polys) in enumerate(_batch_jobs(case)):
            s["items"].append((_field((polys, 1 << lg), seed * 1009 + j), rate, 4, HASHES["poseidon"], zk.CommitBuffers(1 << (lg + rate), polys, 4)))
    elif k == "tree":
        n = 1 << case["lg"]
        nd, nc = zk.merkle_sizes(n, case["cap"])
        s["leaves"] = _field((n, case["width"]), seed)
        s["digests"] = torch.zeros((max(nd, 1), 4), dtype=torch.int64, device="cuda").view(torch.uint64)
        s["cap"] = torch.zeros((nc, 4), dtype=torch.int64, device="cuda").view(torch.uint64)
    elif k == "ntt":
        s["values"] = _field((case["polys"], 1 << case["lg"]), seed)
        s["work"] = torch.empty_like(s["values"])
    elif k == "lde":
        n, big = case["polys"], 1 << (case["lg"] + case["rate"])
        s["coeffs"] = _field((n, 1 << case["lg"]), seed)
        s["rows"] = torch.empty((n, big), dtype=torch.uint64, device="cuda")
        s["leaves"] = torch.empty((big, n), dtype=torch.uint64, device="cuda")
    else:
        s["coeffs"] = _field((2, 1 << case["lg"]), seed)
        big = 1 << (case["lg"] + case["rate"])
        g = torch.Generator().manual_seed(seed)
        s["queries"] = torch.randint(0, big, (case["queries"],), generator=g)
    return s


def _i64(*tensors):
    return [t.view(torch.int64) for t in tensors]


def _challenge(i, cap):
    """Stands for the transcript: two words of the round's cap."""
    words = cap.reshape(-1)
    return int(words[0]) % P, int(words[(i + 1) % words.size]) % P


def run(s):
    case = s["case"]
    k = case["kind"]
    if k == "commit":
        o = zk.commit(s["coeffs"], case["rate"], case["cap"], HASHES[case["hash"]], out=s["out"])
        return _i64(o.leaves, o.digests, o.cap)
    if k == "batch":
        zk.commit_batch(s["items"])
        return [t for item in s["items"] for t in _i64(item[4].leaves, item[4].digests, item[4].cap)]
    if k == "tree":
        return _i64(*zk.merkle_tree(s["leaves"], case["cap"], HASHES[case["hash"]], digests=s["digests"], cap=s["cap"]))
    if k == "ntt":
        # in place, on a copy: the program keeps its values
        s["work"].copy_(s["values"])
        cfg = capi.NTTConfig.default()
        cfg.batches, cfg.are_inputs_on_device, cfg.are_outputs_on_device, cfg.with_coset = case["polys"], True, True, case["coset"]
        (zk.intt_batch if case["inverse"] else zk.ntt_batch)(0, s["work"].data_ptr(), case["lg"], cfg)
        return _i64(s["work"])
    if k == "lde":
        zk.lde(s["coeffs"], case["rate"], out=s["rows"])
        zk.transpose_rev(s["rows"], out=s["leaves"])
        return _i64(s["rows"], s["leaves"])
    if k == "dropin":
        lg, lg_big, n = case["lg"], case["lg"] + case["rate"], case["polys"]
        cfg = capi.NTTConfig.default()
        cfg.batches, cfg.extension_rate_bits, cfg.are_outputs_on_device, cfg.with_coset = n, case["rate"], True, True
        zk.lde_batch(0, s["lde"].data_ptr(), s["host_in"].data_ptr(), lg, cfg)
        t = capi.TransposeConfig.default()
        t.batches, t.are_inputs_on_device, t.are_outputs_on_device = n, True, True
        zk.transpose_rev_batch(0, s["leaves"].data_ptr(), s["lde"].data_ptr(), lg_big, t)
        nd, nc = zk.merkle_sizes(1 << lg_big, case["cap"])
        zk.fill_digests_buf_linear_gpu_with_gpu_ptr(s["digests"].data_ptr(), s["cap"].data_ptr(), s["leaves"].data_ptr(), nd, nc, 1 << lg_big, n, case["cap"],
                                                    HASHES[case["hash"]])
        s["host_digests"].copy_(s["digests"].view(torch.int64), non_blocking=True)
        s["host_cap"].copy_(s["cap"].view(torch.int64), non_blocking=True)
        torch.cuda.current_stream().synchronize()
        return [s["lde"].view(torch.int64), s["leaves"].view(torch.int64), s["host_digests"], s["host_cap"]]
    c = zk.fri_commit(s["coeffs"], case["rate"], _arity(case), case["cap"], _challenge)
    outs = _i64(c.final_poly)
    for r in c.rounds:
        outs += _i64(r.leaves, r.digests, r.cap)
    for rows, siblings in zk.fri_open(c, s["queries"]):
        outs += _i64(rows, siblings)
    return outs


def tolerance(case):
    return "exact"

"""Workloads of the Basefold prover, sized as its users run it.

Every case goes through the package's public entry points: commit, evaluate
and open one polynomial or a matrix of them over either field, from device or
host memory, with the library's transcript or the caller's own; the standalone
product sumcheck; a batch of jobs on the engine; a batch of proofs verified.

`listed()` are the fixed cases, `draw(rng)` gives others of the same ranges,
`prepare(case, seed)` makes a case's inputs and handles, `run(state)` is one
pass and `work(case)` counts what a pass cannot do without.  All outputs are
bytes (roots, field values, proofs, transcript states): there is no rounding,
so `exact` has no value to give.
"""
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "learn-zkp_gb300"))

import basefold_gpu as bg  # noqa: E402
from basefold_gpu import prime  # noqa: E402

LAMBDA = 128  # security parameter of the tests and the benchmark


def listed():
    return [
        # one small polynomial: launches, dependent hashes and round trips
        {"name": "prove_2p10", "kind": "prove", "n": 10, "log2_c": 1, "input": "device", "open": "library"},
        # the plain configuration: 2^16 evaluations, blowup 2
        {"name": "prove_2p16", "kind": "prove", "n": 16, "log2_c": 1, "input": "device", "open": "library"},
        # the trait's route at blowup 4: evaluations in host memory, and an
        # open whose every round waits for the caller's own transcript
        {"name": "trait_2p20_c4", "kind": "prove", "n": 20, "log2_c": 2, "input": "host", "open": "caller"},
        # the largest single polynomial of the benchmark
        {"name": "prove_2p24", "kind": "prove", "n": 24, "log2_c": 1, "input": "device", "open": "library"},
        # the reference's own benchmark shape: 256 binary-field columns
        {"name": "matrix_2p16x256", "kind": "matrix", "n": 16, "width": 256, "log2_c": 1},
        # the same shape over BabyBear, Reed-Solomon code, its largest size
        {"name": "prime_2p19x256", "kind": "prime", "n": 19, "width": 256, "log2_c": 1, "log2_k0": -1},
        # a few short BabyBear columns: an odd, narrow matrix
        {"name": "prime_2p13x5", "kind": "prime", "n": 13, "width": 5, "log2_c": 1, "log2_k0": -1},
        # the random foldable code at the benchmark's smallest shape
        {"name": "generic_2p16x256", "kind": "prime", "n": 16, "width": 256, "log2_c": 1, "log2_k0": 3},
        # the sumcheck prover alone: product of two and of three polynomials
        {"name": "sumcheck2_2p20", "kind": "sumcheck", "n": 20, "k": 2},
        {"name": "sumcheck3_2p24", "kind": "sumcheck", "n": 24, "k": 3},
        # many proofs of one size checked at once
        {"name": "verify_64x2p14", "kind": "verify", "n": 14, "log2_c": 1, "count": 64},
        # independent proofs of mixed sizes in flight together
        {"name": "engine_32_mixed", "kind": "engine", "lo": 10, "hi": 18, "count": 32},
    ]


def draw(rng):
    kind = rng.choice(["prove", "prove", "matrix", "matrix", "prime", "prime", "sumcheck", "verify", "engine"])
    if kind == "prove":
        return {"kind": kind, "n": rng.randint(8, 22), "log2_c": rng.choice([1, 1, 2]),
                "input": rng.choice(["device", "host"]), "open": rng.choice(["library", "library", "caller"])}
    if kind == "matrix":
        n = rng.randint(5, 17)
        width = max(2, int(2 ** rng.uniform(1, min(8.3, 24 - n))))
        return {"kind": kind, "n": n, "width": width, "log2_c": rng.choice([1, 1, 2])}
    if kind == "prime":
        n, k0 = rng.randint(6, 19), rng.choice([-1, -1, 0, 1, 2, 3, 4])
        if k0 >= 0:
            n = min(n, 17)
        width = max(1, int(2 ** rng.uniform(0, min(8.3, 26 - n))))
        return {"kind": kind, "n": n, "width": width, "log2_c": rng.choice([1, 1, 2]), "log2_k0": k0}
    if kind == "sumcheck":
        return {"kind": kind, "n": rng.randint(8, 23), "k": rng.choice([2, 3])}
    if kind == "verify":
        return {"kind": kind, "n": rng.randint(8, 17), "log2_c": 1, "count": int(2 ** rng.uniform(1, 6.5))}
    return {"kind": kind, "lo": rng.randint(8, 11), "hi": rng.randint(13, 18), "count": int(2 ** rng.uniform(2, 5.3))}


def _device_elems(n, seed):
    """n uniform field elements of GF(2^128) in device memory."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    lo = -(1 << 63)
    return torch.randint(lo, -(lo + 1), (n, 2), dtype=torch.int64, device="cuda", generator=g)


def _host_elems(n, seed):
    return np.random.default_rng([seed, 7]).integers(0, 256, (n, 16), dtype=np.uint8)


def _pcs(n, log2_c):
    return bg.Basefold.setup(bg.BasefoldConfig(bg.BinaryReedSolomonCode(LAMBDA, log2_c, n)), device=0)


def _job_sizes(case):
    """The engine's mix: sizes lo..hi, as many of each as fit, in a fixed shuffled order."""
    span = case["hi"] - case["lo"] + 1
    sizes = [case["lo"] + i % span for i in range(case["count"])]
    order = np.random.default_rng(case["count"]).permutation(case["count"])
    return [sizes[i] for i in order]


def prepare(case, seed):
    kind = case["kind"]
    st = {"kind": kind, "case": case}
    if kind in ("prove", "matrix"):
        n, width = case["n"], case.get("width", 1)
        st["pcs"], st["width"] = _pcs(n, case["log2_c"]), width
        data = _device_elems(width << n, seed)
        st["point"] = _host_elems(n, seed)
        if case.get("input") == "host":  # pinned, as a service keeps its request buffers
            pinned = torch.empty(data.shape, dtype=data.dtype, pin_memory=True)
            pinned.copy_(data)
            st["pinned"], st["data"] = pinned, pinned.numpy().view(np.uint8).reshape(-1, 16)
        else:
            st["data"] = data
    elif kind == "prime":
        n, width, k0 = case["n"], case["width"], case["log2_k0"]
        rng = np.random.default_rng([seed, 9])
        if k0 < 0:
            code = prime.ReedSolomonCode(LAMBDA, case["log2_c"], n)
        else:
            n0 = 1 << (case["log2_c"] + k0)
            ts = rng.integers(1, prime.P, n0 * ((1 << (n - k0)) - 1), dtype=np.uint32)
            code = prime.GenericRandomFoldableCode(LAMBDA, case["log2_c"], k0, n - k0, ts)
        st["pcs"] = prime.BabyBearBasefold.setup(bg.BasefoldConfig(code), device=0)
        st["width"] = width
        g = torch.Generator(device="cuda").manual_seed(seed)
        st["data"] = torch.randint(0, prime.P, (1 << n, width), dtype=torch.int32, device="cuda", generator=g)
        st["point"] = rng.integers(0, prime.P, (n, 5), dtype=np.uint32)
    elif kind == "sumcheck":
        st["pcs"] = _pcs(1, 1)  # the handle a device-resident sumcheck runs on
        st["data"] = _device_elems(case["k"] << case["n"], seed)
        st["claim"] = _host_elems(1, seed)
    elif kind == "verify":
        n, count = case["n"], case["count"]
        st["pcs"] = _pcs(n, case["log2_c"])
        st["items"] = []
        for i in range(count):
            data, point = _device_elems(1 << n, seed * 1000 + i), _host_elems(n, seed * 1000 + i)
            torch.cuda.synchronize()
            comm = st["pcs"].commit_device(data.data_ptr(), 1, keep=data)
            ch = bg.GenericChallenger.keccak256()
            ch.observe(comm.root)
            values = st["pcs"].eval(comm, point)
            ch.observe_ext_slice(values)
            evals = [bg.PolyEvals(values, point)]
            proof = st["pcs"].open(comm, evals, ch.clone())
            if i == count // 2:  # one proof of the batch does not verify
                bad = bytearray(proof)
                bad[-20] ^= 1
                proof = bytes(bad)
            st["items"].append((comm.root, evals, proof, ch))
    else:
        st["engine"] = bg.Engine(device=0, lambda_=LAMBDA, log2_c=1, max_inflight=32)
        st["keep"], st["jobs"] = [], []
        for i, n in enumerate(_job_sizes(case)):
            data = _device_elems(1 << n, seed * 1000 + i)
            st["keep"].append(data)
            st["jobs"].append((n, data.data_ptr(), _host_elems(n, seed * 1000 + i)))
    torch.cuda.synchronize()  # the library runs on streams of its own
    return st


def _bytes(b):
    return np.frombuffer(b, dtype=np.uint8)


def _prove(st):
    pcs, case = st["pcs"], st["case"]
    if case.get("input") == "host":
        comm = pcs.commit(st["data"], width=st["width"])
    else:
        comm = pcs.commit_device(st["data"].data_ptr(), st["width"], keep=st["data"])
    ch = bg.GenericChallenger.keccak256()
    ch.observe(comm.root)
    values = pcs.eval(pcs.data(comm), st["point"])
    ch.observe_ext_slice(values)
    evals = bg.PolyEvals(values, st["point"])
    if case.get("open") == "caller":
        proof = pcs.open_session(comm, evals).prove(ch)
    else:
        proof = pcs.open(comm, [evals], ch)
    return {"root": _bytes(comm.root), "values": values, "proof": _bytes(proof), "transcript": _bytes(ch.state())}


def _prove_prime(st):
    pcs = st["pcs"]
    comm = pcs.commit_device(st["data"].data_ptr(), st["width"], keep=st["data"])
    ch = bg.GenericChallenger.keccak256()
    ch.observe(comm.root)
    values = pcs.eval(comm, st["point"])
    prime.observe_ext_slice(ch, values)
    proof = pcs.open(comm, [prime.PrimePolyEvals(values, st["point"])], ch)
    return {"root": _bytes(comm.root), "values": values.view(np.int32), "proof": _bytes(proof),
            "transcript": _bytes(ch.state())}


def run(state):
    kind, case = state["kind"], state["case"]
    if kind in ("prove", "matrix"):
        return _prove(state)
    if kind == "prime":
        return _prove_prime(state)
    if kind == "sumcheck":
        ch = bg.GenericChallenger.keccak256()
        polys, point, finals, claim = state["pcs"].prove_sumcheck_device(case["k"], case["n"], state["data"].data_ptr(),
                                                                        state["claim"], ch)
        return {"polys": polys, "point": point, "finals": finals, "claim": claim, "transcript": _bytes(ch.state())}
    if kind == "verify":
        items = [(root, evals, proof, ch.clone()) for root, evals, proof, ch in state["items"]]
        codes = state["pcs"].verify_batch(items)
        return {"codes": np.array(codes, dtype=np.int64),
                "transcripts": _bytes(b"".join(ch.state() for _, _, _, ch in items))}
    results = state["engine"].prove(state["jobs"], device_input=True)
    return {"roots": _bytes(b"".join(r["root"] for r in results)),
            "values": np.concatenate([r["value"] for r in results]),
            "proofs": _bytes(b"".join(r["proof"] for r in results))}


# 32-bit integer operations: a Keccak-f[1600] permutation (24 rounds of 75
# theta, 48 rho and 50 chi operations on 32-bit halves), a product in
# GF(2^128) (nine 32 x 32 carry-less products and the reduction), a BabyBear
# butterfly and multiply-add.
_KECCAK, _GF, _BB_BFLY, _BB_MAC = 24 * 173, 420, 9, 3


def _queries(log2_c):
    return int(np.ceil(LAMBDA / -np.log2((1 + 1 / (1 << log2_c)) / 2)))


def _binary_work(n, width, log2_c):
    N, c = 1 << n, 1 << log2_c
    rows = N * c
    blocks = 16 * width // 136 + 1  # permutations of a row's leaf
    perms = rows * (blocks + 1) + 2 * rows
    mults = c * n // 2 * N * width + (2 * c + 3) * N + (2 * N * width if width > 1 else 0)
    # evaluations read, codeword and tree written, folded codewords and their
    # trees written; the fold and the sumcheck read what they fold
    data = 16 * N * width * (1 + c) + 64 * rows + (112 * c + 72) * N
    proof = _queries(log2_c) * (16 * width + 32 * (n + log2_c) + 16 * n * (n + 1))
    return {"bytes": data + proof, "flops": perms * _KECCAK + mults * _GF}


def work(case):
    kind = case["kind"]
    if kind in ("prove", "matrix"):
        return _binary_work(case["n"], case.get("width", 1), case["log2_c"])
    if kind == "prime":
        n, w, c = case["n"], case["width"], 1 << case["log2_c"]
        N = 1 << n
        rows = N * c
        perms = rows * (4 * w // 136 + 2) + 2 * rows
        layers = n + case["log2_c"]
        ops = perms * _KECCAK + rows * w * layers // 2 * _BB_BFLY + 2 * 5 * N * w * _BB_MAC
        return {"bytes": 4 * N * w * (1 + c) + 64 * rows + 20 * 6 * rows, "flops": ops}
    if kind == "sumcheck":
        N, k = 1 << case["n"], case["k"]
        # the input read once, each fixed half written and read once
        return {"bytes": 16 * N * k * 3, "flops": (4 if k == 2 else 10) * N * _GF}
    if kind == "verify":
        n, q = case["n"], _queries(case["log2_c"])
        L = n + case["log2_c"]
        perms = case["count"] * q * (L + 1 + sum(case["log2_c"] + i + 1 for i in range(n)))
        size = case["count"] * q * (16 + 32 * L + sum(24 + 32 * (case["log2_c"] + i) for i in range(n)))
        return {"bytes": size, "flops": perms * _KECCAK + case["count"] * q * 2 * n * _GF}
    parts = [_binary_work(n, 1, 1) for n in _job_sizes(case)]
    return {"bytes": sum(p["bytes"] for p in parts), "flops": sum(p["flops"] for p in parts)}

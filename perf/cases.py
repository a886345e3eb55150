"""The work that users of this prover have it do, as cases to be timed.

Each case goes through the public entry points (the Python API over the C ABI
of include/virgo_b200.h) as a program using them would: contexts, commitment
states, sessions and circuits are made once and kept, every pass is one
complete call.  A case is a dict of plain values; `kind` says which path:

  mle     vg_mle_eval: the multilinear extension of a table at a point (the
          value a verifier or an application asks for)
  ntt     vg_ntt: batched transforms, forward (Reed-Solomon encoding, zero
          padded) or inverse (interpolation)
  leaves  vg_leaf_chain + vg_merkle_tree: the Merkle commitment of one
          codeword set, as an opening or a single FRI level needs it
  tree    vg_merkle_tree over leaves that are there already, any number
  commit  vg_pc_commit_all: one polynomial commitment with its FRI phase and
          query answers, from host arrays (a caller with its data in memory)
          or from device arrays (a caller whose data the GPU made)
  prove   a whole proof of a resident circuit for a new witness
          (Session.set_inputs from pinned memory, Session.prove, transcript)
  batch   several such proofs in flight at once (prove_batch)
  job     a whole circuit loaded from host arrays and proven
          (Session.load + Session.prove), what a proof server does per job

All outputs are whole numbers or bytes: field elements of F_p2, digests and
transcripts, equal bit for bit whatever the implementation.
"""
import ctypes
import hashlib

import numpy as np
import torch

import virgo_b200 as vb
from virgo_b200 import circuits, sha256_circuit

P = vb.P
HASHES = {"sha3": 0, "sha256": 1}
MASK = 300   # private mask entries, as the prover's own proofs and the benchmark use

# 32-bit integer operations of one F_p2 product (three 61-bit products of four
# 32x32 multiplies each, their reductions mod 2^61 - 1 and the sums), of one
# F_p2 addition, of one Keccak-f[1600] (24 rounds of 180 on 32-bit halves,
# the last one cut to the digest) and of SHA-256 over one 64-byte message
MUL_OPS, ADD_OPS, KECCAK_OPS, SHA256_OPS = 60, 8, 4200, 3000


def listed():
    return [
        # smallest call: one evaluation of a 2^10-entry table, all latency
        {"name": "mle_2e10", "kind": "mle", "log_n": 10, "host": False},
        # the encoding step of the headline commitment: 65 slices of 2^16 from 2^11 coefficients
        {"name": "ntt_encode_65x2e16", "kind": "ntt", "log_n": 16, "batch": 65, "in_len": 2048, "inverse": False},
        # one large interpolation, beyond the full twiddle tables
        {"name": "ntt_inverse_2e22", "kind": "ntt", "log_n": 22, "batch": 1, "in_len": 1 << 22, "inverse": True},
        # a small FRI level's commitment: 2048 chains, few enough to leave the GPU idle
        {"name": "leaves_65x2e12", "kind": "leaves", "n": 4096, "slices": 65, "hash": "sha3"},
        # ragged number of leaves, the SHA-256 build of the reference
        {"name": "tree_70001_sha256", "kind": "tree", "n": 70001, "hash": "sha256"},
        # the commitment of a small circuit (at most three file layers pad to 2^15), data on the device
        {"name": "commit_2e15_device", "kind": "commit", "log_len": 15, "host": False, "hash": "sha3"},
        # the commitment path as benchmarked: 2^20 values from host memory
        {"name": "commit_2e20_host", "kind": "commit", "log_len": 20, "host": True, "hash": "sha3"},
        # a small circuit, one proof at a time: latency of a whole proof
        {"name": "prove_matmul16", "kind": "prove", "circuit": "matmul", "size": 16, "depth": 0, "bits": 16},
        # the headline workload: 256x256 matmul, 2^24 product gates, one proof at a time
        {"name": "prove_matmul256", "kind": "prove", "circuit": "matmul", "size": 256, "depth": 0, "bits": 32},
        # the same in flight: throughput of a proving service
        {"name": "batch8_matmul256", "kind": "batch", "circuit": "matmul", "size": 256, "depth": 0, "bits": 32, "copies": 8},
        # server jobs: random wiring (scattered gathers), and a ragged SHA-256 circuit with summation gates
        {"name": "job_random_2e22", "kind": "job", "circuit": "random", "size": 22, "depth": 16, "bits": 31},
        {"name": "job_sha256_4", "kind": "job", "circuit": "sha256", "size": 4, "depth": 0, "bits": 1},
    ]


def _log_uniform(rng, lo, hi):
    return max(lo, min(hi, int(round(2 ** rng.uniform(np.log2(lo), np.log2(hi))))))


def draw(rng):
    kind = rng.choice(["mle", "ntt", "leaves", "tree", "commit", "prove", "batch", "job"])
    if kind == "mle":
        host = rng.random() < 0.3
        return {"kind": kind, "log_n": rng.randint(2, 20 if host else 24), "host": host}
    if kind == "ntt":
        log_n = rng.randint(1, 22)
        batch = _log_uniform(rng, 1, max(1, min(4096, 1 << (22 - log_n))))
        inverse = rng.random() < 0.4
        in_len = (1 << log_n) if inverse or rng.random() < 0.3 else _log_uniform(rng, 1, 1 << log_n)
        return {"kind": kind, "log_n": log_n, "batch": batch, "in_len": in_len, "inverse": inverse}
    if kind == "leaves":
        return {"kind": kind, "n": 1 << rng.randint(3, 18), "slices": rng.choice([65, 65, 65, rng.randint(1, 64)]),
                "hash": rng.choice(["sha3", "sha3", "sha256"])}
    if kind == "tree":
        return {"kind": kind, "n": _log_uniform(rng, 3, 1 << 20), "hash": rng.choice(["sha3", "sha256"])}
    if kind == "commit":
        return {"kind": kind, "log_len": rng.randint(11, 21), "host": rng.random() < 0.5,
                "hash": rng.choice(["sha3", "sha3", "sha256"])}
    which = rng.choice(["matmul", "random", "random", "sha256"])
    if which == "matmul":
        c = {"circuit": which, "size": 1 << rng.randint(1, 8 if kind == "prove" else 7), "depth": 0,
             "bits": rng.randint(8, 32)}
    elif which == "random":
        c = {"circuit": which, "size": rng.randint(12, 22 if kind != "batch" else 20), "depth": rng.randint(8, 32),
             "bits": 31}
    else:
        c = {"circuit": which, "size": rng.randint(1, 12), "depth": 0, "bits": 1}
    if kind == "batch":
        c["copies"] = rng.randint(2, 8)
    return {"kind": kind, **c}


# ------------------------------------------------------------------- inputs
def _field(n, seed, device="cuda"):
    """n uniform field elements, (n, 2) int64 holding (img, real)."""
    g = torch.Generator(device=device)
    g.manual_seed(seed)
    return torch.randint(0, P, (n, 2), dtype=torch.int64, device=device, generator=g)


def _bytes(n, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return torch.randint(0, 256, (n, 32), dtype=torch.uint8, device="cuda", generator=g)


def _host_field(n, seed):
    return np.random.default_rng(seed).integers(0, P, (n, 2), dtype=np.int64)


def _layers(case, seed):
    if case["circuit"] == "matmul":
        return circuits.matmul_addtree(case["size"], case["bits"], seed)
    if case["circuit"] == "random":
        return circuits.random_by_gates(case["size"], case["depth"], seed)
    return sha256_circuit.sha256_blocks(case["size"], seed)


def _input_values(case, seed):
    """A new witness for the case's circuit: the values of its input layer."""
    rng = np.random.default_rng(seed)
    if case["circuit"] == "matmul":
        return rng.integers(0, 1 << case["bits"], 2 * case["size"] ** 2, dtype=np.int64)
    if case["circuit"] == "random":
        return rng.integers(0, 1 << case["bits"], len(_layers(case, 1)[0][0]), dtype=np.int64)
    return _layers(case, seed)[0][1]


def _index32(layers):
    """The layers as a loader holds them: wires of layers >= 1 as uint32."""
    return [(t, u if i == 0 else u.astype(np.uint32), v if i == 0 else v.astype(np.uint32))
            for i, (t, u, v) in enumerate(layers)]


def _root(log_n, inverse):
    """A root of unity of order 2^log_n in F_p2 (the reference's generator of
    the 2-adic subgroup of order 2^62, squared down), as (img, real)."""
    re, im = 2147483648, 1033321771269002680
    for _ in range(62 - log_n):
        re, im = (re * re - im * im) % P, 2 * re * im % P
    return (-im % P, re) if inverse else (im, re)   # norm 1: the inverse is the conjugate


# ------------------------------------------------------------------- states
class _State:
    """What a program keeps between calls; released with the last reference."""

    def __init__(self, case):
        self.case, self._close = case, []

    def owns(self, close):
        self._close.append(close)

    def __del__(self):
        for close in reversed(self._close):
            close()


_bases = {}


def _base_session(case):
    """The session that loaded the circuit; programs proving it for many
    witnesses fork it.  One circuit is kept at a time."""
    key = (case["circuit"], case["size"], case["depth"], case["bits"])
    if key not in _bases:
        for s in _bases.values():
            s.close()
        _bases.clear()
        s = vb.Session(_layers(case, 1))
        _bases[key] = s
    return _bases[key]


def _fork(state, case, seed):
    s = _base_session(case).fork()
    state.owns(s.close)
    return s, torch.from_numpy(_input_values(case, seed)).pin_memory()


def prepare(case, seed):
    st = _State(case)
    kind = case["kind"]
    if kind in ("prove", "batch"):
        pairs = [_fork(st, case, 16 * seed + k) for k in range(case.get("copies", 1))]
        st.sessions, st.values = [p[0] for p in pairs], [p[1] for p in pairs]
        st.seeds = [(seed * 1000003 + k) % (1 << 31) + 1 for k in range(len(pairs))]
        return st
    if kind == "job":
        h = ctypes.c_void_p()
        vb.check(vb.lib().vg_session_new(ctypes.byref(h)), "vg_session_new")
        st.session = vb.Session.__new__(vb.Session)
        st.session.h = h
        st.owns(st.session.close)
        st.layers = _index32(_layers(case, seed))
        st.seed = (seed * 1000003) % (1 << 31) + 1
        return st
    ctx = st.ctx = vb.Context(0, HASHES[case.get("hash", "sha3")])
    st.owns(ctx.close)
    if kind == "mle":
        n = 1 << case["log_n"]
        st.vals = _host_field(n, seed) if case["host"] else _field(n, seed)
        st.r = _host_field(case["log_n"], seed + 1)
        st.out = np.zeros((1, 2), np.int64)
    elif kind == "ntt":
        n = 1 << case["log_n"]
        st.inp = _field(case["batch"] * case["in_len"], seed)
        st.out = torch.empty((case["batch"] * n, 2), dtype=torch.int64, device="cuda")
        st.root = vb.to_fe(_root(case["log_n"], case["inverse"]))
    elif kind == "leaves":
        st.cw = _field(case["slices"] * case["n"], seed)
        st.leaves = torch.empty((case["n"] // 2, 32), dtype=torch.uint8, device="cuda")
        st.tree = torch.empty((case["n"], 32), dtype=torch.uint8, device="cuda")
    elif kind == "tree":
        st.leaves = _bytes(case["n"], seed)
        st.tree = torch.empty((2 << (case["n"] - 1).bit_length(), 32), dtype=torch.uint8, device="cuda")
    elif kind == "commit":
        _prepare_commit(st, case, seed)
    torch.cuda.synchronize()
    return st


def _commit_sizes(case):
    log_len = case["log_len"]
    S, levels = 1 << (log_len - 1), log_len - 6
    gap = 1
    while gap * 2 <= S // MASK:
        gap *= 2
    return S, levels, S // gap


def _prepare_commit(st, case, seed):
    log_len = case["log_len"]
    n = 1 << log_len
    S, levels, M = _commit_sizes(case)
    st.pc = ctypes.c_void_p()
    vb.check(vb.lib().vg_pc_create(st.ctx.h, ctypes.byref(st.pc)), "vg_pc_create")
    st.owns(lambda pc=st.pc: vb.lib().vg_pc_destroy(pc))
    made = _host_field if case["host"] else _field
    st.priv, st.pub = made(n, seed), made(n, seed + 1)
    st.mask, st.pub_mask, st.fri_r = (_host_field(k, seed + 2 + i) for i, k in enumerate((MASK, M, levels)))
    st.levels, st.M = levels, M
    # one query of each committed oracle and of each FRI level
    st.which = np.array([0, 1] + [2 + t for t in range(levels)], np.int32)
    half = np.array([S // 2, S // 2] + [max(1, (S >> (t + 1)) // 2) for t in range(levels)], np.int64)
    st.pos = (np.random.default_rng(seed).integers(0, 1 << 62, len(half)) % half).astype(np.int64)
    nq = len(st.which)
    st.out = {"roots": np.zeros((2 + levels, 32), np.uint8), "all_sum": np.zeros((65, 2), np.int64),
              "inner": np.zeros(2, np.int64), "final": np.zeros((65 * (S >> levels), 2), np.int64),
              "values": np.zeros((nq * 130, 2), np.int64), "paths": np.zeros((nq * 32, 32), np.uint8)}
    # path digests beyond a query's own depth are not part of the answer
    depth = np.array([log_len - 2, log_len - 2] + [log_len - 3 - t for t in range(levels)])
    st.path_rows = np.concatenate([32 * q + np.arange(d + 1) for q, d in enumerate(depth)])


def _addr(x):
    return ctypes.c_void_p(x.data_ptr() if isinstance(x, torch.Tensor) else x.ctypes.data)


# --------------------------------------------------------------------- run
def run(st):
    case, kind = st.case, st.case["kind"]
    if kind == "prove":
        st.sessions[0].set_inputs(st.values[0])
        _, transcript = st.sessions[0].prove(st.seeds[0])
        return np.frombuffer(transcript, np.uint8)
    if kind == "batch":
        for s, v in zip(st.sessions, st.values):
            s.set_inputs(v)
        return [np.frombuffer(t, np.uint8) for _, t in vb.prove_batch(st.sessions, st.seeds)]
    if kind == "job":
        st.session.load(st.layers, index_bytes=4)
        _, transcript = st.session.prove(st.seed)
        return np.frombuffer(transcript, np.uint8)
    L, ctx = vb.lib(), st.ctx
    if kind == "mle":
        vb.check(L.vg_mle_eval(ctx.h, _addr(st.vals), len(st.vals), _addr(st.r), case["log_n"], _addr(st.out)),
                 "vg_mle_eval")
        return st.out
    if kind == "ntt":
        vb.check(L.vg_ntt(ctx.h, _addr(st.inp), case["in_len"], case["in_len"], _addr(st.out), case["log_n"],
                          1 << case["log_n"], case["batch"], st.root, 1 if case["inverse"] else 0), "vg_ntt")
        return st.out
    if kind == "leaves":
        vb.check(L.vg_leaf_chain(ctx.h, _addr(st.cw), case["slices"], case["n"], _addr(st.leaves)), "vg_leaf_chain")
        vb.check(L.vg_merkle_tree(ctx.h, _addr(st.leaves), case["n"] // 2, _addr(st.tree)), "vg_merkle_tree")
        return st.tree
    if kind == "tree":
        vb.check(L.vg_merkle_tree(ctx.h, _addr(st.leaves), case["n"], _addr(st.tree)), "vg_merkle_tree")
        return st.tree
    o = st.out
    vb.check(L.vg_pc_commit_all(st.pc, _addr(st.priv), case["log_len"], _addr(st.mask), MASK, _addr(st.pub),
                                _addr(st.pub_mask), st.M, _addr(st.fri_r), st.levels, len(st.which), _addr(st.which),
                                _addr(st.pos), _addr(o["roots"]), _addr(o["all_sum"]), _addr(o["inner"]),
                                _addr(o["final"]), _addr(o["values"]), _addr(o["paths"])), "vg_pc_commit_all")
    return {**o, "paths": o["paths"][st.path_rows]}


# -------------------------------------------------------------------- exact
def exact(case, seed):
    """The hashes and evaluations that Python's own integers and hashlib give
    in little time; the other kinds have no such value."""
    if case["kind"] == "mle" and case["log_n"] <= 16:
        vals = _host_field(1 << case["log_n"], seed) if case["host"] else _field(1 << case["log_n"], seed).cpu().numpy()
        t = [(int(re), int(im)) for im, re in vals]
        for im, re in _host_field(case["log_n"], seed + 1):
            c, d = int(re), int(im)
            t = [((x[0] + (y[0] - x[0]) * c - (y[1] - x[1]) * d) % P, (x[1] + (y[0] - x[0]) * d + (y[1] - x[1]) * c) % P)
                 for x, y in zip(t[::2], t[1::2])]
        return np.array([[t[0][1], t[0][0]]], np.int64)
    if case["kind"] in ("leaves", "tree"):
        h = hashlib.sha3_256 if case["hash"] == "sha3" else hashlib.sha256
        if case["kind"] == "tree":
            rows = [r.tobytes() for r in _bytes(case["n"], seed).cpu().numpy()]
        else:
            n, half = case["n"], case["n"] // 2
            if half * case["slices"] > 4 << 20:
                return None
            cw = _field(case["slices"] * n, seed).cpu().numpy().reshape(case["slices"], n, 2)
            rows = [bytes(32)] * half
            for s in range(case["slices"]):
                rows = [h(cw[s, k].tobytes() + cw[s, k + half].tobytes() + rows[k]).digest() for k in range(half)]
        size = 1 << (len(rows) - 1).bit_length()
        tree = [bytes(32)] * size + rows + [h(bytes(64)).digest()] * (size - len(rows))
        for i in range(size - 1, 0, -1):
            tree[i] = h(tree[2 * i] + tree[2 * i + 1]).digest()
        return np.frombuffer(b"".join(tree), np.uint8).reshape(-1, 32)
    return None


# --------------------------------------------------------------------- work
def _hash_ops(case):
    return KECCAK_OPS if case.get("hash", "sha3") == "sha3" else SHA256_OPS


def _commit_work(log_len, hash_ops, in_bytes):
    """Two encodings, the quotient and the virtual oracle of 65 slices of S,
    FRI folds to 64 entries and a chain and a node hash per leaf of every set."""
    S = 1 << (log_len - 1)
    butterflies = 3 * 65 * S * (log_len - 1) // 2 + 3 * 65 * S // 32 * (log_len - 6)
    leaves = 2 * (S // 2) + S // 2
    return {"bytes": in_bytes + 65 * 16 * (2 * S + S) + 64 * leaves,
            "flops": butterflies * (MUL_OPS + 2 * ADD_OPS) + 65 * S * 6 * MUL_OPS + 66 * leaves * hash_ops}


def _proof_work(widths, load):
    """Per gate the evaluation, two edge terms of two products in each phase;
    per table entry and phase the rounds' folds and sums (3 + 2 products per
    entry, every round halving the tables); the commitment of the padded
    input."""
    padded = max(widths[0], 1 << (17 if len(widths) > 3 else 15))
    log_len = (padded - 1).bit_length()
    widths = [padded, padded] + widths[1:]
    gates = sum(widths[1:])
    entries = 2 * sum(widths[:-1])   # phase 1 and 2 of every layer
    c = _commit_work(log_len, KECCAK_OPS, 0)
    return {"bytes": c["bytes"] + 9 * gates + 16 * gates + 2 * 10 * gates + 48 * entries + (9 * gates if load else 0),
            "flops": c["flops"] + gates * (5 * MUL_OPS + 4 * ADD_OPS) + entries * (5 * MUL_OPS + 6 * ADD_OPS)}


def work(case):
    kind = case["kind"]
    if kind == "mle":
        n = 1 << case["log_n"]
        return {"bytes": 16 * n, "flops": n * (MUL_OPS + 2 * ADD_OPS)}
    if kind == "ntt":
        n, b = 1 << case["log_n"], case["batch"]
        return {"bytes": 16 * b * (n + case["in_len"]),
                "flops": b * n * case["log_n"] // 2 * (MUL_OPS + 2 * ADD_OPS) + b * n}
    if kind == "leaves":
        n, s = case["n"], case["slices"]
        return {"bytes": 16 * n * s + 32 * n, "flops": (n // 2 * s + n // 2) * _hash_ops(case)}
    if kind == "tree":
        size = 1 << (case["n"] - 1).bit_length()
        return {"bytes": 32 * (case["n"] + 2 * size), "flops": size * _hash_ops(case)}
    if kind == "commit":
        return _commit_work(case["log_len"], _hash_ops(case), 2 * (16 << case["log_len"]))
    if case["circuit"] == "matmul":
        n = case["size"]
        widths = [2 * n * n] + [n ** 3 >> k for k in range(n.bit_length())]
    elif case["circuit"] == "random":
        lw = max(1, case["size"] - int(np.log2(case["depth"])))
        widths = [1 << lw] * case["depth"]
    else:
        k = case["size"] - 1
        widths = [1 << (w + k.bit_length()) for w in (14, 16, 15, 14, 12, 10, 10, 10, 9, 9)]
    one = _proof_work(widths, kind == "job")
    return {key: v * case.get("copies", 1) for key, v in one.items()}

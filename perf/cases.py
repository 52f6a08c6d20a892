"""Performance cases of the prove phase, through the entry points a program calls.

The cases cover what a user of the library has it do: whole proves
(``Context.prove``, ``Context.prove_into``), polynomial commitments with their
evaluations and openings (``lg_commit``, ``Committed.eval``,
``Context.open_batches``) and the single operations of the C ABI
(Reed-Solomon encoding, Merkle trees, FRI folds, grand products, DEEP
quotients), from the sizes of the tests to those of the benchmark and its
kernel sweep.  ``listed()`` names twelve of them and ``draw(rng)`` gives others
of the same ranges.

Every output is made of whole field words or proof bytes, so two builds agree
when they give the same bits; ``exact`` therefore has no values to add.
"""
from __future__ import annotations

import ctypes
import functools
import math

import numpy as np
import torch

from loom_b200 import Context, _lib
from loom_b200 import field as F
from loom_b200.program import Builder, Module, col, copy_constraint, range_check

RANGE_BOUND = 256  # the range table of the mixed-size programs
MAX_QUERIES = 200
MAX_WORDS = 1 << 25  # input words of a single operation
# field operations of one width-24 Poseidon2 permutation: 144 + 21 cubes, 483
# diagonal products, the additions of 7 external and 21 internal layers
PERM_OPS = 2 * 165 + 21 * 23 + 165 + 7 * 110 + 21 * 46


def listed():
    return [
        # one small circuit proven from host memory, as the tests do: latency
        {"name": "prove_small", "kind": "prove", "logs": "6", "lookup": False, "queries": 8, "device": False},
        # the benchmark's workload, witness resident on the GPU
        {"name": "prove_40x2e14", "kind": "prove", "logs": ",".join(["14"] * 40), "lookup": False, "queries": 200,
         "device": True},
        # modules of uneven sizes with a range lookup, witness in page-locked
        # host memory: the benchmark's mixed program at a tenth of its rows
        {"name": "prove_mixed", "kind": "prove", "logs": "17,16,12,15,10,18,13,11,14,12", "lookup": True,
         "queries": 200, "device": False},
        # a small batch from host memory: commit, evaluate at zeta, open
        {"name": "commit_small", "kind": "commit", "groups": "9x4+0,7x3+1", "shifts": 2, "queries": 20, "device": False},
        # wide batches of three sizes on the GPU with extension columns
        {"name": "commit_large", "kind": "commit", "groups": "16x48+2,14x30+1,12x9+3", "shifts": 2, "queries": 200,
         "device": True},
        # encoding of a few short columns: latency
        {"name": "encode_small", "kind": "encode", "logn": 9, "cols": 3},
        # a wide batch of long columns (four-step transforms)
        {"name": "encode_large", "kind": "encode", "logn": 18, "cols": 128},
        # a tall tree with injections near the leaves, midway and at the top
        {"name": "merkle_large", "kind": "merkle", "log_leaves": 20, "inject": "18,18,15,3"},
        # one fold of a long layer (the first rounds of FRI)
        {"name": "fold_large", "kind": "fold", "logn": 22},
        # grand product over a row count that is not a power of two
        {"name": "product_ragged", "kind": "product", "rows": 1000003, "noalloc": False},
        # the allocation-free grand product at the benchmark's module size
        {"name": "product_noalloc", "kind": "product", "rows": 16384, "noalloc": True},
        # DEEP quotient of a wide batch at one point
        {"name": "deep_large", "kind": "deep", "log_rows": 20, "cols": 48},
    ]


def draw(rng):
    """One more case: sizes uniform in their logarithm, odd counts included."""

    def log_int(lo, hi):
        return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))

    kind = rng.choice(["prove", "prove", "mixed", "commit", "encode", "merkle", "fold", "product", "deep"])
    if kind == "prove":  # equal modules, at most the benchmark's 40 x 2^14 rows
        logn = rng.randint(4, 16)
        count = log_int(1, max(1, min(40, (40 << 14) >> logn)))
        return {"kind": "prove", "logs": ",".join([str(logn)] * count), "lookup": False,
                "queries": log_int(1, MAX_QUERIES), "device": rng.random() < 0.5}
    if kind == "mixed":  # uneven modules with a lookup
        logs, rows = [], 0
        for _ in range(log_int(2, 12)):
            lg = rng.randint(5, 17)
            if rows + (1 << lg) <= 1 << 18:
                logs.append(lg)
                rows += 1 << lg
        return {"kind": "prove", "logs": ",".join(map(str, logs or [8])), "lookup": True,
                "queries": log_int(1, MAX_QUERIES), "device": rng.random() < 0.5}
    if kind == "commit":
        groups = []
        for lg in sorted(rng.sample(range(4, 17), rng.randint(1, 4)), reverse=True):
            cap = max(1, (MAX_WORDS >> 3) >> lg)
            groups.append("%dx%d+%d" % (lg, log_int(1, min(48, cap)), rng.randint(0, 3)))
        return {"kind": "commit", "groups": ",".join(groups), "shifts": rng.randint(1, 3),
                "queries": log_int(1, MAX_QUERIES), "device": rng.random() < 0.5}
    if kind == "encode":
        logn = rng.randint(4, 20)
        return {"kind": "encode", "logn": logn, "cols": log_int(1, min(1024, MAX_WORDS >> logn))}
    if kind == "merkle":
        top = rng.randint(3, 20)
        widths = sorted((rng.randint(0, top) for _ in range(rng.randint(0, 5))), reverse=True)
        return {"kind": "merkle", "log_leaves": top, "inject": ",".join(map(str, widths))}
    if kind == "fold":
        return {"kind": "fold", "logn": rng.randint(4, 23)}
    if kind == "product":
        noalloc = rng.random() < 0.5
        return {"kind": "product", "rows": log_int(16, 1 << 20), "noalloc": noalloc}
    log_rows = rng.randint(6, 20)
    return {"kind": "deep", "log_rows": log_rows, "cols": log_int(1, min(256, (48 << 20) >> log_rows))}


# ---------------------------------------------------------------- inputs
@functools.lru_cache(maxsize=None)
def _context() -> Context:
    """The process's one context, as a program keeps one per GPU."""
    return Context(0)


class _Inputs:
    """Field words from a seed, on the GPU."""

    def __init__(self, seed: int):
        self.g = torch.Generator(device="cuda")
        self.g.manual_seed(seed)

    def words(self, *shape) -> torch.Tensor:
        return torch.randint(0, F.P, shape, dtype=torch.int32, device="cuda", generator=self.g)


def _u32(t: torch.Tensor) -> np.ndarray:
    return np.ascontiguousarray(t.cpu().numpy().view(np.uint32))


def _check(ctx: Context, rc: int):
    if rc != _lib.LG_OK:
        raise _lib.LoomError(rc, ctx.L.lg_last_error(ctx.h).decode())


def _logs(case):
    return [int(x) for x in case["logs"].split(",")]


def _groups(case):
    out = []
    for g in case["groups"].split(","):
        lg, cols = g.split("x")
        nb, ne = cols.split("+")
        out.append((int(lg), int(nb), int(ne)))
    return out


def _widths(case):
    return [int(x) for x in case["inject"].split(",") if x]


@functools.lru_cache(maxsize=8)
def _program(logs: str, lookup: bool):
    """The compiled program of plonk-like modules (gate, copy constraint over
    the wires, optionally a range lookup) and its columns that do not depend
    on the witness.  The permutation columns are made with the witness."""
    b = Builder()
    for i, lg in enumerate(int(x) for x in logs.split(",")):
        n = 1 << lg
        m = Module(f"plonk_{i}", n)
        L, R, O, QL, QR, QM, QO, QK = (col(f"{s}_{i}") for s in ("L", "R", "O", "QL", "QR", "QM", "QO", "QK"))
        m.assert_zero(QL * L + QR * R + QM * L * R + QO * O + QK)
        b.add_module(m)
        copy_constraint(b, m.name, [L, R, O], np.arange(3 * n), f"plonk.S_{i}")
        if lookup:
            range_check(b, col(f"RC_{i}"), m.name, RANGE_BOUND)
    return b.compile(), dict(b.generated)


def _plonk_columns(i: int, n: int, rng, fixed, lookup: bool):
    """Canonical columns of module i: random wires made equal along random
    copy cycles of two to four positions over half of them, 0/1 selectors,
    the output wire solved from the gate."""
    p = np.uint64(F.P)
    vals = rng.integers(0, F.P, 2 * n, dtype=np.uint64)
    S = np.arange(3 * n)
    perm, at = rng.permutation(2 * n), 0
    for k in (2, 3, 4):
        cnt = (n // 3) // k
        cyc = perm[at:at + cnt * k].reshape(cnt, k)
        at += cnt * k
        S[cyc] = np.roll(cyc, -1, axis=1)
        vals[cyc] = vals[cyc[:, :1]]
    a, b = vals[:n], vals[n:]
    ql, qr, qm, qk = rng.integers(0, 2, (4, n), dtype=np.uint64)
    qo = np.maximum(ql | qr | qm | qk, rng.integers(0, 2, n, dtype=np.uint64))
    lin = (ql * a + qr * b + qm * (a * b % p) + qk) % p
    c = np.where(qo == 1, (p - lin) % p, rng.integers(0, F.P, n, dtype=np.uint64))
    cols = {"L": a, "R": b, "O": c, "QL": ql, "QR": qr, "QM": qm, "QO": qo, "QK": qk}
    cols = {f"{k}_{i}": v for k, v in cols.items()}
    ident = np.concatenate([fixed[Module(f"plonk_{i}", n).id_support_name(k)] for k in range(3)])
    for k in range(3):
        cols[f"plonk.S_{i}_{k}"] = ident[S[k * n:(k + 1) * n]]
    if lookup:
        cols[f"RC_{i}"] = rng.integers(0, RANGE_BOUND, n, dtype=np.uint64)
    return cols


def _prepare_prove(case, seed):
    comp, fixed = _program(case["logs"], case["lookup"])
    rng = np.random.Generator(np.random.PCG64(seed))
    trace = dict(fixed)
    for i, lg in enumerate(_logs(case)):
        trace.update(_plonk_columns(i, 1 << lg, rng, fixed, case["lookup"]))
    cols = [F.to_mont(trace[name]) for name, _, _ in comp.witness_columns]
    total = sum(c.size for c in cols)
    # columns back to back in descriptor order, as a program that allocates
    # its trace once holds them; page-locked when they stay on the host
    flat = torch.empty(total, dtype=torch.int32, pin_memory=True)
    words, views, off = flat.numpy().view(np.uint32), [], 0
    for c in cols:
        words[off:off + c.size] = c
        views.append(words[off:off + c.size])
        off += c.size
    st = {"words": comp.words, "flat": flat, "witness": views}
    if case["device"]:
        st["flat"] = flat.cuda()
        base = st["flat"].data_ptr()
        at = np.concatenate([[0], np.cumsum([c.size for c in cols])[:-1]])
        st["witness"] = [base + 4 * int(a) for a in at]
    # the caller's proof buffer, page-locked, with room to spare
    st["proof"] = torch.empty((1 << 16) + 2 * _proof_bytes(case), dtype=torch.uint8, pin_memory=True).numpy()
    return st


def _proof_bytes(case):
    """About the bytes of the proof: per query the FRI layers' row pairs and
    paths, three committed batches' paths with their injected digests, and
    every module's row pairs; per module its claimed values."""
    logs = _logs(case)
    top, cols = max(logs), 14 + 6 * 6 if case["lookup"] else 14 + 5 * 6
    fri = sum(8 * (k + 1) + 18 for k in range(1, top + 1))
    batches = 3 * 8 * (top + len(logs)) + len(logs) * (2 * cols + 30)
    return 4 * case["queries"] * (fri + batches) + 24 * 30 * len(logs)


def prepare(case, seed):
    st = {"case": dict(case), "ctx": _context()}
    kind = case["kind"]
    gen = _Inputs(seed)
    if kind == "prove":
        st.update(_prepare_prove(case, seed))
    elif kind == "commit":
        groups = _groups(case)
        data = [[gen.words(1 << lg) for _ in range(nb)] + [gen.words(1 << lg, 6) for _ in range(ne)]
                for lg, nb, ne in groups]
        if case["device"]:
            cols = [t for g in data for t in g]
            st["cols"] = cols
            st["ptrs"] = (ctypes.c_void_p * len(cols))(*[t.data_ptr() for t in cols])
            st["rows"] = np.array([1 << lg for lg, _, _ in groups], dtype=np.uint64)
            st["nb"] = np.array([nb for _, nb, _ in groups], dtype=np.uint32)
            st["ne"] = np.array([ne for _, _, ne in groups], dtype=np.uint32)
        else:
            st["groups"] = [{"rows": 1 << lg, "base": [_u32(t) for t in g[:nb]], "ext": [_u32(t) for t in g[nb:]]}
                            for (lg, nb, ne), g in zip(groups, data)]
        st["zeta"] = _u32(gen.words(6))
        st["positions"] = np.random.Generator(np.random.PCG64(seed)).integers(0, 1 << 24, case["queries"],
                                                                              dtype=np.uint32)
    elif kind == "encode":
        st["in"] = gen.words(case["cols"], 1 << case["logn"])
        st["out"] = torch.empty(case["cols"], 4 << case["logn"], dtype=torch.int32, device="cuda")
    elif kind == "merkle":
        st["leaves"] = gen.words(1 << case["log_leaves"], 8)
        widths = [1 << w for w in _widths(case)]
        st["widths"] = np.array(widths, dtype=np.uint64)
        st["inj"] = gen.words(max(1, sum(widths)), 8)
    elif kind == "fold":
        n = 1 << case["logn"]
        st["in"], st["alpha"] = gen.words(n, 6), _u32(gen.words(6))
        st["out"] = torch.empty(n // 2, 6, dtype=torch.int32, device="cuda")
    elif kind == "product":
        n = case["rows"]
        st["num"], st["den"] = gen.words(n, 6), gen.words(n, 6)
        st["out"] = torch.empty(n, 6, dtype=torch.int32, device="cuda")
    else:
        rows = 1 << case["log_rows"]
        st["in"], st["values"] = gen.words(case["cols"], rows), gen.words(case["cols"], 6)
        st["alpha"], st["z"] = _u32(gen.words(6)), _u32(gen.words(6))
        st["out"] = torch.empty(rows, 6, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()  # the library works on a stream of its own
    return st


# ---------------------------------------------------------------- passes
def _dev(t: torch.Tensor):
    return ctypes.c_void_p(t.data_ptr())


def _host(a: np.ndarray, ptr=_lib.u32p):
    return a.ctypes.data_as(ptr)


def run(st):
    case, ctx = st["case"], st["ctx"]
    L, kind = ctx.L, case["kind"]
    if kind == "prove":
        n = ctx.prove_into(st["proof"], st["words"], st["witness"], case["queries"], on_device=case["device"])
        return st["proof"][:n]
    if kind == "commit":
        if case["device"]:
            root, h = np.zeros(8, dtype=np.uint32), ctypes.c_void_p()
            _check(ctx, L.lg_commit(ctx.h, len(st["rows"]), _host(st["rows"], _lib.u64p), _host(st["nb"]),
                                    _host(st["ne"]), st["ptrs"], 1, ctypes.byref(h), _host(root)))
            batch = _lib.Committed(ctx, h, root, st["nb"].tolist(), st["ne"].tolist())
        else:
            batch = ctx.commit(st["groups"])
        values = batch.eval(st["zeta"], list(range(case["shifts"])))
        opening = ctx.open_batches([batch], st["positions"])
        batch.release()
        return {"root": batch.root, "values": values, "opening": np.frombuffer(opening, dtype=np.uint8)}
    if kind == "encode":
        _check(ctx, L.lg_rs_encode(ctx.h, _dev(st["in"]), 1 << case["logn"], case["cols"], _dev(st["out"]), 1))
        return st["out"]
    if kind == "merkle":
        root = np.zeros(8, dtype=np.uint32)
        _check(ctx, L.lg_merkle_root(ctx.h, _dev(st["leaves"]), 1 << case["log_leaves"], st["widths"].size,
                                     _host(st["widths"], _lib.u64p), _dev(st["inj"]), 1, _host(root)))
        return root
    if kind == "fold":
        _check(ctx, L.lg_fri_fold(ctx.h, _dev(st["in"]), 1 << case["logn"], _host(st["alpha"]), _dev(st["out"]), 1))
        return st["out"]
    if kind == "product":
        num, den, out, n = _dev(st["num"]), _dev(st["den"]), _dev(st["out"]), case["rows"]
        if case["noalloc"]:
            rc = L.lg_grand_product_noalloc(num, den, n, out, ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
            if rc != _lib.LG_OK:
                raise _lib.LoomError(rc, "lg_grand_product_noalloc failed")
        else:
            _check(ctx, L.lg_grand_product(ctx.h, num, den, n, out, 1))
        return st["out"]
    _check(ctx, L.lg_deep_quotient(ctx.h, _dev(st["in"]), case["cols"], 1 << case["log_rows"], _host(st["alpha"]),
                                   _host(st["z"]), _dev(st["values"]), _dev(st["out"]), 1))
    return st["out"]


def exact(case, seed):
    """Nothing to give: every output is a whole field word or a proof byte."""
    return None


# ---------------------------------------------------------------- work
def _commit_ops(rows, base, ext, from_coeffs=False):
    """Field operations of one group's encoding and leaf hashing (a butterfly:
    one product, two additions) and of as many tree nodes as it has leaves."""
    lanes = base + 6 * ext
    transforms = 4  # the inverse and three cosets, or four cosets
    ntt = transforms * (rows // 2) * int(math.log2(rows)) * 3
    leaves = 2 * rows
    perms = leaves * (-(-(3 + 2 * lanes) // 16)) + leaves
    return lanes * ntt + perms * PERM_OPS


def work(case):
    kind = case["kind"]
    if kind == "prove":
        nbytes, ops = 0, 0
        for lg in _logs(case):
            n = 1 << lg
            base, ext = 14, 1
            if case["lookup"]:
                base, ext = 15, 2
            nbytes += 4 * n * base
            ops += _commit_ops(n, 9, 0) + _commit_ops(n, base - 9, ext) + _commit_ops(n, 0, 4)
            # constraint evaluation, claimed values and DEEP over every column
            ops += 4 * n * 60 + 4 * n * (base * 12 + (ext + 4) * 60)
        return {"bytes": nbytes + _proof_bytes(case), "flops": ops}
    if kind == "commit":
        nbytes, ops, row_bytes = 0, 0, 0
        for lg, nb, ne in _groups(case):
            n, lanes = 1 << lg, nb + 6 * ne
            nbytes += 4 * n * lanes + 24 * case["shifts"] * (nb + ne)
            ops += _commit_ops(n, nb, ne) + case["shifts"] * lanes * n * 12
            row_bytes += 8 * lanes
        return {"bytes": nbytes + case["queries"] * (row_bytes + 32 * 18), "flops": ops}
    if kind == "encode":
        n = 1 << case["logn"]
        return {"bytes": 20 * n * case["cols"], "flops": case["cols"] * 4 * (n // 2) * case["logn"] * 3}
    if kind == "merkle":
        leaves, inj = 1 << case["log_leaves"], sum(1 << w for w in _widths(case))
        return {"bytes": 32 * (leaves + inj + 1), "flops": (leaves + inj) * PERM_OPS}
    if kind == "fold":
        n = 1 << case["logn"]
        return {"bytes": 36 * n, "flops": (n // 2) * 80}
    if kind == "product":
        # a product for the inverse's share, the quotient and the scan per row
        return {"bytes": 72 * case["rows"], "flops": case["rows"] * 4 * 60}
    rows = 1 << case["log_rows"]
    return {"bytes": (4 * case["cols"] + 24) * rows, "flops": rows * (12 * case["cols"] + 300)}

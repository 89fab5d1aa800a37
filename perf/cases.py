"""Performance cases of the table-commitment library: what they run and on what.

Each case is one call path that a prover or a commitment service takes, through
the Python binding's public entry points (tvmc.py, a thin mirror of the C ABI).
Tables hold uniform field elements, the widths are those of the master tables
(379 base columns; 88 XFieldElement columns = 264 limbs) unless a case says
otherwise, and the evaluation offset is 7.

Every output is a residue mod p, compared bit for bit (tolerance "exact"); no
output is a rounded number, so there is no 64-bit reference to give.
"""
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "triton-vm-prover_b200"))
import tvmc  # noqa: E402

P = tvmc.P
OFFSET = 7
OPENINGS = 80  # leaf indices opened per served commitment
DEV = "cuda"


def listed():
    return [
        # The smallest call: the Merkle tree over one late FRI round's codeword.
        {"name": "fri_tree_2p10", "op": "fri_tree", "logn": 10},
        # The shortest padded height a program runs at: latency of one commit.
        {"name": "commit_2p8x379", "op": "commit", "logn": 8, "width": 379, "exp": 4},
        # A service's small requests: host traces in, root and openings out.
        {"name": "serve_2p10_2p12", "op": "serve", "lo": 10, "hi": 12, "count": 12},
        # The zero-knowledge commitment of a small aux table.
        {"name": "commit_rand_2p12x264", "op": "commit_rand", "logn": 12, "width": 264, "exp": 4, "rand": 98,
         "trace_offset": 3},
        # Row hashing alone: an odd number of rows of an odd width.
        {"name": "hash_rows_50001x88xfe", "op": "hash_rows", "rows": 50001, "width": 88, "xfe": True},
        # A row-major table (the CPU prover's layout) at a larger blowup.
        {"name": "commit_rowmajor_2p13x379", "op": "commit", "logn": 13, "width": 379, "exp": 8, "row_major": True},
        # Interpolation of a whole table's columns.
        {"name": "intt_2p16x379", "op": "ntt", "logn": 16, "width": 379, "inverse": True},
        # Many tables of uneven heights, one graph launch.
        {"name": "batch_2p12_2p16", "op": "batch", "lo": 12, "hi": 16, "count": 16},
        # A mid-size program's main table.
        {"name": "commit_2p16x379", "op": "commit", "logn": 16, "width": 379, "exp": 4},
        # The LDE alone on a tall table's columns.
        {"name": "lde_2p20x96", "op": "lde", "logn": 20, "width": 96, "exp": 4},
        # The large main table.
        {"name": "commit_2p20x379", "op": "commit", "logn": 20, "width": 379, "exp": 4},
        # The streaming commit of a table whose LDE is not kept.
        {"name": "frugal_2p21x379", "op": "commit", "logn": 21, "width": 379, "exp": 4, "frugal": True},
    ]


def _log_size(rng, lo, hi):
    return int(round(rng.uniform(lo, hi)))


def _width(rng):
    """The two master tables' widths half of the time, else any width up to 400."""
    return rng.choice((379, 264)) if rng.random() < 0.5 else int(round(2 ** rng.uniform(0.0, 8.6)))


def draw(rng):
    op = rng.choice(("fri_tree", "commit", "commit", "commit", "commit_rand", "serve", "hash_rows", "ntt", "lde",
                     "batch", "multi", "coset"))
    if op == "fri_tree":
        return {"op": op, "logn": _log_size(rng, 8, 22)}
    if op in ("commit", "commit_rand"):
        exp = rng.choice((2, 4, 4, 8))
        logn = _log_size(rng, 8, 19)
        case = {"op": op, "logn": logn, "width": _width(rng), "exp": exp}
        if op == "commit_rand":
            case.update(rand=rng.randint(1, 200), trace_offset=rng.choice((1, 3)))
        else:
            case.update(row_major=rng.random() < 0.3, frugal=logn >= 16 and rng.random() < 0.3)
        return case
    if op in ("serve", "batch", "multi"):
        lo = rng.randint(8, 12)
        return {"op": op, "lo": lo, "hi": lo + rng.randint(1, 4), "count": rng.randint(3, 16), "shape": rng.randint(0, 999)}
    if op == "hash_rows":
        xfe = rng.random() < 0.5
        return {"op": op, "rows": int(round(2 ** rng.uniform(6, 20))), "width": rng.randint(1, 120 if xfe else 380),
                "xfe": xfe}
    if op == "coset":
        return {"op": op, "logn": _log_size(rng, 8, 20), "width": rng.randint(1, 64), "exp": rng.choice((1, 2, 4))}
    case = {"op": op, "logn": _log_size(rng, 8, 20), "width": rng.randint(1, 200)}
    case.update({"inverse": rng.random() < 0.5} if op == "ntt" else {"exp": rng.choice((2, 4, 8))})
    return case


def _elements(seed, *shape):
    """Uniform canonical field elements as the int64 words of a CUDA tensor."""
    g = torch.Generator(device=DEV).manual_seed(seed)
    x = torch.randint(-2**63, 2**63 - 2**32 + 1, shape, dtype=torch.int64, device=DEV, generator=g)
    return x.bitwise_xor_(-2**63)


def _shapes(case):
    """(trace length, width) of the tables of a many-table case: heights spread
    over [2^lo, 2^hi], main and aux widths in turn."""
    lo, hi, count, twist = case["lo"], case["hi"], case["count"], case.get("shape", 1)
    return [(1 << (lo + (5 * i + twist) % (hi - lo + 1)), 379 if (i + twist) % 2 else 264) for i in range(count)]


class _Words:
    """Device words owned by a tvmc object, viewed by torch without a copy."""

    def __init__(self, owner, ptr, *shape):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": shape, "typestr": "<i8", "data": (ptr, False), "version": 3}


def _view(owner, ptr, *shape):
    return torch.as_tensor(_Words(owner, ptr, *shape), device=DEV)


def _commitment_out(c, lde=True, owner=None):
    """The heap tree (node 0 is unused) and, where it is kept, the LDE, which
    `owner` (the commitment, unless a batch holds its memory) keeps alive."""
    owner = owner or c
    out = {"nodes": _view(owner, c.device_tree() + 40, 2 * c.lde_len - 1, 5)}
    if lde:
        out["lde"] = _view(owner, c.device_lde(), c.width, c.lde_len)
    return out


def prepare(case, seed):
    op = case["op"]
    st = {"case": case}
    if op == "fri_tree":
        st["x"] = _elements(seed, 1 << case["logn"], 3)
    elif op in ("commit", "commit_rand"):
        n, w = 1 << case["logn"], case["width"]
        st["x"] = _elements(seed, n, w) if case.get("row_major") else _elements(seed, w, n)
        if op == "commit_rand":
            st["r"] = _elements(seed + 10**6, w, case["rand"])
    elif op == "serve":
        shapes = _shapes(case)
        st["x"] = [_elements(1000 * seed + i, w, n).cpu().pin_memory().numpy().view(np.uint64)
                   for i, (n, w) in enumerate(shapes)]
        rng = np.random.default_rng(seed)
        st["idx"] = [rng.integers(0, 4 * n, OPENINGS) for n, _ in shapes]
        st["server"] = tvmc.Server()
    elif op == "batch":
        st["batch"] = b = tvmc.Batch(_shapes(case))
        for i, (n, w) in enumerate(_shapes(case)):
            _view(b, b.input_ptr(i), w, n).copy_(_elements(1000 * seed + i, w, n))
    elif op == "multi":
        st["x"] = [_elements(1000 * seed + i, w, n) for i, (n, w) in enumerate(_shapes(case))]
    elif op == "hash_rows":
        w = case["width"] * (3 if case["xfe"] else 1)
        st["x"] = _elements(seed, w, case["rows"])
        st["out"] = torch.empty(case["rows"], 5, dtype=torch.int64, device=DEV)
    elif op == "ntt":
        st["x"] = _elements(seed, case["width"], 1 << case["logn"])
        st["out"] = torch.empty_like(st["x"])
    else:  # lde, coset
        n, w = 1 << case["logn"], case["width"]
        st["x"] = _elements(seed, w, n)
        st["out"] = torch.empty(w, n * case["exp"], dtype=torch.int64, device=DEV)
    return st


def run(st):
    case = st["case"]
    op = case["op"]
    if op == "fri_tree":
        if "c" in st:
            st["c"].free()
        st["c"] = c = tvmc.Commitment.from_digests(st["x"].data_ptr(), xfe=True, count=1 << case["logn"],
                                                   device_ptr=True)
        return _commitment_out(c, lde=False)
    if op in ("commit", "commit_rand"):
        if "c" in st:
            st["c"].free()
        frugal = case.get("frugal", False)
        rand = (st["r"].data_ptr(), case["rand"]) if op == "commit_rand" else None
        st["c"] = c = tvmc.Commitment(st["x"].data_ptr(), width=case["width"], trace_len=1 << case["logn"],
                                      expansion=case["exp"], offset=OFFSET, row_major=case.get("row_major", False),
                                      device_ptr=True, frugal=frugal, randomizers=rand,
                                      trace_offset=case.get("trace_offset", 1))
        return _commitment_out(c, lde=not frugal)
    if op == "serve":
        s = st["server"]
        ids = [s.submit(x, offset=OFFSET) for x in st["x"]]
        out = []
        for rid, idx in zip(ids, st["idx"]):
            root = s.wait(rid)
            out.append((root, s.open(rid, idx)))
            s.release(rid)
        return out
    if op == "batch":
        b = st["batch"]
        b.run()
        return [_commitment_out(t, owner=b) for t in b.tables]
    if op == "multi":
        for c in st.get("c", ()):
            c.free()
        st["c"] = tvmc.commit_multi([x.data_ptr() for x in st["x"]], offset=OFFSET, device_ptr=True,
                                    shapes=[(x.shape[1], x.shape[0]) for x in st["x"]])
        return [_commitment_out(c) for c in st["c"]]
    x, out = st["x"], st["out"]
    if op == "hash_rows":
        f = tvmc.hash_xfield_rows_gpu if case["xfe"] else tvmc.hash_rows_gpu
        f(x.data_ptr(), case["rows"], case["width"], out.data_ptr())
    elif op == "ntt":  # in place on a copy: a program keeps its trace
        out.copy_(x)
        tvmc.ntt_gpu(out.data_ptr(), x.shape[1], x.shape[0], inverse=case["inverse"])
    elif op == "lde":
        tvmc.lde_gpu(x.data_ptr(), x.shape[0], x.shape[1], out.data_ptr(), out.shape[1], OFFSET)
    else:
        w, n = x.shape
        rc = tvmc.lib().tvmc_evaluate_on_coset_gpu(x.data_ptr(), n, w, out.data_ptr(), out.shape[1], OFFSET, None)
        if rc != tvmc.OK:
            raise RuntimeError(tvmc.lib().tvmc_last_error().decode())
    return out


# 32-bit integer operations of the cost model that the benchmark reports: one
# Tip5 permutation, and one butterfly or scale product of an NTT.
PERM_OPS = 8320
NTT_OPS = 24


def _lde_work(n, w, e):
    L = n * e
    ops = w * (n // 2 * (n.bit_length() - 1) + n + L // 2 * (L.bit_length() - 1)) * NTT_OPS
    return 8 * w * (n + L), ops


def _commit_work(n, w, e, keep=True):
    L = n * e
    b, ops = _lde_work(n, w, e)
    b = (b if keep else 8 * w * n) + 40 * (2 * L - 1)
    return b, ops + PERM_OPS * (L * (w // 10 + 1) + L - 1)


def work(case):
    op = case["op"]
    if op == "fri_tree":
        n = 1 << case["logn"]
        b, ops = 24 * n + 40 * (2 * n - 1), PERM_OPS * (n - 1)
    elif op in ("commit", "commit_rand"):
        b, ops = _commit_work(1 << case["logn"], case["width"], case["exp"], not case.get("frugal"))
        b += 8 * case["width"] * case.get("rand", 0)
    elif op in ("serve", "batch", "multi"):
        each = [_commit_work(n, w, 4, op != "serve") for n, w in _shapes(case)]
        b, ops = sum(x[0] for x in each), sum(x[1] for x in each)
    elif op == "hash_rows":
        w = case["width"] * (3 if case["xfe"] else 1)
        b, ops = case["rows"] * (8 * w + 40), PERM_OPS * case["rows"] * (w // 10 + 1)
    elif op == "ntt":
        n, w = 1 << case["logn"], case["width"]
        b, ops = 16 * n * w, w * (n // 2 * case["logn"] + (n if case["inverse"] else 0)) * NTT_OPS
    elif op == "lde":
        b, ops = _lde_work(1 << case["logn"], case["width"], case["exp"])
    else:
        n, w, L = 1 << case["logn"], case["width"], (1 << case["logn"]) * case["exp"]
        b, ops = 8 * w * (n + L), w * (n + L // 2 * (L.bit_length() - 1)) * NTT_OPS
    return {"bytes": b, "flops": ops}


def tolerance(case):
    return "exact"

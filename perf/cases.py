"""Timed cases of the library: what a user's program has it do, through its public entry points.

Every case names an operation ("op"), the Hamiltonian or matrix it works on ("kind" and its size),
the precision and the options.  Hamiltonians:
  tfim   transverse-field Ising chain, open, J ~ U[0.5, 1.5], h ~ U[0.2, 2]: 2n+1 real diagonals
  xxz    periodic XXZ chain, J ~ U[0.5, 1.5], delta 0.8, fields U[-1, 1]: 2n+1 real diagonals
  pauli  random Pauli strings of weight <= 3 with N(0,1) coefficients, 3n of them: complex values,
         a hundred or more sparsely filled diagonals
  band   a rows x cols matrix with nd random diagonals, every stored value a complex Gaussian (a
         matrix that is not a spin chain, of any size)
"""
import ctypes
import math

import numpy as np
import torch

from diaq_gb300 import capi

PREC = {"c128": capi.C128, "c64": capi.C64, "c128f2": capi.C128F2}
MODE = {"c128": capi.EVOLVE_C128, "mixed": capi.EVOLVE_MIXED, "horner": capi.EVOLVE_HORNER}
SIZE = {"c128": 16, "c64": 8, "c128f2": 16}


def listed():
    return [
        # one product on the 12-qubit Ising chain: the smallest call a user makes; latency
        {"name": "spmv_tfim12_c128", "op": "spmv", "kind": "tfim", "n": 12, "prec": "c128", "nrhs": 1},
        # H psi on the 20-qubit chain in the reference's arithmetic (power iterations, Krylov chains)
        {"name": "spmv_xxz20_c128", "op": "spmv", "kind": "xxz", "n": 20, "prec": "c128", "nrhs": 1},
        # the same product on a matrix held as float pairs
        {"name": "spmv_xxz20_c128f2", "op": "spmv", "kind": "xxz", "n": 20, "prec": "c128f2", "nrhs": 1},
        # several right-hand sides, single precision, a general banded matrix of odd shape
        {"name": "spmm_band_c64", "op": "spmv", "kind": "band", "rows": 250007, "cols": 250013, "nd": 37,
         "prec": "c64", "nrhs": 5},
        # the reference's time evolution call on a small chain: 10 steps of 12 terms, one state
        {"name": "ham_sim_tfim12", "op": "ham_sim", "kind": "tfim", "n": 12, "steps": 10, "m": 12, "dt": 0.05},
        # many states under one large Hamiltonian: two steps of a float32 Horner plan
        {"name": "evolve_horner_xxz20_k8", "op": "evolve", "mode": "horner", "kind": "xxz", "n": 20, "nrhs": 8,
         "steps": 2, "s": 0, "m": 12, "dt": 0.05},
        # a few states under a general Pauli Hamiltonian, compensated sums, two sub-steps
        {"name": "evolve_mixed_pauli15_k3", "op": "evolve", "mode": "mixed", "kind": "pauli", "n": 15, "nrhs": 3,
         "steps": 2, "s": 1, "m": 8, "dt": 0.02},
        # many chains of uneven size with 1, 4 or 16 states each, advanced together
        {"name": "batch_c64_24", "op": "batch", "prec": "c64", "horner": True, "inst": 24, "lo": 10, "hi": 17,
         "steps": 2, "m": 8, "dt": 0.02},
        # H H of the 18-qubit chain, structure and values, fetched into device arrays
        {"name": "spgemm_xxz18_c128", "op": "spgemm", "kind": "xxz", "n": 18, "prec": "c128"},
        # the evolution operator exp(-i t H) of a 10-qubit chain as a matrix
        {"name": "expm_tfim10", "op": "expm", "kind": "tfim", "n": 10, "t": 0.1},
        # a diagonal-format matrix times a tall dense block (row-aligned device arrays)
        {"name": "spmm_dia_z_65536x16", "op": "spmm_dia", "rows": 65536, "cols": 65536, "nd": 33, "right": 16,
         "cplx": True},
        # training the (s, m) proposer: four steps of the trainer's batch size, weights read back
        {"name": "mlp_train_1024", "op": "mlp", "batch": 1024, "steps": 4},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["spmv", "spmv", "spmv", "ham_sim", "evolve", "evolve", "batch", "spgemm", "expm", "spmm_dia", "mlp"])
    chain = rng.choice(["tfim", "xxz"])
    dt = round(rng.uniform(0.01, 0.05), 4)
    if op == "spmv":
        prec = rng.choice(["c128", "c64", "c128f2"])
        nrhs = rng.choice([1, 1, 2, 3, 5, 8, 11])
        if rng.random() < 0.5:
            kind = rng.choice([chain, chain, "pauli"])
            n = rng.randint(10, 20 if kind != "pauli" else 17)
            return {"op": op, "kind": kind, "n": n, "prec": prec, "nrhs": nrhs if n <= 18 else min(nrhs, 2)}
        rows = _log_int(rng, 1000, 800000)
        return {"op": op, "kind": "band", "rows": rows, "cols": max(1000, rows + rng.randint(-300, 300)),
                "nd": rng.randint(3, 45), "prec": prec, "nrhs": nrhs}
    if op == "ham_sim":
        return {"op": op, "kind": rng.choice([chain, chain, "pauli"]), "n": rng.randint(9, 16),
                "steps": rng.randint(3, 15), "m": rng.randint(8, 14), "dt": dt}
    if op == "evolve":
        mode = rng.choice(["c128", "mixed", "horner", "horner"])
        kind = rng.choice([chain, chain, "pauli"])
        n = rng.randint(11, 17 if mode == "c128" or kind == "pauli" else 19)
        return {"op": op, "mode": mode, "kind": kind, "n": n, "nrhs": rng.choice([1, 2, 3, 4, 6, 8, 12, 16]),
                "steps": rng.randint(1, 3), "s": rng.randint(0, 1), "m": rng.randint(4, 12), "dt": dt}
    if op == "batch":
        lo = rng.randint(8, 12)
        return {"op": op, "prec": rng.choice(["c64", "c64", "c128"]), "horner": rng.random() < 0.7,
                "inst": rng.randint(3, 28), "lo": lo, "hi": rng.randint(lo, 16), "steps": rng.randint(1, 3),
                "m": rng.randint(4, 9), "dt": dt}
    if op == "spgemm":
        kind = rng.choice([chain, chain, "pauli"])
        return {"op": op, "kind": kind, "n": rng.randint(8, 17 if kind != "pauli" else 10),
                "prec": rng.choice(["c128", "c128", "c64"])}
    if op == "expm":
        return {"op": op, "kind": chain, "n": rng.randint(5, 10), "t": round(rng.uniform(0.02, 0.2), 3)}
    if op == "spmm_dia":
        rows = _log_int(rng, 1000, 100000)
        return {"op": op, "rows": rows, "cols": max(1000, rows + rng.randint(-300, 300)), "nd": rng.randint(3, 41),
                "right": rng.randint(1, 20), "cplx": rng.random() < 0.6}
    return {"op": "mlp", "batch": _log_int(rng, 64, 4096), "steps": rng.randint(1, 6)}


# ---- inputs ----------------------------------------------------------------------------------------------


def _strings(kind, n, seed):
    """(coefficients, flip masks, phase masks) of the Hamiltonian's Pauli strings; qubit q is bit n-1-q."""
    r = np.random.default_rng(seed)
    bit = [1 << (n - 1 - q) for q in range(n)]
    out = []
    if kind == "tfim":
        J, h = r.uniform(0.5, 1.5, n), r.uniform(0.2, 2.0, n)
        out += [(-J[i], 0, bit[i] | bit[i + 1]) for i in range(n - 1)]
        out += [(-h[i], bit[i], 0) for i in range(n)]
    elif kind == "xxz":
        J, h = r.uniform(0.5, 1.5, n), r.uniform(-1.0, 1.0, n)
        for i in range(n):
            p = bit[i] | bit[(i + 1) % n]
            out += [(J[i], p, 0), (J[i], p, p), (0.8 * J[i], 0, p), (h[i], 0, bit[i])]
    else:
        for _ in range(3 * n):
            x = z = 0
            for q in r.choice(n, size=int(r.integers(1, 4)), replace=False):
                p = int(r.integers(0, 3))  # X, Y, Z
                x |= bit[q] if p < 2 else 0
                z |= bit[q] if p > 0 else 0
            out.append((r.standard_normal(), x, z))
    return (np.array([c for c, _, _ in out]), np.array([x for _, x, _ in out], dtype=np.uint64),
            np.array([z for _, _, z in out], dtype=np.uint64))


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _states(k, n, seed):
    """k normalised complex Gaussian states as two float64 planes (k, n)."""
    g = _gen(seed)
    re = torch.randn(k, n, generator=g, device="cuda", dtype=torch.float64)
    im = torch.randn(k, n, generator=g, device="cuda", dtype=torch.float64)
    norm = (re.square().sum(1, keepdim=True) + im.square().sum(1, keepdim=True)).sqrt()
    return re.div_(norm), im.div_(norm)


def _band(case, seed):
    """(ascending offsets, packed float64 re, im) with values exact in the case's precision."""
    rows, cols = case["rows"], case["cols"]
    r = np.random.default_rng(seed)
    off = np.unique(np.concatenate([[0], r.integers(-(rows - 1), cols, case["nd"] - 1)])).astype(np.int32)
    total = sum(_length(rows, cols, int(d)) for d in off)
    g = _gen(seed + 1)
    re = torch.randn(total, generator=g, device="cuda", dtype=torch.float64)
    im = torch.randn(total, generator=g, device="cuda", dtype=torch.float64)
    if case.get("prec") == "c64":
        re, im = re.float().double(), im.float().double()
    return off, re, im


def _length(rows, cols, d):
    return min(rows, cols - d) if d >= 0 else min(rows + d, cols)


def _shape(case):
    return (case["rows"], case["cols"]) if "rows" in case else (1 << case["n"], 1 << case["n"])


def _matrix(case, seed):
    prec = PREC[case.get("prec", "c128")]
    if case["kind"] == "band":
        off, re, im = _band(case, seed)
        return capi.Matrix.create(*_shape(case), off, re, im, precision=prec, on_device=True)
    return capi.Matrix.from_pauli(case["n"], *_strings(case["kind"], case["n"], seed), precision=prec)


def _vectors(case, seed):
    """The right-hand sides of a product: (k, cols) planes in the vectors' precision."""
    re, im = _states(case["nrhs"], _shape(case)[1], seed + 2)
    return (re.float(), im.float()) if case["prec"] == "c64" else (re, im)


def _instances(case, seed):
    r = np.random.default_rng(12345)  # the same mix of sizes whatever the seed of the values
    return [{"kind": "xxz" if i % 2 else "tfim", "n": int(r.integers(case["lo"], case["hi"] + 1)),
             "nrhs": int(r.choice([1, 4, 16])), "prec": case["prec"], "seed": seed + 100 * i}
            for i in range(case["inst"])]


def _dia(case, seed):
    rows, cols = case["rows"], case["cols"]
    r = np.random.default_rng(seed)
    off = torch.from_numpy(np.unique(np.concatenate([[0], r.integers(-(rows - 1), cols, case["nd"] - 1)]))).cuda()
    g = _gen(seed + 1)
    dt = torch.complex128 if case["cplx"] else torch.float64
    vals = torch.randn(len(off), rows, generator=g, device="cuda", dtype=dt)
    B = torch.randn(cols, case["right"], generator=g, device="cuda", dtype=dt)
    return off, vals, B


def _network(case, seed):
    """Starting weights (flat, the library's order) and the mini-batches of features and labels."""
    r = np.random.default_rng(seed)
    parts = []
    for fan_in, fan_out in ((16, 64), (64, 64), (64, 51)):
        parts += [r.normal(0, math.sqrt(2.0 / fan_in), fan_in * fan_out), np.zeros(fan_out)]
    g = _gen(seed)
    B = case["batch"]
    batches = [(torch.randn(B, 16, generator=g, device="cuda"),
                torch.randint(0, 5, (B,), generator=g, device="cuda", dtype=torch.int32),
                torch.randint(4, 25, (B,), generator=g, device="cuda", dtype=torch.int32))
               for _ in range(case["steps"])]
    return np.concatenate(parts).astype(np.float32), batches


def prepare(case, seed):
    op = case["op"]
    st = {"case": case, "L": capi.lib()}
    if op == "spmv":
        st["A"] = _matrix(case, seed)
        st["x"] = _vectors(case, seed)
        st["y"] = tuple(torch.empty(case["nrhs"], _shape(case)[0], device="cuda", dtype=st["x"][0].dtype) for _ in "ri")
    elif op == "ham_sim":
        st["A"] = _matrix(case, seed)
        st["x"] = _states(1, 1 << case["n"], seed + 2)
        st["y"] = tuple(torch.empty_like(x) for x in st["x"])
    elif op == "evolve":
        st["E"] = capi.Evolve(_matrix(case, seed), case["nrhs"], MODE[case["mode"]])
        st["psi"] = _states(case["nrhs"], 1 << case["n"], seed + 2)
    elif op == "batch":
        inst = _instances(case, seed)
        psi = [_states(i["nrhs"], 1 << i["n"], i["seed"] + 2) for i in inst]
        st["psi"] = psi
        st["B"] = capi.Batch([_matrix(i, i["seed"]) for i in inst], [p[0] for p in psi], [p[1] for p in psi])
        st["B"].set_horner(case["horner"])
    elif op in ("spgemm", "expm"):
        st["A"] = _matrix(case, seed)
    elif op == "spmm_dia":
        st["dia"] = _dia(case, seed)
        st["C"] = torch.empty(case["rows"], case["right"], device="cuda", dtype=st["dia"][2].dtype)
    elif op == "mlp":
        w, st["batches"] = _network(case, seed)
        st["net"] = capi.Mlp(0)
        st["net"].set_params(w)
        st["loss"] = [torch.empty(case["batch"], device="cuda") for _ in st["batches"]]
    return st


# ---- one pass --------------------------------------------------------------------------------------------


def run(st):
    case, L = st["case"], st["L"]
    op = case["op"]
    if op == "spmv":
        (xr, xi), (yr, yi), A = st["x"], st["y"], st["A"]
        if case["nrhs"] > 1:
            capi.check(L.diaq_spmm(A.h, case["nrhs"], xr.data_ptr(), xi.data_ptr(), xr.shape[1], yr.data_ptr(),
                                   yi.data_ptr(), yr.shape[1], None))
        else:
            f = L.diaq_spmv_c if case["prec"] == "c64" else L.diaq_spmv_z
            capi.check(f(A.h, xr.data_ptr(), xi.data_ptr(), yr.data_ptr(), yi.data_ptr(), None))
        return [yr, yi]
    if op == "ham_sim":
        (xr, xi), (yr, yi) = st["x"], st["y"]
        capi.check(L.diaq_ham_sim(st["A"].h, xr.data_ptr(), xi.data_ptr(), case["dt"] * case["steps"], case["steps"],
                                  case["m"], yr.data_ptr(), yi.data_ptr(), None))
        return [yr, yi]
    if op == "evolve":
        pr, pi = st["psi"]
        st["E"].run(pr, pi, pr.shape[1], case["dt"], case["steps"], case["s"], case["m"])
        return [pr, pi]
    if op == "batch":
        k = case["inst"]
        st["B"].run(case["dt"], [0] * k, [case["m"]] * k, case["steps"])
        return [list(p) for p in st["psi"]]
    if op == "spgemm":
        out = ctypes.c_void_p()
        capi.check(L.diaq_spgemm(st["A"].h, st["A"].h, 0, None, ctypes.byref(out)))
        C = capi.Matrix(out)
        total = C.info()[3]
        re = torch.empty(total, device="cuda", dtype=torch.float64)
        im = torch.empty(total, device="cuda", dtype=torch.float64)
        capi.check(L.diaq_matrix_download(C.h, re.data_ptr(), im.data_ptr(), 1, None))
        return [C.offsets(), re, im]
    if op == "expm":
        out = ctypes.c_void_p()
        capi.check(L.diaq_expm_negative(st["A"].h, case["t"], 100, 1.0, 1e-12, 1, None, ctypes.byref(out), None, None))
        U = capi.Matrix(out)
        N = 1 << case["n"]
        dense = torch.empty(N, N, device="cuda", dtype=torch.complex128)
        capi.check(L.diaq_matrix_to_dense(U.h, dense.data_ptr(), 1, None))
        return [dense]
    if op == "spmm_dia":
        off, vals, B = st["dia"]
        capi.check(L.diaq_spmm_dia_device(off.data_ptr(), vals.data_ptr(), len(off), case["rows"], case["cols"],
                                          B.data_ptr(), case["right"], st["C"].data_ptr(), 1 if case["cplx"] else 0,
                                          None))
        return [st["C"]]
    for (X, ys, ym), loss in zip(st["batches"], st["loss"]):
        st["net"].train_step(X, ys, ym, 2e-3, loss)
    return [st["net"].params(), st["loss"]]


# ---- the work of a pass ------------------------------------------------------------------------------------


def _nonzeros(case):
    """(nonzeros, multiply-adds per nonzero and state, values per nonzero): real entries need one
    value and two multiply-adds, complex ones two and four."""
    if case["kind"] == "band":
        off = _band_offsets(case)
        return sum(_length(case["rows"], case["cols"], d) for d in off), 4, 2
    n, N = case["n"], 1 << case["n"]
    if case["kind"] == "xxz":
        return N + n * N // 2, 2, 1
    if case["kind"] == "tfim":
        return N + n * N, 2, 1
    return len(set(_strings("pauli", n, 1)[1].tolist())) * N, 4, 2


def _band_offsets(case):
    r = np.random.default_rng(1)
    return np.unique(np.concatenate([[0], r.integers(-(case["rows"] - 1), case["cols"], case["nd"] - 1)])).tolist()


def _product_work(case, word, k):
    """One product of the matrix with k vectors, the matrix in words of `word` bytes."""
    nnz, macs, vals = _nonzeros(case)
    rows, cols = _shape(case)
    return nnz * vals * word, 2 * macs * nnz * k, (rows + cols) * k


def _passes(operands, terms):
    """Bytes of `terms` Taylor terms, each a product over all rows: the operands come from memory
    once if they stay on the chip between terms, else for every term."""
    return operands * (terms if operands > 100e6 else 1)


def work(case):
    op = case["op"]
    if op == "spmv":
        word = SIZE[case["prec"]] // 2
        m, f, v = _product_work(case, word, case["nrhs"])
        return {"bytes": m + 2 * word * v, "flops": f}
    if op in ("ham_sim", "evolve"):
        word = 8 if case.get("mode", "c128") == "c128" else 4
        m, f, v = _product_work(case, word, case.get("nrhs", 1))
        terms = case["steps"] * case["m"] * (1 << case.get("s", 0))
        return {"bytes": _passes(m + 2 * word * v, terms), "flops": terms * f}
    if op == "batch":
        word = SIZE[case["prec"]] // 2
        total = {"bytes": 0, "flops": 0}
        for i in _instances(case, 1):
            m, f, v = _product_work(i, word, i["nrhs"])
            total["bytes"] += _passes(m + 2 * word * v, case["steps"] * case["m"])
            total["flops"] += case["steps"] * case["m"] * f
        return total
    if op == "spgemm":  # H read, and the result's stored values written as float64 planes
        N, n = 1 << case["n"], case["n"]
        nnz, macs, vals = _nonzeros(case)
        per_row = nnz / N
        x = set(_strings(case["kind"], n, 1)[1].tolist())
        offs = set()
        for a in x:
            bits = [1 << p for p in range(n) if a >> p & 1]
            sums = {0}
            for b in bits:
                sums = {s + b for s in sums} | {s - b for s in sums}
            offs |= {s for s in sums if case["kind"] != "xxz" or len(bits) < 2 or abs(s) == abs(bits[0] - bits[-1])}
        out = sum(_length(N, N, d) for d in {a + b for a in offs for b in offs} if abs(d) < N)
        return {"bytes": nnz * vals * SIZE[case["prec"]] // 2 + 16 * out, "flops": 2 * (macs // 2) ** 2 * nnz * per_row}
    if op == "expm":  # the operator written once; at least one product of two full matrices
        N = 1 << case["n"]
        return {"bytes": 16 * N * N, "flops": 8 * N ** 3}
    if op == "spmm_dia":
        w = 16 if case["cplx"] else 8
        off = _band_offsets(case)
        stored = sum(_length(case["rows"], case["cols"], d) for d in off)
        return {"bytes": w * (stored + (case["rows"] + case["cols"]) * case["right"]),
                "flops": (8 if case["cplx"] else 2) * stored * case["right"]}
    macs = 16 * 64 + 64 * 64 + 64 * 51
    return {"bytes": case["steps"] * (case["batch"] * (16 + 3) * 4 + 7 * 4 * macs), "flops": case["steps"] * 6 * macs * case["batch"]}


# ---- the same in 64 bits, in plain torch ---------------------------------------------------------------------


class _Pauli:
    """H as one factor vector per flip mask: (H v)[b ^ x] += D_x[b] v[b]."""

    def __init__(self, kind, n, seed):
        c, xs, zs = _strings(kind, n, seed)
        self.b = torch.arange(1 << n, device="cuda")
        self.D = {}
        for ck, x, z in zip(c.tolist(), xs.tolist(), zs.tolist()):
            p = self.b & z
            for s in (32, 16, 8, 4, 2, 1):
                p = p ^ (p >> s)
            f = ck * 1j ** (bin(x & z).count("1") % 4)
            d = (1 - 2 * (p & 1)).to(torch.complex128) * f
            self.D[x] = self.D[x] + d if x in self.D else d

    def apply(self, v):
        y = torch.zeros_like(v)
        for x, d in self.D.items():
            y += (d * v)[..., self.b ^ x]
        return y

    def diagonals(self):
        """{offset: values by row} (zero where the diagonal has no row)."""
        out = {}
        for x, d in self.D.items():
            rows_val = d[self.b ^ x]     # the value of (row, row ^ x)
            off = (self.b ^ x) - self.b
            for o in torch.unique(off).tolist():
                v = torch.where(off == o, rows_val, torch.zeros_like(rows_val))
                out[o] = out[o] + v if o in out else v
        return {o: v for o, v in out.items() if bool((v != 0).any())}


def _taylor(H, v, dt, steps, s, m):
    tau = dt / (1 << s)
    for _ in range(steps << s):
        term, acc = v, v.clone()
        for k in range(1, m + 1):
            term = H.apply(term) * (-1j * tau / k)
            acc += term
        v = acc
    return v


def _planes(v):
    return [v.real.contiguous(), v.imag.contiguous()]


def exact(case, seed):
    op = case["op"]
    if op == "spmv":
        xr, xi = _vectors(case, seed)
        x = torch.complex(xr.double(), xi.double())
        if case["kind"] != "band":
            return _planes(_Pauli(case["kind"], case["n"], seed).apply(x))
        rows, cols = _shape(case)
        off, re, im = _band(case, seed)
        y = torch.zeros(case["nrhs"], rows, device="cuda", dtype=torch.complex128)
        p = 0
        for d in off.tolist():
            n, lo = _length(rows, cols, d), max(0, -d)
            y[:, lo:lo + n] += torch.complex(re[p:p + n], im[p:p + n]) * x[:, lo + d:lo + d + n]
            p += n
        return _planes(y)
    if op in ("ham_sim", "evolve"):
        v = torch.complex(*_states(case.get("nrhs", 1), 1 << case["n"], seed + 2))
        H = _Pauli(case["kind"], case["n"], seed)
        return _planes(_taylor(H, v, case["dt"], case["steps"], case.get("s", 0), case["m"]))
    if op == "batch":
        out = []
        for i in _instances(case, seed):
            v = torch.complex(*_states(i["nrhs"], 1 << i["n"], i["seed"] + 2))
            out.append(_planes(_taylor(_Pauli(i["kind"], i["n"], i["seed"]), v, case["dt"], case["steps"], 0, case["m"])))
        return out
    if op == "spgemm":
        N = 1 << case["n"]
        A = _Pauli(case["kind"], case["n"], seed).diagonals()
        C = {}
        for da, a in A.items():
            lo, hi = max(0, -da), min(N, N - da)
            for db, b in A.items():
                if abs(da + db) >= N:
                    continue
                c = C.get(da + db)
                if c is None:
                    c = C[da + db] = torch.zeros(N, device="cuda", dtype=torch.complex128)
                c[lo:hi] += a[lo:hi] * b[lo + da:hi + da]
        parts = [C[d][max(0, -d):max(0, -d) + _length(N, N, d)] for d in sorted(C)]
        C.clear()
        re = torch.cat([p.real for p in parts])
        return [None, re, torch.cat([p.imag for p in parts])]
    if op == "expm":
        N = 1 << case["n"]
        H = torch.zeros(N, N, device="cuda", dtype=torch.complex128)
        r = torch.arange(N, device="cuda")
        for x, d in _Pauli(case["kind"], case["n"], seed).D.items():
            H[r ^ x, r] += d
        return [torch.linalg.matrix_exp(-1j * case["t"] * H)]
    if op == "spmm_dia":
        off, vals, B = _dia(case, seed)
        C = torch.zeros(case["rows"], case["right"], device="cuda", dtype=B.dtype)
        for k, d in enumerate(off.tolist()):
            n, lo = _length(case["rows"], case["cols"], d), max(0, -d)
            C[lo:lo + n] += vals[k, lo:lo + n, None] * B[lo + d:lo + d + n]
        return [C]
    return _train64(case, seed)


def _train64(case, seed):
    flat, batches = _network(case, seed)
    p, at = [], 0
    for shape in ((16, 64), (64,), (64, 64), (64,), (64, 51), (51,)):
        k = math.prod(shape)
        p.append(torch.from_numpy(flat[at:at + k].astype(np.float64).reshape(shape)).cuda().requires_grad_())
        at += k
    m, v, losses = [torch.zeros_like(w) for w in p], [torch.zeros_like(w) for w in p], []
    ce = torch.nn.functional.cross_entropy
    for t, (X, ys, ym) in enumerate(batches, 1):
        a = torch.relu(X.double() @ p[0] + p[1])
        lg = torch.relu(a @ p[2] + p[3]) @ p[4] + p[5]
        loss = ce(lg[:, :21], ys.long(), reduction="none") + ce(lg[:, 21:], ym.long() - 1, reduction="none")
        losses.append(loss.detach())
        grads = torch.autograd.grad(loss.mean(), p)
        with torch.no_grad():
            for w, g, mi, vi in zip(p, grads, m, v):
                mi.mul_(0.9).add_(g, alpha=0.1)
                vi.mul_(0.999).addcmul_(g, g, value=0.001)
                w -= 2e-3 * (mi / (1 - 0.9 ** t)) / ((vi / (1 - 0.999 ** t)).sqrt() + 1e-8)
    return [torch.cat([w.detach().reshape(-1) for w in p]), losses]

"""What a user of this framework has it do, as measurable cases.

Each case is one call (or the one short sequence of calls) that a program
makes through `spined`: products with a prepared Hamiltonian, ground-state and
few-lowest-states solves, the batched solve, and the passes of the learned
start vector. `exact` gives the same results in 64 bits from plain torch code
over the whole space of spin configurations, where that is small enough.
"""
from __future__ import annotations

import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "spin-ed_gb300"))

from spined import internal as I  # noqa: E402
from spined import lattices  # noqa: E402
from spined.learned import Mlp, Samples  # noqa: E402
from spined.model import build_model  # noqa: E402

DTYPES = {"f32": torch.float32, "f64": torch.float64, "c64": torch.complex64, "c128": torch.complex128}


def listed():
    return [
        # One product with a small ring's Hamiltonian (the README-sized
        # observables, a step of a user's own iteration): latency is what counts.
        {"name": "apply_f64_chain24", "kind": "apply", "lattice": "chain", "n": 24, "dtype": "f64", "block": 1},
        # The product that the headline 6x6 solve consists of.
        {"name": "apply_f64_square6", "kind": "apply", "lattice": "square", "n": 36, "dtype": "f64", "block": 1},
        # datatype: float32 of a configuration file.
        {"name": "apply_f32_chain32", "kind": "apply", "lattice": "chain", "n": 32, "dtype": "f32", "block": 1},
        # A block of vectors (max_primme_block_size), J1-J2 ring.
        {"name": "apply_f64x8_chain30", "kind": "apply", "lattice": "chain", "n": 30, "dtype": "f64", "block": 8,
         "j2": 0.3},
        # A momentum sector: complex characters and vectors.
        {"name": "apply_c128_chain28_k3", "kind": "apply", "lattice": "chain", "n": 28, "dtype": "c128", "block": 1,
         "momentum": 3},
        # The whole small solve: basis, operator, ground state, from nothing.
        {"name": "solve_chain24", "kind": "solve", "lattice": "chain", "n": 24, "nev": 1},
        # The headline: the 6x6 torus from nothing to its ground state.
        {"name": "solve_square6", "kind": "solve", "lattice": "square", "n": 36, "nev": 1},
        # Several lowest states (number_vectors) of a prepared J1-J2 ring.
        {"name": "eigh4_chain28", "kind": "eigh", "lattice": "chain", "n": 28, "nev": 4, "j2": 0.3},
        # Thick restart with few stored vectors, FP32-stored with FP64
        # refinement: the form for systems whose Krylov basis fills the memory.
        {"name": "eigh_thick_mixed_chain32", "kind": "eigh", "lattice": "chain", "n": 32, "nev": 1,
         "max_basis": 16, "mixed": True},
        # Many rings of uneven size at once, four lowest states each.
        {"name": "batch128_16to28", "kind": "batch", "count": 128, "n_min": 16, "n_max": 28},
        # One training batch of the learned start vector: forward and backward.
        {"name": "mlp_grad_h256_4096", "kind": "mlp_grad", "n": 36, "hidden": 256, "samples": 4096},
        # Its inference over every representative of the 6x6 torus.
        {"name": "mlp_start_h256_square6", "kind": "mlp_start", "lattice": "square", "n": 36, "hidden": 256},
    ]


def draw(rng):
    kind = rng.choice(["apply"] * 5 + ["solve"] * 2 + ["eigh"] * 2 + ["batch", "mlp_grad", "mlp_start"])
    if kind == "apply":
        c = {"kind": kind, "lattice": "chain", "n": rng.randint(20, 32)}
        c["dtype"] = rng.choice(["f64", "f64", "f64", "f32", "c128", "c64"])
        c["block"] = rng.choice([1, 1, 2, 3, 4, 5, 7, 8, 12, 16])
        if rng.random() < 0.3:
            c["lattice"], c["n"] = "rect", rng.choice([20, 24, 28, 30])
        elif rng.random() < 0.5:
            c["j2"] = round(rng.uniform(0.05, 0.6), 3)
        if c["lattice"] == "chain" and c["dtype"].startswith("c") and rng.random() < 0.6:
            c["n"] = min(c["n"], 28)
            c["momentum"] = rng.randint(1, c["n"] // 2)
        if c["block"] > 4:
            c["n"] = min(c["n"], 30)
        return c
    if kind == "solve":
        if rng.random() < 0.4:
            return {"kind": kind, "lattice": "rect", "n": rng.choice([16, 20, 24, 28, 30]), "nev": rng.choice([1, 2])}
        return {"kind": kind, "lattice": "chain", "n": rng.randint(14, 32), "nev": 1,
                "j2": round(rng.uniform(0.05, 0.5), 3)}
    if kind == "eigh":
        c = {"kind": kind, "lattice": "chain", "n": rng.randint(18, 30), "nev": rng.choice([1, 2, 3, 4, 6]),
             "j2": round(rng.uniform(0.05, 0.45), 3)}
        if rng.random() < 0.4:
            c.update(nev=1, max_basis=rng.choice([12, 16, 24, 32]), mixed=rng.random() < 0.5)
        return c
    if kind == "batch":
        a = rng.choice([12, 14, 16, 18])
        return {"kind": kind, "count": rng.randint(8, 128), "n_min": a, "n_max": rng.choice([20, 22, 24, 26])}
    if kind == "mlp_grad":
        return {"kind": kind, "n": rng.randint(16, 40), "hidden": rng.choice([128, 256, 512]),
                "samples": int(2 ** rng.uniform(8, 16))}
    return {"kind": kind, "lattice": rng.choice(["chain", "rect"]), "n": rng.choice([24, 28, 30]),
            "hidden": rng.choice([128, 256, 512])}


# ------------------------------------------------------------------ models --

def _model(case, rng):
    """The lattice description: couplings from the seed, J1 near 1."""
    n, j1, j2 = case["n"], float(rng.uniform(0.8, 1.2)), case.get("j2", 0.0)
    kind = case["lattice"]
    if kind == "chain":
        k = case.get("momentum", 0)
        m = lattices.heisenberg_chain(n, momentum=k, parity=None if k else 0, spin_inversion=1, j2=j2)
    elif kind == "square":
        m = lattices.heisenberg_square(math.isqrt(n), j2=j2)
    else:
        ly = max(d for d in range(3, math.isqrt(n) + 1) if n % d == 0)
        lx = n // ly
        m = lattices.Model(f"rect{lx}x{ly}", n, n // 2, 1, [(g, 0) for g in lattices.rect_translations(lx, ly)],
                           [(lattices.HEISENBERG, lattices.rect_bonds(lx, ly))])
    m.terms = [([[j1 * v for v in row] for row in mat], sites) for mat, sites in m.terms]
    return m


def _dimension(case):
    """About how many representatives the sector has."""
    n, kind = case["n"], case["lattice"]
    order = n if case.get("momentum") else {"chain": 2 * n, "square": 8 * n, "rect": n}[kind]
    return max(1.0, math.comb(n, n // 2) / (order * (2 if n % 2 == 0 else 1)))


def _elements(case):
    """About how many off-diagonal elements one product has."""
    n = case["n"]
    bonds = (n if case["lattice"] == "chain" else 2 * n) * (2 if case.get("j2") else 1)
    return _dimension(case) * bonds * 2 * (n // 2) * (n - n // 2) / (n * (n - 1))


def _batch_models(case, rng):
    sizes = np.random.default_rng(case["count"])  # the mix of sizes belongs to the case
    ns = sizes.choice(np.arange(case["n_min"], case["n_max"] + 1, 2), size=case["count"])
    return [lattices.heisenberg_chain(int(n), j2=float(j))
            for n, j in zip(ns, rng.uniform(0.02, 0.6, size=case["count"]))]


def _words(n, count, rng):
    """Random configurations of n spins with n // 2 up."""
    up = np.argsort(rng.random((count, n)), axis=1)[:, : n // 2]
    return np.bitwise_or.reduce(np.uint64(1) << up.astype(np.uint64), axis=1)


def _input_vectors(case, D, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    dt = DTYPES[case["dtype"]]
    real = torch.float64 if dt in (torch.float64, torch.complex128) else torch.float32
    shape = (case["block"], D) + ((2,) if dt.is_complex else ())
    x = torch.randn(shape, generator=g, device="cuda", dtype=real)
    x = torch.view_as_complex(x) if dt.is_complex else x
    x = (x / x.abs().square().sum(dim=1, keepdim=True).sqrt()).to(dt)
    return x[0] if case["block"] == 1 else x.t()  # column-major block


def _weights(case, seed):
    rng = np.random.default_rng([seed, 7])
    n, h = case["n"], case["hidden"]
    parts = [rng.standard_normal((h, n)) / math.sqrt(n), 0.1 * rng.standard_normal(h),
             rng.standard_normal((h, h)) / math.sqrt(h), 0.1 * rng.standard_normal(h),
             rng.standard_normal((2, h)) / math.sqrt(h), 0.1 * rng.standard_normal(2)]
    return np.concatenate([p.ravel() for p in parts]).astype(np.float32)


def _samples(case, seed):
    rng = np.random.default_rng([seed, 11])
    s = case["samples"]
    return Samples(_words(case["n"], s, rng), rng.normal(-4.0, 1.5, s).astype(np.float32),
                   (rng.random(s) < 0.5).astype(np.float32))


# --------------------------------------------------------------- the cases --

def prepare(case, seed):
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    if kind == "apply":
        b = build_model(_model(case, rng))
        b.hamiltonian.prepare()
        x = _input_vectors(case, I.get_number_states(b.basis), seed)
        y = torch.empty_like(x)  # keeps the block's column-major layout
        return {"case": case, "built": b, "x": x, "y": y}
    if kind == "solve":
        return {"case": case, "model": _model(case, rng), "seed": int(rng.integers(1, 1 << 30))}
    if kind == "eigh":
        b = build_model(_model(case, rng))
        b.hamiltonian.prepare()
        out = torch.empty((case["nev"], I.get_number_states(b.basis)), dtype=torch.float64, device="cuda").t()
        return {"case": case, "built": b, "out": out, "seed": int(rng.integers(1, 1 << 30))}
    if kind == "batch":
        built = [build_model(m) for m in _batch_models(case, rng)]
        for b in built:
            b.hamiltonian.prepare()
        return {"case": case, "built": built, "seed": int(rng.integers(1, 1 << 30))}
    net = Mlp(case["n"], case["hidden"], sign_mask=0x5555555555555555 & ((1 << case["n"]) - 1))
    net.set_params(_weights(case, seed))
    if kind == "mlp_grad":
        return {"case": case, "net": net, "samples": _samples(case, seed)}
    b = build_model(_model(case, rng))
    out = torch.empty(I.get_number_states(b.basis), dtype=torch.float64, device="cuda")
    return {"case": case, "net": net, "built": b, "out": out}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "apply":
        I.inplace_apply(state["built"].hamiltonian, state["x"], state["y"])
        return state["y"]
    if kind == "solve":
        b = build_model(state["model"])
        r = I.eigh(b.hamiltonian, nev=case["nev"], seed=state["seed"])
        return {"states": I.basis_get_states(b.basis).view(np.int64), "eigenvalues": r.eigenvalues,
                "eigenvectors": r.eigenvectors}
    if kind == "eigh":
        r = I.eigh(state["built"].hamiltonian, nev=case["nev"], seed=state["seed"], out=state["out"],
                   max_basis=case.get("max_basis", 0),
                   precision=I.L.SED_PRECISION_MIXED if case.get("mixed") else I.L.SED_PRECISION_FP64)
        return {"eigenvalues": r.eigenvalues, "eigenvectors": state["out"]}
    if kind == "batch":
        # a scan of the lowest levels: the program wants the eigenvalues
        r = I.eigh_batched([b.hamiltonian for b in state["built"]], nev=4, seed=state["seed"], vectors=False)
        return r.eigenvalues
    if kind == "mlp_grad":
        loss, grads = state["net"].loss_grad(state["samples"])
        return {"loss": loss, "grads": grads}
    return state["net"].start_vector(state["built"].basis, out=state["out"])


def work(case):
    kind = case["kind"]
    if kind in ("mlp_grad", "mlp_start"):
        n, h = case["n"], case["hidden"]
        params = h * n + h + h * h + h + 2 * h + 2
        if kind == "mlp_grad":
            s = case["samples"]
            return {"bytes": 16.0 * s + 8.0 * params, "flops": 6.0 * s * (h * n + h * h + 2 * h)}
        D = _dimension(case)
        return {"bytes": 16.0 * D + 4.0 * params, "flops": 2.0 * D * (h * n + h * h + 2 * h)}
    if kind == "batch":
        total = {"bytes": 0.0, "flops": 0.0}
        for m in _batch_models(case, np.random.default_rng(0)):
            w = _product({"lattice": "chain", "n": m.number_spins, "j2": 0.3}, 8, 4)
            total = {k: total[k] + 40 * w[k] for k in total}  # some 40 block products each
        return total
    size = {"f32": 4, "f64": 8, "c64": 8, "c128": 16}[case.get("dtype", "f64")]
    w = _product(case, size, case.get("block", 1))
    if kind == "apply":
        return w
    steps = 50 + 25 * (case["nev"] - 1)  # about the products that a Krylov method needs
    return {"bytes": steps * w["bytes"] + 8 * _dimension(case) * (1 + case["nev"]), "flops": steps * w["flops"]}


def _product(case, size, block):
    """One product: an index per element, the diagonal, x and y once; a
    multiplication per element and column is an addition where the element is
    plus or minus a common factor."""
    D, E = _dimension(case), _elements(case)
    return {"bytes": 4 * E + D * (8 + 2 * size * block), "flops": 2 * E * block * (2 if size == 16 else 1)}


# ------------------------------------------------------- the same in 64 bits --

_DEV = "cuda" if torch.cuda.is_available() else "cpu"
_MOST_WORDS = 610_000_000  # the largest space that is enumerated here


def _all_words(n, k):
    """All n-bit words with k bits set, ascending."""
    table = {(0, 0): torch.zeros(1, dtype=torch.int64, device=_DEV)}
    for m in range(1, n + 1):
        new = {}
        for w in range(max(0, k - (n - m)), min(m, k) + 1):
            low, high = table.get((m - 1, w)), table.get((m - 1, w - 1))
            parts = ([low] if low is not None else []) + ([high | (1 << (m - 1))] if high is not None else [])
            new[(m, w)] = torch.cat(parts)
        table = new
    return table[(n, k)]


def _group(model):
    """All (permutation, flip, character) of the symmetry group: a word x goes
    to the word whose bit i is bit permutation[i] of x."""
    n = model.number_spins
    elements = {tuple(range(n)): 1.0 + 0.0j}
    gens = []
    for p, sector in model.symmetries:
        q, period = list(p), 1
        while q != list(range(n)):
            q, period = [q[i] for i in p], period + 1
        gens.append((tuple(p), np.exp(-2j * np.pi * sector / period)))
    todo = list(elements)
    while todo:
        a = todo.pop()
        for p, c in gens:
            b = tuple(a[i] for i in p)
            if b not in elements:
                elements[b] = elements[a] * c
                todo.append(b)
    flips = [(False, 1.0)] + ([(True, float(model.spin_inversion))] if model.spin_inversion else [])
    return [(p, f, c * s) for p, c in elements.items() for f, s in flips]


def _image(words, p, flip, n):
    out = torch.zeros_like(words)
    runs, i = [], 0  # runs of consecutive bits move together
    while i < n:
        j = i
        while j + 1 < n and p[j + 1] == p[j] + 1:
            j += 1
        runs.append((i, p[i], j - i + 1))
        i = j + 1
    for to, at, length in runs:
        out |= ((words >> at) & ((1 << length) - 1)) << to
    return out ^ ((1 << n) - 1) if flip else out


class _Sector:
    """Representatives (orbit minima), norms, and every word's representative
    and character, from the whole space of words."""

    def __init__(self, model):
        n = model.number_spins
        group = _group(model)
        words = _all_words(n, model.hamming_weight)
        cand = words
        for p, f, _ in group:
            cand = cand[_image(cand, p, f, n) >= cand]
        total = torch.zeros(len(cand), dtype=torch.complex128, device=_DEV)
        for p, f, c in group:
            total += (_image(cand, p, f, n) == cand).to(torch.complex128) * complex(c)
        keep = total.real > 0.5
        self.reps = cand[keep]
        self.norms = (total.real[keep] / len(group)).sqrt()
        self.words = words
        self.index = torch.full((len(words),), -1, dtype=torch.int64, device=_DEV)
        self.chi = torch.zeros(len(words), dtype=torch.complex128, device=_DEV)
        at = torch.arange(len(self.reps), device=_DEV)
        for p, f, c in group:  # the element that takes the representative to the word
            k = torch.searchsorted(words, _image(self.reps, p, f, n))
            self.index[k] = at
            self.chi[k] = complex(np.conj(c))
        self.n = n

    def matrix(self, terms):
        """(row, column, value) of the off-diagonal elements, and the diagonal."""
        rows, cols, vals = [], [], []
        diag = torch.zeros(len(self.reps), dtype=torch.float64, device=_DEV)
        at = torch.arange(len(self.reps), device=_DEV)
        for mat, sites in terms:
            for i, j in sites:
                anti = ((self.reps >> i) ^ (self.reps >> j)) & 1 == 1
                diag += float(mat[0][0]) + (float(mat[1][1]) - float(mat[0][0])) * anti.double()
                s = torch.searchsorted(self.words, self.reps[anti] ^ ((1 << i) | (1 << j)))
                r, c, chi = at[anti], self.index[s], self.chi[s]
                ok = c >= 0
                r, c, chi = r[ok], c[ok], chi[ok]
                rows.append(r)
                cols.append(c)
                vals.append(float(mat[1][2]) * chi * self.norms[c] / self.norms[r])
        return torch.cat(rows), torch.cat(cols), torch.cat(vals), diag


def _csr(sector, terms, real):
    r, c, v, d = sector.matrix(terms)
    D = len(sector.reps)
    at = torch.arange(D, device=_DEV)
    v = torch.cat([v.real if real else v, d if real else d.to(torch.complex128)])
    m = torch.sparse_coo_tensor(torch.stack([torch.cat([r, at]), torch.cat([c, at])]), v, (D, D))
    return m.coalesce().to_sparse_csr()


def _lowest(matrix, nev):
    """Lowest eigenvalues by Lanczos with full reorthogonalisation."""
    D = matrix.shape[0]
    if D <= 1500:
        return torch.linalg.eigvalsh(matrix.to_dense())[:nev].cpu().numpy()
    g = torch.Generator(device=_DEV).manual_seed(1)
    v = torch.randn(D, generator=g, dtype=torch.float64, device=_DEV)
    V = torch.empty((401, D), dtype=torch.float64, device=_DEV)
    V[0] = v / v.norm()
    alpha, beta = [], []
    for k in range(400):
        w = matrix @ V[k]
        alpha.append(float(V[k] @ w))
        for _ in range(2):
            w = w - V[: k + 1].t() @ (V[: k + 1] @ w)
        beta.append(float(w.norm()))
        V[k + 1] = w / beta[-1]
        if k % 20 == 19:
            T = np.diag(alpha) + np.diag(beta[:-1], 1) + np.diag(beta[:-1], -1)
            ev, S = np.linalg.eigh(T)
            if np.all(np.abs(beta[-1] * S[-1, :nev]) < 1e-9):
                return ev[:nev]
    return None


def exact(case, seed):
    kind = case["kind"]
    if kind == "mlp_grad":
        return _exact_grad(case, seed)
    if kind in ("mlp_start", "batch") or math.comb(case["n"], case["n"] // 2) > _MOST_WORDS:
        return None
    model = _model(case, np.random.default_rng(seed))
    sector = _Sector(model)
    if kind == "apply":
        real = not case.get("momentum")
        x = _input_vectors(case, len(sector.reps), seed).to(torch.complex128)
        r, c, v, d = sector.matrix(model.terms)
        x = x.reshape(len(x), -1)
        y = torch.empty((x.shape[1], x.shape[0]), dtype=torch.complex128, device=_DEV)
        for k in range(x.shape[1]):
            y[k] = (d * x[:, k]).index_add_(0, r, v * x[c, k])
        y = y[0] if case["block"] == 1 else y.t()
        return y.real.contiguous() if real and not case["dtype"].startswith("c") else y
    ev = _lowest(_csr(sector, model.terms, True), case["nev"])
    if kind == "solve":
        return {"states": sector.reps, "eigenvalues": ev, "eigenvectors": None}
    return {"eigenvalues": ev, "eigenvectors": None}


def _exact_grad(case, seed):
    n, h, s = case["n"], case["hidden"], _samples(case, seed)
    p = torch.tensor(_weights(case, seed), dtype=torch.float64, device=_DEV, requires_grad=True)
    w1, b1, w2, b2, w3, b3 = torch.split(p, [h * n, h, h * h, h, 2 * h, 2])
    states = torch.from_numpy(s.states.view(np.int64)).to(_DEV)
    bits = ((states[:, None] >> torch.arange(n, device=_DEV)) & 1).double()
    h1 = torch.tanh((2.0 * bits - 1.0) @ w1.view(h, n).t() + b1)
    h2 = torch.tanh(h1 @ w2.view(h, h).t() + b2)
    out = h2 @ w3.view(2, h).t() + b3
    mask = 0x5555555555555555 & ((1 << n) - 1)
    odd = torch.from_numpy(np.array([bin(int(v) & mask).count("1") & 1 for v in s.states])).to(_DEV)
    positive = torch.from_numpy(s.t_sign).to(_DEV).double()
    agrees = torch.where(odd == 1, 1.0 - positive, positive)
    t = torch.from_numpy(s.t_abs).to(_DEV).double()
    loss = ((out[:, 0] - t).square()
            + torch.nn.functional.binary_cross_entropy_with_logits(out[:, 1], agrees, reduction="none")).mean()
    loss.backward()
    return {"loss": float(loss.detach()), "grads": p.grad}

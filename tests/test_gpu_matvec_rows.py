"""Products row by row: factors with few significant bits, vectors whose
entries differ much in size, columns alone and in blocks
(src/SpinED/Internal.hs:411-429), against the oracle's matrix."""
import numpy as np
import pytest

from _models import both
from spined import lattices
from spined import _lib as L

pytestmark = pytest.mark.gpu


def f32(v):
    return float(np.float32(v))


def ring(n, j1, j2, k=0, dm=0.0, inversion=None, parity=None):
    """Ring with exchange j1, j2 and a Dzyaloshinskii-Moriya term along z on the nearest bonds."""
    bond = [[j1, 0, 0, 0], [0, -j1, 2 * j1 + 1j * dm, 0], [0, 2 * j1 - 1j * dm, -j1, 0], [0, 0, 0, j1]]
    terms = [(bond, lattices.chain_bonds(n, 1))]
    if j2:
        terms.append(([[j2 * v for v in row] for row in lattices.HEISENBERG], lattices.chain_bonds(n, 2)))
    syms = [(lattices.chain_translation(n), k)] + ([(lattices.chain_parity(n), parity)] if parity is not None else [])
    return lattices.Model(f"ring{n}k{k}", n, n // 2, inversion, syms, terms)


class Case:
    def __init__(self, sed, oracle, model):
        self.built, ob, oop = both(sed, oracle, model)
        self.op, self.D, self.A = self.built.hamiltonian, len(ob.reps), oop.sparse()
        self.op.prepare(L.SED_FORM_STREAM)
        self.abs = abs(self.A)
        self.R = int(np.diff(self.A.tocsr().indptr).max())

    def check(self, x, y):
        """Every part of every entry: both sides' FP64 sums err by at most (R +
        8) 2^-53 of the absolute terms (R + 1 products and additions, the
        factors by a few units), and an FP32 part is rounded once (2^-24) from
        a value that is within 2^-30 of that."""
        single = y.dtype in (np.float32, np.complex64)
        want = self.A @ x.astype(np.complex128)
        real = not np.iscomplexobj(self.A.data) or not np.any(self.A.data.imag)
        # complex factors mix the parts of x
        size = np.abs(x).astype(np.float64)
        for part in ("real", "imag") if np.iscomplexobj(y) else ("real",):
            terms = self.abs @ (np.abs(getattr(x, part)).astype(np.float64) if real else size)
            w = getattr(want, part)
            tol = (self.R + 8) * 2.0 ** -52 * terms
            if single:
                tol = tol + (2.0 ** -24 + 2.0 ** -29) * np.abs(w) + 2.0 ** -149
            d = np.abs(getattr(y, part).astype(np.float64) - w)
            worst = np.argmax(d - tol)
            assert d[worst] <= tol[worst], (part, worst, d[worst], tol[worst], w[worst])


_cases = {}


@pytest.fixture
def case(sed, oracle):
    def get(name, make):
        if name not in _cases:
            _cases[name] = Case(sed, oracle, make())
        return _cases[name]
    yield get


@pytest.fixture(scope="module", autouse=True)
def _drop():
    yield
    _cases.clear()


# 2.8 M elements: complex64 products take integer sums. Imaginary factors whose FP64 value has 23 or 24 significant bits.
FEW_BITS = {
    "k6_0.3": lambda: ring(24, f32(0.3), f32(0.9), k=6),
    "k6_1+2^-22": lambda: ring(24, 1 + 2.0 ** -22, 0.5, k=6),
    "dm_0.6": lambda: ring(24, f32(0.3), f32(0.9), k=1, dm=f32(0.6)),
}


@pytest.mark.parametrize("dtype", ["complex64", "complex128"])
@pytest.mark.parametrize("name", list(FEW_BITS))
def test_factors_of_few_bits(sed, case, name, dtype):
    import torch
    c = case(name, FEW_BITS[name])
    gen = torch.Generator(device="cuda").manual_seed(5)
    x = torch.randn(c.D, dtype=getattr(torch, dtype), device="cuda", generator=gen)
    y = sed.apply(c.op, x)
    c.check(x.cpu().numpy(), y.cpu().numpy())


# integer sums: FP32 from 2^21 elements of a real operator, complex64 from 2^20 of any
RANGE_MODELS = {
    "real_one": lambda: lattices.heisenberg_chain(28),
    "real_two": lambda: lattices.heisenberg_chain(26, j2=0.3),
    "real_signed": lambda: lattices.heisenberg_chain(26, momentum=13, parity=None, j2=0.4),
    "complex": lambda: ring(24, 1.0, 0.37, k=5),
    "complex_far": lambda: ring(24, 1.0, 0.3 / 300, k=6, dm=0.7),
    "imaginary": lambda: ring(26, 0.0, 0.0, dm=1.1),
}


def vector(kind, D, dtype, seed):
    rng = np.random.default_rng(seed)
    x = rng.normal(size=D) + (1j * rng.normal(size=D) if dtype.startswith("complex") else 0)
    big = rng.random(D) < 1e-3
    if kind == "small":  # most rows couple to entries of 1e-25 only
        x[~big] *= 1e-25
    elif kind == "half":
        x[int(0.6 * D):] *= 1e-25
    elif kind == "sparse":
        x[~big] = 0.0
    elif kind == "small_parts" and dtype.startswith("complex"):
        x = x.real + 1e-22j * x.imag
    elif kind == "zero_part":
        x = x.real + 0j if dtype.startswith("complex") else 0 * x
    return x.astype(dtype)


def with_dtypes(models):
    """FP32 vectors for real operators only."""
    return [(name, dtype) for name in models for dtype in ("float32", "complex64", "complex128")
            if dtype != "float32" or name in ("chain24", "real_one", "real_two", "real_signed")]


@pytest.mark.parametrize("kind", ["plain", "small", "half", "sparse", "small_parts", "zero_part"])
@pytest.mark.parametrize("name,dtype", with_dtypes(RANGE_MODELS))
def test_entries_of_different_size(sed, case, name, dtype, kind):
    """Rows that couple to small entries of the vector only keep the digits
    of those, and rows that couple to zeros are zero."""
    import torch
    c = case(name, RANGE_MODELS[name])
    x = vector(kind, c.D, dtype, 6)
    y = sed.apply(c.op, torch.tensor(x, device="cuda"))
    c.check(x, y.cpu().numpy())


@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
@pytest.mark.parametrize("name,dtype", with_dtypes(["real_two", "complex"]))
def test_non_finite_entry(sed, case, name, dtype, bad):
    """A NaN or an infinity reaches the rows that couple to its entry, and the
    others are as they would be with a zero in its place."""
    import torch
    c = case(name, RANGE_MODELS[name])
    x = vector("plain", c.D, dtype, 8)
    j = c.D // 3
    x[j] = 0
    reached = np.asarray((c.A[:, [j]] != 0).todense()).ravel()
    reached[j] = True
    t = torch.tensor(x, device="cuda")
    t[j] = bad
    y = sed.apply(c.op, t).cpu().numpy()
    assert np.array_equal(np.isfinite(y), ~reached)
    want = sed.apply(c.op, torch.tensor(x, device="cuda")).cpu().numpy()
    y[reached] = want[reached]
    c.check(x, y)


BLOCK_MODELS = {
    "chain24": lambda: lattices.heisenberg_chain(24),
    "real_two": RANGE_MODELS["real_two"],
    "complex": RANGE_MODELS["complex"],
}


@pytest.mark.parametrize("bad", [None, float("nan")])
@pytest.mark.parametrize("name,dtype", with_dtypes(BLOCK_MODELS))
def test_columns_do_not_depend_on_their_block(sed, case, name, dtype, bad):
    """A column's product is the same alone and in a block of any width, also
    beside a column with a NaN."""
    import torch
    c = case(name, BLOCK_MODELS[name])
    gen = torch.Generator(device="cuda").manual_seed(7)
    x = torch.randn(16, c.D, dtype=getattr(torch, dtype), device="cuda", generator=gen).t()
    if bad is not None:
        x[c.D // 3, 1] = bad
    alone = [sed.apply(c.op, x[:, q].contiguous()) for q in range(16)]
    for width in (2, 3, 8, 16):
        y = sed.apply(c.op, x[:, :width])
        for q in range(width):
            assert torch.equal(y[:, q].nan_to_num(123.0), alone[q].nan_to_num(123.0)), (width, q)


def test_wide_products_leave_a_bounded_workspace(sed):
    """Blocks of FP32 and complex vectors: what stays with the operator after
    the call is at most 1 GiB (15.8 M rows: 16 columns would take 2 GB)."""
    import torch
    from spined.model import build_model
    built = build_model(lattices.heisenberg_square(6))
    op, lib = built.hamiltonian, L.load()
    op.prepare(L.SED_FORM_STREAM)
    D = sed.get_number_states(built.basis)
    lib.sed_release_workspace()
    before = lib.sed_device_memory_in_use()
    x = torch.randn(16, D, dtype=torch.float32, device="cuda").t()
    sed.apply(op, x)
    assert lib.sed_device_memory_in_use() - before <= 1 << 30
    x = torch.view_as_complex(torch.randn(4, D, 2, dtype=torch.float32, device="cuda")).t()
    sed.apply(op, x)
    assert lib.sed_device_memory_in_use() - before <= 1 << 30


def test_products_beside_a_captured_one(sed):
    """A captured FP64 product keeps its workspace: FP32 blocks run beside it,
    and replays give the product of what x holds."""
    import ctypes as C
    import torch
    from spined.model import build_model
    lib = L.load()
    plain, held = (build_model(lattices.heisenberg_chain(28)).hamiltonian for _ in range(2))
    held.prepare(L.SED_FORM_STREAM)
    D = sed.get_number_states(held.basis)
    gen = torch.Generator(device="cuda").manual_seed(9)
    x = torch.randn(D, dtype=torch.float64, device="cuda", generator=gen)
    y = torch.zeros_like(x)
    graph = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, capture_error_mode="thread_local"):
        stream = torch.cuda.current_stream().cuda_stream
        sed.check_status(lib.sed_operator_matmat_device(held.ptr, 1, D, 1, C.c_void_p(x.data_ptr()), D,
                                                        C.c_void_p(y.data_ptr()), D, C.c_void_p(stream)))
    z = torch.randn(8, D, dtype=torch.float32, device="cuda", generator=gen).t()
    for scale in (1.0, 1e6, 1e-6):
        x.mul_(scale)
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(y, sed.apply(plain, x))
        w = sed.apply(held, z)
        want = sed.apply(plain, z)
        assert (w - want).abs().max() <= 2.0 ** -22 * want.abs().max()  # both rounded to FP32

"""Precision of the split mixed product output by output: rows of a vector whose elements spread too far for fixed-point
words stay with the FP64 kernel, and the others lose nothing against it."""
import numpy as np
import pytest

from conftest import dev

pytestmark = pytest.mark.gpu

NORB, NA, NB = 8, 4, 4


@pytest.fixture(scope="module")
def system():
    import torch
    from binsim_b200 import cuotf, network as nw
    net = nw.hamiltonian_network(NORB, seed=3, native=True)
    B = cuotf.CuBasis(NORB, NA, NB)
    f = cuotf.CuOTFFunctions(B, cuotf.CuNetwork(net))
    # the matrix that the FP64 kernels apply, column by column: products with one are exact
    H = torch.empty(B.dim, B.dim, dtype=torch.float64, device="cuda")
    e = torch.zeros(B.dim, dtype=torch.float64, device="cuda")
    mp = pytest.MonkeyPatch()
    mp.setenv("BSIM_SIGMA_SPLIT", "0")
    for i in range(B.dim):
        e.zero_()
        e[i] = 1.0
        f.hvec(e, H[i])
    mp.undo()
    return B, f, H.cpu().numpy().T


def _vector(kind, dim):
    rng = np.random.default_rng(4)
    x = rng.normal(size=dim)
    rows = x.reshape(70, 70)
    if kind == "lognormal":
        x *= np.exp(rng.normal(size=dim))
    elif kind == "three_decades":
        x *= 10.0 ** rng.uniform(-3, 0, dim)
    elif kind == "six_decades":
        x *= 10.0 ** rng.uniform(-6, 0, dim)
    elif kind == "leading":           # one leading element in every row, a tail far below
        x *= 10.0 ** rng.uniform(-12, -6, dim)
        rows[np.arange(70), rng.integers(0, 70, 70)] = 1.0
    elif kind == "leading_3":
        x *= 1e-3
        rows[:, 0] = 1.0
    elif kind == "noise":             # a few elements of rounding noise in place of zeros
        rows[:, ::10] *= 1e-17
    return x


@pytest.mark.parametrize("kind", ["normal", "lognormal", "three_decades", "six_decades", "leading", "leading_3", "noise"])
def test_error_against_the_terms_of_each_output(cuda, system, monkeypatch, kind):
    """|error| <= 40 x 2^-53 x sum |H_ij x_j| for every output i: each kernel rounds its sums of at most a few hundred
    terms once a term, to a random walk of about twenty of them, and the words of an accepted row lose less."""
    B, f, H = system
    x = _vector(kind, B.dim)
    ref = (H.astype(np.longdouble) * x).sum(1)
    terms = np.abs(H) @ np.abs(x)
    y = cuda.empty(B.dim, dtype=cuda.float64, device="cuda")
    for split in ("0", "1"):
        monkeypatch.setenv("BSIM_SIGMA_SPLIT", split)
        f.hvec(dev(cuda, x), y)
        assert float((np.abs(y.cpu().numpy() - ref) / terms).max()) <= 40 * 2.0 ** -53, split


@pytest.mark.parametrize("kind", ["six_decades", "leading", "leading_3", "noise"])
def test_wide_rows_are_those_of_the_fp64_kernel(cuda, system, monkeypatch, kind):
    B, f, _ = system
    x = dev(cuda, _vector(kind, B.dim))
    y, z = cuda.empty_like(x), cuda.empty_like(x)
    monkeypatch.setenv("BSIM_SIGMA_SPLIT", "0")
    f.hvec(x, z)
    monkeypatch.setenv("BSIM_SIGMA_SPLIT", "1")
    f.hvec(x, y)
    assert cuda.equal(y, z)


def test_non_finite_elements_reach_what_they_reached(cuda, system, monkeypatch):
    """An infinity or a NaN spoils the outputs that it spoils in the FP64 kernel, and no other."""
    B, f, _ = system
    x = dev(cuda, _vector("normal", B.dim))
    y, z = cuda.empty_like(x), cuda.empty_like(x)
    for bad in (np.inf, -np.inf, np.nan):
        x[1234] = bad
        monkeypatch.setenv("BSIM_SIGMA_SPLIT", "0")
        f.hvec(x, z)
        monkeypatch.setenv("BSIM_SIGMA_SPLIT", "1")
        f.hvec(x, y)
        assert bool(cuda.isfinite(z).any())
        assert cuda.equal(cuda.isfinite(y), cuda.isfinite(z))
        assert cuda.equal(cuda.isnan(y), cuda.isnan(z))


def test_a_wait_that_runs_out_costs_no_result(cuda, system, monkeypatch):
    """The producers of one row fill nothing: its waits run out (20 ms, counted), the row and those after it go to the FP64
    kernel, and the next call is as before."""
    import ctypes as C
    from binsim_b200.cuotf import lib
    B, f, _ = system
    x = dev(cuda, _vector("normal", B.dim))
    y, z, w = (cuda.full_like(x, float("nan")) for _ in range(3))

    def timeouts(reset):
        n = C.c_int32()
        assert lib().bsim_tensor_core_timeouts(C.byref(n), reset) == 0
        return n.value
    timeouts(1)
    monkeypatch.setenv("BSIM_SIGMA_SPLIT", "1")
    f.hvec(x, z)
    for row in (0, 33, 69):
        monkeypatch.setenv("BSIM_SPLIT_DROP_ROW", str(row))
        f.hvec(x, y)
        # the row's elements are its words, within 2^-63 of its largest; both kernels as in the test above
        assert float((y - z).abs().max()) <= 1e-13 * float(z.abs().max())
        assert timeouts(1) >= 1
    monkeypatch.delenv("BSIM_SPLIT_DROP_ROW")
    f.hvec(x, w)
    assert cuda.equal(w, z)
    assert timeouts(0) == 0


@pytest.mark.parametrize("count", [1, 2, 30, 147, 149, 286])
def test_wide_rows_among_others(cuda, monkeypatch, count):
    """A few rows that stay in FP64 share their column chunks among the CTAs, many take one each: 286 rows of 715 columns
    (six chunks), K of 78, thirty singles a row; the rows' elements spread over nine decades, their largest as the others'."""
    from binsim_b200 import cuotf, network as nw
    norb, na, nb = 13, 3, 4
    B = cuotf.CuBasis(norb, na, nb)
    f = cuotf.CuOTFFunctions(B, cuotf.CuNetwork(nw.hamiltonian_network(norb, seed=3, native=True)))
    rng = np.random.default_rng(count)
    x = rng.normal(size=(286, 715))
    rows = rng.permutation(286)[:count]
    x[rows] *= 10.0 ** rng.uniform(-9, 0, (count, 715))
    x = dev(cuda, x.ravel())
    y, z = cuda.full_like(x, float("nan")), cuda.empty_like(x)
    monkeypatch.setenv("BSIM_SIGMA_SPLIT", "0")
    f.hvec(x, z)
    monkeypatch.setenv("BSIM_SIGMA_SPLIT", "1")
    f.hvec(x, y)
    assert float((y - z).abs().max()) <= 1e-13 * float(z.abs().max())
    if count == 286:
        assert cuda.equal(y, z)
    # two windows of Z and column bands find the rows again
    nB = 715
    w = cuda.full_like(x, float("nan"))
    for lo, hi in ((0, 384), (384, nB)):
        f.hvec_cols(x, w, lo, hi)
    assert float((y - w).abs().max()) <= 1e-13 * float(z.abs().max())

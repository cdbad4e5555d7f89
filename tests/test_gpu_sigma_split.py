"""FP64 sigma with its mixed product as split products on the tensor cores (BSIM_SIGMA_SPLIT=1: at every size) against
the oracle and the DMMA kernels (BSIM_SIGMA_SPLIT=0), at the edges of its tiles and on vectors that stress the
fixed-point rows."""
import math

import numpy as np
import pytest

from conftest import dev

pytestmark = pytest.mark.gpu


def _setup(norb, na, nb, seed=3):
    from binsim_b200 import cuotf, network as nw
    net = nw.hamiltonian_network(norb, seed=seed, native=True)
    B = cuotf.CuBasis(norb, na, nb)
    return net, B, cuotf.CuOTFFunctions(B, cuotf.CuNetwork(net))


# connected singles per string: 16 (one 16-row half), 30, 36 (32 + 16), 49 (32 + 32), 65 (passes of 64 + 1); slices of
# 32 K rows: 1 to 3 (all in stages), 5 (slice by slice); columns that end inside a chunk of 128, one to eight chunks
@pytest.mark.parametrize("norb,na,nb", [(8, 4, 4), (10, 2, 6), (11, 5, 5), (12, 6, 5), (14, 7, 2), (18, 5, 1), (18, 2, 2),
                                        (13, 3, 4)])
def test_matches_oracle_and_dmma(cuda, oracle, monkeypatch, norb, na, nb):
    net, B, f = _setup(norb, na, nb)
    x = np.random.default_rng(norb).normal(size=B.dim)
    x /= np.linalg.norm(x)
    ref = oracle.hvec(oracle.basis(norb, na, nb), oracle.network(net), x)
    monkeypatch.setenv("BSIM_SIGMA_SPLIT", "1")   # at every size
    y = cuda.full((B.dim,), float("nan"), dtype=cuda.float64, device="cuda")
    f.hvec(dev(cuda, x), y)
    monkeypatch.setenv("BSIM_SIGMA_SPLIT", "0")
    z = cuda.empty_like(y)
    f.hvec(dev(cuda, x), z)
    scale = np.abs(ref).max()
    # the DMMA kernel with the source row in global memory: the same bits
    monkeypatch.setenv("BSIM_MIXED_ROW_SMEM", "1")
    w = cuda.empty_like(y)
    f.hvec(dev(cuda, x), w)
    monkeypatch.delenv("BSIM_MIXED_ROW_SMEM")
    assert cuda.equal(w, z)
    assert np.abs(y.cpu().numpy() - ref).max() <= 1e-12 * scale
    # both round their sums at 2^-53 of terms no larger than the largest element of H x
    assert float((y - z).abs().max()) <= 1e-13 * scale
    # in column bands (their starts multiples of 128; the beta doubles take another route)
    monkeypatch.setenv("BSIM_SIGMA_SPLIT", "1")
    nB = math.comb(norb, nb)
    w.fill_(float("nan"))
    for lo, hi in ((0, min(nB, 128)), (128, nB)):
        if lo < hi:
            f.hvec_cols(dev(cuda, x), w, lo, hi)
    assert float((y - w).abs().max()) <= 1e-13 * scale


@pytest.mark.parametrize("kind", ["decades", "unit", "tiny", "huge", "zero_rows"])
def test_dynamic_range(cuda, oracle, monkeypatch, kind):
    """Rows of very different size, a unit vector (its products are exact), and vectors near the ends of the exponent
    range: the error stays below that of FP64 sums against the oracle, relative to the largest output."""
    norb, na, nb = 10, 5, 4
    net, B, f = _setup(norb, na, nb)
    rng = np.random.default_rng(2)
    x = rng.normal(size=B.dim)
    if kind == "decades":
        x *= 10.0 ** rng.uniform(-12, 0, B.dim)
    elif kind == "unit":
        x[:] = 0.0
        x[B.hf_index()] = 1.0
    elif kind == "tiny":
        x *= 1e-290
    elif kind == "huge":
        x *= 1e290
    else:
        x.reshape(-1, 210)[::3] = 0.0
    monkeypatch.setenv("BSIM_SIGMA_SPLIT", "1")
    y = cuda.empty(B.dim, dtype=cuda.float64, device="cuda")
    f.hvec(dev(cuda, x), y)
    ref = oracle.hvec(oracle.basis(norb, na, nb), oracle.network(net), x)
    assert np.abs(y.cpu().numpy() - ref).max() <= 1e-13 * np.abs(ref).max()


def test_non_finite_rows_give_nan(cuda, monkeypatch):
    """An infinity or a NaN reaches every output that it reached in the DMMA kernels (as NaN), and the next call on a
    finite vector is clean."""
    net, B, f = _setup(10, 5, 4)
    x = np.random.default_rng(5).normal(size=B.dim)
    y, z, w = (cuda.empty(B.dim, dtype=cuda.float64, device="cuda") for _ in range(3))
    for bad in (np.inf, np.nan):
        xb = x.copy()
        xb[1234] = bad
        monkeypatch.setenv("BSIM_SIGMA_SPLIT", "0")
        f.hvec(dev(cuda, xb), z)
        monkeypatch.setenv("BSIM_SIGMA_SPLIT", "1")
        f.hvec(dev(cuda, xb), y)
        lost = ~cuda.isfinite(z) & cuda.isfinite(y)
        assert not bool(lost.any())
    f.hvec(dev(cuda, x), w)
    assert bool(cuda.isfinite(w).all())


def test_no_wait_gave_up(cuda):
    from binsim_b200.cuotf import lib
    import ctypes as C
    n = C.c_int()
    assert lib().bsim_tensor_core_timeouts(C.byref(n), 0) == 0
    assert n.value == 0

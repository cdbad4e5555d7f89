"""Pure-spin rows with the entries divided among warps (small bases) and one CTA per even chunk of columns (larger
ones): both sides of the line, columns that end inside a tile, FP64 and FP32 bulk, against the oracle."""
import numpy as np
import pytest

from conftest import dev

pytestmark = pytest.mark.gpu


# rows x 1024-column tiles: 2, 70, 462, 495 (below the line of 512), 715 and 792 (above it), 715 x 2: rows of 1287
# columns, two chunks of 161 quads in FP64 and one of 322 in FP32
@pytest.mark.parametrize("norb,na,nb", [(2, 1, 1), (8, 4, 4), (11, 5, 5), (12, 4, 2), (13, 4, 3), (12, 5, 5), (13, 4, 5)])
def test_matches_oracle(cuda, oracle, norb, na, nb):
    from binsim_b200 import cuotf, network as nw
    net = nw.hamiltonian_network(norb, seed=7, native=True)
    B = cuotf.CuBasis(norb, na, nb)
    f = cuotf.CuOTFFunctions(B, cuotf.CuNetwork(net))
    x = np.random.default_rng(norb).normal(size=B.dim)
    x /= np.linalg.norm(x)
    ref = oracle.hvec(oracle.basis(norb, na, nb), oracle.network(net), x)
    scale = np.abs(ref).max()
    y = cuda.full((B.dim,), float("nan"), dtype=cuda.float64, device="cuda")
    f.hvec(dev(cuda, x), y)
    assert np.abs(y.cpu().numpy() - ref).max() <= 1e-12 * scale
    # FP32 bulk: sums of at most a few hundred products of FP32 factors, each rounded at 2^-24
    f.hvec_mixed(dev(cuda, x), y)
    assert np.abs(y.cpu().numpy() - ref).max() <= 1e-5 * scale
    # repeated calls give the same bits: the warps' sums are added in a fixed order
    z = cuda.empty_like(y)
    f.hvec(dev(cuda, x), y)
    f.hvec(dev(cuda, x), z)
    assert bool((y == z).all())


@pytest.mark.parametrize("norb,na,nb", [(12, 5, 5), (13, 3, 6)])
def test_column_bands_give_the_same_bits(cuda, norb, na, nb):
    """Bands whose own rows fall below the line, cut in two ways: the kernel is chosen by the whole side."""
    import math
    from binsim_b200 import cuotf, network as nw
    B = cuotf.CuBasis(norb, na, nb)
    f = cuotf.CuOTFFunctions(B, cuotf.CuNetwork(nw.hamiltonian_network(norb, seed=7, native=True)))
    x = dev(cuda, np.random.default_rng(norb).normal(size=B.dim))
    nB = math.comb(norb, nb)
    out = []
    for cuts in ((0, 128, nB), (0, 640, nB)):
        y = cuda.empty_like(x)
        for lo, hi in zip(cuts, cuts[1:]):
            f.hvec_cols(x, y, lo, hi)
        out.append(y)
    assert cuda.equal(out[0], out[1])

"""Sigma on symmetry-blocked bases (per-row lists) against the oracle."""
import numpy as np
import pytest

from conftest import dev

pytestmark = pytest.mark.gpu


def _masked(norb, sym, seed):
    """A Hamiltonian whose integrals respect the point group."""
    from binsim_b200 import network as nw
    h, g, _ = nw.synthetic_integrals(norb, seed)
    s = np.asarray(sym)
    h = h * ((s[:, None] ^ s[None, :]) == 0)
    g = g * ((s[:, None, None, None] ^ s[None, :, None, None] ^ s[None, None, :, None] ^ s[None, None, None, :]) == 0)
    x, z, c = nw.jw_hamiltonian_terms(h, g)
    return nw.compress_groups(*nw.split_aabb(x, z, norb), c, norb, orbsym=s)


# electron counts at the ends, unequal spins, odd irreps, one- and two-block bases, rows longer than a CTA's 128 columns
@pytest.mark.parametrize("norb,na,nb,sym,nirr,tsym,bits", [
    (4, 1, 3, [0, 1, 0, 1], 2, 1, 32), (5, 0, 2, [0, 1, 1, 0, 1], 2, 0, 32), (6, 6, 1, [0, 1, 2, 3, 0, 1], 4, 2, 64),
    (9, 4, 5, [0, 1, 2, 3, 4, 5, 6, 7, 0], 8, 5, 32), (11, 5, 6, [0, 0, 1, 1, 0, 1, 0, 0, 1, 1, 0], 2, 1, 32),
    (10, 5, 5, [0, 1, 2, 3, 0, 1, 2, 3, 0, 1], 4, 0, 64)])
@pytest.mark.parametrize("symmetric", [True, False])
def test_blocked_sigma(cuda, oracle, norb, na, nb, sym, nirr, tsym, bits, symmetric):
    from binsim_b200 import cuotf, network as nw
    sym = np.asarray(sym, np.int64)
    if symmetric:
        net = _masked(norb, sym, norb)
    else:   # integrals of every irrep: the terms that leave the total irrep drop out
        net = nw.hamiltonian_network(norb, seed=norb)
        net.orbsym = sym
    kw = dict(orbsym=sym, total_sym=tsym, num_irreps=nirr)
    Bo, No = oracle.basis(norb, na, nb, **kw), oracle.network(net)
    B = cuotf.CuBasis(norb, na, nb, string_bits=bits, **kw)
    f = cuotf.CuOTFFunctions(B, cuotf.CuNetwork(net, string_bits=bits))
    assert B.dim == Bo.dim and f.sigma_path()[0] == 0
    x = np.random.default_rng(norb).normal(size=B.dim)
    ref = oracle.hvec(Bo, No, x)
    scale = max(np.abs(ref).max(), 1e-300)
    for call, tol in ((f.hvec, 1e-13), (f.hvec_mixed, 2e-6)):
        y = cuda.full((B.dim,), float("nan"), dtype=cuda.float64, device="cuda")
        call(dev(cuda, x), y)
        assert np.abs(y.cpu().numpy() - ref).max() <= tol * scale


def test_blocked_sigma_with_other_groups(cuda, oracle):
    """Groups that are no part of a two-body Hamiltonian (antisymmetric generators) go through the tile kernel."""
    from binsim_b200 import cuotf, network as nw
    norb, na, nb, sym = 6, 3, 2, np.array([0, 1, 0, 1, 1, 0], np.int64)
    net = nw.ucc_pool(norb).network
    net.orbsym = sym
    kw = dict(orbsym=sym, total_sym=1, num_irreps=2)
    Bo, No = oracle.basis(norb, na, nb, **kw), oracle.network(net)
    B = cuotf.CuBasis(norb, na, nb, **kw)
    f = cuotf.CuOTFFunctions(B, cuotf.CuNetwork(net))
    x = np.random.default_rng(1).normal(size=B.dim)
    ref = oracle.hvec(Bo, No, x)
    y = cuda.empty(B.dim, dtype=cuda.float64, device="cuda")
    f.hvec(dev(cuda, x), y)
    assert np.abs(y.cpu().numpy() - ref).max() <= 1e-13 * np.abs(ref).max()


def test_first_call_inside_a_capture(cuda, oracle):
    """The first sigma inside a stream capture takes the tile kernel, which makes nothing (its tile table comes from the
    diagonal); the captured graph stays good after later calls have made the lists."""
    from binsim_b200 import cuotf
    norb, sym = 6, np.array([0, 1, 0, 1, 1, 0], np.int64)
    net = _masked(norb, sym, 3)
    kw = dict(orbsym=sym, num_irreps=2)
    Bo, No = oracle.basis(norb, 3, 2, **kw), oracle.network(net)
    B = cuotf.CuBasis(norb, 3, 2, **kw)
    f = cuotf.CuOTFFunctions(B, cuotf.CuNetwork(net))
    x = np.random.default_rng(2).normal(size=B.dim)
    ref = oracle.hvec(Bo, No, x)
    f.get_diags(cuda.zeros(B.dim, dtype=cuda.float64, device="cuda"))
    xd = dev(cuda, x)
    y, z = cuda.zeros_like(xd), cuda.zeros_like(xd)
    s = cuda.cuda.Stream()
    with cuda.cuda.stream(s):
        g = cuda.cuda.CUDAGraph()
        with cuda.cuda.graph(g, stream=s):
            f.hvec(xd, y, stream=s.cuda_stream)
    f.hvec(xd, z)
    g.replay()
    cuda.cuda.synchronize()
    for out in (y, z):
        assert np.abs(out.cpu().numpy() - ref).max() <= 1e-13 * np.abs(ref).max()


def test_first_call_is_no_slower_than_the_tile_kernel(cuda):
    """What the first call on a handle pays for the lists: compared with one call that needs none (hvec_tiles over every
    tile).  Made by the host they took twenty times that at this size; three times is the line."""
    import time
    from binsim_b200 import cuotf
    norb, sym = 14, np.array([0, 5, 0, 6, 7, 0, 2, 3, 5, 1, 4, 0, 5, 6], np.int64)
    net = _masked(norb, sym, 0)
    B = cuotf.CuBasis(norb, 7, 7, orbsym=sym, num_irreps=8)
    x = cuda.randn(B.dim, dtype=cuda.float64, device="cuda")
    y = cuda.empty_like(x)

    def ms(call, *args):
        cuda.cuda.synchronize()
        t = time.perf_counter()
        call(*args)
        cuda.cuda.synchronize()
        return 1e3 * (time.perf_counter() - t)
    first, tiles = [], []
    for _ in range(4):
        f = cuotf.CuOTFFunctions(B, cuotf.CuNetwork(net))
        first.append(ms(f.hvec, x, y))
        tiles.append(ms(f.hvec_tiles, x, y, 0, f.num_tiles()))
    assert min(first[1:]) <= 3.0 * min(tiles[1:]), (first, tiles)


def test_lists_stay_within_the_scratch_limit(cuda, oracle, monkeypatch):
    """Lists and frame vector above the limit: the tile kernel serves the call and no memory is taken.  Unsymmetric
    integrals on one alpha electron, whose beta columns make the longest lists, within it."""
    from binsim_b200 import cuotf, network as nw
    sym = np.array([0, 1] * 7, np.int64)
    net = _masked(14, sym, 0)
    B = cuotf.CuBasis(14, 7, 7, orbsym=sym, num_irreps=2)
    assert 8 * B.dim < 50e6 < 1.1 * 8 * B.dim   # the vector alone is just below the lowest limit, 0.05 GB
    f = cuotf.CuOTFFunctions(B, cuotf.CuNetwork(net))
    x = cuda.randn(B.dim, dtype=cuda.float64, device="cuda")
    y, z = cuda.empty_like(x), cuda.empty_like(x)
    f.hvec_tiles(x, z, 0, f.num_tiles())
    monkeypatch.setenv("BSIM_SIGMA_SCRATCH_GB", "0.05")
    cuda.cuda.synchronize()
    free = cuda.cuda.mem_get_info()[0]
    f.hvec(x, y)
    cuda.cuda.synchronize()
    assert free - cuda.cuda.mem_get_info()[0] < 8e6
    assert cuda.equal(y, z)
    monkeypatch.delenv("BSIM_SIGMA_SCRATCH_GB")
    sym = np.array([0, 1, 2, 3, 0, 1, 2, 3, 0], np.int64)
    net = nw.hamiltonian_network(9, seed=1)
    net.orbsym = sym
    Bo = oracle.basis(9, 1, 4, orbsym=sym, num_irreps=4)
    B = cuotf.CuBasis(9, 1, 4, orbsym=sym, num_irreps=4)
    f = cuotf.CuOTFFunctions(B, cuotf.CuNetwork(net))
    x = np.random.default_rng(9).normal(size=B.dim)
    y = cuda.empty(B.dim, dtype=cuda.float64, device="cuda")
    f.hvec(dev(cuda, x), y)
    ref = oracle.hvec(Bo, oracle.network(net), x)
    assert np.abs(y.cpu().numpy() - ref).max() <= 1e-13 * np.abs(ref).max()

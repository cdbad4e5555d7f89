"""Plans that a network keeps for a basis are not found again for another basis: a basis is made, used and destroyed,
and the next one of equal dimension (which often gets its address) computes with the same networks."""
import numpy as np
import pytest

from conftest import dev

pytestmark = pytest.mark.gpu

SYM = [0, 1, 2, 3, 0, 1, 2]


def _sectors(oracle, norb, blocked):
    """Sectors of equal dimension: swapped electron counts, and total irreps of one pair of counts."""
    if not blocked:
        yield from (((4, 3), 0), ((3, 4), 0), ((4, 3), 0), ((3, 4), 0))
        return
    kw = dict(orbsym=np.asarray(SYM, np.int64), num_irreps=4)
    dims = {}
    for t in range(4):
        dims.setdefault(oracle.basis(norb, 4, 3, total_sym=t, **kw).dim, []).append(t)
    pair = max(dims.values(), key=len)[:2]
    assert len(pair) == 2
    yield from (((4, 3), pair[0]), ((4, 3), pair[1]), ((4, 3), 0), ((3, 4), 0), ((4, 3), pair[0]))


@pytest.mark.parametrize("blocked", [False, True])
def test_sectors_in_turn_with_one_network(cuda, oracle, blocked):
    from binsim_b200 import cuotf, network as nw
    norb = 7
    ham, pool = nw.hamiltonian_network(norb, seed=5), nw.ucc_pool(norb)
    osym = np.asarray(SYM if blocked else [0] * norb, np.int64)
    ham.orbsym = pool.network.orbsym = osym
    rng = np.random.default_rng(0)
    wa, wb = (w * np.exp(1j * rng.uniform(-1, 1, len(w))) for w in (ham.flat_wa, ham.flat_wb))
    H, P, Z = cuotf.CuNetwork(ham), cuotf.CuNetwork(pool.network), cuotf.CuNetworkC64(ham, wa, wb)
    Ho, Po, Zo = oracle.network(ham), oracle.network(pool.network), oracle.network_c64(ham, wa, wb)
    kw = dict(orbsym=osym, num_irreps=4 if blocked else 1)
    for (na, nb), tsym in _sectors(oracle, norb, blocked):
        B = cuotf.CuBasis(norb, na, nb, total_sym=tsym, **kw)
        Bo = oracle.basis(norb, na, nb, total_sym=tsym, **kw)
        f, fz = cuotf.CuOTFFunctions(B, H, P), cuotf.CuOTFC64(B, Z)
        x = rng.normal(size=B.dim)
        y = cuda.empty(B.dim, dtype=cuda.float64, device="cuda")
        ref = oracle.hvec(Bo, Ho, x)
        scale = np.abs(ref).max()
        f.hvec(dev(cuda, x), y)
        assert np.abs(y.cpu().numpy() - ref).max() <= 1e-13 * scale
        f.hvec_mixed(dev(cuda, x), y)
        assert np.abs(y.cpu().numpy() - ref).max() <= 2e-6 * scale
        z = x + 1j * rng.normal(size=B.dim)
        out = cuda.empty(B.dim, dtype=cuda.complex128, device="cuda")
        fz.hvec(cuda.as_tensor(z, device="cuda"), out)
        zref = oracle.hvec_c64(Bo, Zo, z)
        assert np.abs(out.cpu().numpy() - zref).max() <= 1e-13 * np.abs(zref).max()
        # pair lists and the theta = 0 gradient
        v = dev(cuda, x)
        f.expm(4, 0.3, v)   # 1-based
        assert np.abs(v.cpu().numpy() - oracle.expm(Bo, Po, 3, 0.3, x)).max() <= 1e-14 * np.abs(x).max()
        for th in (0.0, 0.2):
            thetas = np.full(pool.network.ngs, th)
            grads = cuda.empty(pool.network.ngs, dtype=cuda.float64, device="cuda")
            f.batchgrad(dev(cuda, x), dev(cuda, ref), grads, dev(cuda, thetas))
            g0 = oracle.batchgrad(Bo, Po, thetas, x, ref)
            assert np.abs(grads.cpu().numpy() - g0).max() <= 1e-12 * max(1.0, np.abs(g0).max())
        cuda.cuda.synchronize()
        del f, fz
        B.close()

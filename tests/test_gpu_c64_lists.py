"""Complex sigma over lists against the oracle's complex restatement."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("norb,na,nb,sym,nirr,bits", [(5, 2, 1, None, 1, 32), (7, 4, 3, None, 1, 64),
                                                      (8, 3, 5, [0, 1, 0, 1, 2, 3, 2, 3], 4, 32)])
def test_complex_sigma_lists(cuda, oracle, norb, na, nb, sym, nirr, bits):
    """Against the oracle's complex restatement, and inside a stream capture of the first call (which takes the kernel
    that needs no lists)."""
    from binsim_b200 import cuotf, network as nw
    net = nw.hamiltonian_network(norb, seed=3)
    net.orbsym = np.zeros(norb, np.int64) if sym is None else np.asarray(sym, np.int64)
    rng = np.random.default_rng(norb)
    wa, wb = (w * np.exp(1j * rng.uniform(-1, 1, len(w))) for w in (net.flat_wa, net.flat_wb))
    kw = dict(orbsym=net.orbsym, num_irreps=nirr)
    Bo = oracle.basis(norb, na, nb, total_sym=0, **kw)
    No = oracle.network_c64(net, wa, wb)
    B = cuotf.CuBasis(norb, na, nb, string_bits=bits, **kw)
    f = cuotf.CuOTFC64(B, cuotf.CuNetworkC64(net, wa, wb, string_bits=bits))
    x = rng.normal(size=B.dim) + 1j * rng.normal(size=B.dim)
    ref = oracle.hvec_c64(Bo, No, x)
    xd = cuda.as_tensor(x, device="cuda")
    y, z = cuda.zeros_like(xd), cuda.zeros_like(xd)
    s = cuda.cuda.Stream()
    with cuda.cuda.stream(s):
        g = cuda.cuda.CUDAGraph()
        with cuda.cuda.graph(g, stream=s):
            f.hvec(xd, z, stream=s.cuda_stream)
        g.replay()
    f.hvec(xd, y)
    cuda.cuda.synchronize()
    for out in (y, z):
        assert np.abs(out.cpu().numpy() - ref).max() <= 1e-13 * np.abs(ref).max()

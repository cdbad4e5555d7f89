"""What a first call on new handles pays for its lists."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_first_pool_gradient_beside_the_first_sigma(cuda):
    """The first pool gradient makes the pair lists of the pool; the first sigma its row lists.  At 20o 3a+3b the gradient
    took 0.6 of the sigma's time while every string was looked up for every mask, and takes 0.2 of it now."""
    from binsim_b200 import cuotf, network as nw
    norb = 20
    B = cuotf.CuBasis(norb, 3, 3)
    ham, pool = nw.hamiltonian_network(norb, seed=0, native=True), nw.ucc_pool(norb, native=True)
    x = cuda.randn(B.dim, dtype=cuda.float64, device="cuda")
    y = cuda.empty_like(x)
    thetas = cuda.zeros(pool.network.ngs, dtype=cuda.float64, device="cuda")
    grads = cuda.empty_like(thetas)

    def ms(call):
        cuda.cuda.synchronize()
        t = time.perf_counter()
        call()
        cuda.cuda.synchronize()
        return 1e3 * (time.perf_counter() - t)
    sigma, grad = [], []
    for _ in range(4):
        f = cuotf.CuOTFFunctions(B, cuotf.CuNetwork(ham), cuotf.CuNetwork(pool.network))
        sigma.append(ms(lambda: f.hvec(x, y)))
        grad.append(ms(lambda: f.batchgrad(x, y, grads, thetas)))
    assert np.min(grad[1:]) <= 0.4 * np.min(sigma[1:]), (sigma, grad)

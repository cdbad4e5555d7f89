"""Two host threads with a basis each and one network: no thread's plan goes while the other works with it, and bases used
in turn keep their plans."""
import threading

import numpy as np
import pytest

from conftest import dev

pytestmark = pytest.mark.gpu

NORB = 7
SYM = np.array([0, 1, 2, 3, 0, 1, 2], np.int64)


def _setup(blocked):
    from binsim_b200 import cuotf, network as nw
    ham = nw.hamiltonian_network(NORB, seed=5)
    ham.orbsym = SYM if blocked else np.zeros(NORB, np.int64)
    rng = np.random.default_rng(0)
    wa, wb = (w * np.exp(1j * rng.uniform(-1, 1, len(w))) for w in (ham.flat_wa, ham.flat_wb))
    return ham, (wa, wb), dict(orbsym=ham.orbsym, num_irreps=4 if blocked else 1)


@pytest.mark.parametrize("blocked", [False, True])
def test_two_threads_one_network(cuda, oracle, blocked):
    from binsim_b200 import cuotf
    ham, w, kw = _setup(blocked)
    H, Z = cuotf.CuNetwork(ham), cuotf.CuNetworkC64(ham, *w)
    Ho, Zo = oracle.network(ham), oracle.network_c64(ham, *w)
    work = []
    for k, (na, nb) in enumerate(((4, 3), (3, 4))):
        x = np.random.default_rng(k).normal(size=oracle.basis(NORB, na, nb, **kw).dim)
        Bo = oracle.basis(NORB, na, nb, **kw)
        work.append(((na, nb), x, oracle.hvec(Bo, Ho, x), oracle.hvec_c64(Bo, Zo, x + 0.5j * x[::-1])))
    errors, out = [], [None, None]

    def run(i):
        try:
            (na, nb), x, ref, zref = work[i]
            stream = cuda.cuda.Stream()
            with cuda.cuda.stream(stream):
                worst = 0.0
                for rep in range(6):
                    B = cuotf.CuBasis(NORB, na, nb, **kw)
                    f, fz = cuotf.CuOTFFunctions(B, H), cuotf.CuOTFC64(B, Z)
                    y, z = dev(cuda, x), cuda.as_tensor(x + 0.5j * x[::-1], device="cuda")
                    hy, hz = cuda.empty_like(y), cuda.empty_like(z)
                    for _ in range(5):
                        f.hvec(y, hy)
                        fz.hvec(z, hz)
                    stream.synchronize()
                    worst = max(worst, np.abs(hy.cpu().numpy() - ref).max() / np.abs(ref).max(),
                                np.abs(hz.cpu().numpy() - zref).max() / np.abs(zref).max())
                    del f, fz
                    B.close()
            out[i] = worst
        except Exception as e:   # handed to the main thread
            errors.append(e)

    threads = [threading.Thread(target=run, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    assert max(out) <= 1e-13


def test_bases_in_turn_make_no_new_plans(cuda):
    """Symmetry blocks and complex sigma: the plans of two irreps stay while both bases live."""
    from binsim_b200 import cuotf
    from binsim_b200.cuotf import lib
    ham, w, kw = _setup(True)
    H, Z = cuotf.CuNetwork(ham), cuotf.CuNetworkC64(ham, *w)
    f = []
    for t in (0, 1):
        B = cuotf.CuBasis(NORB, 4, 3, total_sym=t, **kw)
        x = cuda.ones(B.dim, dtype=cuda.float64, device="cuda")
        z = cuda.ones(B.dim, dtype=cuda.complex128, device="cuda")
        f.append((cuotf.CuOTFFunctions(B, H), x, cuda.empty_like(x), cuotf.CuOTFC64(B, Z), z, cuda.empty_like(z)))

    def both():
        for g, x, y, gz, z, u in f:
            g.hvec(x, y)
            gz.hvec(z, u)
        cuda.cuda.synchronize()
    both()
    n = lib().bsim_device_alloc_count()
    both()
    assert lib().bsim_device_alloc_count() == n


def test_a_plan_goes_with_its_basis(cuda):
    """Lists of the complex sigma at 10o 5+5 (tens of megabytes) are given back when the basis is destroyed, the network
    still alive."""
    from binsim_b200 import cuotf, network as nw
    ham = nw.hamiltonian_network(10, seed=1, native=True)
    Z = cuotf.CuNetworkC64(ham, ham.flat_wa.astype(complex), ham.flat_wb.astype(complex))
    z = cuda.ones(252 * 252, dtype=cuda.complex128, device="cuda")
    u = cuda.empty_like(z)

    def free():
        cuda.cuda.synchronize()
        return cuda.cuda.mem_get_info()[0]
    for _ in range(2):   # the first round also loads the kernels
        before = free()
        B = cuotf.CuBasis(10, 5, 5)
        f = cuotf.CuOTFC64(B, Z)
        f.hvec(z, u)
        used = before - free()
        del f
        B.close()
        left = before - free()
    assert used > 8e6 and left < 4e6, (used, left)


def test_shapes_of_two_threads(cuda):
    """Kernels launched with one thread's shared memory while another launches them with less (or more)."""
    from binsim_b200 import cuotf, network as nw
    errors = []
    sizes = ((8, 3, 4), (11, 4, 3))
    fs = [cuotf.CuOTFFunctions(cuotf.CuBasis(*n), cuotf.CuNetwork(nw.hamiltonian_network(n[0], seed=1, native=True)))
          for n in sizes]

    def run(f):
        try:
            stream = cuda.cuda.Stream()
            with cuda.cuda.stream(stream):
                x = cuda.randn(f.basis.dim, dtype=cuda.float64, device="cuda")
                y = cuda.empty_like(x)
                for _ in range(300):
                    f.hvec(x, y)
                    f.hvec_mixed(x, y)
                stream.synchronize()
        except Exception as e:
            errors.append(e)

    threads = [threading.Thread(target=run, args=(f,)) for f in fs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors

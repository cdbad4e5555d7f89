"""Rotation sequences applied several components per pass: prepare_state and the adjoint sweep against the oracle,
for op orders that make units of one to four components, diagonal and unclassified groups, and odd sizes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _sequences(pool, rng):
    n = pool.network.ngs
    gens = [pool.components[i] for i in rng.integers(0, len(pool.components), 24)]
    yield [c for g in gens for c in g]                                   # whole generators
    yield [int(i) for i in rng.integers(0, n, 40)]                       # unrelated components
    yield [c for g in gens[:6] for c in (list(g) + list(g[::-1]))]       # a generator forwards and backwards


@pytest.mark.parametrize("norb,na,nb,bits", [(4, 1, 2, 32), (5, 4, 1, 32), (7, 3, 4, 32), (8, 4, 4, 64), (9, 2, 7, 32)])
def test_sequences_match_oracle(cuda, oracle, norb, na, nb, bits):
    from binsim_b200 import cuotf, network as nw
    ham, pool = nw.hamiltonian_network(norb, seed=norb), nw.ucc_pool(norb)
    Bo, Ho, Po = oracle.basis(norb, na, nb), oracle.network(ham), oracle.network(pool.network)
    B = cuotf.CuBasis(norb, na, nb, string_bits=bits)
    f = cuotf.CuOTFFunctions(B, cuotf.CuNetwork(ham, string_bits=bits), cuotf.CuNetwork(pool.network, string_bits=bits))
    rng = np.random.default_rng(norb)
    ref_idx = np.unique(rng.integers(0, B.dim, 5))
    ref_val = rng.normal(size=len(ref_idx))
    lv = cuda.empty(B.dim, dtype=cuda.float64, device="cuda")
    rv = cuda.empty_like(lv)
    for ops in _sequences(pool, rng):
        ops = np.array(ops)
        par = np.arange(len(ops)) // 3
        th = rng.normal(0.0, 0.4, par[-1] + 1)
        l0 = np.zeros(B.dim)
        l0[ref_idx] = ref_val
        for i, p in zip(ops, par):
            l0 = oracle.expm(Bo, Po, int(i), th[p], l0)
        f.prepare_state(ops, par, th, ref_idx, ref_val, lv)
        # every rotation rounds each of its two products once: eps per operator and unit norm
        tol = 4e-16 * len(ops) * np.linalg.norm(ref_val)
        np.testing.assert_allclose(lv.cpu().numpy(), l0, rtol=0, atol=tol)
        r0 = oracle.hvec(Bo, Ho, l0)
        ll, e0, g0 = l0 @ l0, l0 @ r0 / (l0 @ l0), np.zeros(len(th))
        for i, p in zip(ops[::-1], par[::-1]):
            g, l0, r0 = oracle.backgrad(Bo, Po, int(i), th[p], l0, r0)
            g0[p] += 2 * g / ll
        for every in (0, 2):
            e, g, _ = f.energy_grad(ops, par, th, ref_idx, ref_val, lv, rv, ckpt_every=every)
            scale = np.abs(r0).max()
            assert abs(e - e0) < 1e-13 * max(1.0, abs(e0)) * len(ops)
            np.testing.assert_allclose(g, g0, rtol=0, atol=1e-14 * len(ops) * max(1.0, scale))
            np.testing.assert_allclose(lv.cpu().numpy(), l0, rtol=0, atol=2 * tol)
            np.testing.assert_allclose(rv.cpu().numpy(), r0, rtol=0, atol=1e-15 * len(ops) * max(1.0, scale))


def test_mixed_forms_fall_back_in_order(cuda, oracle):
    """Diagonal groups and groups that are no excitation (those of a Hamiltonian network) between excitations, and a
    basis of several symmetry blocks, take the pair kernels in their place of the sequence."""
    from binsim_b200 import cuotf, network as nw
    norb, na, nb = 6, 3, 2
    ham = nw.hamiltonian_network(norb, seed=2)
    ref = np.array([1]), np.array([1.0])
    for sym in (None, np.array([0, 1, 0, 1, 1, 0])):
        osym = np.zeros(norb, np.int64) if sym is None else sym
        ham.orbsym = osym
        kw = dict(orbsym=osym, num_irreps=1 if sym is None else 2)
        Bo, Ho = oracle.basis(norb, na, nb, total_sym=0, **kw), oracle.network(ham)
        B = cuotf.CuBasis(norb, na, nb, **kw)
        H = cuotf.CuNetwork(ham)
        f = cuotf.CuOTFFunctions(B, H, H)
        ops = np.array([5, 0, 9, 12, 0, 0, 30, 31, 7])
        th = np.linspace(-0.3, 0.4, len(ops))
        v = cuda.empty(B.dim, dtype=cuda.float64, device="cuda")
        f.prepare_state(ops, np.arange(len(ops)), th, *ref, v)
        v0 = np.zeros(B.dim)
        v0[1] = 1.0
        for i, t in zip(ops, th):
            v0 = oracle.expm(Bo, Ho, int(i), t, v0)
        np.testing.assert_allclose(v.cpu().numpy(), v0, rtol=0, atol=1e-14 * max(1.0, np.abs(v0).max()))

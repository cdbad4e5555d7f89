"""The work a user of the library has it do, as cases that can be timed and checked.

Every case goes through the public Python layer (binsim_b200.cuotf), which is one ctypes call per
operator.  ``prepare`` makes what a program holds before the call (basis and network handles, device
vectors), ``run`` is one pass, ``exact`` recomputes its outputs in FP64 torch from the second-quantised
operators (E_pq link tables in the alpha-first determinant frame), without the library.
"""
import functools
import itertools
import math

import numpy as np
import torch

from binsim_b200 import cuotf
from binsim_b200 import network as nw

D2H = (0, 5, 0, 6, 7, 0, 2, 3, 5, 1, 4, 0, 5, 6, 7, 2)   # irreps of a minimal-basis-like orbital list


def listed():
    return [
        # one sigma of a model-sized space: a single call, bound by launches and latency
        {"name": "sigma_8o_f64", "op": "sigma", "norb": 8, "na": 4, "nb": 4, "mixed": False, "irreps": 1,
         "vec": "normal"},
        # the FCI size of the Davidson configuration: every Davidson step is one of these
        {"name": "sigma_12o_f64", "op": "sigma", "norb": 12, "na": 6, "nb": 6, "mixed": False, "irreps": 1,
         "vec": "normal"},
        # an open-shell, odd-sized space with a decaying CI vector
        {"name": "sigma_13o_7a5b_f64", "op": "sigma", "norb": 13, "na": 7, "nb": 5, "mixed": False, "irreps": 1,
         "vec": "ci"},
        # a molecule with point-group symmetry: only the determinants of one irrep
        {"name": "sigma_14o_d2h_f64", "op": "sigma", "norb": 14, "na": 7, "nb": 7, "mixed": False, "irreps": 8,
         "vec": "normal"},
        # the headline sigma microbenchmark, plain FP64 and FP32 bulk
        {"name": "sigma_16o_f64", "op": "sigma", "norb": 16, "na": 8, "nb": 8, "mixed": False, "irreps": 1,
         "vec": "normal"},
        {"name": "sigma_16o_f32", "op": "sigma", "norb": 16, "na": 8, "nb": 8, "mixed": True, "irreps": 1,
         "vec": "normal"},
        # the FCI ground state to convergence, FP64 and with FP32 subspace storage
        {"name": "davidson_12o_f64", "op": "davidson", "norb": 12, "na": 6, "nb": 6, "mixed": False},
        {"name": "davidson_12o_mixed", "op": "davidson", "norb": 12, "na": 6, "nb": 6, "mixed": True},
        # one VQE optimiser step (energy and adjoint gradient): a short ansatz on a small space, and the
        # UCCGSD configuration with 2000 generators
        {"name": "vqe_10o_200", "op": "vqe", "norb": 10, "na": 5, "nb": 5, "gens": 200},
        {"name": "vqe_14o_2000", "op": "vqe", "norb": 14, "na": 7, "nb": 7, "gens": 2000},
        # one ADAPT screening step (H psi and the gradient of every pool operator) on 64-bit strings
        {"name": "adapt_20o_3a3b", "op": "adapt", "norb": 20, "na": 3, "nb": 3, "bits": 64},
        # sigma with complex weights (periodic systems)
        {"name": "sigma_c64_10o", "op": "sigma_c64", "norb": 10, "na": 5, "nb": 5},
    ]


def draw(rng):
    """One more case of the listed ranges; electron counts around half filling, sizes spread over their logarithm."""
    op = rng.choice(["sigma", "sigma", "sigma", "sigma", "davidson", "vqe", "adapt", "sigma_c64"])

    def electrons(norb, far):
        return [max(1, min(norb - 1, norb // 2 + rng.randint(-far, far))) for _ in (0, 1)]
    if op == "sigma":
        norb = rng.randint(6, 15)
        na, nb = electrons(norb, 2)
        return {"op": op, "norb": norb, "na": na, "nb": nb, "mixed": rng.random() < 0.35,
                "irreps": rng.choice([1, 1, 2, 4, 8]), "vec": rng.choice(["normal", "ci"])}
    if op == "davidson":
        norb = rng.randint(8, 12)
        na, nb = electrons(norb, 1)
        return {"op": op, "norb": norb, "na": na, "nb": nb, "mixed": rng.random() < 0.5}
    if op == "vqe":
        norb = rng.randint(6, 13)
        na, nb = electrons(norb, 1)
        return {"op": op, "norb": norb, "na": na, "nb": nb, "gens": int(round(math.exp(rng.uniform(math.log(20), math.log(600)))))}
    if op == "adapt":
        norb = rng.randint(8, 18)
        return {"op": op, "norb": norb, "na": rng.randint(2, 3), "nb": rng.randint(2, 3), "bits": rng.choice([32, 64])}
    norb = rng.randint(6, 10)
    na, nb = electrons(norb, 1)
    return {"op": op, "norb": norb, "na": na, "nb": nb}


# ---- inputs ---------------------------------------------------------------------------------------


def _orbsym(case):
    k = case.get("irreps", 1)
    return np.array([D2H[p % len(D2H)] % k for p in range(case["norb"])], np.int64)


def _integrals(case, seed):
    """The seeded benchmark integrals (one molecule) moved a little by the seed (a nearby geometry), with the
    integrals that the point group forbids set to zero."""
    norb = case["norb"]
    h, g, _ = nw.synthetic_integrals(norb, 0)
    dh, dg, _ = nw.synthetic_integrals(norb, seed + 1)
    h, g = h + 0.02 * dh, g + 0.02 * dg
    s = _orbsym(case)
    h = h * ((s[:, None] ^ s[None, :]) == 0)
    g = g * ((s[:, None, None, None] ^ s[None, :, None, None] ^ s[None, None, :, None] ^ s[None, None, None, :]) == 0)
    return h, np.ascontiguousarray(g)


def _hamiltonian(case, seed):
    h, g = _integrals(case, seed)
    x, z, c = nw.jw_hamiltonian_terms(h, g)
    return cuotf.compress_groups_native(*nw.split_aabb(x, z, case["norb"]), c, case["norb"], orbsym=_orbsym(case))


def _complex_weights(net, seed):
    r = np.random.default_rng(seed)
    return [w * np.exp(1j * r.uniform(-1.0, 1.0, len(w))) for w in (net.flat_wa, net.flat_wb)]


def _vector(case, seed, dim, dtype=torch.float64):
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randn(dim, dtype=dtype, device="cuda", generator=g)
    if case.get("vec") == "ci":   # amplitudes over six decades under one leading determinant
        x *= 10.0 ** (-6.0 * torch.rand(dim, dtype=torch.float64, device="cuda", generator=g))
        x[0] = 0.9 * torch.linalg.vector_norm(x)
    return x / torch.linalg.vector_norm(x)


def _ansatz(case, seed):
    pool = nw.ucc_pool(case["norb"], native=True)
    return (pool,) + nw.draw_generators(pool, case.get("gens", 40), seed=seed, amp_sigma=0.05)


def prepare(case, seed):
    op, norb = case["op"], case["norb"]
    bits = case.get("bits")
    basis = cuotf.CuBasis(norb, case["na"], case["nb"], orbsym=_orbsym(case), num_irreps=case.get("irreps", 1),
                          string_bits=bits)
    if op == "sigma_c64":
        net = _hamiltonian(case, seed)
        f = cuotf.CuOTFC64(basis, cuotf.CuNetworkC64(net, *_complex_weights(net, seed)))
        x = _vector(case, seed, basis.dim, torch.complex128)
        return {"op": op, "f": f, "x": x, "y": torch.empty_like(x)}
    pool = None
    if op in ("vqe", "adapt"):
        pool, op_idx, param_idx, thetas = _ansatz(case, seed)
        pool = cuotf.CuNetwork(pool.network, string_bits=bits)
    f = cuotf.CuOTFFunctions(basis, cuotf.CuNetwork(_hamiltonian(case, seed), string_bits=bits), pool)
    state = {"op": op, "f": f, "mixed": case.get("mixed", False)}
    if op == "sigma":
        state["x"] = _vector(case, seed, basis.dim)
        state["y"] = torch.empty_like(state["x"])
    elif op == "davidson":
        state["diags"] = torch.zeros(basis.dim, dtype=torch.float64, device="cuda")
        f.get_diags(state["diags"])
        state["v0"] = 0.05 * _vector(case, seed, basis.dim)
        state["hf"] = basis.hf_index()
        state["v0"][state["hf"]] += 1.0
        state["x"] = torch.empty_like(state["v0"])
    elif op == "vqe":
        state.update(ansatz=(op_idx, param_idx, thetas), ref=(np.array([basis.hf_index()]), np.array([1.0])),
                     lv=torch.empty(basis.dim, dtype=torch.float64, device="cuda"),
                     rv=torch.empty(basis.dim, dtype=torch.float64, device="cuda"))
    else:
        state["x"] = torch.empty(basis.dim, dtype=torch.float64, device="cuda")
        f.prepare_state(op_idx, param_idx, thetas, np.array([basis.hf_index()]), np.array([1.0]), state["x"])
        state["y"] = torch.empty_like(state["x"])
        state["thetas"] = torch.zeros(pool.ngs, dtype=torch.float64, device="cuda")
        state["grads"] = torch.empty_like(state["thetas"])
    return state


DAV_TOL = 1e-5


def run(state):
    f, op = state["f"], state["op"]
    if op in ("sigma", "sigma_c64"):
        (f.hvec_mixed if state.get("mixed") else f.hvec)(state["x"], state["y"])
        return state["y"]
    if op == "davidson":
        st = f.davidson(state["v0"], state["diags"], state["x"], tol=DAV_TOL, maxiter=300, ncv=3, maxspace=8,
                        mixed=state["mixed"])
        return {"energy": np.float64(st["energy"]), "x": state["x"] * torch.sign(state["x"][state["hf"]])}
    if op == "vqe":
        e, g, var = f.energy_grad(*state["ansatz"], *state["ref"], state["lv"], state["rv"], ckpt_every=64)
        return {"energy": np.float64(e), "variance": np.float64(var), "grad": g, "l": state["lv"], "r": state["rv"]}
    f.hvec(state["x"], state["y"])
    f.batchgrad(state["x"], state["y"], state["grads"], state["thetas"])
    return {"hpsi": state["y"], "grads": state["grads"]}


# ---- work and tolerance ---------------------------------------------------------------------------


def _dim(case):
    return math.comb(case["norb"], case["na"]) * math.comb(case["norb"], case["nb"])


def _connected(case):
    """Determinants that a two-body Hamiltonian connects to one determinant (itself included)."""
    n = case["norb"]
    single = [k * (n - k) for k in (case["na"], case["nb"])]
    double = [math.comb(k, 2) * math.comb(n - k, 2) for k in (case["na"], case["nb"])]
    return 1 + sum(single) + sum(double) + single[0] * single[1]


def work(case):
    """Vectors read and written once; two flops per connected pair of determinants (four times that for complex
    numbers); for the rotations of an ansatz, its pairs' updates."""
    dim, conn, op = _dim(case), _connected(case), case["op"]
    k = case.get("irreps", 1)
    if op == "sigma":
        return {"bytes": 16.0 * dim / k, "flops": 2.0 * dim * conn / (k * k)}
    if op == "sigma_c64":
        return {"bytes": 32.0 * dim, "flops": 8.0 * dim * conn}
    if op == "davidson":
        steps = 25
        return {"bytes": steps * 32.0 * dim, "flops": steps * 2.0 * dim * conn}
    if op == "vqe":
        comps = 3.4 * case["gens"]
        return {"bytes": 48.0 * dim, "flops": 2.0 * dim * conn + comps * 0.25 * dim * 30}
    pairs = 8.0 * case["norb"] ** 4 / 4
    return {"bytes": 24.0 * dim + 16.0 * pairs, "flops": 2.0 * dim * conn + 4.0 * pairs * dim / 20}


def tolerance(case):
    op = case["op"]
    if op == "sigma" and case["mixed"]:
        return {"rel": 1e-6}        # FP32 products, FP64 sums across batches
    if op == "davidson":
        return {"rel": 5e-5, "max": 2e-2}   # the eigenvector of a residual of DAV_TOL over the spectral gap
    if op == "vqe":
        return {"rel": 1e-12, "max": 1e-9}  # thousands of rotations, one after another
    return {"rel": 4e-14, "max": 4e-12}     # FP64 sums of thousands of terms


# ---- exact ----------------------------------------------------------------------------------------


def _strings(norb, n):
    return np.array(sorted(sum(1 << p for p in c) for c in itertools.combinations(range(norb), n)), np.int64)


def _parity(x):
    x = np.asarray(x, np.uint64)
    return (nw.popcount_u64(x) & 1).astype(np.int64)


def _apply(strs, norb, ops):
    """Ladder operators [(orbital, creates), ...], the rightmost first, on every string: (source index, target index,
    sign) of the strings that survive."""
    s, sign, ok = strs.copy(), np.ones(len(strs)), np.ones(len(strs), bool)
    for p, creates in reversed(ops):
        bit = np.int64(1) << np.int64(p)
        occ = (s & bit) != 0
        ok &= occ != creates
        sign *= 1 - 2 * _parity(s & (bit - 1))
        s = s ^ bit
    src = np.flatnonzero(ok)
    dst = np.searchsorted(strs, s[ok])
    cu = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    return cu(src), cu(dst), cu(sign[ok])


class _Space:
    """All determinants of (norb, na, nb) in the alpha-first frame: c~[a, b] = eps(a, b) c(a, b)."""

    def __init__(self, case):
        self.norb, self.na, self.nb = case["norb"], case["na"], case["nb"]
        self.A, self.B = _strings(self.norb, self.na), _strings(self.norb, self.nb)
        K = np.zeros(len(self.A), np.int64)
        for i in range(self.norb):
            K ^= np.where(self.A >> i & 1, (1 << i) - 1, 0)
        par = torch.zeros(len(self.A), len(self.B), dtype=torch.float64, device="cuda")
        Kt, Bt = torch.from_numpy(K).cuda(), torch.from_numpy(self.B).cuda()
        for i in range(self.norb):
            par += ((Kt >> i & 1)[:, None] * (Bt >> i & 1)[None, :]).double()
        self.eps = 1.0 - 2.0 * torch.remainder(par, 2.0)
        # the library's order: blocks by the alpha irrep, determinants outside the total symmetry left out
        sym = _orbsym(case)
        sa, sb = ([int(functools.reduce(lambda x, y: x ^ y, [int(sym[p]) for p in range(self.norb) if s >> p & 1], 0))
                   for s in T] for T in (self.A, self.B))
        sa, sb, order = np.array(sa), np.array(sb), []
        for k in range(case.get("irreps", 1)):
            a, b = np.flatnonzero(sa == k), np.flatnonzero(sb == k)
            order.append((a[:, None] * len(self.B) + b[None, :]).ravel())
        self.order = torch.from_numpy(np.concatenate(order)).cuda()
        E = [(p, q) for p in range(self.norb) for q in range(self.norb)]
        self.ea = [_apply(self.A, self.norb, [(p, True), (q, False)]) for p, q in E]
        self.eb = [_apply(self.B, self.norb, [(p, True), (q, False)]) for p, q in E]

    def frame(self, v):
        out = torch.zeros(len(self.A) * len(self.B), dtype=torch.float64, device="cuda")
        out[self.order] = v
        return out.view(len(self.A), len(self.B)) * self.eps

    def back(self, v):
        return (v * self.eps).reshape(-1)[self.order]

    def excite(self, c, alpha=True, beta=True):
        """E_pq c for every p, q: [norb^2, nA, nB]."""
        D = torch.zeros(self.norb ** 2, *c.shape, dtype=torch.float64, device="cuda")
        for k in range(self.norb ** 2):
            if alpha:
                s, d, g = self.ea[k]
                D[k][d] += g[:, None] * c[s]
            if beta:
                s, d, g = self.eb[k]
                D[k][:, d] += g[None, :] * c[:, s]
        return D

    def sigma(self, h, g, c):
        """H = sum k_ps E_ps + 1/2 sum (ps|qr) E_ps E_qr with g[p,q,r,s] = (ps|qr)."""
        n = self.norb
        k = torch.from_numpy(h - 0.5 * np.einsum("pqrq->pr", g)).cuda()
        G = torch.from_numpy(np.ascontiguousarray(0.5 * g.transpose(0, 3, 1, 2)).reshape(n * n, n * n)).cuda()
        D = self.excite(c)
        out = (k.reshape(1, -1) @ D.view(n * n, -1)).view(c.shape)
        D = (G @ D.view(n * n, -1)).view(n * n, *c.shape)
        for j in range(n * n):
            s, d, q = self.ea[j]
            out[d] += q[:, None] * D[j][s]
            s, d, q = self.eb[j]
            out[:, d] += q[None, :] * D[j][:, s]
        return out

    def rotation(self, cre, ann):
        """The generator's index blocks: t |src> = sign |dst> on alpha and beta strings."""
        ops = [(o, True) for o in cre] + [(o, False) for o in ann]
        inv = sum(1 for i in range(len(ops)) for j in range(i) if ops[i][0] % 2 == 0 and ops[j][0] % 2 == 1)
        parts = [_apply(T, self.norb, [(o // 2, c) for o, c in ops if o % 2 == s])
                 for s, T in ((0, self.A), (1, self.B))]
        return parts, -1.0 if inv % 2 else 1.0


def _rotate(part, v, c, s):
    """exp(theta (t - t^+)) v in place."""
    ((sa, da, ga), (sb, db, gb)), sign = part
    src, dst = (sa[:, None], sb[None, :]), (da[:, None], db[None, :])
    w = sign * ga[:, None] * gb[None, :]
    x, y = v[src], v[dst]
    v[src], v[dst] = c * x - s * w * y, c * y + s * w * x


def _generator(part, l, r):
    """<r| t - t^+ |l>."""
    ((sa, da, ga), (sb, db, gb)), sign = part
    src, dst = (sa[:, None], sb[None, :]), (da[:, None], db[None, :])
    w = sign * ga[:, None] * gb[None, :]
    return (w * (l[src] * r[dst] - l[dst] * r[src])).sum()


def _exact_vqe(case, seed, S, h, g):
    pool, op_idx, param_idx, thetas = _ansatz(case, seed)
    parts = {i: S.rotation(*pool.excitations[i]) for i in set(op_idx.tolist())}
    l = torch.zeros(len(S.A), len(S.B), dtype=torch.float64, device="cuda")
    l[0, 0] = 1.0
    l = l * S.eps
    for i, p in zip(op_idx.tolist(), param_idx.tolist()):
        _rotate(parts[i], l, math.cos(thetas[p]), math.sin(thetas[p]))
    r = S.sigma(h, g, l)
    ll, lr, rr = (l * l).sum(), (l * r).sum(), (r * r).sum()
    grad = torch.zeros(len(thetas), dtype=torch.float64, device="cuda")
    for i, p in zip(op_idx[::-1].tolist(), param_idx[::-1].tolist()):
        grad[p] += 2.0 * _generator(parts[i], l, r) / ll
        for v in (l, r):
            _rotate(parts[i], v, math.cos(thetas[p]), -math.sin(thetas[p]))
    return {"energy": lr / ll, "variance": rr / ll - (lr / ll) ** 2, "grad": grad, "l": S.back(l), "r": S.back(r)}


def _exact_adapt(case, seed, S, h, g):
    """Pool gradients <H psi| t - t^+ |psi> through <E_q1p1 H psi| E_p2q2 psi>, the excitations of each spin apart."""
    pool, op_idx, param_idx, thetas = _ansatz(case, seed)
    parts = {i: S.rotation(*pool.excitations[i]) for i in set(op_idx.tolist())}
    psi = torch.zeros(len(S.A), len(S.B), dtype=torch.float64, device="cuda")
    psi[0, 0] = 1.0
    psi = psi * S.eps
    for i, p in zip(op_idx.tolist(), param_idx.tolist()):
        _rotate(parts[i], psi, math.cos(thetas[p]), math.sin(thetas[p]))
    hpsi = S.sigma(h, g, psi)
    n, nn = S.norb, S.norb ** 2
    stack = lambda v: torch.cat([S.excite(v, beta=False), S.excite(v, alpha=False)]).view(2 * nn, -1)
    L, R = stack(psi), stack(hpsi)
    # M[x, y] = <H psi| E_x^+ E_y |psi>, M2 the same with the vectors exchanged; one[x] = <.|E_x|.>
    M, M2 = R @ L.T, L @ R.T
    one, one2 = L @ hpsi.reshape(-1), R @ psi.reshape(-1)
    e = lambda p, q: (p % 2) * nn + (p // 2) * n + q // 2
    cu = lambda a: torch.from_numpy(np.asarray(a, np.int64)).cuda()
    grads = torch.zeros(len(pool.excitations), dtype=torch.float64, device="cuda")
    single = [(i, e(c[0], a[0])) for i, (c, a) in enumerate(pool.excitations) if len(c) == 1]
    double = [(i, e(a[1], c[0]), e(c[1], a[0]), e(c[0], a[0]) if c[1] == a[1] else -1)
              for i, (c, a) in enumerate(pool.excitations) if len(c) == 2]
    i, x = (cu(v) for v in zip(*single))
    grads[i] = one[x] - one2[x]
    i, x, y, d = (cu(v) for v in zip(*double))
    # t = E_{c0 a1} E_{c1 a0} - delta(a1, c1) E_{c0 a0}
    dl = torch.where(d >= 0, one[d.clamp(min=0)] - one2[d.clamp(min=0)], torch.zeros((), dtype=torch.float64, device="cuda"))
    grads[i] = M[x, y] - M2[x, y] - dl
    return {"hpsi": S.back(hpsi), "grads": grads}


def _exact_davidson(case, seed, S, h, g):
    """Lowest eigenpair by Lanczos with full re-orthogonalisation."""
    dim = len(S.A) * len(S.B)
    v = 0.05 * _vector(case, seed, dim)
    v[0] += 1.0
    V = [S.frame(v).reshape(-1)]
    V[0] /= torch.linalg.vector_norm(V[0])
    al, be = [], []
    for k in range(120):
        w = S.sigma(h, g, V[k].view(len(S.A), len(S.B))).reshape(-1)
        al.append(float(w @ V[k]))
        Q = torch.stack(V)
        for _ in range(2):
            w = w - Q.T @ (Q @ w)
        be.append(float(torch.linalg.vector_norm(w)))
        T = torch.diag(torch.tensor(al, dtype=torch.float64)) + sum(
            torch.diag(torch.tensor(be[:-1], dtype=torch.float64), o) for o in (1, -1)) if k else torch.tensor([[al[0]]], dtype=torch.float64)
        ev, U = torch.linalg.eigh(T)
        if be[-1] < 1e-12 or abs(float(U[-1, 0])) * be[-1] < 1e-10:
            break
        V.append(w / be[-1])
    x = S.back((torch.stack(V[:len(al)]).T @ U[:, 0].cuda()).view(len(S.A), len(S.B)))
    return {"energy": np.float64(ev[0]), "x": x * torch.sign(x[0])}


def _exact_c64(case, seed):
    """Group by group: <a^ax, b^bx|H_g|a, b> = sum_r PA_r(a) PB_r(b)."""
    net = _hamiltonian(case, seed)
    wa, wb = _complex_weights(net, seed)
    A, B = _strings(case["norb"], case["na"]), _strings(case["norb"], case["nb"])
    x = _vector(case, seed, len(A) * len(B), torch.complex128).view(len(A), len(B))
    y = torch.zeros_like(x)
    za = zb = oa = ob = 0

    def side(strs, mask, zs, w):
        to = strs ^ np.int64(mask)
        src = np.flatnonzero(np.isin(to, strs))
        P = (1 - 2 * _parity(strs[src][:, None] & zs.astype(np.int64)[None, :])) @ w
        return torch.from_numpy(src).cuda(), torch.from_numpy(np.searchsorted(strs, to[src])).cuda(), torch.from_numpy(P).cuda()
    for k in range(net.ngs):
        na, nb, r = int(net.num_zas[k]), int(net.num_zbs[k]), int(net.ranks[k])
        sa, da, pa = side(A, int(net.axs[k]), net.flat_zas[za:za + na], wa[oa:oa + na * r].reshape(r, na).T)
        sb, db, pb = side(B, int(net.bxs[k]), net.flat_zbs[zb:zb + nb], wb[ob:ob + nb * r].reshape(r, nb).T)
        y[da[:, None], db[None, :]] += (pa @ pb.T) * x[sa[:, None], sb[None, :]]
        za, zb, oa, ob = za + na, zb + nb, oa + na * r, ob + nb * r
    return y.reshape(-1)


def exact(case, seed):
    op, dim = case["op"], _dim(case)
    if op == "sigma_c64":
        return _exact_c64(case, seed)
    if dim * 8.0 * case["norb"] ** 2 > 2.5e10 or (op == "vqe" and dim * case["gens"] > 2.5e9):
        return None
    h, g = _integrals(case, seed)
    S = _Space(case)
    if op == "sigma":
        return S.back(S.sigma(h, g, S.frame(_vector(case, seed, len(S.order)))))
    return {"davidson": _exact_davidson, "vqe": _exact_vqe, "adapt": _exact_adapt}[op](case, seed, S, h, g)

// Sigma on symmetry-blocked bases (several (alpha irrep, beta irrep) blocks).
//
// In the alpha-first frame c~ = eps c (fastplan.h) a group of a two-body
// Hamiltonian is one of: the diagonal; a pure-alpha or pure-beta term, a row or a
// column of the coefficient block times a factor of the other spin; a mixed
// single-single term Lam[E][F] sA_E sB_F.  A group moves irreps by (asym, bsym)
// and stays inside the basis only where asym = bsym, so with point-group
// integrals a destination row meets few excitations E, and each only the F of its
// own irrep: too few for the dense products of sigma_fast.cu.  One CTA computes one
// destination row a, a thread one column b at a time:
//   sigma~[a, b] = D(a, b) c~[a, b]
//     + sum over the row's pure-alpha entries   f(b) c~[a', b]       (coalesced)
//     + sum over the column's pure-beta entries f(a) c~[a, b']       (the row is in L1)
//     + sum_F sB_F(b') sum_{E of F's irrep, a^E valid} Lam[E][F] sA_E(a') c~[a^E, b^F]
// with the row's Lam_conn staged in shared memory and the column indices b^F read
// once per F for all E.
// Bound: L1 (67 % of its throughput; ~300 gathers per determinant at 14o in eight
// irreps, issue slots 53 %).  At 14o 7a+7b in eight irreps 1.10 ms; the tile kernel
// (sigma.cu), which finds partners and phases of every group inside each tile, 5.05
// ms.  The beta entries lie by entry, not by column, so that a warp reads them in one
// piece (by column: 1.31 ms).
#include "fastplan.h"
#include "ops.h"

#include <algorithm>
#include <cmath>
#include <cstring>
#include <memory>
#include <unordered_map>

namespace bsim {

namespace {

constexpr int kBlkThreads = 128;
constexpr size_t kBlkSmem = 96 * 1024;    // Lam_conn and the row factors of one row

// a constant-factor entry of an alpha row: source row (element offset), coefficient
struct BEnt {
    long long src;
    double coef;
};
// a table-factor entry of an alpha row: source, first table row << 3 | rank, row phases
struct BTab {
    long long src;
    int t, pad;
    double p[kSideMaxRank];
};
// a connected alpha single of a row: source row offset, excitation << 1 | sign
struct BExc {
    long long src;
    int e, pad;
};

struct BlkView {
    int nirr, nAt, nBt, rank_d, nF, ntA, ntB;
    const int *row_blk;                   // [nAt]
    const i64 *off;                       // blocks
    const int *nb, *astart, *bstart;
    const u64 *Ka;                        // [nAt]
    const double *PAd, *PBd;              // [nAt][rank_d], [rank_d][nBt]
    const i64 *acp, *atp;                 // CSR over alpha rows: constant, table entries
    const BEnt *ac;
    const BTab *at;
    // entries of the beta columns, entry e of column b at e * nBt + b (lanes read
    // neighbouring columns), source -1 past a column's last
    int nbc, nbt;                         // most constant, table entries of a column
    const int *bcs, *bts, *btt;           // local source; table row << 3 | rank
    const double *bcc, *btp;              // coefficient; phases [entry][r][nBt]
    const double *tabB, *tabA;            // [ntB][nBt] factors of alpha entries, [nAt][ntA] factors of beta entries
    const int *ep;                        // [nAt][nirr + 1] into ex
    const BExc *ex;
    const int *fp;                        // [nirr + 1]: F sorted by irrep
    const double *Lam;                    // [nE][nF]
    const int *gidx;                      // [nF][nBt]: (local index of b^F) << 1 | sign, or -1
};

template <typename Ti, typename Tin>
__global__ void __launch_bounds__(256)
blk_frame_kernel(const BlkView V, const Ti *__restrict__ bstr, const Tin *__restrict__ c, double *__restrict__ ct)
{
    const int a = blockIdx.x, k = V.row_blk[a], nb = V.nb[k];
    const i64 row = V.off[k] + (i64)(a - V.astart[k]) * nb;
    const u64 K = V.Ka[a];
    for (int b = threadIdx.x; b < nb; b += 256) {
        const double v = (double)c[row + b];
        ct[row + b] = par((u64)bstr[V.bstart[k] + b] & K) ? -v : v;
    }
}

template <typename Ti>
__global__ void __launch_bounds__(kBlkThreads)
blk_sigma_kernel(const BlkView V, const Ti *__restrict__ bstr, const double *__restrict__ ct, double *__restrict__ dst)
{
    extern __shared__ double sm[];
    const int a = blockIdx.x, k = V.row_blk[a], nb = V.nb[k];
    const i64 row = V.off[k] + (i64)(a - V.astart[k]) * nb;
    const int *ep = V.ep + (i64)a * (V.nirr + 1);
    // staged once per row: the constant alpha entries, the sources of the connected
    // singles, Lam_conn per irrep [F][E], the row's factors of the beta tables
    const i64 ac0 = V.acp[a];
    const int nac = (int)(V.acp[a + 1] - ac0), ne_all = ep[V.nirr] - ep[0];
    double *acc_c = sm;
    long long *acc_s = reinterpret_cast<long long *>(sm + nac), *exs = acc_s + nac;
    double *ta = reinterpret_cast<double *>(exs + ne_all), *lam = ta + V.ntA;
    for (int i = threadIdx.x; i < nac; i += kBlkThreads) {
        const BEnt x = V.ac[ac0 + i];
        acc_c[i] = x.coef;
        acc_s[i] = x.src;
    }
    for (int i = threadIdx.x; i < ne_all; i += kBlkThreads) exs[i] = V.ex[ep[0] + i].src;
    for (int i = threadIdx.x; i < V.ntA; i += kBlkThreads) ta[i] = V.tabA[(i64)a * V.ntA + i];
    int nl = 0;
    for (int g = 0; g < V.nirr; ++g) {
        const int e0 = ep[g], ne = ep[g + 1] - e0, f0 = V.fp[g], nf = V.fp[g + 1] - f0;
        for (int i = threadIdx.x; i < ne * nf; i += kBlkThreads) {
            const int x = V.ex[e0 + i % ne].e;
            const double v = V.Lam[(i64)(x >> 1) * V.nF + f0 + i / ne];
            lam[nl + i] = (x & 1) ? -v : v;
        }
        nl += ne * nf;
    }
    __syncthreads();
    const u64 K = V.Ka[a];
    const double *self = ct + row;
    for (int b = threadIdx.x; b < nb; b += kBlkThreads) {
        const int gb = V.bstart[k] + b;
        double acc = 0.0;
        for (int r = 0; r < V.rank_d; ++r) acc += V.PAd[(i64)a * V.rank_d + r] * __ldg(V.PBd + (i64)r * V.nBt + gb);
        acc *= self[b];
#pragma unroll 4
        for (int e = 0; e < nac; ++e) acc += acc_c[e] * __ldg(ct + acc_s[e] + b);
        for (i64 e = V.atp[a]; e < V.atp[a + 1]; ++e) {
            const BTab t = V.at[e];
            double f = 0.0;
            for (int r = 0; r < (t.t & 7); ++r) f += t.p[r] * __ldg(V.tabB + (i64)((t.t >> 3) + r) * V.nBt + gb);
            acc += f * __ldg(ct + t.src + b);
        }
#pragma unroll 4
        for (int e = 0; e < V.nbc; ++e) {
            const int s = __ldg(V.bcs + (i64)e * V.nBt + gb);
            if (s >= 0) acc += __ldg(V.bcc + (i64)e * V.nBt + gb) * __ldg(self + s);
        }
        for (int e = 0; e < V.nbt; ++e) {
            const int s = __ldg(V.bts + (i64)e * V.nBt + gb);
            if (s < 0) continue;
            const int t = __ldg(V.btt + (i64)e * V.nBt + gb);
            double f = 0.0;
            for (int r = 0; r < (t & 7); ++r) f += __ldg(V.btp + (i64)(e * kSideMaxRank + r) * V.nBt + gb) * ta[(t >> 3) + r];
            acc += f * __ldg(self + s);
        }
        const double *lg = lam;
        const long long *ex = exs;
        for (int g = 0; g < V.nirr; ++g) {
            const int ne = ep[g + 1] - ep[g];
#pragma unroll 2
            for (int f = V.fp[g]; f < V.fp[g + 1]; ++f, lg += ne) {
                const int gi = __ldg(V.gidx + (i64)f * V.nBt + gb);
                if (gi < 0) continue;
                const double *col = ct + (gi >> 1);
                double s = 0.0;
#pragma unroll 4
                for (int e = 0; e < ne; ++e) s += lg[e] * __ldg(col + ex[e]);
                acc += (gi & 1) ? -s : s;
            }
            ex += ne;
        }
        dst[row + b] = par((u64)bstr[gb] & K) ? -acc : acc;
    }
}

template <typename Ti>
struct BlkPlan {
    bool ok = false;
    Arena arena;
    BlkView v{};
    size_t smem = 0;
    const int *d_resid = nullptr;
    const int4 *d_resid_chunks = nullptr;
    int n_resid_chunks = 0;
    double *ct = nullptr;                 // the frame vector, allocated with the first call
    ~BlkPlan()
    {
        arena.release();
        if (ct) cudaFree(ct);
    }
};

inline int popc(u64 x) { return __builtin_popcountll(x); }

u64 mask_below_odd(u64 x, int norb)   // orbitals with an odd number of x bits below them
{
    u64 m = 0;
    for (int i = 0; i < norb; ++i)
        if (popc(x & ((1ull << i) - 1)) & 1) m |= 1ull << i;
    return m;
}
u64 mask_above_odd(u64 x, int norb)   // orbitals with an odd number of x bits above them
{
    u64 m = 0;
    for (int j = 0; j < norb; ++j)
        if (popc(x >> (j + 1)) & 1) m |= 1ull << j;
    return m;
}

template <typename Ti>
int build(const DevBasis<Ti> *B, const DevNet<Ti> *N, BlkPlan<Ti> *P)
{
    P->ok = false;
    const int norb = B->norb, nirr = B->num_irreps;
    if (B->num_blocks < 2 || norb > 63 || N->norb > norb || N->cplx) return BSIM_OK;
    const u64 full = (1ull << norb) - 1;
    const int nAt = (int)B->astrs.size(), nBt = (int)B->bstrs.size();
    // string -> block, local index, per spin
    struct Where { int blk, loc; };
    auto index = [&](const std::vector<Ti> &strs, const std::vector<int> &start, const std::vector<int> &cnt) {
        std::unordered_map<u64, Where> m;
        m.reserve(strs.size() * 2);
        for (int k = 0; k < B->num_blocks; ++k)
            for (int i = 0; i < cnt[k]; ++i) m[(u64)strs[start[k] + i]] = Where{k, i};
        return m;
    };
    const auto amap = index(B->astrs, B->astart, B->na), bmap = index(B->bstrs, B->bstart, B->nb);
    std::vector<int> row_blk(nAt), col_blk(nBt);
    std::vector<u64> Ka(nAt);
    for (int k = 0; k < B->num_blocks; ++k) {
        for (int i = 0; i < B->na[k]; ++i) row_blk[B->astart[k] + i] = k;
        for (int i = 0; i < B->nb[k]; ++i) col_blk[B->bstart[k] + i] = k;
    }
    for (int a = 0; a < nAt; ++a)
        for (int i = 0; i < norb; ++i)
            if (((u64)B->astrs[a] >> i) & 1u) Ka[a] ^= (1ull << i) - 1;
    const Ti *z = N->z.data();
    const double *w = N->w.data();
    auto phase = [&](u64 s, i64 zo, i64 wo, int nz, int r, u64 zxor) {
        double v = 0.0;
        for (int q = 0; q < nz; ++q) {
            const double x = w[wo + (i64)r * nz + q];
            v += (popc(s & ((u64)z[zo + q] ^ zxor)) & 1) ? -x : x;
        }
        return v;
    };

    std::vector<int> residual;
    std::vector<double> PAd, PBd;
    int rank_d = 0, diag = -1;
    // pure groups of one spin: own masks and weights, other-spin factor constant or tabled
    struct Side {
        std::vector<int> g, tab;              // group, first table row or -1
        std::vector<double> c;                // constant factors [kSideMaxRank]
        std::vector<double> tabs;             // [rows][other strings]
        int nt = 0;
    } sd[2];
    struct Rec { int E, F; double v; };
    std::vector<Rec> recs;
    std::unordered_map<u64, int> eid, fid;
    std::vector<u64> Em, Fm, mA, mB;
    std::vector<int> Firr, Eirr;
    for (i64 gi = 0; gi < N->ngs; ++gi) {
        const GroupDev &G = N->groups[(size_t)gi];
        if (G.rank == 0) continue;
        if (G.asym != G.bsym) continue;       // leaves the total irrep: reaches no determinant of the basis
        if (G.type == 0) {
            if (diag >= 0) { residual.push_back((int)gi); continue; }
            diag = (int)gi;
            rank_d = G.rank;
            PAd.resize((size_t)nAt * rank_d);
            PBd.resize((size_t)nBt * rank_d);
            for (int r = 0; r < rank_d; ++r) {
                for (int a = 0; a < nAt; ++a) PAd[(size_t)a * rank_d + r] = phase((u64)B->astrs[a], G.za_off, G.wa_off, G.nza, r, 0);
                for (int b = 0; b < nBt; ++b) PBd[(size_t)r * nBt + b] = phase((u64)B->bstrs[b], G.zb_off, G.wb_off, G.nzb, r, 0);
            }
        } else if (G.type == 1 || G.type == 2) {
            if (G.rank > kSideMaxRank) { residual.push_back((int)gi); continue; }
            Side &S = sd[G.type - 1];
            const bool al = G.type == 1;
            const u64 cm = al ? mask_above_odd(G.ax, norb) : mask_below_odd(G.bx, norb);
            const i64 zo = al ? G.zb_off : G.za_off, wo = al ? G.wb_off : G.wa_off;
            const int nz = al ? G.nzb : G.nza;
            const auto &other = al ? B->bstrs : B->astrs;
            bool constant = true;             // every mask empty or full in the frame
            for (int q = 0; q < nz; ++q) {
                const u64 m = ((u64)z[zo + q] ^ cm) & full;
                if (m != 0 && m != full) constant = false;
            }
            S.g.push_back((int)gi);
            S.tab.push_back(constant ? -1 : S.nt);
            for (int r = 0; r < kSideMaxRank; ++r)
                S.c.push_back(constant && r < G.rank ? phase((u64)other[0], zo, wo, nz, r, cm) : 0.0);
            if (!constant) {
                for (int r = 0; r < G.rank; ++r)
                    for (size_t s = 0; s < other.size(); ++s) S.tabs.push_back(phase((u64)other[s], zo, wo, nz, r, cm));
                S.nt += G.rank;
            }
        } else {
            if (G.rank != 1 || popc(G.ax) != 2 || popc(G.bx) != 2) { residual.push_back((int)gi); continue; }
            const u64 ma = mask_below_odd(G.bx, norb), mb = mask_above_odd(G.ax, norb);
            // lam (-1)^popc(s & m) on the strings that hold one of the two flipped
            // orbitals: the masks agree outside them, and the two values agree up to
            // the sign that the excitation's sign mask m gives them
            auto factor = [&](u64 x, i64 zo, i64 wo, int nz, u64 zx, u64 m, double *out) {
                for (int q = 0; q < nz; ++q)
                    if ((((u64)z[zo + q] ^ zx ^ m) & full & ~x) != 0) return false;
                const u64 p = x & (~x + 1), q = x ^ p;
                double v[2];
                const u64 s[2] = {p, q};
                for (int i = 0; i < 2; ++i) {
                    v[i] = phase(s[i], zo, wo, nz, 0, zx);
                    if (popc(s[i] & m) & 1) v[i] = -v[i];
                }
                *out = v[0];
                return std::fabs(v[0] - v[1]) <= 1e-12 * std::max(1.0, std::fabs(v[0]));
            };
            const auto ei = eid.find(G.ax);
            const auto fi = fid.find(G.bx);
            const u64 sa = ei == eid.end() ? (u64)z[G.za_off] ^ ma : mA[ei->second];
            const u64 sb = fi == fid.end() ? (u64)z[G.zb_off] ^ mb : mB[fi->second];
            double lam, mu;
            if (G.nza < 1 || G.nzb < 1 || !factor(G.ax, G.za_off, G.wa_off, G.nza, ma, sa, &lam) ||
                !factor(G.bx, G.zb_off, G.wb_off, G.nzb, mb, sb, &mu)) {
                residual.push_back((int)gi);
                continue;
            }
            int E = ei == eid.end() ? -1 : ei->second, F = fi == fid.end() ? -1 : fi->second;
            if (E < 0) {
                E = (int)Em.size();
                eid[G.ax] = E;
                Em.push_back(G.ax);
                mA.push_back(sa);
                Eirr.push_back(G.asym);
            }
            if (F < 0) {
                F = (int)Fm.size();
                fid[G.bx] = F;
                Fm.push_back(G.bx);
                mB.push_back(sb);
                Firr.push_back(G.bsym);
            }
            recs.push_back({E, F, ((popc(G.ax & ma) & 1) ? -1.0 : 1.0) * lam * mu});
        }
    }
    const int nE = (int)Em.size(), nF = (int)Fm.size();
    // F sorted by irrep
    std::vector<int> forder(nF), fpos(nF), fp(nirr + 1, 0);
    for (int f = 0; f < nF; ++f) forder[f] = f;
    std::stable_sort(forder.begin(), forder.end(), [&](int x, int y) { return Firr[x] < Firr[y]; });
    for (int i = 0; i < nF; ++i) {
        fpos[forder[i]] = i;
        if (Firr[forder[i]] >= nirr) return BSIM_OK;
        ++fp[Firr[forder[i]] + 1];
    }
    for (int g = 0; g < nirr; ++g) fp[g + 1] += fp[g];
    std::vector<double> Lam((size_t)nE * nF, 0.0);
    for (const Rec &r : recs) Lam[(size_t)r.E * nF + fpos[r.F]] += r.v;
    std::vector<int> gidx((size_t)nF * nBt, -1);
    for (int i = 0; i < nF; ++i) {
        const u64 fm = Fm[forder[i]], sm = mB[forder[i]];
        for (int b = 0; b < nBt; ++b) {
            const u64 s = (u64)B->bstrs[b];
            if (popc(s & fm) != 1) continue;
            const auto it = bmap.find(s ^ fm);
            if (it != bmap.end()) gidx[(size_t)i * nBt + b] = (it->second.loc << 1) | (popc((s ^ fm) & sm) & 1);
        }
    }
    // connected alpha singles per row, by irrep, where the source block exists
    std::vector<int> ep((size_t)nAt * (nirr + 1), 0);
    std::vector<BExc> ex;
    std::vector<int> eorder(nE);
    for (int e = 0; e < nE; ++e) eorder[e] = e;
    std::stable_sort(eorder.begin(), eorder.end(), [&](int x, int y) { return Eirr[x] < Eirr[y]; });
    size_t lam_max = 0;
    for (int a = 0; a < nAt; ++a) {
        const u64 s = (u64)B->astrs[a];
        int *p = &ep[(size_t)a * (nirr + 1)];
        size_t nl = 0, i = 0;
        for (int g = 0; g < nirr; ++g) {
            p[g] = (int)ex.size();
            for (; i < eorder.size() && Eirr[eorder[i]] <= g; ++i) {
                const int e = eorder[i];
                if (popc(s & Em[e]) != 1) continue;
                const auto it = amap.find(s ^ Em[e]);
                if (it == amap.end()) continue;
                const int ks = it->second.blk;
                ex.push_back(BExc{B->off[ks] + (i64)it->second.loc * B->nb[ks], (e << 1) | (popc((s ^ Em[e]) & mA[e]) & 1), 0});
            }
            nl += (size_t)((int)ex.size() - p[g]) * (fp[g + 1] - fp[g]);
        }
        p[nirr] = (int)ex.size();
        lam_max = std::max(lam_max, nl);
    }
    if (ex.size() > ((size_t)1 << 30)) return BSIM_OK;
    // pure entries of every alpha row and of every beta column
    std::vector<i64> cp[2], tp[2];
    std::vector<BEnt> ce[2];
    std::vector<BTab> te[2];
    for (int side = 0; side < 2; ++side) {
        const Side &S = sd[side];
        const auto &strs = side == 0 ? B->astrs : B->bstrs;
        const auto &map = side == 0 ? amap : bmap;
        const auto &blk = side == 0 ? row_blk : col_blk;
        cp[side].assign(1, 0);
        tp[side].assign(1, 0);
        for (size_t i = 0; i < strs.size(); ++i) {
            const u64 s = (u64)strs[i];
            for (size_t q = 0; q < S.g.size(); ++q) {
                const GroupDev &G = N->groups[(size_t)S.g[q]];
                const u64 x = side == 0 ? G.ax : G.bx;
                if (2 * popc(s & x) != popc(x)) continue;
                const auto it = map.find(s ^ x);
                if (it == map.end() || it->second.blk != blk[i]) continue;
                const i64 zo = side == 0 ? G.za_off : G.zb_off, wo = side == 0 ? G.wa_off : G.wb_off;
                const int nz = side == 0 ? G.nza : G.nzb, k = it->second.blk;
                const long long src = side == 0 ? B->off[k] + (i64)it->second.loc * B->nb[k] : it->second.loc;
                double p[kSideMaxRank] = {0, 0, 0, 0}, c = 0.0;
                for (int r = 0; r < G.rank; ++r) {
                    p[r] = phase(s ^ x, zo, wo, nz, r, 0);
                    c += p[r] * S.c[q * kSideMaxRank + r];
                }
                if (S.tab[q] < 0) ce[side].push_back(BEnt{src, c});
                else te[side].push_back(BTab{src, (S.tab[q] << 3) | G.rank, 0, {p[0], p[1], p[2], p[3]}});
            }
            cp[side].push_back((i64)ce[side].size());
            tp[side].push_back((i64)te[side].size());
        }
    }
    size_t max_ac = 0, max_ex = 0, nbc = 0, nbt = 0;
    for (int a = 0; a < nAt; ++a) {
        max_ac = std::max(max_ac, (size_t)(cp[0][a + 1] - cp[0][a]));
        max_ex = std::max(max_ex, (size_t)(ep[(size_t)a * (nirr + 1) + nirr] - ep[(size_t)a * (nirr + 1)]));
    }
    for (int b = 0; b < nBt; ++b) {
        nbc = std::max(nbc, (size_t)(cp[1][b + 1] - cp[1][b]));
        nbt = std::max(nbt, (size_t)(tp[1][b + 1] - tp[1][b]));
    }
    P->smem = (lam_max + (size_t)sd[1].nt + 2 * max_ac + max_ex) * sizeof(double);
    if (P->smem > kBlkSmem) return BSIM_OK;
    // the beta entries by column
    std::vector<int> bcs(nbc * nBt, -1), bts(nbt * nBt, -1), btt(nbt * nBt, 0);
    std::vector<double> bcc(nbc * nBt, 0.0), btp(nbt * kSideMaxRank * nBt, 0.0);
    for (int b = 0; b < nBt; ++b) {
        for (i64 i = cp[1][b]; i < cp[1][b + 1]; ++i) {
            const size_t o = (size_t)(i - cp[1][b]) * nBt + b;
            bcs[o] = (int)ce[1][(size_t)i].src;
            bcc[o] = ce[1][(size_t)i].coef;
        }
        for (i64 i = tp[1][b]; i < tp[1][b + 1]; ++i) {
            const size_t e = (size_t)(i - tp[1][b]);
            const BTab &t = te[1][(size_t)i];
            bts[e * nBt + b] = (int)t.src;
            btt[e * nBt + b] = t.t;
            for (int r = 0; r < kSideMaxRank; ++r) btp[(e * kSideMaxRank + r) * nBt + b] = t.p[r];
        }
    }
    // factors of beta entries by alpha row
    std::vector<double> tabA((size_t)nAt * sd[1].nt);
    for (int t = 0; t < sd[1].nt; ++t)
        for (int a = 0; a < nAt; ++a) tabA[(size_t)a * sd[1].nt + t] = sd[1].tabs[(size_t)t * nAt + a];
    // residual groups through the tile kernel
    std::stable_sort(residual.begin(), residual.end(), [&](int x, int y) {
        const GroupDev &p = N->groups[x], &q = N->groups[y];
        return p.type != q.type ? p.type < q.type : p.rank < q.rank;
    });
    std::vector<int4> chunks;
    for (size_t i = 0; i < residual.size();) {
        const GroupDev &G = N->groups[residual[i]];
        size_t j = i + 1;
        if (G.rank <= 2)
            while (j < residual.size() && j - i < 32 && N->groups[residual[j]].rank == G.rank &&
                   N->groups[residual[j]].type == G.type)
                ++j;
        chunks.push_back(make_int4((int)i, (int)(j - i), G.rank, G.type));
        i = j;
    }

    std::vector<char> blob;
    auto put = [&](const auto &v) {   // offset of the vector in the one upload
        using T = typename std::decay_t<decltype(v)>::value_type;
        const size_t o = (blob.size() + 255) & ~size_t(255);
        blob.resize(o + std::max<size_t>(v.size(), 1) * sizeof(T));
        if (!v.empty()) memcpy(blob.data() + o, v.data(), v.size() * sizeof(T));
        return o;
    };
    const size_t o_rb = put(row_blk), o_off = put(B->off), o_nb = put(B->nb), o_as = put(B->astart), o_bs = put(B->bstart),
                 o_Ka = put(Ka), o_PA = put(PAd), o_PB = put(PBd), o_acp = put(cp[0]), o_atp = put(tp[0]),
                 o_bcs = put(bcs), o_bts = put(bts), o_btt = put(btt), o_bcc = put(bcc), o_btp = put(btp),
                 o_ac = put(ce[0]), o_at = put(te[0]), o_tB = put(sd[0].tabs), o_tA = put(tabA), o_ep = put(ep), o_ex = put(ex),
                 o_fp = put(fp), o_L = put(Lam), o_g = put(gidx), o_r = put(residual), o_rc = put(chunks);
    int st = P->arena.reserve(blob.size());
    if (st != BSIM_OK) return st;
    char *d = P->arena.template take<char>(blob.size());
    BSIM_CUDA(cudaMemcpy(d, blob.data(), blob.size(), cudaMemcpyHostToDevice));
    auto at = [&](auto *type, size_t o) { return reinterpret_cast<decltype(type)>(d + o); };
    using I = const int *;
    using L = const i64 *;
    using D = const double *;
    P->v = BlkView{nirr, nAt, nBt, rank_d, nF, sd[1].nt, sd[0].nt,
                   at(I(), o_rb), at(L(), o_off), at(I(), o_nb), at(I(), o_as), at(I(), o_bs),
                   reinterpret_cast<const u64 *>(d + o_Ka), at(D(), o_PA), at(D(), o_PB), at(L(), o_acp), at(L(), o_atp),
                   reinterpret_cast<const BEnt *>(d + o_ac), reinterpret_cast<const BTab *>(d + o_at), (int)nbc, (int)nbt,
                   at(I(), o_bcs), at(I(), o_bts), at(I(), o_btt), at(D(), o_bcc), at(D(), o_btp),
                   at(D(), o_tB), at(D(), o_tA), at(I(), o_ep),
                   reinterpret_cast<const BExc *>(d + o_ex), at(I(), o_fp), at(D(), o_L), at(I(), o_g)};
    P->d_resid = at(I(), o_r);
    P->d_resid_chunks = reinterpret_cast<const int4 *>(d + o_rc);
    P->n_resid_chunks = (int)chunks.size();
    P->ok = true;
    return BSIM_OK;
}

}  // namespace

// sigma over every block; *used = false when the tile kernel must run.  Products
// and sums are FP64 for both precisions of the call (the FP32-bulk call asks for
// speed, and FP32 would not make this kernel faster).
template <typename Ti>
int sigma_blocks(const DevBasis<Ti> *B, const DevNet<Ti> *N, const double *src, const float *src32, double *dst,
                 bool mixed, cudaStream_t s, bool *used)
{
    *used = false;
    if (B->num_blocks < 2) return BSIM_OK;
    std::shared_ptr<BlkPlan<Ti>> P = N->blk_plans.template find<BlkPlan<Ti>>(B->serial);
    if (!P) {   // making the lists allocates and waits: not inside a capture, whose call the tile kernel serves
        cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
        BSIM_CUDA(cudaStreamIsCapturing(s, &cap));
        if (cap != cudaStreamCaptureStatusNone) return BSIM_OK;
    }
    const int st = P ? BSIM_OK : N->blk_plans.get(B->serial, &P, [&](std::shared_ptr<BlkPlan<Ti>> &plan) {
        auto p = std::make_shared<BlkPlan<Ti>>();
        int rc = build(B, N, p.get());
        if (rc == BSIM_OK && p->ok) {
            const cudaError_t e = dmalloc(&p->ct, sizeof(double) * B->dim);
            if (e != cudaSuccess) {
                p->ct = nullptr;
                rc = e == cudaErrorMemoryAllocation ? BSIM_ERR_ALLOC : cuda_status(e, "symmetry-blocked sigma");
            }
        }
        if (rc == BSIM_ERR_ALLOC) {   // no room for the lists: the tile kernel needs none
            (void)cudaGetLastError();
            p->ok = false;
            rc = BSIM_OK;
        }
        if (rc == BSIM_OK) plan = p;
        return rc;
    });
    if (st != BSIM_OK) return st;
    if (!P->ok) return BSIM_OK;
    if (src32) blk_frame_kernel<Ti, float><<<P->v.nAt, 256, 0, s>>>(P->v, B->view.bstrs, src32, P->ct);
    else blk_frame_kernel<Ti, double><<<P->v.nAt, 256, 0, s>>>(P->v, B->view.bstrs, src, P->ct);
    BSIM_CUDA(allow_smem(blk_sigma_kernel<Ti>));
    blk_sigma_kernel<Ti><<<P->v.nAt, kBlkThreads, P->smem, s>>>(P->v, B->view.bstrs, P->ct, dst);
    BSIM_CUDA(cudaGetLastError());
    if (P->n_resid_chunks > 0) {
        const int rc = sigma_generic_accumulate(B, N, P->d_resid, P->d_resid_chunks, P->n_resid_chunks, src, src32, dst,
                                                mixed, s);
        if (rc != BSIM_OK) return rc;
    }
    *used = true;
    return BSIM_OK;
}

template int sigma_blocks<unsigned>(const DevBasis<unsigned> *, const DevNet<unsigned> *, const double *, const float *,
                                    double *, bool, cudaStream_t, bool *);
template int sigma_blocks<unsigned long long>(const DevBasis<unsigned long long> *, const DevNet<unsigned long long> *,
                                              const double *, const float *, double *, bool, cudaStream_t, bool *);

}  // namespace bsim

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
constexpr size_t kBlkLists = (size_t)2 << 30;   // larger lists: the tile kernel

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

// ---- the lists, made on the device -----------------------------------------------------
// The host sorts the groups into forms; a warp per string finds the string's partners
// by its index tables, first to count its entries, then to write them in the order of
// the groups.  At 14o 7a+7b in eight irreps the first sigma takes 2.7 ms with them;
// with lists made by the host it took 105 ms, and through the tile kernel 5.1 ms.

// a pure group: own-spin flip mask, masks and weights; first row of its table of
// other-spin factors, or -1 and the constant factors
struct PureG {
    u64 x;
    i64 zo, wo;
    int nz, rank, tab, pad;
    double c[kSideMaxRank];
};
// a row of a factor table: masks and weights of the other spin, the frame's mask
struct TabG {
    i64 zo, wo;
    u64 cm;
    int nz, r;
};
// an excitation of one spin: flipped orbitals, sign mask, irrep
struct ExcG {
    u64 x, m;
    int irr, pad;
};

template <typename Ti>
__device__ __forceinline__ double blk_phase(const NetView<Ti> &N, u64 s, i64 zo, i64 wo, int nz, int r, u64 zxor)
{
    double v = 0.0;
    for (int q = 0; q < nz; ++q) {
        const double x = N.w[wo + (i64)r * nz + q];
        v += par(s & ((u64)N.z[zo + q] ^ zxor)) ? -x : x;
    }
    return v;
}
// block of a string's index in the list of all blocks' strings
__device__ __forceinline__ int blk_of(const int *start, int nblk, int i)
{
    int k = 0;
    while (k + 1 < nblk && start[k + 1] <= i) ++k;
    return k;
}
// place of string t in block k, or -1
template <typename Ti>
__device__ __forceinline__ int blk_find(const BasisView<Ti> &B, bool beta, int k, u64 t)
{
    const int loc = string_index(B, beta ? B.bmap : B.amap, beta ? B.nel_b : B.nel_a, (Ti)t);
    if (loc < 0 || loc >= (beta ? B.blk_nb : B.blk_na)[k]) return -1;
    const int i = (beta ? B.blk_bstart : B.blk_astart)[k] + loc;
    return (u64)(beta ? B.bstrs : B.astrs)[i] == t ? loc : -1;
}

// per row: its block, frame mask and diagonal factors; per column: its diagonal factors
template <typename Ti>
__global__ void blk_strings_kernel(const BasisView<Ti> B, const NetView<Ti> N, int diag, int nAt, int nBt,
                                   int *__restrict__ row_blk, u64 *__restrict__ Ka, double *__restrict__ PAd,
                                   double *__restrict__ PBd)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    GroupDev g{};
    if (diag >= 0) g = N.g[diag];
    if (i < nAt) {
        const u64 s = (u64)B.astrs[i];
        u64 K = 0;
        for (u64 y = s; y; y &= y - 1) K ^= (y & (~y + 1)) - 1;
        row_blk[i] = blk_of(B.blk_astart, B.num_blocks, i);
        Ka[i] = K;
        for (int r = 0; r < g.rank; ++r) PAd[(i64)i * g.rank + r] = blk_phase(N, s, g.za_off, g.wa_off, g.nza, r, 0);
    } else if (i < nAt + nBt) {
        const int b = i - nAt;
        for (int r = 0; r < g.rank; ++r)
            PBd[(i64)r * nBt + b] = blk_phase(N, (u64)B.bstrs[b], g.zb_off, g.wb_off, g.nzb, r, 0);
    }
}

// factor tables: entry (row t, string s) at t * rs + s * ss
template <typename Ti>
__global__ void blk_tab_kernel(const NetView<Ti> N, const Ti *__restrict__ strs, int n, const TabG *__restrict__ tabs,
                               i64 rs, i64 ss, double *__restrict__ out)
{
    const TabG t = tabs[blockIdx.y];
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        out[(i64)blockIdx.y * rs + (i64)i * ss] = blk_phase(N, (u64)strs[i], t.zo, t.wo, t.nz, t.r, t.cm);
}

template <typename Ti>
__global__ void blk_gidx_kernel(const BasisView<Ti> B, int nBt, const ExcG *__restrict__ F, int *__restrict__ gidx)
{
    const ExcG f = F[blockIdx.y];
    for (int b = blockIdx.x * blockDim.x + threadIdx.x; b < nBt; b += gridDim.x * blockDim.x) {
        const u64 s = (u64)B.bstrs[b], t = s ^ f.x;
        int g = -1;
        if (__popcll(s & f.x) == 1) {
            const int loc = string_index(B, B.bmap, B.nel_b, (Ti)t);
            if (loc >= 0) g = (loc << 1) | par(t & f.m);
        }
        gidx[(i64)blockIdx.y * nBt + b] = g;
    }
}

constexpr int kBuildWarps = 8;

// Connected alpha singles of every row, E sorted by irrep; out == nullptr: counts per
// irrep (zeroed before) into cnt[row][nirr], else entries from ep[row][0].
template <typename Ti>
__global__ void __launch_bounds__(32 * kBuildWarps)
blk_singles_kernel(const BasisView<Ti> B, int nAt, int nirr, int nE, const ExcG *__restrict__ E, int *__restrict__ cnt,
                   const int *__restrict__ ep, BExc *__restrict__ out)
{
    const int a = blockIdx.x * kBuildWarps + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (a >= nAt) return;
    const u64 s = (u64)B.astrs[a];
    const int asym = B.blk_asym[blk_of(B.blk_astart, B.num_blocks, a)];
    int at = out ? ep[(i64)a * (nirr + 1)] : 0;
    for (int e0 = 0; e0 < nE; e0 += 32) {
        const int e = e0 + lane;
        int ks = -1, loc = -1;
        ExcG x{};
        if (e < nE && __popcll(s & (x = E[e]).x) == 1) {
            for (int k = 0; k < B.num_blocks; ++k)
                if (B.blk_asym[k] == (asym ^ x.irr)) ks = k;
            if (ks >= 0) loc = blk_find(B, false, ks, s ^ x.x);
        }
        const unsigned on = __ballot_sync(0xffffffffu, loc >= 0);
        if (loc >= 0) {
            if (out)
                out[at + __popc(on & ((1u << lane) - 1))] =
                    BExc{B.blk_off[ks] + (i64)loc * B.blk_nb[ks], (e << 1) | par((s ^ x.x) & x.m), 0};
            else
                atomicAdd(cnt + (i64)a * nirr + x.irr, 1);
        }
        at += __popc(on);
    }
}

// where the entries of one spin's strings go: rows of alpha strings by CSR, beta
// columns by entry (BlkView)
struct PureOut {
    const i64 *acp, *atp;
    BEnt *ac;
    BTab *at;
    int nBt;
    int *bcs, *bts, *btt;
    double *bcc, *btp;
};

// Pure entries of every string of one spin; W.ac == W.bcs == nullptr: counts of
// constant and table entries into cnt[string].
template <typename Ti, bool BETA, bool COUNT>
__global__ void __launch_bounds__(32 * kBuildWarps)
blk_pure_kernel(const BasisView<Ti> B, const NetView<Ti> N, int n, int ng, const PureG *__restrict__ G,
                int2 *__restrict__ cnt, const PureOut W)
{
    const int i = blockIdx.x * kBuildWarps + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (i >= n) return;
    const u64 s = (u64)(BETA ? B.bstrs : B.astrs)[i];
    const int k = blk_of(BETA ? B.blk_bstart : B.blk_astart, B.num_blocks, i);
    int nc = 0, nt = 0;
    for (int q0 = 0; q0 < ng; q0 += 32) {
        const int q = q0 + lane;
        int loc = -1, tab = 0;
        u64 x = 0;
        if (q < ng) {
            x = G[q].x;
            tab = G[q].tab;
            if (2 * __popcll(s & x) == __popcll(x)) loc = blk_find(B, BETA, k, s ^ x);
        }
        const unsigned c = __ballot_sync(0xffffffffu, loc >= 0 && tab < 0);
        const unsigned t = __ballot_sync(0xffffffffu, loc >= 0 && tab >= 0);
        if (!COUNT && loc >= 0) {
            const PureG g = G[q];
            const int pos = tab < 0 ? nc + __popc(c & ((1u << lane) - 1)) : nt + __popc(t & ((1u << lane) - 1));
            const i64 src = BETA ? loc : B.blk_off[k] + (i64)loc * B.blk_nb[k];
            double p[kSideMaxRank] = {0.0, 0.0, 0.0, 0.0}, coef = 0.0;
            for (int r = 0; r < g.rank; ++r) {
                p[r] = blk_phase(N, s ^ x, g.zo, g.wo, g.nz, r, 0);
                coef += p[r] * g.c[r];
            }
            if (BETA) {
                const i64 o = (i64)pos * W.nBt + i;
                if (tab < 0) {
                    W.bcs[o] = (int)src;
                    W.bcc[o] = coef;
                } else {
                    W.bts[o] = (int)src;
                    W.btt[o] = (tab << 3) | g.rank;
                    for (int r = 0; r < kSideMaxRank; ++r) W.btp[((i64)pos * kSideMaxRank + r) * W.nBt + i] = p[r];
                }
            } else if (tab < 0) {
                W.ac[W.acp[i] + pos] = BEnt{src, coef};
            } else {
                W.at[W.atp[i] + pos] = BTab{src, (tab << 3) | g.rank, 0, {p[0], p[1], p[2], p[3]}};
            }
        }
        nc += __popc(c);
        nt += __popc(t);
    }
    if (COUNT && lane == 0) cnt[i] = make_int2(nc, nt);
}

// pieces of one device allocation
struct Blob {
    size_t n = 0;
    template <typename T>
    size_t add(size_t count)
    {
        const size_t o = (n + 255) & ~size_t(255);
        n = o + std::max<size_t>(count, 1) * sizeof(T);
        return o;
    }
};
struct TempMem {
    char *p = nullptr;
    ~TempMem() { if (p) cudaFree(p); }
};

template <typename Ti>
int build(const DevBasis<Ti> *B, const DevNet<Ti> *N, BlkPlan<Ti> *P, cudaStream_t s)
{
    P->ok = false;
    const int norb = B->norb, nirr = B->num_irreps;
    if (B->num_blocks < 2 || norb > 63 || N->norb > norb || N->cplx) return BSIM_OK;
    const u64 full = (1ull << norb) - 1;
    const int nAt = (int)B->astrs.size(), nBt = (int)B->bstrs.size();
    const Ti *z = N->z.data();
    const double *w = N->w.data();
    auto phase = [&](u64 x, i64 zo, i64 wo, int nz, int r, u64 zxor) {
        double v = 0.0;
        for (int q = 0; q < nz; ++q) {
            const double y = w[wo + (i64)r * nz + q];
            v += (popc(x & ((u64)z[zo + q] ^ zxor)) & 1) ? -y : y;
        }
        return v;
    };

    std::vector<int> residual;
    int rank_d = 0, diag = -1;
    struct Side {   // pure groups of one spin, their tables of other-spin factors
        std::vector<PureG> g;
        std::vector<TabG> tabs;
    } sd[2];
    struct Rec { int E, F; double v; };
    std::vector<Rec> recs;
    std::unordered_map<u64, int> eid, fid;
    std::vector<ExcG> Eg, Fg;
    for (i64 gi = 0; gi < N->ngs; ++gi) {
        const GroupDev &G = N->groups[(size_t)gi];
        if (G.rank == 0) continue;
        if (G.asym != G.bsym) continue;       // leaves the total irrep: reaches no determinant of the basis
        if (G.type == 0) {
            if (diag >= 0) { residual.push_back((int)gi); continue; }
            diag = (int)gi;
            rank_d = G.rank;
        } else if (G.type == 1 || G.type == 2) {
            if (G.rank > kSideMaxRank) { residual.push_back((int)gi); continue; }
            Side &S = sd[G.type - 1];
            const bool al = G.type == 1;
            const u64 cm = al ? mask_above_odd(G.ax, norb) : mask_below_odd(G.bx, norb);
            const i64 zo = al ? G.zb_off : G.za_off, wo = al ? G.wb_off : G.wa_off;
            const int nz = al ? G.nzb : G.nza;
            const u64 other = (u64)(al ? B->bstrs : B->astrs)[0];
            bool constant = true;             // every mask empty or full in the frame
            for (int q = 0; q < nz; ++q) {
                const u64 m = ((u64)z[zo + q] ^ cm) & full;
                if (m != 0 && m != full) constant = false;
            }
            PureG p{al ? G.ax : G.bx, al ? G.za_off : G.zb_off, al ? G.wa_off : G.wb_off, al ? G.nza : G.nzb, G.rank,
                    constant ? -1 : (int)S.tabs.size(), 0, {0.0, 0.0, 0.0, 0.0}};
            for (int r = 0; r < G.rank; ++r) {
                if (constant) p.c[r] = phase(other, zo, wo, nz, r, cm);
                else S.tabs.push_back(TabG{zo, wo, cm, nz, r});
            }
            S.g.push_back(p);
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
                const u64 one[2] = {p, q};
                for (int i = 0; i < 2; ++i) {
                    v[i] = phase(one[i], zo, wo, nz, 0, zx);
                    if (popc(one[i] & m) & 1) v[i] = -v[i];
                }
                *out = v[0];
                return std::fabs(v[0] - v[1]) <= 1e-12 * std::max(1.0, std::fabs(v[0]));
            };
            const auto ei = eid.find(G.ax);
            const auto fi = fid.find(G.bx);
            const u64 sa = ei == eid.end() ? (u64)z[G.za_off] ^ ma : Eg[ei->second].m;
            const u64 sb = fi == fid.end() ? (u64)z[G.zb_off] ^ mb : Fg[fi->second].m;
            double lam, mu;
            if (G.nza < 1 || G.nzb < 1 || !factor(G.ax, G.za_off, G.wa_off, G.nza, ma, sa, &lam) ||
                !factor(G.bx, G.zb_off, G.wb_off, G.nzb, mb, sb, &mu)) {
                residual.push_back((int)gi);
                continue;
            }
            int E = ei == eid.end() ? -1 : ei->second, F = fi == fid.end() ? -1 : fi->second;
            if (E < 0) {
                E = (int)Eg.size();
                eid[G.ax] = E;
                Eg.push_back(ExcG{G.ax, sa, G.asym, 0});
            }
            if (F < 0) {
                F = (int)Fg.size();
                fid[G.bx] = F;
                Fg.push_back(ExcG{G.bx, sb, G.bsym, 0});
            }
            recs.push_back({E, F, ((popc(G.ax & ma) & 1) ? -1.0 : 1.0) * lam * mu});
        }
    }
    const int nE = (int)Eg.size(), nF = (int)Fg.size(), nt0 = (int)sd[0].tabs.size(), nt1 = (int)sd[1].tabs.size();
    if (nt0 > 65535 || nt1 > 65535) return BSIM_OK;   // a grid dimension of blk_tab_kernel
    // E and F sorted by irrep
    auto by_irrep = [&](std::vector<ExcG> &v, std::vector<int> &pos) {
        std::vector<int> order(v.size());
        for (size_t i = 0; i < order.size(); ++i) order[i] = (int)i;
        std::stable_sort(order.begin(), order.end(), [&](int x, int y) { return v[x].irr < v[y].irr; });
        std::vector<ExcG> t(v.size());
        pos.resize(v.size());
        for (size_t i = 0; i < order.size(); ++i) {
            t[i] = v[order[i]];
            pos[order[i]] = (int)i;
        }
        v.swap(t);
        return v.empty() || v.back().irr < nirr;
    };
    std::vector<int> epos, fpos, fp(nirr + 1, 0);
    if (!by_irrep(Eg, epos) || !by_irrep(Fg, fpos)) return BSIM_OK;
    for (const ExcG &f : Fg) ++fp[f.irr + 1];
    for (int g = 0; g < nirr; ++g) fp[g + 1] += fp[g];
    std::vector<double> Lam((size_t)nE * nF, 0.0);
    for (const Rec &r : recs) Lam[(size_t)epos[r.E] * nF + fpos[r.F]] += r.v;
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

    // counts
    auto upload = [](char *d, const auto &v) {
        return v.empty() ? cudaSuccess : cudaMemcpy(d, v.data(), v.size() * sizeof(v[0]), cudaMemcpyHostToDevice);
    };
    Blob T;
    const size_t t_g[2] = {T.add<PureG>(sd[0].g.size()), T.add<PureG>(sd[1].g.size())};
    const size_t t_t[2] = {T.add<TabG>(nt0), T.add<TabG>(nt1)};
    const size_t t_e = T.add<ExcG>(nE), t_f = T.add<ExcG>(nF);
    const size_t t_c = T.add<int2>((size_t)nAt + nBt), t_n = T.add<int>((size_t)nAt * nirr);
    TempMem tmp;
    cudaError_t e = dmalloc(&tmp.p, T.n);
    if (e != cudaSuccess) {
        tmp.p = nullptr;
        return e == cudaErrorMemoryAllocation ? BSIM_ERR_ALLOC : cuda_status(e, "symmetry-blocked sigma");
    }
    for (int side = 0; side < 2; ++side) {
        BSIM_CUDA(upload(tmp.p + t_g[side], sd[side].g));
        BSIM_CUDA(upload(tmp.p + t_t[side], sd[side].tabs));
    }
    BSIM_CUDA(upload(tmp.p + t_e, Eg));
    BSIM_CUDA(upload(tmp.p + t_f, Fg));
    const PureG *dG[2] = {reinterpret_cast<PureG *>(tmp.p + t_g[0]), reinterpret_cast<PureG *>(tmp.p + t_g[1])};
    const TabG *dT[2] = {reinterpret_cast<TabG *>(tmp.p + t_t[0]), reinterpret_cast<TabG *>(tmp.p + t_t[1])};
    const ExcG *dE = reinterpret_cast<ExcG *>(tmp.p + t_e), *dF = reinterpret_cast<ExcG *>(tmp.p + t_f);
    int2 *d_cnt = reinterpret_cast<int2 *>(tmp.p + t_c);
    int *d_ne = reinterpret_cast<int *>(tmp.p + t_n);
    const unsigned gA = (unsigned)((nAt + kBuildWarps - 1) / kBuildWarps), gB = (unsigned)((nBt + kBuildWarps - 1) / kBuildWarps);
    constexpr int kBT = 32 * kBuildWarps;
    BSIM_CUDA(cudaMemsetAsync(d_ne, 0, sizeof(int) * (size_t)nAt * nirr, s));
    blk_singles_kernel<Ti><<<gA, kBT, 0, s>>>(B->view, nAt, nirr, nE, dE, d_ne, nullptr, nullptr);
    blk_pure_kernel<Ti, false, true><<<gA, kBT, 0, s>>>(B->view, N->view, nAt, (int)sd[0].g.size(), dG[0], d_cnt, PureOut{});
    blk_pure_kernel<Ti, true, true><<<gB, kBT, 0, s>>>(B->view, N->view, nBt, (int)sd[1].g.size(), dG[1], d_cnt + nAt,
                                                       PureOut{});
    BSIM_CUDA(cudaGetLastError());
    std::vector<int2> cnt((size_t)nAt + nBt);
    std::vector<int> ne((size_t)nAt * nirr);
    BSIM_CUDA(cudaMemcpyAsync(cnt.data(), d_cnt, cnt.size() * sizeof(int2), cudaMemcpyDeviceToHost, s));
    BSIM_CUDA(cudaMemcpyAsync(ne.data(), d_ne, ne.size() * sizeof(int), cudaMemcpyDeviceToHost, s));
    BSIM_CUDA(cudaStreamSynchronize(s));
    std::vector<i64> acp(nAt + 1, 0), atp(nAt + 1, 0);
    std::vector<int> ep((size_t)nAt * (nirr + 1));
    i64 nex = 0;
    size_t max_ac = 0, max_ex = 0, lam_max = 0, nbc = 0, nbt = 0;
    for (int a = 0; a < nAt; ++a) {
        acp[a + 1] = acp[a] + cnt[a].x;
        atp[a + 1] = atp[a] + cnt[a].y;
        const i64 first = nex;
        size_t nl = 0;
        for (int g = 0; g <= nirr; ++g) {
            ep[(size_t)a * (nirr + 1) + g] = (int)nex;
            if (g == nirr) break;
            const int k = ne[(size_t)a * nirr + g];
            nex += k;
            nl += (size_t)k * (fp[g + 1] - fp[g]);
        }
        if (nex > ((i64)1 << 30)) return BSIM_OK;
        max_ac = std::max(max_ac, (size_t)cnt[a].x);
        max_ex = std::max(max_ex, (size_t)(nex - first));
        lam_max = std::max(lam_max, nl);
    }
    for (int b = 0; b < nBt; ++b) {
        nbc = std::max(nbc, (size_t)cnt[(size_t)nAt + b].x);
        nbt = std::max(nbt, (size_t)cnt[(size_t)nAt + b].y);
    }
    P->smem = (lam_max + (size_t)nt1 + 2 * max_ac + max_ex) * sizeof(double);
    if (P->smem > kBlkSmem) return BSIM_OK;

    // the lists; what the host made comes first and goes up in one copy
    Blob D;
    const size_t o_fp = D.add<int>(nirr + 1), o_L = D.add<double>(Lam.size()), o_acp = D.add<i64>(nAt + 1),
                 o_atp = D.add<i64>(nAt + 1), o_ep = D.add<int>(ep.size()), o_r = D.add<int>(residual.size()),
                 o_rc = D.add<int4>(chunks.size());
    const size_t host_bytes = D.n;
    const size_t o_rb = D.add<int>(nAt), o_Ka = D.add<u64>(nAt), o_PA = D.add<double>((size_t)nAt * rank_d),
                 o_PB = D.add<double>((size_t)nBt * rank_d), o_ac = D.add<BEnt>((size_t)acp[nAt]),
                 o_at = D.add<BTab>((size_t)atp[nAt]), o_bcs = D.add<int>(nbc * nBt), o_bts = D.add<int>(nbt * nBt),
                 o_btt = D.add<int>(nbt * nBt), o_bcc = D.add<double>(nbc * nBt),
                 o_btp = D.add<double>(nbt * kSideMaxRank * nBt), o_tB = D.add<double>((size_t)nt0 * nBt),
                 o_tA = D.add<double>((size_t)nt1 * nAt), o_ex = D.add<BExc>((size_t)nex),
                 o_g = D.add<int>((size_t)nF * nBt);
    // The tile kernel needs no memory: it serves where the lists would be larger than
    // kBlkLists (14o 7a+7b in eight irreps takes 18 MB, 16o 8a+8b 90 MB), or lists and
    // frame vector larger than sigma's scratch limit or half of the free memory.
    size_t free_b = 0, total_b = 0;
    BSIM_CUDA(cudaMemGetInfo(&free_b, &total_b));
    if (D.n > kBlkLists || D.n + sizeof(double) * (size_t)B->dim > std::min(scratch_limit(), free_b / 2)) return BSIM_OK;
    int st = P->arena.reserve(D.n);
    if (st != BSIM_OK) return st;
    char *d = P->arena.template take<char>(D.n);
    std::vector<char> host(host_bytes, 0);
    auto put = [&](size_t o, const auto &v) {
        if (!v.empty()) memcpy(host.data() + o, v.data(), v.size() * sizeof(v[0]));
    };
    put(o_fp, fp); put(o_L, Lam); put(o_acp, acp); put(o_atp, atp); put(o_ep, ep); put(o_r, residual); put(o_rc, chunks);
    BSIM_CUDA(cudaMemcpy(d, host.data(), host_bytes, cudaMemcpyHostToDevice));
    auto at = [&](auto *type, size_t o) { return reinterpret_cast<decltype(type)>(d + o); };
    using I = int *;
    using L = i64 *;
    using R = double *;
    blk_strings_kernel<Ti><<<(unsigned)((nAt + nBt + 255) / 256), 256, 0, s>>>(
        B->view, N->view, diag, nAt, nBt, at(I(), o_rb), reinterpret_cast<u64 *>(d + o_Ka), at(R(), o_PA), at(R(), o_PB));
    const unsigned xB = (unsigned)std::min(256, (nBt + 255) / 256), xA = (unsigned)std::min(256, (nAt + 255) / 256);
    if (nt0 > 0) blk_tab_kernel<Ti><<<dim3(xB, nt0), 256, 0, s>>>(N->view, B->view.bstrs, nBt, dT[0], nBt, 1, at(R(), o_tB));
    if (nt1 > 0) blk_tab_kernel<Ti><<<dim3(xA, nt1), 256, 0, s>>>(N->view, B->view.astrs, nAt, dT[1], 1, nt1, at(R(), o_tA));
    if (nF > 0) blk_gidx_kernel<Ti><<<dim3(xB, nF), 256, 0, s>>>(B->view, nBt, dF, at(I(), o_g));
    BSIM_CUDA(cudaMemsetAsync(d + o_bcs, 0xff, sizeof(int) * nbc * nBt, s));   // -1: no entry
    BSIM_CUDA(cudaMemsetAsync(d + o_bts, 0xff, sizeof(int) * nbt * nBt, s));
    PureOut W{at(L(), o_acp), at(L(), o_atp), reinterpret_cast<BEnt *>(d + o_ac), reinterpret_cast<BTab *>(d + o_at), nBt,
              at(I(), o_bcs), at(I(), o_bts), at(I(), o_btt), at(R(), o_bcc), at(R(), o_btp)};
    blk_singles_kernel<Ti><<<gA, kBT, 0, s>>>(B->view, nAt, nirr, nE, dE, nullptr, at(I(), o_ep),
                                              reinterpret_cast<BExc *>(d + o_ex));
    blk_pure_kernel<Ti, false, false><<<gA, kBT, 0, s>>>(B->view, N->view, nAt, (int)sd[0].g.size(), dG[0], nullptr, W);
    blk_pure_kernel<Ti, true, false><<<gB, kBT, 0, s>>>(B->view, N->view, nBt, (int)sd[1].g.size(), dG[1], nullptr, W);
    BSIM_CUDA(cudaGetLastError());
    BSIM_CUDA(cudaStreamSynchronize(s));   // the group tables are freed on return
    P->v = BlkView{nirr, nAt, nBt, rank_d, nF, nt1, nt0,
                   at(I(), o_rb), B->view.blk_off, B->view.blk_nb, B->view.blk_astart, B->view.blk_bstart,
                   reinterpret_cast<const u64 *>(d + o_Ka), at(R(), o_PA), at(R(), o_PB), at(L(), o_acp), at(L(), o_atp),
                   W.ac, W.at, (int)nbc, (int)nbt, W.bcs, W.bts, W.btt, W.bcc, W.btp, at(R(), o_tB), at(R(), o_tA),
                   at(I(), o_ep), reinterpret_cast<const BExc *>(d + o_ex), at(I(), o_fp), at(R(), o_L), at(I(), o_g)};
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
        int rc = build(B, N, p.get(), s);
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

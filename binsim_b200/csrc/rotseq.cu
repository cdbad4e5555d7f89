// Rotation sequences exp(theta_m G_m) ... exp(theta_1 G_1) of excitation
// generators, up to four components per pass over the state.
//
// A component G = f sA sB (|dst><src| - |src><dst|) pairs a determinant with the
// one whose strings are flipped by the masks (ax, bx).  The components of one
// spin-adapted generator flip the same few orbitals: their alpha masks lie in
// the span of two masks ga, their beta masks in the span of two masks gb, so
// they act inside closed sets of 4 x 4 determinants, (alpha orbit
// {a, a^g1, a^g2, a^g1^g2}) x (beta orbit).  One thread owns such a set and
// rotates the pairs of one component after another; what the components share
// stays in L1.  The pair kernels (pairlist.cu) stream the state once per
// component, and stream every string pair that the flip masks connect, two
// thirds of which a double excitation multiplies by a phase of zero.
//
// Which members a component moves depends only on the occupation of the orbitals
// it looks at, so the orbits of one spin are listed sorted by that pattern: the
// threads of a warp (consecutive beta orbits, one alpha orbit) take the same
// branches.  The lists are made on the device for a batch of units at a time:
// the size of a pattern's bucket is a binomial coefficient and a string's place
// in it is the rank of its other orbitals, so every string finds its place
// alone.
//
// Bound: at 14o 7a+7b the latency and traffic of scattered 8-byte accesses (3.3 TB/s
// of HBM, the sectors that neighbouring patterns share are fetched more than once;
// L1 and L2 hit 40 % and 60 %); at small sizes the launch
// latency, of which programmatic dependent launch hides a part (a unit's CTAs
// read their lists while the previous unit finishes).
// Measured and not kept: the 16 members in registers, every component over all of
// them (the same time at 14o, instruction-bound there).
#include "rotseq.h"

#include <algorithm>
#include <cmath>
#include <mutex>

namespace bsim {

namespace {

constexpr int kRotMaxBits = 8;         // orbitals of one spin that a unit looks at
constexpr size_t kRotListBytes = (size_t)128 << 20;   // orbit lists of one batch

// what the list kernel needs of a unit
struct RotUnitDev {
    u64 g[2][2];                       // [spin][flip mask]
    u64 um[2];                         // [spin] every orbital looked at
    u64 x[2][kRotComps], src[2][kRotComps], z[2][kRotComps];   // orbitals looked at, source pattern, sign mask
    int m, pad;
};

// Members of the orbit of s under the flip masks g1, g2 (bit 0, bit 1 of the
// member's number): valid when the string has the same electron count and is
// not a repeat of another member.
__host__ __device__ __forceinline__ u64 rot_member(const u64 *g, u64 s, int e)
{
    return s ^ ((e & 1) ? g[0] : 0ull) ^ ((e & 2) ? g[1] : 0ull);
}
__host__ __device__ __forceinline__ int popc64(u64 x)
{
#ifdef __CUDA_ARCH__
    return __popcll(x);
#else
    return __builtin_popcountll(x);
#endif
}
__host__ __device__ __forceinline__ bool rot_valid(const u64 *g, u64 s, int e)
{
    if (((e & 1) && !g[0]) || ((e & 2) && !g[1])) return false;
    return popc64(rot_member(g, s, e)) == popc64(s);
}
// The bucket key of an occupation pattern s of the orbitals looked at: valid
// members << 16 | bit 4 k + e where component k moves member e as its source;
// 0 when another string lists the orbit (the smallest member does) or nothing
// moves it.
__host__ __device__ __forceinline__ unsigned rot_key(const RotUnitDev &U, int sp, u64 s)
{
    unsigned a = 0;
    int nv = 0;
    for (int e = 0; e < 4; ++e) {
        if (!rot_valid(U.g[sp], s, e)) continue;
        const u64 t = rot_member(U.g[sp], s, e);
        if (t < s) return 0;
        ++nv;
        for (int k = 0; k < U.m; ++k)
            if ((t & U.x[sp][k]) == U.src[sp][k]) a |= 1u << (4 * k + e);
    }
    return a ? ((unsigned)nv << 16) | a : 0u;
}
// pattern number p (bit i: the i-th orbital of um is occupied) as a string
__host__ __device__ __forceinline__ u64 rot_pattern(u64 um, int p)
{
    u64 s = 0;
    for (int i = 0; um; ++i, um &= um - 1)
        if ((p >> i) & 1) s |= um & (~um + 1);
    return s;
}

// Orbit lists: per unit nA alpha then nB beta slots of {member index or -1} x 4
// and a word of bits 4 k + e: component k moves member e as its source;
// bits 16 + 4 k + e: the sign of component k on member e.
template <typename Ti>
__global__ void __launch_bounds__(256)
rot_list_kernel(const BasisView<Ti> B, const RotUnitDev *__restrict__ units, int nA, int nB, int4 *__restrict__ idx,
                unsigned *__restrict__ bits)
{
    __shared__ unsigned key[256];
    __shared__ int cnt[256], off[256];
    const int unit = blockIdx.y >> 1, sp = blockIdx.y & 1;
    const RotUnitDev &U = units[unit];
    const u64 um = U.um[sp];
    const int nu = __popcll(um), nel = sp ? B.nel_b : B.nel_a, m = U.m;
    {   // one thread per occupation pattern: its key and how many strings show it
        const int p = threadIdx.x;
        unsigned kp = 0;
        int c = 0;
        if (p < (1 << nu)) {
            const u64 s = rot_pattern(um, p);
            const int rest = nel - __popcll(s), room = B.norb - nu;
            if (rest >= 0 && rest <= room && (kp = rot_key(U, sp, s)) != 0) c = (int)B.binom[room * 65 + rest];
        }
        key[p] = kp;
        cnt[p] = c;
    }
    __syncthreads();
    const int n = sp ? nB : nA;
    const i64 base = (i64)unit * (nA + nB) + (sp ? nA : 0);
    const Ti *strs = sp ? B.bstrs : B.astrs;
    const int *map = sp ? B.bmap : B.amap;
    {   // buckets in the order of their keys, the largest orbits first
        const int p = threadIdx.x;
        int o = 0;
        for (int q = 0; q < (1 << nu); ++q)
            if (key[q] > key[p] || (key[q] == key[p] && q < p)) o += cnt[q];
        off[p] = o;
    }
    __syncthreads();
    for (int i = blockIdx.x * 256 + threadIdx.x; i < n; i += gridDim.x * 256) {
        const u64 s = (u64)strs[i];
        int p = 0, q = 0;
        for (u64 y = um; y; y &= y - 1, ++q)
            if (s & (y & (~y + 1))) p |= 1 << q;
        if (key[p] == 0) continue;
        i64 r = off[p];
        q = 1;
        for (u64 y = s & ~um; y; y &= y - 1, ++q) {   // colex rank of the other orbitals among themselves
            const u64 low = (y & (~y + 1)) - 1;
            r += B.binom[(__popcll(low) - __popcll(low & um)) * 65 + q];
        }
        int id[4];
        unsigned b = key[p] & 0xffffu;
        for (int e = 0; e < 4; ++e) {
            id[e] = -1;
            if (!rot_valid(U.g[sp], s, e)) continue;
            const u64 t = rot_member(U.g[sp], s, e);
            id[e] = e == 0 ? i : string_index(B, map, nel, (Ti)t);
            for (int k = 0; k < m; ++k)
                if (par(t & U.z[sp][k])) b |= 1u << (16 + 4 * k + e);
        }
        idx[base + r] = make_int4(id[0], id[1], id[2], id[3]);
        bits[base + r] = b;
    }
}

struct RotOps { int op0, m, na, pad; };   // of a unit: first operator, components, alpha orbits

// angle terms of a unit's components: c, s rotate; gd, go weight the gradient
struct RotArgs {
    int m, nB, nb;                     // components, row length, beta orbits
    unsigned char xa[kRotComps], xb[kRotComps];
    double c[kRotComps], s[kRotComps], gd[kRotComps], go[kRotComps];
};

// bit e -> bit 4 e
__device__ __forceinline__ unsigned spread4(unsigned n)
{
    return (n & 1u) | ((n & 2u) << 3) | ((n & 4u) << 6) | ((n & 8u) << 9);
}

// One CTA per alpha orbit: the rows of its members are walked in the order of
// the beta lists, all of a row's beta patterns close in time.  256 threads: at 14o
// 7a+7b a 2000-generator energy and gradient takes 277 ms with them, 2 % more with
// 512, 16 % with 1024; more registers or shared memory to hold fewer CTAs on an SM, or
// fewer registers to hold more, cost 7-75 %, and beta orbits in ascending order
// instead of sorted by pattern 8 %.
// BACK: the components in reverse order on l and r, the gradient terms summed
// into part[CTA][component]; else in order on l.
template <bool BACK, int NT>
__global__ void __launch_bounds__(NT)
rot_apply_kernel(const RotArgs A, const int4 *__restrict__ ia, const unsigned *__restrict__ ba,
                 const int4 *__restrict__ ib, const unsigned *__restrict__ bb, double *__restrict__ l,
                 double *__restrict__ r, double *__restrict__ part)
{
    __shared__ double red[kRotComps][NT / 32];
    const int4 ca = __ldg(ia + blockIdx.x);
    const unsigned aw = __ldg(ba + blockIdx.x);
    int j = threadIdx.x;
    int4 cb = make_int4(-1, -1, -1, -1);
    unsigned bw = 0;
    if (j < A.nb) { cb = __ldg(ib + j); bw = __ldg(bb + j); }
    __shared__ i64 row[4];
    if (threadIdx.x < 4) {
        const int id[4] = {ca.x, ca.y, ca.z, ca.w};
        row[threadIdx.x] = (i64)id[threadIdx.x] * A.nB;
    }
    unsigned sa[kRotComps], sg[kRotComps];   // sources among the alpha members at bits 4 e, signs as 16 member bits
#pragma unroll
    for (int k = 0; k < kRotComps; ++k) {
        sa[k] = spread4((aw >> (4 * k)) & 15u);
        sg[k] = spread4((aw >> (16 + 4 * k)) & 15u) * 15u;
    }
    auto any4 = [](unsigned w) {   // bit 4 k: component k has a source among the members
        w |= w >> 1;
        w |= w >> 2;
        return w & 0x1111u;
    };
    const unsigned any_a = any4(aw);
    __syncthreads();
    // the lists were complete before the previous unit's CTAs passed this point;
    // l and r are that unit's results
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    double a0 = 0.0, a1 = 0.0, a2 = 0.0, a3 = 0.0;
    while (j < A.nb) {
        const int rb[4] = {cb.x, cb.y, cb.z, cb.w};
        const unsigned b = bw;
        j += NT;
        if (j < A.nb) { cb = __ldg(ib + j); bw = __ldg(bb + j); }
        if ((any_a & any4(b)) == 0) continue;
#pragma unroll
        for (int q = 0; q < kRotComps; ++q) {
            const int k = BACK ? kRotComps - 1 - q : q;
            const int x = A.xa[k] * 4 + A.xb[k];
            const unsigned neg = sg[k] ^ (((b >> (16 + 4 * k)) & 15u) * 0x1111u);
            double g = 0.0;
            for (unsigned m = sa[k] * ((b >> (4 * k)) & 15u); m; m &= m - 1) {   // its sources
                const int i = __ffs((int)m) - 1, t = i ^ x;
                auto at = [&](int e) {
                    return row[e >> 2] + ((e & 2) ? ((e & 1) ? rb[3] : rb[2]) : ((e & 1) ? rb[1] : rb[0]));
                };
                const i64 oi = at(i), oj = at(t);
                const bool minus = (neg >> i) & 1u;
                const double c = A.c[k], sv = minus ? -A.s[k] : A.s[k];
                const double vi = l[oi], vj = l[oj];
                double wi = 0.0, wj = 0.0;
                if (BACK) { wi = r[oi]; wj = r[oj]; }
                const double ni = vi * c - vj * sv, nj = vj * c + vi * sv;
                l[oi] = ni;
                l[oj] = nj;
                if (BACK) {   // backgrad_update, core/math.hpp:187-215
                    const double gd = A.gd[k], go = minus ? -A.go[k] : A.go[k];
                    g += ni * (wi * gd + wj * go) + nj * (wj * gd - wi * go);
                    r[oi] = wi * c - wj * sv;
                    r[oj] = wj * c + wi * sv;
                }
            }
            if (BACK) {
                if (k == 0) a0 += g;
                else if (k == 1) a1 += g;
                else if (k == 2) a2 += g;
                else a3 += g;
            }
        }
    }
    if (!BACK) return;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    a0 = warp_sum(a0); a1 = warp_sum(a1); a2 = warp_sum(a2); a3 = warp_sum(a3);
    if (lane == 0) { red[0][wid] = a0; red[1][wid] = a1; red[2][wid] = a2; red[3][wid] = a3; }
    __syncthreads();
    if (threadIdx.x < kRotComps) {
        double t = 0.0;
        for (int i = 0; i < NT / 32; ++i) t += red[threadIdx.x][i];
        part[(i64)blockIdx.x * kRotComps + threadIdx.x] = t;
    }
}

// terms[op0 + k] = the partial sums of a unit's component k in CTA order
__global__ void __launch_bounds__(128)
rot_terms_kernel(const double *__restrict__ part, int stride, const RotOps *__restrict__ ops,
                 double *__restrict__ terms)
{
    const int u = blockIdx.x, k = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (k >= ops[u].m) return;
    const double *p = part + (i64)u * stride * kRotComps + k;
    double t = 0.0;
    for (int i = lane; i < ops[u].na; i += 32) t += p[(i64)i * kRotComps];
    t = warp_sum(t);
    if (lane == 0) terms[ops[u].op0 + k] = t;
}

// ---- host: groups as excitations ------------------------------------------------------

template <typename Ti>
RotComp classify(const DevNet<Ti> *N, const GroupDev &G)
{
    RotComp C;
    C.kind = 0;
    if (G.type == 0) { C.kind = 2; return C; }
    const int ka = __builtin_popcountll(G.ax), kb = __builtin_popcountll(G.bx);
    if (ka > 4 || kb > 4 || (ka & 1) || (kb & 1) || G.nza < 1 || G.nzb < 1) return C;
    const Ti *za = N->z.data() + G.za_off, *zb = N->z.data() + G.zb_off;
    const double *wa = N->w.data() + G.wa_off, *wb = N->w.data() + G.wb_off;
    // orbitals looked at: those flipped and those on which the Z masks differ (an
    // occupation that the element depends on); elsewhere the masks agree, so a
    // string's other orbitals give one sign
    C.ax = G.ax; C.bx = G.bx;
    C.am = G.ax; C.bm = G.bx;
    for (int q = 1; q < G.nza; ++q) C.am |= (u64)za[q] ^ (u64)za[0];
    for (int q = 1; q < G.nzb; ++q) C.bm |= (u64)zb[q] ^ (u64)zb[0];
    C.az = (u64)za[0] & ~C.am;
    C.bz = (u64)zb[0] & ~C.bm;
    if (__builtin_popcountll(C.am) > 4 || __builtin_popcountll(C.bm) > 4) return C;
    // the matrix element of every pattern that keeps the electron count
    auto patterns = [](u64 m, u64 x, u64 *out) {
        int n = 0;
        for (int p = 0; p < (1 << __builtin_popcountll(m)); ++p) {
            const u64 s = rot_pattern(m, p);
            if (2 * __builtin_popcountll(s & x) == __builtin_popcountll(x)) out[n++] = s;
        }
        return n;
    };
    u64 pa[16], pb[16];
    const int na = patterns(C.am, G.ax, pa), nb = patterns(C.bm, G.bx, pb);
    double v[16][16], vmax = 0.0;
    for (int i = 0; i < na; ++i)
        for (int j = 0; j < nb; ++j) {
            double t = 0.0;
            for (int r = 0; r < G.rank; ++r) {
                double a = 0.0, b = 0.0;
                for (int q = 0; q < G.nza; ++q)
                    a += __builtin_parityll(pa[i] & (u64)za[q]) ? -wa[(i64)r * G.nza + q] : wa[(i64)r * G.nza + q];
                for (int q = 0; q < G.nzb; ++q)
                    b += __builtin_parityll(pb[j] & (u64)zb[q]) ? -wb[(i64)r * G.nzb + q] : wb[(i64)r * G.nzb + q];
                t += a * b;
            }
            v[i][j] = t;
            vmax = std::max(vmax, std::fabs(t));
        }
    if (!(vmax > 0.0) || !std::isfinite(vmax)) return C;
    // an excitation: one pattern, and its target with the opposite element; the
    // rest zero to the rounding of the sums above
    const double noise = 1e-14 * vmax;
    int si[2] = {0, 0}, sj[2] = {0, 0}, nz = 0;
    for (int i = 0; i < na; ++i)
        for (int j = 0; j < nb; ++j)
            if (std::fabs(v[i][j]) > noise) {
                if (nz < 2) { si[nz] = i; sj[nz] = j; }
                ++nz;
            }
    if (nz != 2 || (pa[si[0]] ^ pa[si[1]]) != G.ax || (pb[sj[0]] ^ pb[sj[1]]) != G.bx) return C;
    if (std::fabs(v[si[0]][sj[0]] + v[si[1]][sj[1]]) > noise) return C;
    C.kind = 1;
    C.as = pa[si[0]];
    C.bs = pb[sj[0]];
    C.f = v[si[0]][sj[0]];
    return C;
}

std::mutex g_rot_mu;

// the group's form, looked at once per network
template <typename Ti>
RotComp component(const DevNet<Ti> *N, i64 g)
{
    auto *tab = static_cast<std::vector<RotComp> *>(N->rot_state);
    RotComp &C = (*tab)[(size_t)g];
    if (C.kind < 0) C = classify(N, N->groups[(size_t)g]);
    return C;
}

// x as a combination of g[0], g[1] (bit 0, bit 1), extending g when it has room; -1 when it has none
int combine(u64 x, u64 (&g)[2])
{
    if (x == 0) return 0;
    for (int c = 1; c < 4; ++c) {
        if (((c & 1) && !g[0]) || ((c & 2) && !g[1])) continue;
        if ((((c & 1) ? g[0] : 0) ^ ((c & 2) ? g[1] : 0)) == x) return c;
    }
    for (int i = 0; i < 2; ++i)
        if (!g[i]) { g[i] = x; return 1 << i; }
    return -1;
}

}  // namespace

// ---- host: units --------------------------------------------------------------------------

template <typename Ti>
int RotSequence<Ti>::init(const DevBasis<Ti> *B, const DevNet<Ti> *P, i64 n_ops, const i64 *op_idx,
                          const i64 *param_idx, const double *thetas, const std::vector<i64> &breaks, cudaStream_t s)
{
    B_ = B; P_ = P; op_idx_ = op_idx; param_idx_ = param_idx; thetas_ = thetas; s_ = s;
    // the lists count strings with binomial coefficients: a single block that holds every string
    auto binom = [](int n, int k) {
        double c = 1.0;
        for (int i = 1; i <= k; ++i) c = c * (n - k + i) / i;
        return c;
    };
    const bool whole = B->num_blocks == 1 && B->dim > 0 && !P->cplx && n_ops < ((i64)1 << 31) &&
                       (double)B->na[0] == std::round(binom(B->norb, B->nel_a)) &&
                       (double)B->nb[0] == std::round(binom(B->norb, B->nel_b));
    {
        std::lock_guard<std::mutex> lk(g_rot_mu);
        if (whole && !P->rot_state) {
            auto *N = const_cast<DevNet<Ti> *>(P);
            N->rot_state = new std::vector<RotComp>((size_t)P->ngs);
            N->rot_free = [](void *q) { delete static_cast<std::vector<RotComp> *>(q); };
        }
        size_t nb = 0;
        i64 fused = 0;
        for (i64 i = 0; i < n_ops; ++i) {
            while (nb < breaks.size() && breaks[nb] < i) ++nb;
            const bool stop = nb < breaks.size() && breaks[nb] == i;
            RotComp C;
            C.kind = 0;
            if (whole && op_idx[i] >= 0 && op_idx[i] < P->ngs) C = component(P, op_idx[i]);
            if (B->norb < 64 && ((C.am | C.bm) >> B->norb)) C.kind = 0;   // orbitals outside the basis
            if (C.kind == 2) continue;   // the exponential of a diagonal group is the identity for real vectors
            if (C.kind == 1 && !stop && !units_.empty()) {
                RotUnit &U = units_.back();
                if (U.m > 0 && U.m < kRotComps && U.op0 + U.m == i) {
                    u64 ga[2] = {U.ga[0], U.ga[1]}, gb[2] = {U.gb[0], U.gb[1]};
                    const int xa = combine(C.ax, ga), xb = combine(C.bx, gb);
                    if (xa >= 0 && xb >= 0 && __builtin_popcountll(U.ua | C.am) <= kRotMaxBits &&
                        __builtin_popcountll(U.ub | C.bm) <= kRotMaxBits) {
                        for (int q = 0; q < 2; ++q) { U.ga[q] = ga[q]; U.gb[q] = gb[q]; }
                        U.ua |= C.am;
                        U.ub |= C.bm;
                        U.c[U.m] = C;
                        U.xa[U.m] = (unsigned char)xa;
                        U.xb[U.m] = (unsigned char)xb;
                        ++U.m;
                        continue;
                    }
                }
            }
            RotUnit U;
            U.op0 = i;
            if (C.kind == 1) {
                U.m = 1;
                U.c[0] = C;
                U.xa[0] = (unsigned char)combine(C.ax, U.ga);
                U.xb[0] = (unsigned char)combine(C.bx, U.gb);
                U.ua = C.am;
                U.ub = C.bm;
                ++fused;
            }
            units_.push_back(U);
        }
        if (fused == 0) return BSIM_OK;
    }
    const int nA = B->na[0], nB = B->nb[0];
    const size_t per_unit = (size_t)(nA + nB) * (sizeof(int4) + sizeof(unsigned));
    batch_ = std::max<i64>(1, std::min<i64>((i64)units_.size(), (i64)(kRotListBytes / per_unit)));
    batch_ = std::min<i64>(batch_, 30000);   // two list CTA rows per unit in one grid dimension
    const size_t nU = units_.size();
    auto al = [](size_t n) { return (n + 255) & ~size_t(255); };
    const size_t b_units = al(nU * sizeof(RotUnitDev)), b_ops = al(nU * sizeof(RotOps));
    std::vector<char> host(b_units + b_ops, 0);
    rows_ = 1;
    for (size_t u = 0; u < nU; ++u) {
        RotUnit &U = units_[u];
        RotUnitDev D{};
        D.m = U.m;
        for (int q = 0; q < 2; ++q) { D.g[0][q] = U.ga[q]; D.g[1][q] = U.gb[q]; }
        D.um[0] = U.ua;
        D.um[1] = U.ub;
        for (int k = 0; k < U.m; ++k) {
            D.x[0][k] = U.c[k].am; D.src[0][k] = U.c[k].as; D.z[0][k] = U.c[k].az;
            D.x[1][k] = U.c[k].bm; D.src[1][k] = U.c[k].bs; D.z[1][k] = U.c[k].bz;
        }
        for (int sp = 0; sp < 2 && U.m > 0; ++sp) {   // list lengths, as the list kernel counts them
            const int nu = __builtin_popcountll(D.um[sp]), nel = sp ? B->nel_b : B->nel_a;
            double c = 0.0;
            for (int p = 0; p < (1 << nu); ++p) {
                const u64 t = rot_pattern(D.um[sp], p);
                const int rest = nel - __builtin_popcountll(t), room = B->norb - nu;
                if (rest >= 0 && rest <= room && rot_key(D, sp, t)) c += std::round(binom(room, rest));
            }
            (sp ? U.nb : U.na) = (int)c;
        }
        rows_ = std::max(rows_, U.na);
        reinterpret_cast<RotUnitDev *>(host.data())[u] = D;
        reinterpret_cast<RotOps *>(host.data() + b_units)[u] = RotOps{(int)U.op0, U.m, U.nb ? U.na : 0, 0};
    }
    const size_t b_idx = al((size_t)batch_ * (nA + nB) * sizeof(int4)), b_bits = al((size_t)batch_ * (nA + nB) * 4);
    const size_t b_part = al((size_t)batch_ * rows_ * kRotComps * sizeof(double));
    cudaError_t e = dmalloc_async(&mem_, b_units + b_ops + b_idx + b_bits + b_part, s);
    if (e == cudaErrorMemoryAllocation) {   // no room for the lists: operator by operator
        (void)cudaGetLastError();
        mem_ = nullptr;
        units_.clear();
        for (i64 i = 0; i < n_ops; ++i) {
            RotUnit U;
            U.op0 = i;
            units_.push_back(U);
        }
        return BSIM_OK;
    }
    if (e != cudaSuccess) { mem_ = nullptr; return cuda_status(e, "rotation lists"); }
    char *p = static_cast<char *>(mem_);
    d_units_ = p;
    d_ops_ = p + b_units;
    p += b_units + b_ops;
    d_idx_ = reinterpret_cast<int4 *>(p); p += b_idx;
    d_bits_ = reinterpret_cast<unsigned *>(p); p += b_bits;
    d_part_ = reinterpret_cast<double *>(p);
    BSIM_CUDA(cudaMemcpyAsync(mem_, host.data(), host.size(), cudaMemcpyHostToDevice, s));
    BSIM_CUDA(cudaStreamSynchronize(s));   // the host array must outlive the copy
    return BSIM_OK;
}

template <typename Ti>
RotSequence<Ti>::~RotSequence()
{
    if (mem_) cudaFreeAsync(mem_, s_);
}

// the orbit lists of unit u and of the units after it (ascending) or before it
template <typename Ti>
int RotSequence<Ti>::lists(i64 u, bool ascending)
{
    if (u >= b0_ && u < b1_) return BSIM_OK;
    const i64 n = (i64)units_.size();
    b0_ = ascending ? u : std::max<i64>(0, u + 1 - batch_);
    b1_ = ascending ? std::min(n, u + batch_) : u + 1;
    const int nA = B_->na[0], nB = B_->nb[0];
    dim3 grid((unsigned)std::max(1, std::min(8, (std::max(nA, nB) + 1023) / 1024)), (unsigned)(2 * (b1_ - b0_)));
    rot_list_kernel<Ti><<<grid, 256, 0, s_>>>(B_->view, static_cast<const RotUnitDev *>(d_units_) + b0_, nA, nB, d_idx_,
                                              d_bits_);
    BSIM_CUDA(cudaGetLastError());
    chained_ = false;
    return BSIM_OK;
}

template <typename Ti>
static RotArgs rot_args(const RotUnit &U, const i64 *param_idx, const double *thetas, int nB, bool back)
{
    RotArgs A{};
    A.m = U.m;
    A.nB = nB;
    A.nb = U.nb;
    for (int k = 0; k < U.m; ++k) {
        const double th = thetas[param_idx[U.op0 + k]], f = U.c[k].f;
        A.xa[k] = U.xa[k];
        A.xb[k] = U.xb[k];
        A.c[k] = 1.0 + (cos(th) - 1.0) * (f * f);
        A.s[k] = (back ? -sin(th) : sin(th)) * f;
        A.gd[k] = -sin(th) * (f * f);
        A.go[k] = cos(th) * f;
    }
    return A;
}

// One unit's pass.  A unit that directly follows another of the same batch is
// launched as its programmatic dependent: its CTAs start while the other's
// finish and wait for them before they touch l and r.
template <typename Ti>
template <bool BACK>
int RotSequence<Ti>::launch(i64 u, double *l, double *r, double *part)
{
    const RotUnit &U = units_[u];
    if (U.na == 0 || U.nb == 0) return BSIM_OK;   // no determinant has the pattern of any component
    const int nA = B_->na[0], nB = B_->nb[0];
    const i64 o = (u - b0_) * (nA + nB);
    const int4 *ia = d_idx_ + o, *ib = ia + nA;
    const unsigned *ba = d_bits_ + o, *bb = ba + nA;
    const RotArgs A = rot_args<Ti>(U, param_idx_, thetas_, nB, BACK);
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)U.na);
    cfg.stream = s_;
    cfg.attrs = &at;
    cfg.numAttrs = chained_ ? 1 : 0;
    auto go = [&](auto kern, int nt) {
        cfg.blockDim = dim3((unsigned)nt);
        return cudaLaunchKernelEx(&cfg, kern, A, ia, ba, ib, bb, l, r, part);
    };
    if (U.nb > 128) BSIM_CUDA(go(rot_apply_kernel<BACK, 256>, 256));
    else BSIM_CUDA(go(rot_apply_kernel<BACK, 128>, 128));
    chained_ = true;
    return BSIM_OK;
}

template <typename Ti>
int RotSequence<Ti>::forward(i64 u, double *v)
{
    const RotUnit &U = units_[u];
    if (U.m == 0) {
        chained_ = false;
        return expm(B_, P_, op_idx_[U.op0], thetas_[param_idx_[U.op0]], v, s_);
    }
    int st = lists(u, true);
    if (st != BSIM_OK) return st;
    return launch<false>(u, v, nullptr, nullptr);
}

template <typename Ti>
int RotSequence<Ti>::backward(i64 u, double *l, double *r, double *terms)
{
    const RotUnit &U = units_[u];
    if (U.m == 0) {
        chained_ = false;
        return backgrad(B_, P_, op_idx_[U.op0], thetas_[param_idx_[U.op0]], l, r, terms + U.op0, false, s_);
    }
    if (u < b0_ || u >= b1_) {   // the partial sums belong to the batch whose lists are in place
        int st = flush(terms);
        if (st == BSIM_OK) st = lists(u, false);
        if (st != BSIM_OK) return st;
    }
    int st = launch<true>(u, l, r, d_part_ + (u - b0_) * (i64)rows_ * kRotComps);
    if (st != BSIM_OK) return st;
    if (pend0_ == pend1_) pend1_ = u + 1;
    pend0_ = u;
    return BSIM_OK;
}

template <typename Ti>
int RotSequence<Ti>::flush(double *terms)
{
    chained_ = false;
    if (pend0_ == pend1_) return BSIM_OK;
    rot_terms_kernel<<<(unsigned)(pend1_ - pend0_), 128, 0, s_>>>(
        d_part_ + (pend0_ - b0_) * (i64)rows_ * kRotComps, rows_, static_cast<const RotOps *>(d_ops_) + pend0_, terms);
    BSIM_CUDA(cudaGetLastError());
    pend0_ = pend1_ = 0;
    return BSIM_OK;
}

template class RotSequence<unsigned>;
template class RotSequence<unsigned long long>;

}  // namespace bsim

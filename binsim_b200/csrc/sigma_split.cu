// The mixed-excitation product of the FP64 structured sigma (the product of
// mixed_dmma_kernel in sigma_fast.cu) as byte products on the 5th-generation tensor
// cores: tcgen05.mma kind::i8, 32-bit integer accumulators in tensor memory.
//
// Every operand is a fixed-point number relative to the largest element of its row
// (a power of two above it), cut into ND = 8 signed bytes x = sum_i d_i 256^(7-i),
// d_i in [-128, 127].  The product is sum_{i+j<8} d_i d'_j 256^(14-i-j), every byte
// product and sum exact in 32-bit integers, the eight diagonals i + j = const summed in
// 64 bits and rounded once (error-free splitting: Ozaki, Ogita, Oishi, Rump 2012; on
// integer tensor cores: Ootomo, Ozaki, Yokota 2024).  The terms left out are below
// 2^-57 of (largest element of the row) x (largest element of the B row) a product, and a
// word's rounding below 2^-62 of its row's largest element.  FP64 rounds at 2^-53 of a
// sum's own terms, so the split is as exact only where most elements of a row are not
// far below its largest: a row of c~ with more than 1/8 of its nonzero elements below
// 2^-12 of it (of the power of two above it) or 1/64 below 2^-30, or with an infinity or
// NaN, stays in FP64 and goes to mixed_dmma_kernel (kWideRow); a Hamiltonian with such a
// row of Lam (1/8 below 2^-10) does not use the split products at all (fastplan.cu).
// An output that only the few small elements of an accepted row reach keeps the bound
// above, relative to the row.  Error over the sum of |terms| of an output, 36 terms, rms
// and max of 4000, the byte products emulated on the host, FP64 / split: normal elements 5.3e-17 3.2e-16 / 1.2e-17 6.1e-17;
// log-normal (sigma 1, 2 % below 2^-12) 7.2e-17 4.6e-16 / 2.4e-17 1.1e-16; log-uniform
// over three decades (10 %) 9.0e-17 7.9e-16 / 2.6e-17 1.2e-16; beyond the line, log-normal
// (sigma 2.5, 60 %) 1.2e-16 8.3e-16 / 3.3e-16 3.1e-15.  Zeros stay exact.
//
// The product is computed transposed, D[b][j], the 128 columns b of a chunk in
// the MMA's M.  A byte plane i of X^T meets every byte plane j < 8 - i of B in
// ONE instruction: the planes of B are stacked along N, and the diagonals i + j
// are consecutive accumulator blocks, so plane i of A starts i blocks further
// right.  An accumulator holds the eight diagonals of up to 32 output rows, 256
// columns of tensor memory; the two halves of 64 rows take two accumulators in turn.
//
// Warp roles (800 threads, one CTA per source row):
//   warps 0-7   epilogue: tcgen05.ld of the diagonals (warp w reads lanes
//               32 (w % 4) ..), 64-bit sums, stores;
//   warps 8-23  producers: gather the fixed-point words of a slice of 32 K rows, two
//               slices ahead in registers, and write their bytes as K-major core
//               matrices, one (column, 8 rows) group per thread;
//   warp 24     TMEM allocation and, by one lane, the MMA issue.
// Handoffs and bounded waits as in sigma_tc.cu; a CTA that gives up a wait, and every
// CTA that starts after it and before the next call, leaves its row to
// mixed_dmma_kernel (row_to_fp64).
//
// Bound: the L1 pipe that the producers' gathers, the byte stores and the epilogue's
// stores share (a slice of 4 K words takes ~3700 cycles, the MMAs of 64 rows 1200 of
// them, the integer tensor pipe ~30 % busy).  What took time out, at 14 orbitals 7a+7b:
// the halves of a pass one after the other over all slices of the chunk, so that one
// accumulator is read out during the other's MMAs, and the epilogue's eight rows at a
// time (8 loads per 8 rows, not per 4): 4.5 -> 3.8 ms; before that, biased words
// (bytes d + 128: a subtraction negates them) and byte offsets in the gather table.
// Against mixed_dmma_kernel, which runs at the FP64 tensor rate: 0.426 -> 0.343 ms at
// 12o 6+6, 1.05 -> 0.78 ms at 13o 7+5, 5.72 -> 3.86 ms at 14o 7+7, 99.8 -> 68.5 ms at
// 16o 8+8, 1.29 -> 0.82 ms at 20o 3+3, with the launch for rows left in FP64.  On a vector
// whose rows all stay in FP64 (six decades under a leading determinant, 13o 7+5) a sigma
// takes 2.16 ms, with all rows split 1.87.
// Measured and not kept: FP16 digits (seven of 9 bits, kind::f16; 110 ms at 16o, for the
// conversion of the digits), the same kernel for the doubles through intermediate
// strings (43 -> 50 ms at 16o: 45 rows of 64, K of 45 in 64, coalesced DMMA operands)
// and for the FP32-bulk sigma with four bytes (36 -> 40 ms against TF32).
#include "mixed.cuh"
#include "ops.h"
#include "tc.cuh"

#include <algorithm>
#include <cstdlib>

namespace bsim {

namespace {

constexpr int kThreads = 800;
constexpr int kEpiWarps = 8, kProdWarps = 16, kMmaWarp = 24;
constexpr int kM = 128;                    // columns per chunk: MMA M
constexpr int kKS = 32;                    // K rows per slice: one MMA K step
constexpr int kStages = 4;                 // A stages, at most
constexpr int kRows = kSplitRows;          // output rows per pass
constexpr uint32_t kPlane = kM * kKS;      // one byte plane of an A stage
constexpr int kZeroExp = -2000;            // exponent of a row of zeros

// instruction descriptor of kind::i8: D S32 (bits 4-5 = 2), A and B signed (bits
// 7-9, 10-12 = 1), both K-major, N >> 3 at bit 17, M >> 4 at bit 24
__host__ __device__ constexpr uint32_t idesc_i8(int n)
{
    return (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(kM >> 4) << 24);
}
__device__ __forceinline__ void umma_i8(uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate)
{
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
                 "l"(a), "l"(b), "r"(idesc), "r"(accumulate)
                 : "memory");
}
// one lane of a converged warp, the same in every call
__device__ __forceinline__ bool elect_lane()
{
    uint32_t e;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.b32 %0, 1, 0, p;\n\t}" : "=r"(e));
    return e != 0;
}
// 8 consecutive 32-bit columns of this thread's lane (not waited for)
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, int (&r)[8])
{
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr)
                 : "memory");
}
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

constexpr int ND = 8;                          // signed bytes of a word
constexpr int kHalf = 256 / ND;                // output rows of one accumulator
constexpr int kBits = 8 * ND - 2;              // |fixed-point word| <= 2^kBits
constexpr uint32_t kStageBytes = (uint32_t)ND * kPlane;
constexpr u64 kBias = 0x8080808080808080ull;   // a word of c~ holds the bytes d + 128
constexpr long long kMagic = 0x4338000000000000ll;   // the bits of 1.5 2^52
constexpr double kMagicD = 6755399441055744.0;

// output rows of part h of a pass: multiples of 16, so that every N = n (ND - i) is one
__host__ __device__ inline int half_rows(int jm, int h)
{
    const int left = jm - kHalf * h;
    if (left <= 0) return 0;
    const int n = (left + 15) & ~15;
    return n > 16 ? 32 : 16;
}

constexpr size_t kStaticSmem = 2048;   // the kernels' static shared memory, and the dynamic base aligned to 1 KB

struct SplitLayout {
    uint32_t b, a, scale, tab, bars, tmem, total;
    int kp;            // K rounded up to whole slices
    int stages;        // A stages
    uint32_t sbo_b;    // byte stride between 8-row groups of B
};
__host__ __device__ inline SplitLayout split_layout(int K, int jm, uint32_t tab_bytes)
{
    SplitLayout L{};
    L.kp = (K + kKS - 1) / kKS * kKS;
    L.sbo_b = (uint32_t)(L.kp / 16) * kCoreBytes;
    uint32_t o = 0;
    L.b = o;
    o = align128(o + (uint32_t)ND * (uint32_t)(half_rows(jm, 0) + half_rows(jm, 1)) * (uint32_t)L.kp);
    const uint32_t rest = kRows * 16u + tab_bytes + 512u;   // what follows, with its alignment
    L.stages = o + kStages * kStageBytes + rest + kStaticSmem <= kSmemMax ? kStages : kStages - 1;
    L.a = o; o = align128(o + (uint32_t)L.stages * kStageBytes);
    L.scale = o; o = align128(o + kRows * 16u);
    L.tab = o; o = align128(o + tab_bytes);
    L.bars = o; o = align128(o + (uint32_t)(2 * kStages + 5) * 8u);
    L.tmem = o; o = align128(o + 4u);
    L.total = o;
    return L;
}
constexpr uint32_t kMixTab = 2u * kMaxConn * 4u;

// smallest e with |x| < 2^e for the largest |x| = m of a row
__device__ __forceinline__ int exp_above(double m)
{
    if (!(m <= 1.7976931348623157e308)) return kWideRow;   // infinite or NaN
    return m > 0.0 ? ilogb(m) + 1 : kZeroExp;
}
// max that keeps a NaN
__device__ __forceinline__ double max_nan(double a, double b) { return (a > b || a != a) ? a : b; }
__device__ __forceinline__ double warp_max_nan(double v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = max_nan(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}
// 2^e as the product of two factors (e beyond one FP64 exponent)
struct Pow2 {
    double a, b;
    __device__ __forceinline__ explicit Pow2(int e) : a(scalbn(1.0, e / 2)), b(scalbn(1.0, e - e / 2)) {}
};
// x times the factors of 2^(kBits - exponent), rounded and biased: bytes d + 128 of
// the signed bytes d.  Zero is the bias, all bytes 128.
__device__ __forceinline__ u64 to_word(double x, const Pow2 &f)
{
    return (u64)__double2ll_rn(x * f.a * f.b) + kBias;
}
// the biased word of -x
__device__ __forceinline__ u64 negate_word(u64 y) { return 2 * kBias - y; }

// 4 x 4 byte transpose: out[t] = byte t of a, b, c, d
__device__ __forceinline__ void transpose4(uint32_t a, uint32_t b, uint32_t c, uint32_t d, uint32_t (&out)[4])
{
    const uint32_t x = __byte_perm(a, b, 0x5140), y = __byte_perm(c, d, 0x5140);
    const uint32_t z = __byte_perm(a, b, 0x7362), w = __byte_perm(c, d, 0x7362);
    out[0] = __byte_perm(x, y, 0x5410);
    out[1] = __byte_perm(x, y, 0x7632);
    out[2] = __byte_perm(z, w, 0x5410);
    out[3] = __byte_perm(z, w, 0x7632);
}

// Rows of c~ to fixed point in place, with the exponent of each; wide rows stay.
__global__ void __launch_bounds__(256)
rows_to_fixed_kernel(double *__restrict__ in, int ld, int *__restrict__ rexp)
{
    chain_wait();
    __shared__ double red[8];
    __shared__ int cnt[3];
    if (threadIdx.x < 3) cnt[threadIdx.x] = 0;
    double *row = in + (i64)blockIdx.x * ld;
    double m = 0.0;
    for (int i = threadIdx.x; i < ld; i += 256) m = max_nan(m, fabs((double)row[i]));
    m = warp_max_nan(m);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
    __syncthreads();
    m = red[0];
    for (int i = 1; i < 8; ++i) m = max_nan(m, red[i]);
    int e = exp_above(m);
    const bool plain = e != kWideRow && e != kZeroExp;
    const Pow2 f(plain ? kBits - e : 0);
    if (plain) {   // nonzero elements, those below 2^(e - kFarBits), those below 2^(e - kLeastBits)
        const double far = ldexp(1.0, kBits - kFarBits), least = ldexp(1.0, kBits - kLeastBits);
        int n = 0, k = 0, l = 0;
        for (int i = threadIdx.x; i < ld; i += 256) {
            const double x = fabs((double)row[i]), y = x * f.a * f.b;
            n += x != 0.0;
            k += x != 0.0 && y < far;
            l += x != 0.0 && y < least;
        }
        n = __reduce_add_sync(0xffffffffu, n);
        k = __reduce_add_sync(0xffffffffu, k);
        l = __reduce_add_sync(0xffffffffu, l);
        if ((threadIdx.x & 31) == 0) {
            atomicAdd(&cnt[0], n);
            atomicAdd(&cnt[1], k);
            atomicAdd(&cnt[2], l);
        }
        __syncthreads();
        if ((i64)cnt[1] * 8 > cnt[0] || (i64)cnt[2] * 64 > cnt[0]) e = kWideRow;
    }
    if (threadIdx.x == 0) rexp[blockIdx.x] = e;
    if (blockIdx.x == 0 && threadIdx.x == 0) g_tc_abort = 0;   // of an earlier call (the flag only saves waits)
    if (e == kWideRow) return;   // uniform across the CTA
    for (int i = threadIdx.x; i < ld; i += 256)
        reinterpret_cast<u64 *>(row)[i] = to_word(plain ? (double)row[i] : 0.0, f);
}

// B = [jm x K] as byte planes: row (half h, plane d, row e of the half) of one
// K-major operand, and per output row the two factors whose product is
// 2^(a_exp + its exponent - 68).  bval(j, k): the FP64 element, row_exp(j) the exponent
// above row j (kZeroExp for a row of zeros).
template <typename BVal, typename RowExp>
__device__ __forceinline__ void stage_b(const SplitLayout &L, unsigned char *smem, int jm, int K, int a_exp, BVal bval,
                                        RowExp row_exp)
{
    __shared__ double2 fj[kRows];
    if ((int)threadIdx.x < jm) {
        const int e = row_exp((int)threadIdx.x);
        const Pow2 f(a_exp + e - 2 * kBits + 8 * (ND - 1)), p(e == kZeroExp ? 0 : kBits - e);
        reinterpret_cast<double2 *>(smem + L.scale)[threadIdx.x] = make_double2(f.a, f.b);
        fj[threadIdx.x] = e == kZeroExp ? make_double2(0.0, 0.0) : make_double2(p.a, p.b);
    }
    __syncthreads();
    const int n0 = half_rows(jm, 0), n1 = half_rows(jm, 1), nk4 = L.kp / 4;
    for (int i = threadIdx.x; i < (n0 + n1) * nk4; i += kThreads) {
        const int j = i / nk4, k = (i % nk4) * 4;
        u64 y[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            double x = 0.0;
            if (j < jm && k + c < K && fj[j].x != 0.0) x = bval(j, k + c) * fj[j].x * fj[j].y;
            y[c] = (u64)(__double2ll_rn(x) + kBias) ^ kBias;
        }
        uint32_t p[8];   // by byte, the least significant first
        transpose4((uint32_t)y[0], (uint32_t)y[1], (uint32_t)y[2], (uint32_t)y[3], reinterpret_cast<uint32_t (&)[4]>(p[0]));
        transpose4((uint32_t)(y[0] >> 32), (uint32_t)(y[1] >> 32), (uint32_t)(y[2] >> 32), (uint32_t)(y[3] >> 32),
                   reinterpret_cast<uint32_t (&)[4]>(p[4]));
        const int h = j >= kHalf, n = h ? n1 : n0, base = (h ? ND * n0 : 0) + (j - kHalf * h);
#pragma unroll
        for (int d = 0; d < ND; ++d) {
            const int r = base + n * d;
            *reinterpret_cast<uint32_t *>(smem + L.b + (uint32_t)(r >> 3) * L.sbo_b + (uint32_t)(k >> 4) * kCoreBytes +
                                          (uint32_t)(r & 7) * 16u + (uint32_t)(k & 15)) = p[ND - 1 - d];
        }
    }
}

// The slice's bytes of this thread: 8 biased words (8 K rows of one column) into the
// byte planes of stage a, at byte offset off of each plane.
__device__ __forceinline__ void put_words(unsigned char *a, uint32_t off, const u64 (&x)[8])
{
    constexpr uint32_t m = (uint32_t)kBias;
    uint32_t q0[4], q1[4];
#pragma unroll
    for (int w = 0; w < 2; ++w) {
        const int s = 32 - 32 * w;   // the upper halves hold planes 0-3
        transpose4((uint32_t)(x[0] >> s), (uint32_t)(x[1] >> s), (uint32_t)(x[2] >> s), (uint32_t)(x[3] >> s), q0);
        transpose4((uint32_t)(x[4] >> s), (uint32_t)(x[5] >> s), (uint32_t)(x[6] >> s), (uint32_t)(x[7] >> s), q1);
#pragma unroll
        for (int d = 0; d < 4; ++d)
            *reinterpret_cast<uint2 *>(a + (4 * w + d) * kPlane + off) = make_uint2(q0[3 - d] ^ m, q1[3 - d] ^ m);
    }
}

// A producer thread's place in every slice: column b of the chunk and K rows
// k .. k + 7.  Lanes 2 i, 2 i + 1 hold the two halves of a 16-byte core-matrix row.
struct ProdPlace {
    int b, k;
    uint32_t off;
    __device__ __forceinline__ ProdPlace(int pw, int lane)
    {
        b = (pw & 7) * 16 + (lane >> 1);
        k = (pw >> 3) * 16 + (lane & 1) * 8;
        off = (uint32_t)(b >> 3) * (kKS / 16) * kCoreBytes + (uint32_t)(pw >> 3) * kCoreBytes + (uint32_t)(b & 7) * 16u +
              (uint32_t)(lane & 1) * 8u;
    }
};

// slice and chunk of a producer's position
struct SlicePos {
    int s = 0, c = 0;
    __device__ __forceinline__ void next(int nsl) { if (++s == nsl) { s = 0; ++c; } }
};

// X^T[b][F] = sB_F c~[a'][b ^ F] through the table of byte offsets into the row (a
// word of zero where b ^ F is no string, and in the rows past K) with the sign in bit
// 31: the words two slices ahead (two sets of registers in turn), the table entries
// three.
struct GatherWords {
    const unsigned *goff;          // [ldG][kp]
    const unsigned char *row;
    int ldG, kp, z0, nsl, nq;
    SlicePos pos;                  // of the table entries
    int left;                      // slices whose entries are still to load
    unsigned gn[8];                // entries of the next slice to gather
    struct Set { u64 x[8]; unsigned neg; } set[2];
    __device__ __forceinline__ void index(const ProdPlace &P)
    {
        if (left <= 0) return;
        --left;
        const int b = min(z0 + pos.c * kM + P.b, ldG - 1);
        const uint4 *t = reinterpret_cast<const uint4 *>(goff + ((i64)b * kp + (pos.s * kKS + P.k)));
        *reinterpret_cast<uint4 *>(gn) = __ldg(t);
        *reinterpret_cast<uint4 *>(gn + 4) = __ldg(t + 1);
        pos.next(nsl);
    }
    __device__ __forceinline__ void words(Set &S)
    {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            S.x[i] = __ldg(reinterpret_cast<const u64 *>(row + (gn[i] & 0x7fffffffu)));
            S.neg = __funnelshift_l(gn[i], S.neg, 1);   // bit 7 - i of the sum
        }
    }
    __device__ __forceinline__ void begin(const ProdPlace &P)
    {
        left = nq;
        set[0].neg = set[1].neg = 0;
        index(P);
        if (nq > 0) words(set[0]);
        index(P);
        if (nq > 1) words(set[1]);
        index(P);
    }
    template <int SET>
    __device__ __forceinline__ void put(int q, const ProdPlace &P, unsigned char *a)
    {
        Set &S = set[SET];
#pragma unroll
        for (int i = 0; i < 8; ++i)
            if (S.neg & (0x80u >> i)) S.x[i] = negate_word(S.x[i]);
        put_words(a, P.off, S.x);
        if (q + 2 < nq) words(S);
        index(P);
    }
};

// Outputs from their diagonals, D_0 the most significant: the 64-bit sums of four
// (below 2^51 in magnitude) start from kMagic and so are the bits of an FP64 number,
// its integer plus 1.5 2^52; the upper sum times 2^32 plus the lower rounds once, the
// factors are powers of two.
__device__ __forceinline__ long long mad_wide(int a, int b, long long c)
{
    long long r;
    asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(r) : "r"(a), "r"(b), "l"(c));
    return r;
}
__device__ __forceinline__ double unmagic(long long x) { return __longlong_as_double(x) - kMagicD; }
__device__ __forceinline__ double sum4(int a, int b, int c, int d)
{
    return unmagic(mad_wide(d, 1, mad_wide(c, 256, mad_wide(b, 65536, mad_wide(a, 16777216, kMagic)))));
}
// mbar_wait with all but its first test out of line where a chunk's slices all have
// stages (FITS): inlined it takes registers (351 against 343 us at 12o, 799 / 779 at
// 13o 7+5).  Slice by slice the waits are longer and the call costs more (20o 3+3: 892
// us with it, 816 inlined and in an instance of its own).
__device__ __noinline__ bool wait_slow(uint32_t bar, uint32_t parity, volatile int *abort_flag)
{
    return mbar_wait(bar, parity, abort_flag);
}
template <bool FITS>
__device__ __forceinline__ bool wait_phase(uint32_t bar, uint32_t parity, volatile int *abort_flag)
{
    if constexpr (FITS) return mbar_try(bar, parity) || wait_slow(bar, parity, abort_flag);
    else return mbar_wait(bar, parity, abort_flag);
}
// wait_phase by every lane of a warp, with one answer for all: what follows it is a
// barrier of the warp or an aligned instruction
template <bool FITS>
__device__ __forceinline__ bool wait_all(uint32_t bar, uint32_t parity, volatile int *abort_flag)
{
    return __all_sync(0xffffffffu, wait_phase<FITS>(bar, parity, abort_flag));
}

// The producers' loop: slice q into A stage q % kStages.
template <bool FITS, typename Src>
__device__ __forceinline__ void produce_slices(const SplitLayout &L, unsigned char *smem, uint32_t bar0, int nq, Src &src,
                                               volatile int *abort_flag)
{
    const ProdPlace P((int)(threadIdx.x >> 5) - kEpiWarps, (int)(threadIdx.x & 31));
    src.begin(P);
    int st = 0;
    uint32_t empty = 1;   // parity before the first release: passes at once
    auto one = [&](auto set, int q) {
        // a wait that gave up is settled for the warp after the stores, beside its barrier
        const bool ok = wait_phase<FITS>(bar0 + 8u * (uint32_t)(kStages + st), empty, abort_flag);
        src.template put<decltype(set)::value>(q, P, smem + L.a + (size_t)st * kStageBytes);
        fence_async_smem();
        if (!__all_sync(0xffffffffu, ok)) return false;
        warp_arrive(bar0 + 8u * (uint32_t)st);
        if (++st == L.stages) { st = 0; empty ^= 1u; }
        return true;
    };
    for (int q = 0; q < nq; q += 2) {
        if (!one(std::integral_constant<int, 0>{}, q)) break;
        if (q + 1 < nq && !one(std::integral_constant<int, 1>{}, q + 1)) break;
    }
}

// The byte planes of an A slice (descriptor da of plane 0) on N output rows of B
// (descriptor db), into the diagonals from column d; keep: add to what they hold.
template <int N>
__device__ __forceinline__ void issue_planes_n(uint64_t da, uint64_t db, uint32_t d, uint32_t keep)
{
#pragma unroll
    for (int i = 0; i < ND; ++i)
        umma_i8(d + (uint32_t)(N * i), da + (uint64_t)(i * (kPlane >> 4)), db, idesc_i8(N * (ND - i)), i == 0 ? keep : 1u);
}
__device__ __forceinline__ void issue_planes(const SplitLayout &L, uint32_t sbase, int st, int s, uint32_t boff, int n,
                                             uint32_t d)
{
    const uint64_t da = umma_desc(sbase + L.a + (uint32_t)st * kStageBytes, kCoreBytes, (kKS / 16) * kCoreBytes);
    const uint64_t db = umma_desc(sbase + L.b + boff + (uint32_t)s * 2u * kCoreBytes, kCoreBytes, L.sbo_b);
    const uint32_t keep = s != 0 ? 1u : 0u;
    if (n == 16) issue_planes_n<16>(da, db, d, keep);
    else issue_planes_n<32>(da, db, d, keep);
}

// Parts u = chunk * (parts per chunk) + half, accumulator u % 2.
template <bool FITS, typename Src>
__device__ __forceinline__ void split_pipeline(const SplitLayout &L, unsigned char *smem, uint32_t sbase, uint32_t tmem,
                                            int ncb, int jm, double *zrow, int zrows, Src &src,
                                            volatile int *abort_flag, bool drop)
{
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t bar0 = sbase + L.bars;   // afull[S], aempty[S], dfull[2], dempty[2], done
    auto afull = [&](int i) { return bar0 + 8u * (uint32_t)i; };
    auto aempty = [&](int i) { return bar0 + 8u * (uint32_t)(kStages + i); };
    auto dfull = [&](int i) { return bar0 + 8u * (uint32_t)(2 * kStages + i); };
    auto dempty = [&](int i) { return bar0 + 8u * (uint32_t)(2 * kStages + 2 + i); };
    const uint32_t done = bar0 + 8u * (uint32_t)(2 * kStages + 4);
    const int nsl = L.kp / kKS;
    const int n0 = half_rows(jm, 0), n1 = half_rows(jm, 1), nh = n1 ? 2 : 1, nu = ncb * nh;

    if (warp >= kEpiWarps && warp < kEpiWarps + kProdWarps) {
        if (!drop) produce_slices<FITS>(L, smem, bar0, ncb * nsl, src, abort_flag);
    } else if (warp == kMmaWarp) {
        // ---- MMA issue (one elected lane).  With a chunk's slices all in stages, half by
        // half, so that one half's accumulator is read out during the other's MMAs; else
        // slice by slice ----
        const bool lead = elect_lane();
        // slices outside the halves' loop (1 where they fit; a constant there made the
        // kernel take 355 us at 12o) and inside
        const int nslow = !FITS || nsl > L.stages ? nsl : 1;
        const int nin = FITS ? nsl / nslow : 1;
        bool ok = true;
        int st0 = 0;
        uint32_t full0 = 0;   // stage and parity of the next slice
        for (int c = 0; c < ncb && ok; ++c)
            for (int so = 0; so < nslow && ok; ++so) {
                int st = st0;
                uint32_t full = full0;
                for (int h = 0; h < nh && ok; ++h) {
                    const int u = c * nh + h, acc = u & 1, n = h ? n1 : n0;
                    const uint32_t boff = h ? (uint32_t)(ND * n0 / 8) * L.sbo_b : 0u;
                    st = st0;
                    full = full0;
                    // the accumulator's previous part was read out
                    if (so == 0 && u >= 2 && !wait_all<FITS>(dempty(acc), (uint32_t)(((u >> 1) - 1) & 1), abort_flag)) {
                        ok = false;
                        break;
                    }
                    for (int si = 0; si < nin; ++si) {
                        const int s = so * nin + si;
                        if (h == 0 && !wait_all<FITS>(afull(st), full, abort_flag)) { ok = false; break; }
                        tc_fence_after();
                        if (lead) {
                            issue_planes(L, sbase, st, s, boff, n, tmem + (uint32_t)(ND * n0 * acc));
                            if (h == nh - 1) umma_commit(aempty(st));   // the stage is free once these MMAs completed
                        }
                        __syncwarp();
                        if (++st == L.stages) { st = 0; full ^= 1u; }
                    }
                    if (ok && so == nslow - 1 && lead) umma_commit(dfull(acc));
                }
                st0 = st;
                full0 = full;
            }
        if (lead) umma_commit(done);   // every issued MMA has completed before TMEM is freed
        __syncwarp();
        if (lane == 0) mbar_wait_drain(done, 0u);
        __syncwarp();
    } else if (warp < kEpiWarps) {
        // ---- epilogue: half of the part's rows per warp, eight at a time ----
        const double2 *scale = reinterpret_cast<const double2 *>(smem + L.scale);
        const uint32_t lanes = tmem + ((uint32_t)((warp & 3) * 32) << 16);
        for (int u = 0; u < nu; ++u) {
            const int c = u / nh, h = u % nh, acc = u & 1;
            if (!wait_all<FITS>(dfull(acc), (uint32_t)((u >> 1) & 1), abort_flag)) break;
            tc_fence_after();
            const int n = h ? n1 : n0, e0 = (warp >> 2) * (n / 2), e1 = min(e0 + n / 2, jm - kHalf * h);
            const uint32_t base = lanes + (uint32_t)(ND * n0 * acc);
            double *zb = zrow + (i64)c * zrows * kM + (warp & 3) * 32 + lane;
            for (int e = e0; e < e1; e += 8) {   // warp-uniform; n / 2 is 8 or 16
                double v[8];
#pragma unroll
                for (int p = 0; p < 2; ++p) {   // the upper four diagonals, the lower four
                    int d[4][8];
#pragma unroll
                    for (int k = 0; k < 4; ++k) tmem_ld8(base + (uint32_t)(n * (4 * p + k) + e), d[k]);
                    tmem_wait_ld();
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const double x = sum4(d[0][i], d[1][i], d[2][i], d[3][i]);
                        v[i] = p ? fma(v[i], 4294967296.0, x) : x;
                    }
                }
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const int j = kHalf * h + e + i;
                    if (j < jm) zb[j * kM] = v[i] * scale[j].x * scale[j].y;
                }
            }
            tc_fence_before();
            if (u + 2 < nu) warp_arrive(dempty(acc));
        }
    }
}

__device__ __forceinline__ uint32_t split_begin(const SplitLayout &L, uint32_t sbase, unsigned char *smem, uint32_t cols,
                                             uint32_t readers, volatile int *abort_flag)
{
    const uint32_t bar0 = sbase + L.bars;
    if (threadIdx.x == 0) {
        for (int i = 0; i < kStages; ++i) {
            mbar_init(bar0 + 8u * (uint32_t)i, kProdWarps);
            mbar_init(bar0 + 8u * (uint32_t)(kStages + i), 1);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(bar0 + 8u * (uint32_t)(2 * kStages + i), 1);
            mbar_init(bar0 + 8u * (uint32_t)(2 * kStages + 2 + i), readers);   // warps that read an accumulator
        }
        mbar_init(bar0 + 8u * (uint32_t)(2 * kStages + 4), 1);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if ((threadIdx.x >> 5) == kMmaWarp) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(sbase + L.tmem), "r"(cols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    fence_async_smem();   // B (generic-proxy stores) is read by the tensor cores
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    return *reinterpret_cast<volatile uint32_t *>(smem + L.tmem);
}

__device__ __forceinline__ void split_end(uint32_t tmem, uint32_t cols)
{
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if ((threadIdx.x >> 5) == kMmaWarp)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(cols) : "memory");
}

// tensor memory of a pass: two accumulators of ND n columns, a power of two
__device__ __forceinline__ uint32_t split_cols(int cols) { return cols > 256 ? 512u : cols > 128 ? 256u : 128u; }

// A row's words back to FP64, and the row to mixed_dmma_kernel: the end of a CTA whose
// waits gave up, so that a stalled device costs time and never a result.  The elements
// are those of the words, within 2^-63 of the row's largest.
// Out of line: inlined, it takes the kernel's registers (72.0 against 67.9 ms at 16o).
__device__ __noinline__ void row_to_fp64(u64 *row, int ld, int e, int *rexp)
{
    const Pow2 f(e - kBits);
    for (int i = threadIdx.x; i < ld; i += kThreads)
        reinterpret_cast<double *>(row)[i] = (double)(long long)(row[i] - kBias) * f.a * f.b;
    if (threadIdx.x == 0) *rexp = kWideRow;
}

template <typename Ti, bool FITS>
__global__ void __launch_bounds__(kThreads, 1)
mixed_gemm_split_kernel(const MixedArgs P, const Ti *__restrict__ astr, u64 *ct, int *rexp, double *__restrict__ Z,
                        int z0, int W, int jbase, int rows, int drop)
{
    chain_wait();
    extern __shared__ __align__(1024) unsigned char smem[];
    const int K = P.nF;
    const int jcap = min(rows, P.M - jbase);
    const SplitLayout L = split_layout(K, jcap, kMixTab);
    int *conn = reinterpret_cast<int *>(smem + L.tab);
    int *sgn = conn + kMaxConn;
    const uint32_t sbase = (uint32_t)__cvta_generic_to_shared(smem);
    __shared__ int wcnt[kThreads / 32], cnt;
    __shared__ volatile int abort_flag;
    __shared__ int skip_all;
    const int a = blockIdx.x, aexp = rexp[a];
    u64 *row = ct + (i64)a * P.ldA;
    if (aexp == kWideRow) return;   // uniform across the CTA: mixed_dmma_kernel computes the row
    if (threadIdx.x == 0) skip_all = *(volatile int *)&g_tc_abort;
    __syncthreads();
    if (skip_all) {   // an earlier CTA gave up a wait
        row_to_fp64(row, P.ldA, aexp, rexp + a);
        return;
    }
    const int m = connected_excitations<kThreads>(P, (u64)astr[a], conn, sgn, wcnt, &cnt);
    const int jm = min(jcap, m - jbase);
    if (jm <= 0) return;   // uniform across the CTA
    const double *Lam = static_cast<const double *>(P.Lam);
    stage_b(
        L, smem, jm, K, aexp,
        [&](int j, int f) { return (double)sgn[jbase + j] * __ldg(Lam + (i64)conn[jbase + j] * K + f); },
        [&](int j) { return __ldg(P.lexp + conn[jbase + j]); });
    const uint32_t cols = split_cols(2 * ND * half_rows(jm, 0));
    const uint32_t tmem = split_begin(L, sbase, smem, cols, kEpiWarps, &abort_flag);
    const int zend = min(P.cend, z0 + W);
    const int ncb = (zend - z0 + kM - 1) / kM;
    GatherWords src;
    src.goff = P.goff;
    src.row = reinterpret_cast<const unsigned char *>(row);
    src.ldG = P.ldG;
    src.kp = L.kp;
    src.z0 = z0;
    src.nsl = L.kp / kKS;
    src.nq = ncb * src.nsl;
    split_pipeline<FITS>(L, smem, sbase, tmem, ncb, jm, zchunk(Z, a, P.M, W, 0) + jbase * kM, P.M, src,
                   &abort_flag, a == drop);
    split_end(tmem, cols);
    if (abort_flag)   // uniform: written before split_end's barrier
        row_to_fp64(ct + (i64)a * P.ldA, P.ldA, rexp[a], rexp + a);
}

}  // namespace

int mixed_split_rows(int nF, int M)
{
    for (int rows : {kRows, kRows / 2})
        if (split_layout(nF, std::min(M, rows), kMixTab).total + kStaticSmem <= kSmemMax) return rows;
    return 0;
}

int rows_to_fixed(double *in, int rows, int ld, int *rexp, cudaStream_t s)
{
    if (rows <= 0) return BSIM_OK;
    launch_chained(rows_to_fixed_kernel, rows, 256, 0, s, in, ld, rexp);
    BSIM_CUDA(cudaGetLastError());
    return BSIM_OK;
}

template <typename Ti>
int mixed_gemm_split(const MixedArgs &ma, const Ti *astr, double *ct, int *rexp, double *Z, int z0, int W, int jbase,
                     int rows, cudaStream_t s)
{
    // BSIM_SPLIT_DROP_ROW (tests): the producers of this row fill nothing, so the row's
    // waits run out
    const char *drop = getenv("BSIM_SPLIT_DROP_ROW");
    const SplitLayout L = split_layout(ma.nF, std::min(rows, ma.M - jbase), kMixTab);
    const size_t smem = L.total;
    auto kern = L.kp / kKS <= L.stages ? mixed_gemm_split_kernel<Ti, true> : mixed_gemm_split_kernel<Ti, false>;
    BSIM_CUDA(allow_smem(kern));
    launch_chained(kern, ma.nA, kThreads, smem, s, ma, astr, reinterpret_cast<u64 *>(ct), rexp, Z, z0, W, jbase, rows,
                   drop ? atoi(drop) : -1);
    BSIM_CUDA(cudaGetLastError());
    return BSIM_OK;
}

int split_timeouts(int *count, bool reset)
{
    int h = 0;
    BSIM_CUDA(cudaMemcpyFromSymbol(&h, g_tc_timeouts, sizeof(int)));
    if (reset) {
        const int z = 0;
        BSIM_CUDA(cudaMemcpyToSymbol(g_tc_timeouts, &z, sizeof(int)));
    }
    *count = h;
    return BSIM_OK;
}

template int mixed_gemm_split<unsigned>(const MixedArgs &, const unsigned *, double *, int *, double *, int, int, int,
                                        int, cudaStream_t);
template int mixed_gemm_split<unsigned long long>(const MixedArgs &, const unsigned long long *, double *, int *, double *,
                                                  int, int, int, int, cudaStream_t);

}  // namespace bsim

// Sequences of generator rotations, several components per pass (rotseq.cu).
#pragma once
#include "ops.h"

#include <vector>

namespace bsim {

constexpr int kRotComps = 4;   // components of one unit (a spin-adapted double has four)

// One group as a directed excitation: G = f sA sB (|dst><src| - |src><dst|) for
// the strings whose orbitals in am, bm hold the pattern as, bs, dst = src ^ (ax,
// bx), ax in am and bx in bm, with the signs sA = (-1)^popc(a & az), sB likewise.
struct RotComp {
    int kind = -1;             // -1 not looked at, 0 another form, 1 an excitation, 2 diagonal (no effect)
    u64 ax = 0, am = 0, as = 0, az = 0, bx = 0, bm = 0, bs = 0, bz = 0;
    double f = 0.0;
};

// Consecutive components [op0, op0 + m) whose alpha masks lie in the span of ga
// and whose beta masks lie in the span of gb; m = 0: the single operator op0
// goes through the pair kernels.
struct RotUnit {
    i64 op0 = 0;
    int m = 0;
    u64 ga[2] = {0, 0}, gb[2] = {0, 0};
    u64 ua = 0, ub = 0;        // orbitals the components look at
    int na = 0, nb = 0;        // alpha and beta orbits
    RotComp c[kRotComps];
    unsigned char xa[kRotComps] = {0}, xb[kRotComps] = {0};   // masks as combinations of ga, gb (bit 0, bit 1)
};

// The units of an operator sequence on one basis, and their application.
template <typename Ti>
class RotSequence {
public:
    // breaks: ascending operator positions that start a new unit
    int init(const DevBasis<Ti> *B, const DevNet<Ti> *P, i64 n_ops, const i64 *op_idx, const i64 *param_idx,
             const double *thetas, const std::vector<i64> &breaks, cudaStream_t s);
    ~RotSequence();
    // other work of the stream follows the last unit: the next one waits for it
    void unchain() { chained_ = false; }
    i64 size() const { return (i64)units_.size(); }
    const RotUnit &unit(i64 u) const { return units_[u]; }
    // v <- the unit's rotations applied in order
    int forward(i64 u, double *v);
    // the inverse rotations in reverse order on l and r; the gradient term of
    // operator i goes to terms[i] once flush() has run
    int backward(i64 u, double *l, double *r, double *terms);
    int flush(double *terms);
private:
    int lists(i64 u, bool ascending);
    template <bool BACK> int launch(i64 u, double *l, double *r, double *part);
    const DevBasis<Ti> *B_ = nullptr;
    const DevNet<Ti> *P_ = nullptr;
    const i64 *op_idx_ = nullptr, *param_idx_ = nullptr;
    const double *thetas_ = nullptr;
    cudaStream_t s_ = nullptr;
    std::vector<RotUnit> units_;
    void *mem_ = nullptr;            // unit descriptors, orbit lists of one batch, partial sums
    void *d_units_ = nullptr, *d_ops_ = nullptr;
    int4 *d_idx_ = nullptr;
    unsigned *d_bits_ = nullptr;
    double *d_part_ = nullptr;
    i64 batch_ = 0, b0_ = -1, b1_ = -1;   // units per batch; the batch whose lists are in place
    i64 pend0_ = 0, pend1_ = 0;           // units whose partial sums wait for flush()
    int rows_ = 1;                        // partial sums of a unit (its alpha orbits, at most)
    bool chained_ = false;                // the last launch was a unit whose lists are in place
};

}  // namespace bsim

// State and stopping rule of the trace-correcting (SP2) purification on the
// device, shared by the single-system path (sp2.cu) and the grouped one
// (sp2_batch.cu).
#pragma once

#include <cmath>
#include <vector>

#include "ptbgpu.h"

namespace ptb {

constexpr int kMaxIt = 255;
// Contraction of the refinement rounds per unit response gain g of the first
// round (measured bounds, see sp2_mixed): the first round leaves at most
// kRho1 * g of its correction, every later one at most kRho2 * g of its own.
constexpr double kRho1 = 6.5e-5;
constexpr double kRho2 = 2.6e-4;
// What pass 1 had not converged when it ended: the replay gives a state that still is f
// away from 0 or 1 a share 1 - f of its response.  f <= ||X - X^2||_F of pass 1's last
// iterate, which is the length of the step that the cleanup takes from it; it can hide
// below the rounding floor of the trace, to 0.03 (2e-5 to 4e-4 in three of four boxes).
// The first round left up to 0.9 of this bound of its correction in 1925 water boxes and
// chains; half of it keeps what is left above 1e-7 to 0.2 % of them and 1.7e-7 (without:
// 1.9 % and 6.3e-7) and takes a second round in 13 % (6.5 %).
constexpr double kRhoF = 0.5;

struct SP2State {
    int active;      // 1 while pass 1 runs; product/decision launches are no-ops at 0
    int next;        // index of the iterate the next decision evaluates
    int converged;
    int status;      // 0 or a PTBGPU_E* code
    int sq_cur;      // branch for the step about to run
    int pad[3];
    double trX[kMaxIt + 1];
    double trX2[kMaxIt + 1];
    double err[kMaxIt + 1];
    int sq[kMaxIt + 1];
};

// Whether the traces leave the occupied states in no doubt.  An idempotency error far
// below one and a trace within half an electron of N put every eigenvalue near 0 or 1 and
// N of them near 1, and both branches keep the eigenvalues' order.  A small error alone
// does not: X^2 at a trace above N + 1/2 can take all states around a small gap down to
// a few hundredths, the highest occupied one among them, which then has to double its way
// back up through an error of order one.
__host__ __device__ __forceinline__ bool sp2_counted(double trX, double N) { return fabs(trX - N) < 0.5; }

// Record iterate k's traces and decide the next step (one thread): the branch
// by the trace (Niklasson's trace correction), the stop at the rounding floor,
// the iteration cap.
__device__ __forceinline__ void sp2_decide(SP2State* st, double trX, double trX2, double N, double tol_abs,
                                           double e_asym, int maxit) {
    const int k = st->next;
    const double e = trX - trX2;
    st->trX[k] = trX;
    st->trX2[k] = trX2;
    st->err[k] = e;
    if (!(e == e)) {
        st->status = PTBGPU_ENAN;
        st->active = 0;
        return;
    }
    const int sq = fabs(trX2 - N) <= fabs(2.0 * trX - trX2 - N) ? 1 : 0;
    st->sq[k] = sq;
    st->sq_cur = sq;
    const double ae = fabs(e);
    // Rounding floor: in the asymptotic regime (every eigenvalue within ~0.1 of 0 or 1
    // and the right ones of them, which e < e_asym and the count imply) two exact steps
    // always lower e, so no decrease over two steps means rounding.  Outside it nothing is
    // read off e: states around a small gap hold it level or let it rise for many steps.
    if (sp2_counted(trX, N) && (ae < tol_abs || (k >= 2 && ae < e_asym && ae >= fabs(st->err[k - 2])))) {
        st->converged = 1;
        st->active = 0;
    } else if (k >= maxit || k >= kMaxIt) {
        st->status = PTBGPU_EITER;   // left to the FP64 path
        st->active = 0;
    } else {
        st->next = k + 1;
    }
}

// FP64 steps (the FP64 path and the cleanup): stop at rounding, or where the error stops
// falling over two steps; both only once the states are counted.
inline bool sp2_floor(const std::vector<double>& hist, double trX, double N, double n) {
    const double e = hist.back();
    return sp2_counted(trX, N) && (e < 1e-13 * n || (hist.size() > 2 && e < 1e-2 && e >= hist[hist.size() - 3]));
}
// The cleanup's result as a projector: its error per state is of the order of e at most.
// Measured floors: 2e-10 with 8 slices at order 11776, 1e-8 with 7.
inline bool sp2_settled(double e, double trX, double N) { return sp2_counted(trX, N) && e < 1e-4; }

}  // namespace ptb

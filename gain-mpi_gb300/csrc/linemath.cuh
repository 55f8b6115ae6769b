// S, A and I of one line (BaseClasses/Output.cpp:52-112), shared by the line
// assembly (k_lines) and the line-list text kernels so both see the same doubles.
#pragma once
#include "gain_internal.h"

namespace gain {

constexpr long long kInfBits = 0x7ff0000000000000ll;
constexpr long long kNuMinBits = 0x37a16c262777579cll;   // 1e-40

struct LineVals {
    double nu, ls, A;
    int keep;   // the reference writes the line: nu in FREQ-WINDOW, nu >= 1e-40, A >= THRESH_LINE
};

// The line strength of the line at amp[off] (and its component slots).
__device__ __forceinline__ double line_ls(const double* amp, long off, const LineParams& p) {
    if (p.nslot == 0) {
        const double a = amp[off];
        return __dmul_rn(a, a);                               // :83, ndegI = ndegF = 1
    }
    double ls = 0.0;
    for (int s = 0; s < p.nslot; ++s) {                       // :78-85
        const double a = amp[off + (long)p.slot[s] * p.slot_stride];
        ls = __dadd_rn(ls, __dmul_rn(a, a));
    }
    ls = __ddiv_rn(ls, (double)p.ndegI);                      // :89
    if (p.reduced_deg) ls = __dmul_rn(ls, (double)p.ndegI);   // :90-91
    return ls;
}

__device__ __forceinline__ LineVals line_eval(const double* amp, long off, double eIr, double eFc,
                                              const LineParams& p) {
    LineVals v;
    v.nu = eFc - eIr;
    v.ls = line_ls(amp, off, p);
    const double anu = fabs(v.nu);
    v.A = __dmul_rn(__dmul_rn(__dmul_rn(__dmul_rn(p.acoef_2jI1, v.ls), anu), anu), anu);   // :93
    // by the bits: A is not negative (or NaN), nu below 1e-40 is not written, and a comparison
    // of doubles costs the FP64 pipe as much as a product
    const long long bn = __double_as_longlong(v.nu), ba = __double_as_longlong(v.A);
    v.keep = (bn >= p.nu_lo && bn <= p.nu_hi && bn <= kInfBits && ba >= p.a_lo && ba <= kInfBits) ? 1 : 0;
    return v;
}

// exp(-beta E''), the intensity's factor that depends on the row only: a caller with several
// lines of a row takes it once (each FP64 exp is about a third of a line's arithmetic).
__device__ __forceinline__ double line_row_factor(double eIr, const LineParams& p) {
    return exp(-p.beta * (eIr - p.zpe));
}

// CMCOEF*A*gns*(2jF+1)*exp(-beta E'')*(1-exp(-beta nu))/(nu^2 Q), :101-102; 0 where nu < 1e-40.
// *e2 is exp(-beta nu).
__device__ __forceinline__ double line_intensity(const LineVals& v, double row_factor, const LineParams& p,
                                                 double* e2) {
    *e2 = 0.0;
    const long long bn = __double_as_longlong(v.nu);
    if (bn < kNuMinBits || bn > kInfBits) return 0.0;
    double t = __dmul_rn(p.cmcoef, v.A);
    t = __dmul_rn(t, p.gnsF);
    t = __dmul_rn(t, p.two_jF1);
    t = __dmul_rn(t, row_factor);
    *e2 = exp(-p.beta * v.nu);
    t = __dmul_rn(t, 1.0 - *e2);
    return __ddiv_rn(t, __dmul_rn(__dmul_rn(v.nu, v.nu), p.q_part));
}

}  // namespace gain

// fdiv.h -- IEEE double division by a divisor shared by several quotients.
//
// One reciprocal of the divisor serves every quotient, and all of it runs on the integer
// pipe (softdbl.h): GB300 runs FP64 at a small fraction of its other rates, and a double
// division is a sequence of several FP64 instructions.  The fast path covers divisors
// with binary exponent in [-125, 125] and numerators that are zero or have exponent in
// [-200, 200); anything else takes the plain division.  Results are the IEEE quotients
// bit for bit, signed zeros included.  Plain C++ on the host, so host tests check the
// same code.
#pragma once

#include "softdbl.h"

#if defined(__CUDACC__)
#define EBB_FDIV_HD __host__ __device__ __forceinline__
#else
#define EBB_FDIV_HD inline
#endif

namespace ebbdiv {

EBB_FDIV_HD uint64_t bits_of(double x) { return ((uint64_t)ebbsoft::hi_of(x) << 32) | ebbsoft::lo_of(x); }

struct Recip {
    double b;
    ebbsoft::Recip r;
    bool ok;  // the fast path applies to this divisor
};

EBB_FDIV_HD Recip recip(double b) { return {b, ebbsoft::recip(b), ebbsoft::divisor_ok(b)}; }

// RN(a / R.b)
EBB_FDIV_HD double div(double a, const Recip &R)
{
    bool bad = !R.ok;
    ebbsoft::check<200>(a, bad);
    return bad ? a / R.b : ebbsoft::div(a, R.r);
}

}  // namespace ebbdiv

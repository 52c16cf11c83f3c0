// word_sum.h -- a running sum of floats that is held no shorter than in 64 bits, on the FP32 pipe.
#pragma once

#include <cmath>

namespace ekg {

#ifdef __CUDACC__
#define EKG_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define EKG_HOST_DEVICE inline
#endif

// The sum, the rounding errors of its additions, and those of their additions (cascaded two-sums; Ogita,
// Rump and Oishi, "Accurate sum and dot product", 2005).  With S = sum |w| and u = 2^-24 the words lose at
// most n^3 u^3 S over n terms, below the n 2^-53 S of a sum in FP64 up to WORD_SUM_MAX terms; value() rounds
// what they hold to a float once more.  An infinite or undefined sum comes out as the plain one does.
constexpr int WORD_SUM_MAX = 512;
struct WordSum {
    float s = 0.f, e = 0.f, f = 0.f;
    // a + b rounded, and its error; no operation may be contracted into another one
    static EKG_HOST_DEVICE float two_sum(float a, float b, float &err) {
#ifdef __CUDA_ARCH__
        const float r = __fadd_rn(a, b), bb = __fsub_rn(r, a);
        err = __fadd_rn(__fsub_rn(a, __fsub_rn(r, bb)), __fsub_rn(b, bb));
#else
        const float r = a + b, bb = r - a;
        err = (a - (r - bb)) + (b - bb);
#endif
        return r;
    }
    // the second term behind a first one that was put into s
    EKG_HOST_DEVICE void second(float w) { s = two_sum(s, w, e); }
    EKG_HOST_DEVICE void add(float w) {
        float d, d2;
        s = two_sum(s, w, d);
        e = two_sum(e, d, d2);
        f += d2;
    }
    EKG_HOST_DEVICE float value() const {
        if (!(fabsf(s) < INFINITY)) return s;
        float d;
        const float r = two_sum(s, e, d);
        return r + (d + f);
    }
    EKG_HOST_DEVICE double wide() const {
        if (!(fabsf(s) < INFINITY)) return (double)s;
        return (double)s + ((double)e + (double)f);
    }
};

}  // namespace ekg

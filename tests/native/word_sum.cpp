// word_sum.cpp -- the resident lead field's running sum (csrc/word_sum.h) for tests/test_word_sum.py
#include "word_sum.h"

extern "C" float word_sum(const float *w, int n) {
    ekg::WordSum a;
    for (int i = 0; i < n; ++i) a.add(w[i]);
    return a.value();
}
// with the short forms of the first two terms
extern "C" float word_sum_short(const float *w, int n) {
    ekg::WordSum a;
    a.s = w[0];
    if (n > 1) a.second(w[1]);
    for (int i = 2; i < n; ++i) a.add(w[i]);
    return a.value();
}
// in parts of WORD_SUM_MAX terms, as for an AP of more voxels
extern "C" float word_sum_parts(const float *w, int n) {
    double wide = 0.0;
    for (int c = 0; c < n; c += ekg::WORD_SUM_MAX) {
        ekg::WordSum a;
        for (int i = c; i < n && i < c + ekg::WORD_SUM_MAX; ++i) a.add(w[i]);
        wide += a.wide();
    }
    return (float)wide;
}

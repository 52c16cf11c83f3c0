// eval_buffers_check.cpp -- the buffers of an evaluation after an allocation that failed, on the host: the
// allocator is replaced by one with a limit, which knows what is allocated.  For tests/test_buffers.py:
//   eval_buffers_check pass|band|dense few many
// takes the buffers of `few` simulations, fails to take those of `many`, takes those of `few` again, and
// reports every buffer that is held but not allocated, or too small for what the last call asked for.
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>

#include "ekg_internal.h"

namespace {
size_t limit = (size_t)-1, total = 0;
std::map<char *, size_t> live;
}  // namespace

extern "C" {
cudaError_t cudaMalloc(void **p, size_t n) {
    if (total + n > limit) return cudaErrorMemoryAllocation;
    // addresses only: nothing reads or writes these buffers here
    static char *next = reinterpret_cast<char *>(uintptr_t(1) << 40);
    live[next] = n;
    total += n;
    *p = next;
    next += (n + 4095) / 4096 * 4096 + 4096;
    return cudaSuccess;
}
cudaError_t cudaFree(void *p) {
    auto it = live.find(static_cast<char *>(p));
    if (it == live.end()) {
        std::printf("freed what was not allocated\n");
        std::exit(1);
    }
    total -= it->second;
    live.erase(it);
    return cudaSuccess;
}
cudaError_t cudaGetLastError(void) { return cudaSuccess; }
const char *cudaGetErrorString(cudaError_t) { return "out of memory"; }
}

using namespace ekg;

static int bad = 0;
template <class T>
static void check(const char *when, const char *name, const DBuf<T> &b, size_t need) {
    if (b.n < need) {
        std::printf("%s: %s holds %zu of %zu\n", when, name, b.n, need);
        ++bad;
    }
    if (!b.n && !b.p) return;
    const char *p = reinterpret_cast<const char *>(b.p);
    auto it = live.upper_bound(const_cast<char *>(p));
    if (it == live.begin() || (--it, p + b.n * sizeof(T) > it->first + it->second)) {
        std::printf("%s: %s is not allocated\n", when, name);
        ++bad;
    }
}
static void check_all(const char *when, const EvalDev &E, const HeartDev &D, const char *form, size_t S) {
    const size_t T = D.steps, L = D.nleads, nl = D.nlayers, nc = S * D.nchunks;
    const bool pass = !std::strcmp(form, "pass"), band = !std::strcmp(form, "band"), dense = !std::strcmp(form, "dense");
    check(when, "layer_c", E.layer_c, pass ? S * nl * 4 : 0);
    check(when, "F", E.F, pass ? S * nl * T : 0);
    check(when, "Ff", E.Ff, pass ? S * nl * T : 0);
    check(when, "k0w", E.k0w, pass ? S * L : 0);
    check(when, "out", E.out, pass && S ? EvalDev::ecg_offset((int)S, (int)L) + S * L * T : 0);
    check(when, "ecg_ff", E.ecg_ff, pass ? S * L * T : 0);
    check(when, "W", E.W, band || dense ? S * L * D.apad : 0);
    check(when, "Wp", E.Wp, dense ? S * L * D.apad : 0);
    check(when, "work", E.work, (band || dense) && S ? 1 : 0);
    check(when, "band", E.band, band ? nc * L * T : 0);
    check(when, "csum", E.csum, band ? nc * L : 0);
    check(when, "cinfo", E.cinfo, band ? nc : 0);
    check(when, "partial", E.partial, dense ? nc * L * T : 0);
    if (pass && E.cap_sims && (size_t)E.cap_sims < S) ++bad;
}

int main(int argc, char **argv) {
    if (argc != 4) return 2;
    const char *form = argv[1];
    const int few = std::atoi(argv[2]), many = std::atoi(argv[3]);
    HeartDev D;
    D.apad = 192;
    D.nlayers = 3;
    D.nleads = 5;
    D.steps = 70;
    D.nchunks = 4;
    EvalDev E;
    auto take = [&](int n) {
        if (!std::strcmp(form, "pass")) E.reserve_pass(D, n);
        else E.reserve_general(D, n, !std::strcmp(form, "band"));
    };
    take(few);
    check_all("at first", E, D, form, few);
    limit = total + total / 4;  // one block more of the size is too much, the old one freed or not
    int code = 0;
    try {
        take(many);
    } catch (const Error &e) {
        code = e.code;
    }
    if (code != EKG_ERR_OUT_OF_MEMORY) {
        std::printf("the larger batch: %d\n", code);
        ++bad;
    }
    check_all("after the failure", E, D, form, 0);
    take(few);
    check_all("again", E, D, form, few);
    limit = (size_t)-1;
    take(many);
    check_all("with room", E, D, form, many);
    return bad ? 1 : 0;
}

// Host build of the FP64 filter (circlepacking_b200/csrc/cp_filter.cuh) for the
// CPU tests: the same code with the host's reciprocal seeds.
#include "cp_filter.cuh"

using namespace cpb::flt;

namespace {
template <int FAM, int NEED>
void run(const double* lo, const double* hi, long n, int order, unsigned char* decided, unsigned char* mask) {
    constexpr bool kThree = FAM != 1 && FAM != 4;
    for (long i = 0; i < n; ++i) {
        FBox b{lo[i], hi[i], lo[n + i], hi[n + i], lo[2 * n + i], hi[2 * n + i], 0.0, 0.0};
        if (kThree) {
            b.l3 = lo[3 * n + i];
            b.h3 = hi[3 * n + i];
            if (b.l2 < b.l3) b.l2 = b.l3;
        }
        if (b.l1 < b.l2) b.l1 = b.l2;
        FOut o{0, 0};
        const bool empty = b.ll > b.lh || b.l1 > b.h1 || b.l2 > b.h2 || (kThree && b.l3 > b.h3);
        decided[i] = !empty && filter_box<FAM, NEED>(ValRef{b}, order, o);
        mask[i] = o.mask;
    }
}
template <int FAM>
void need(int n_, const double* lo, const double* hi, long n, int order, unsigned char* d, unsigned char* m) {
    if (n_ == NEED_VERDICT) run<FAM, NEED_VERDICT>(lo, hi, n, order, d, m);
    if (n_ == NEED_HANDLES) run<FAM, NEED_HANDLES>(lo, hi, n, order, d, m);
    if (n_ == NEED_MASK) run<FAM, NEED_MASK>(lo, hi, n, order, d, m);
    if (n_ == NEED_FULL) run<FAM, NEED_FULL>(lo, hi, n, order, d, m);
}
}  // namespace

extern "C" {
void filter_boxes(int fam, int need_, const double* lo, const double* hi, long n, int order, unsigned char* decided,
                  unsigned char* mask) {
    switch (fam) {
    case 0: return need<0>(need_, lo, hi, n, order, decided, mask);
    case 1: return need<1>(need_, lo, hi, n, order, decided, mask);
    case 2: return need<2>(need_, lo, hi, n, order, decided, mask);
    case 3: return need<3>(need_, lo, hi, n, order, decided, mask);
    case 4: return need<4>(need_, lo, hi, n, order, decided, mask);
    default: return need<5>(need_, lo, hi, n, order, decided, mask);
    }
}
// asin of n / d the two ways the filter takes it
void filter_asin(const double* n, const double* d, long count, double* out, unsigned char* ok) {
    for (long i = 0; i < count; ++i) {
        bool k = true;
        out[i] = asin_quot(n[i], d[i], rcp_(d[i]), k);
        ok[i] = k;
    }
}
}

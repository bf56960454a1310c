// The split of rows over threads that with_split() chooses (host code only): prints
// "<operator> <rows> <split> <split of whole rows>" per line.
#include <cstdio>

#include "qmb_ham.cuh"

template <class Op>
static void show(const char* name, int64_t n, int n_ext = 1) {
    Op op{};
    op.n = n;
    if constexpr (qmb::OpMaxSplit<Op>::value == 8) op.rg.g.n_ext = n_ext;
    int s = 0, w = 0;
    qmb::with_split(op, [&](auto k) { s = decltype(k)::value; });
    qmb::with_split(op, [&](auto k) { w = decltype(k)::value; }, true);
    std::printf("%s %lld %d %d\n", name, (long long)n, s, w);
}

int main() {
    for (int64_t n : {1, 16383, 16384, 39999, 40000, 131071, 131072, 299999, 300000, 399999, 400000, 639999, 640000}) {
        show<qmb::SellOp<float>>("sell", n);
        show<qmb::SellOp<double2>>("sell_c64", n);
        show<qmb::MfOp<double>>("mf", n, 24);
        show<qmb::MfOp<float, true>>("mf_no_group", n, 1);
        show<qmb::RefEllOp<float2>>("ref_ell", n);
        show<qmb::CbSellOp<float>>("coded", n);
    }
    return 0;
}

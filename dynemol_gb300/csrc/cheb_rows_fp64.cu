// cheb_rows_kernel in FP64, and the choice among the three arithmetics.
#include "cheb_rows.cuh"

namespace elhl {
using namespace rows;

namespace {
// rows per CTA with an instance: FP64 and DF64 are bound by their products above a
// few hundred AOs, so every count has one; FP32 is not, so a few serve
constexpr int kMaxRows = 13;
constexpr int kRows32[] = {1, 2, 3, 4, 5, 6, 8, 10, 13, 16};

template <typename A>
bool fits(int N, int m, int R) {
    return (m == 2 ? smem_bytes<A, 2 * A::kPerColumn>(N, R) : smem_bytes<A, 4 * A::kPerColumn>(N, R)) <= kSmemLimit;
}
}  // namespace

// Where the kernel pays: with FP64 or DF64 words the exchange (16 bytes a word, every
// word read by every CTA) overtakes what the barrier and the lane sums cost cheb_kernel
// at about 5,000 row-columns.  Propagation of one step in ms, cheb_kernel / this kernel:
// FP64 four columns 1.01 / 0.22 at N = 62, 2.30 / 1.46 at 620, 3.68 / 3.13 at 1032,
// 5.26 / 5.36 at 1395; two columns 0.297 / 0.106 at 465, 0.89 / 0.71 at 1240; DF64 0.62 /
// 0.25 at 62, 1.91 / 1.73 at 1032, 2.51 / 2.78 at 1395; FP32 0.52 / 0.18 at 62, 0.85 /
// 0.50 at 744, 1.44 / 1.26 at 1860, level where its rows end (2,432).
constexpr int kMaxWide = 5000;

int cheb_rows_fit(int precision, int N, int m, int sms) {
    if (N < 2 || sms < 1 || (m != 2 && m != 4)) return 0;
    const int R = (N + sms - 1) / sms;
    if ((precision == ELHL_PREC_FP64 || precision == ELHL_PREC_DF64) && N * m > kMaxWide) return 0;
    if (precision == ELHL_PREC_FP64) return R <= kMaxRows && fits<F64>(N, m, R) ? R : 0;
    if (precision == ELHL_PREC_DF64) return R <= kMaxRows && fits<DF64>(N, m, R) ? R : 0;
    for (int r : kRows32)
        if (r >= R) return fits<F32>(N, m, r) ? r : 0;
    return 0;
}

size_t cheb_rows_words(int precision, int N, int m) {
    return (size_t)N * m * (precision == ELHL_PREC_FP64 || precision == ELHL_PREC_DF64 ? 2 : 1);
}

cudaError_t launch_cheb_rows_fp64(const RowsLaunch &L, int rows, cudaStream_t st) {
#define ELHL_ROWS(R_) \
    case R_: return L.m == 2 ? launch<F64, 4, R_>(L, st) : launch<F64, 8, R_>(L, st);
    switch (rows) {
        ELHL_ROWS(1) ELHL_ROWS(2) ELHL_ROWS(3) ELHL_ROWS(4) ELHL_ROWS(5) ELHL_ROWS(6) ELHL_ROWS(7)
        ELHL_ROWS(8) ELHL_ROWS(9) ELHL_ROWS(10) ELHL_ROWS(11) ELHL_ROWS(12) ELHL_ROWS(13)
    }
#undef ELHL_ROWS
    return cudaErrorInvalidValue;
}

cudaError_t launch_cheb_rows(const RowsLaunch &L, int precision, int rows, cudaStream_t st) {
    if (precision == ELHL_PREC_FP64) return launch_cheb_rows_fp64(L, rows, st);
    if (precision == ELHL_PREC_DF64) return launch_cheb_rows_df64(L, rows, st);
    return launch_cheb_rows_fp32(L, rows, st);
}

}  // namespace elhl

// cheb_rows_kernel in FP32 pairs (DF64).
#include "cheb_rows.cuh"

namespace elhl {
using namespace rows;

cudaError_t launch_cheb_rows_df64(const RowsLaunch &L, int rows, cudaStream_t st) {
#define ELHL_ROWS(R_) \
    case R_: return L.m == 2 ? launch<DF64, 4, R_>(L, st) : launch<DF64, 8, R_>(L, st);
    switch (rows) {
        ELHL_ROWS(1) ELHL_ROWS(2) ELHL_ROWS(3) ELHL_ROWS(4) ELHL_ROWS(5) ELHL_ROWS(6) ELHL_ROWS(7)
        ELHL_ROWS(8) ELHL_ROWS(9) ELHL_ROWS(10) ELHL_ROWS(11) ELHL_ROWS(12) ELHL_ROWS(13)
    }
#undef ELHL_ROWS
    return cudaErrorInvalidValue;
}

}  // namespace elhl

// cheb_rows_kernel in FP32 (FP64 sums of c_k v_k).
#include "cheb_rows.cuh"

namespace elhl {
using namespace rows;

cudaError_t launch_cheb_rows_fp32(const RowsLaunch &L, int rows, cudaStream_t st) {
#define ELHL_ROWS(R_) \
    case R_: return L.m == 2 ? launch<F32, 2, R_>(L, st) : launch<F32, 4, R_>(L, st);
    switch (rows) {
        ELHL_ROWS(1) ELHL_ROWS(2) ELHL_ROWS(3) ELHL_ROWS(4) ELHL_ROWS(5) ELHL_ROWS(6) ELHL_ROWS(8)
        ELHL_ROWS(10) ELHL_ROWS(13) ELHL_ROWS(16)
    }
#undef ELHL_ROWS
    return cudaErrorInvalidValue;
}

}  // namespace elhl

// Row kernels of the SpMM for __nv_bfloat16 rows.
#include "spmm_stream.cuh"

namespace apt {
APT_DEFINE_SPMM_ROWS(__nv_bfloat16)
}  // namespace apt

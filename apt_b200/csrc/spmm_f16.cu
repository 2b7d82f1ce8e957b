// Row kernels of the SpMM for __half rows.
#include "spmm_bulk.cuh"

namespace apt {
APT_DEFINE_SPMM_ROWS(__half)
}  // namespace apt

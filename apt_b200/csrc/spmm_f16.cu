// Row kernels of the SpMM for __half rows.
#include "spmm_stream.cuh"

namespace apt {
APT_DEFINE_SPMM_ROWS(__half)
}  // namespace apt

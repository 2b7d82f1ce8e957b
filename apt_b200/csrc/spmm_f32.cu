// Row kernels of the SpMM for float rows.
#include "spmm_stream.cuh"

namespace apt {
APT_DEFINE_SPMM_ROWS(float)
}  // namespace apt

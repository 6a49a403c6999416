// bin_single.cu -- the row-binning kernel for one field (bin_rows.cuh).
#include "bin_rows.cuh"

namespace genpk {

cudaError_t bin_rows_single(const BinParams &p, const BinDevice &d, double *partial, int ctas,
                            size_t smem, cudaStream_t stream)
{
    return launch_bin_rows<1, false>(p, d, partial, ctas, smem, stream);
}

}  // namespace genpk

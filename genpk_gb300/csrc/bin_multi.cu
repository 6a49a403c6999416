// bin_multi.cu -- the row-binning kernel for two to four fields (bin_rows.cuh).
#include "bin_rows.cuh"

namespace genpk {

cudaError_t bin_rows_multi(int nf, bool cross1, const BinParams &p, const BinDevice &d,
                           double *partial, int ctas, size_t smem, cudaStream_t stream)
{
    if (cross1)
        return launch_bin_rows<2, true>(p, d, partial, ctas, smem, stream);
    if (nf == 2)
        return launch_bin_rows<2, false>(p, d, partial, ctas, smem, stream);
    if (nf == 3)
        return launch_bin_rows<3, false>(p, d, partial, ctas, smem, stream);
    return launch_bin_rows<4, false>(p, d, partial, ctas, smem, stream);
}

}  // namespace genpk

// columns.h -- result columns that lie side by side in one block, to the host.
#pragma once

#include "common.cuh"

namespace fgss {

// `cols` columns of `width` bytes, spitch bytes apart on the device, to the host dpitch
// bytes apart.  One copy while both pitches are at most `most` (Ctx::max_pitch: CUDA
// refuses a 2-D copy of a larger one, which a column of 2^29 pairs has), else one for
// each column.  (One copy instead of six: a call on 1,000 titles 303 -> 291 us.)
inline void columns_to_host(void* dst, size_t dpitch, const void* src, size_t spitch, size_t width, int cols, size_t most,
                            cudaStream_t stream) {
    if (dpitch <= most && spitch <= most) {
        FGSS_CK(cudaMemcpy2DAsync(dst, dpitch, src, spitch, width, cols, cudaMemcpyDeviceToHost, stream));
        return;
    }
    for (int k = 0; k < cols; k++)
        FGSS_CK(cudaMemcpyAsync(static_cast<char*>(dst) + k * dpitch, static_cast<const char*>(src) + k * spitch, width,
                                cudaMemcpyDeviceToHost, stream));
}

}  // namespace fgss

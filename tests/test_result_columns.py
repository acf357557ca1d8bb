"""Columns of a result to the host (csrc/columns.h): one 2-D copy while the runtime takes the pitch, else
one copy a column.  On the CPU, with a runtime that refuses pitches above its limit as CUDA does."""
import fake_util

PROGRAM = r"""
#include <stdio.h>
#include <string.h>
#include <vector>
#include "columns.h"
static size_t limit;
static int one, two;
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "invalid pitch argument"; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
    memcpy(d, s, n);
    one++;
    return cudaSuccess;
}
cudaError_t cudaMemcpy2DAsync(void* d, size_t dp, const void* s, size_t sp, size_t w, size_t h, cudaMemcpyKind, cudaStream_t) {
    if (dp > limit || sp > limit || w > dp || w > sp) return cudaErrorInvalidPitchValue;
    for (size_t k = 0; k < h; k++) memcpy((char*)d + k * dp, (const char*)s + k * sp, w);
    two++;
    return cudaSuccess;
}
int main() {
    const size_t cases[][4] = {{1024, 1024, 1000, 1024}, {1024, 1024, 1024, 1023}, {1024, 2048, 1000, 1024},
                               {2048, 1024, 4, 2047},    {256, 512, 256, 512},     {256, 512, 0, 511}};
    for (auto& c : cases) {
        const size_t dp = c[0], sp = c[1], w = c[2];
        limit = c[3];
        std::vector<unsigned char> src(6 * sp), dst(6 * dp, 0xee);
        for (size_t i = 0; i < src.size(); i++) src[i] = (unsigned char)(i * 7 + i / 256);
        one = two = 0;
        bool ok = true;
        try {
            fgss::columns_to_host(dst.data(), dp, src.data(), sp, w, 6, limit, nullptr);
        } catch (const fgss::Error&) {
            ok = false;
        }
        for (size_t k = 0; k < 6 && ok; k++)
            for (size_t i = 0; i < dp; i++) ok &= dst[k * dp + i] == (i < w ? src[k * sp + i] : 0xee);
        printf("%d %d %d\n", (int)ok, one, two);
    }
}
"""


def test_one_copy_up_to_the_largest_pitch(tmp_path):
    out = fake_util.run(tmp_path, PROGRAM).splitlines()
    assert out == ["1 0 1", "1 6 0", "1 6 0", "1 6 0", "1 0 1", "1 6 0"]


def test_results_go_to_the_host_through_it():
    import os
    src = open(os.path.join(fake_util.CSRC, "api.cu")).read()
    assert "cudaMemcpy2DAsync" not in src and src.count("columns_to_host(") == 2

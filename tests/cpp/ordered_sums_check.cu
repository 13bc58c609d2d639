// ordered_column_sum and ordered_sum (mlp.cuh) against a loop over the rows, bit for bit. The matrix is
// allocated to its last element and its rows past the end hold nothing that may be added.
#include <cstdio>
#include <cstring>
#include <vector>

#include "mlp.cuh"

using namespace lsp;

__global__ void k_sums(const float* m, int rows, int width, const float* v, int n, float* out)
{
    __shared__ SumBuffer buf;
    if (blockIdx.x == gridDim.x - 1) {
        const float s = ordered_sum(v, n, buf);
        if (threadIdx.x == 0) out[width] = s;
        return;
    }
    const float s = ordered_column_sum(m, rows, width, blockIdx.x * kSumCols, buf);
    const int c = blockIdx.x * kSumCols + (int)threadIdx.x;
    if (threadIdx.x < kSumCols && c < width) out[c] = s;
}

static uint32_t g_seed = 1;
static float next()
{
    g_seed = g_seed * 1664525u + 1013904223u;
    // Magnitudes over twelve binades and both signs, so that a row lost, doubled or out of order shows.
    const int e = (int)(g_seed >> 28) - 6;
    const float f = (float)(int32_t)(g_seed << 4) / 2147483648.f;
    return ldexpf(f, e);
}

int main()
{
    const int rows_of[] = {1, 31, 32, 33, 255, 256, 257, 511, 512, 513, 1000, 2048, 2368};
    const int widths[] = {1, 7, 8, 9, kMlpParams};
    const int lengths[] = {1, 31, 33, 2079, 2080, 2081, 2368, 5000};
    int checked = 0;
    long long bad = 0;
    for (int rows : rows_of)
        for (int width : widths) {
            const int n = lengths[checked % 8];
            std::vector<float> m((size_t)rows * width), v(n), want(width + 1, 0.f), got(width + 1);
            for (float& x : m) x = next();
            for (float& x : v) x = next();
            for (int r = 0; r < rows; r++)
                for (int c = 0; c < width; c++) want[c] += m[(size_t)r * width + c];
            for (float x : v) want[width] += x;
            float *dm, *dv, *out;
            cudaMalloc(&dm, m.size() * 4);
            cudaMalloc(&dv, v.size() * 4);
            cudaMalloc(&out, got.size() * 4);
            cudaMemcpy(dm, m.data(), m.size() * 4, cudaMemcpyHostToDevice);
            cudaMemcpy(dv, v.data(), v.size() * 4, cudaMemcpyHostToDevice);
            k_sums<<<sum_blocks(width), kSumThreads>>>(dm, rows, width, dv, n, out);
            const cudaError_t e = cudaMemcpy(got.data(), out, got.size() * 4, cudaMemcpyDeviceToHost);
            if (e != cudaSuccess) {
                printf("%s\n", cudaGetErrorString(e));
                return 1;
            }
            for (int c = 0; c <= width; c++)
                if (std::memcmp(&got[c], &want[c], 4)) {
                    if (bad < 10) printf("rows %d width %d column %d (vector of %d): %g, not %g\n", rows, width, c, n, got[c], want[c]);
                    bad++;
                }
            cudaFree(dm);
            cudaFree(dv);
            cudaFree(out);
            checked++;
        }
    printf("%d shapes, %lld mismatches\n", checked, bad);
    return bad ? 1 : 0;
}

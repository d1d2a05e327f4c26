// Builds a graph on the device, multiplies and frees it, resets the device, and
// does it all again in the new context.  Prints "ok".
#include <cmath>
#include <cstdio>
#include <vector>

#include <cuda_runtime_api.h>

#include "cola_spmm.h"

static bool cu(cudaError_t e, const char *what)
{
    if (e != cudaSuccess)
        std::printf("%s: %s\n", what, cudaGetErrorString(e));
    return e == cudaSuccess;
}
static bool co(cola_status s, const char *what)
{
    if (s != COLA_SUCCESS)
        std::printf("%s: %s\n", what, cola_last_error());
    return s == COLA_SUCCESS;
}

static bool once(int K)
{
    const int n = 1000, m = 40 * n;
    std::vector<int32_t> row(m), col(m);
    std::vector<float> val(m), x((size_t)n * K), y((size_t)n * K);
    std::vector<double> want((size_t)n * K, 0.0);
    for (int i = 0; i < m; i++) {
        row[i] = i % n;
        col[i] = (i * 7 + i / n * 13) % n;
        val[i] = 1.0f + (i % 5);
    }
    for (size_t i = 0; i < x.size(); i++)
        x[i] = (float)(i % 11) - 5.0f;
    for (int i = 0; i < m; i++)
        for (int k = 0; k < K; k++)
            want[(size_t)row[i] * K + k] += (double)val[i] * x[(size_t)col[i] * K + k];
    void *d[5] = {};
    const void *src[4] = {row.data(), col.data(), val.data(), x.data()};
    const size_t bytes[5] = {row.size() * 4, col.size() * 4, val.size() * 4, x.size() * 4, y.size() * 4};
    for (int i = 0; i < 5; i++)
        if (!cu(cudaMalloc(&d[i], bytes[i]), "cudaMalloc"))
            return false;
    for (int i = 0; i < 4; i++)
        if (!cu(cudaMemcpy(d[i], src[i], bytes[i], cudaMemcpyHostToDevice), "copy in"))
            return false;
    cola_graph *g = nullptr;
    if (!co(cola_graph_build_device(n, m, (const int32_t *)d[0], (const int32_t *)d[1], (const float *)d[2], 2, nullptr,
                                    nullptr, &g), "build"))
        return false;
    if (!co(cola_spmm(g, d[3], COLA_FLOAT32, K, d[4], COLA_FLOAT32, K, K, nullptr, nullptr), "spmm"))
        return false;
    if (!cu(cudaMemcpy(y.data(), d[4], bytes[4], cudaMemcpyDeviceToHost), "copy out") || !co(cola_graph_free(g), "free"))
        return false;
    for (void *p : d)
        cudaFree(p);
    for (size_t i = 0; i < y.size(); i++)
        if (std::fabs(y[i] - want[i]) > 1e-3) {
            std::printf("value %zu: %g instead of %g\n", i, y[i], want[i]);
            return false;
        }
    return true;
}

int main()
{
    for (int rep = 0; rep < 3; rep++) {
        if (!once(33) || !once(64))
            return 1;
        if (!cu(cudaDeviceReset(), "reset"))
            return 1;
    }
    std::printf("ok\n");
    return 0;
}

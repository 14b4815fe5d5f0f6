// Folds the partials of n blocks with csrc/common.cuh's reduce_partials, as the
// last block of a reduction does, and prints the entries: sums, then maxima.
#include <cstdio>
#include <cstdlib>
#include <vector>

#include "common.cuh"

using namespace ibm;

template <int NV, int NS>
__global__ void fold(const double *partials, int nblocks, double *out) {
    __shared__ double smem[8 * NV];
    double v[NV];
    reduce_partials<NV, NS>(partials, nblocks, v, smem);
    if (threadIdx.x == 0)
        for (int q = 0; q < NV; q++) out[q] = v[q];
}

template <int NV, int NS>
static int run(int nblocks) {
    // Quarters of small whole numbers: their sums are exact in any order.
    std::vector<double> h((size_t)nblocks * NV), r(NV);
    for (int b = 0; b < nblocks; b++)
        for (int q = 0; q < NV; q++) h[(size_t)b * NV + q] = 0.25 * ((b * 37LL + q * 101LL + 11) % 4093);
    double *p, *o;
    if (cudaMalloc(&p, sizeof(double) * h.size()) != cudaSuccess || cudaMalloc(&o, sizeof(double) * NV) != cudaSuccess)
        return 1;
    cudaMemcpy(p, h.data(), sizeof(double) * h.size(), cudaMemcpyHostToDevice);
    fold<NV, NS><<<1, 256>>>(p, nblocks, o);
    if (cudaMemcpy(r.data(), o, sizeof(double) * NV, cudaMemcpyDeviceToHost) != cudaSuccess) return 1;
    cudaFree(p);
    cudaFree(o);
    for (int q = 0; q < NV; q++) {
        double want = 0.0;
        for (int b = 0; b < nblocks; b++) {
            const double x = h[(size_t)b * NV + q];
            want = q < NS ? want + x : (x > want ? x : want);
        }
        if (r[q] != want) {
            printf("%d blocks, entry %d of %d: %.17g, not %.17g\n", nblocks, q, NV, r[q], want);
            return 1;
        }
    }
    return 0;
}

int main() {
    int bad = 0;
    for (int n : {1, 7, 31, 33, 608, 1024, 1025, 2201, 65537})
        bad += run<1, 1>(n) + run<2, 1>(n) + run<3, 2>(n) + run<3, 3>(n) + run<4, 4>(n) + run<6, 6>(n) + run<7, 6>(n);
    printf(bad ? "%d wrong\n" : "equal\n", bad);
    return bad != 0;
}

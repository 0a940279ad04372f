// Both inverses of the one-CTA IPM on one matrix, for test_inverse_bits_gpu.py:
// the 8 x 8 tile form (form 1, n <= 120) and the sweep by single columns (form 0).
#include "reg_linalg.cuh"
#include "sym_tiles.cuh"

using namespace bqb;

__global__ void __launch_bounds__(ST_THREADS, 1) inverse_kernel(const double* A, int n, int form, double* out, int* ok)
{
    const int T = st_tiles(n), lane = threadIdx.x & 31;
    bool pd;
    if (form) {
        pd = st_inverse(
            T, st_smem, reinterpret_cast<int*>(st_smem + st_buffers(T)),
            [&](int I, int J, int r, int c) {
                const int i = 8 * I + r, j = 8 * J + 2 * c;
                double2 v = make_double2(i == j ? 1.0 : 0.0, i == j + 1 ? 1.0 : 0.0);
                if (i < n && j < n) v.x = A[i + j * n];
                if (i < n && j + 1 < n) v.y = A[i + (j + 1) * n];
                return v;
            },
            [&](int I, int J, double a, double b) {
                const int i = 8 * I + (lane >> 2), j = 8 * J + 2 * (lane & 3);
                if (i < n && j < n) out[i + j * n] = a;
                if (i < n && j + 1 < n) out[i + (j + 1) * n] = b;
            });
    } else {
        RegMat R;
        rm_fill(R, n, [&](int r, int c) { return A[r + c * n]; });
        pd = rm_spd_inverse(R, n, st_smem);
        if (pd) rm_store(R, out, n);
    }
    if (threadIdx.x == 0) *ok = pd ? 1 : 0;
}

// 1: positive definite, 0: not, -1: a CUDA error.
extern "C" __attribute__((visibility("default"))) int inverse(const double* A, int n, int form, double* out)
{
    const size_t bytes = (size_t)n * n * sizeof(double);
    const int smem = (st_buffers(st_tiles(n)) + 2) * (int)sizeof(double);
    double *dA = nullptr, *dout = nullptr;
    int *dok = nullptr, ok = -1;
    bool good = cudaMalloc(&dA, bytes) == cudaSuccess && cudaMalloc(&dout, bytes) == cudaSuccess &&
                cudaMalloc(&dok, sizeof(int)) == cudaSuccess &&
                cudaFuncSetAttribute(inverse_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) == cudaSuccess &&
                cudaMemcpy(dA, A, bytes, cudaMemcpyHostToDevice) == cudaSuccess &&
                cudaMemset(dout, 0, bytes) == cudaSuccess;
    if (good) {
        inverse_kernel<<<1, ST_THREADS, smem>>>(dA, n, form, dout, dok);
        good = cudaGetLastError() == cudaSuccess &&
               cudaMemcpy(out, dout, bytes, cudaMemcpyDeviceToHost) == cudaSuccess &&
               cudaMemcpy(&ok, dok, sizeof(int), cudaMemcpyDeviceToHost) == cudaSuccess;
    }
    cudaFree(dA);
    cudaFree(dout);
    cudaFree(dok);
    return good ? ok : -1;
}

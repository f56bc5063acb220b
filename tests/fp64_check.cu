// The functions of ht_fp64.cuh over arrays (compiled and called by test_gpu_fp64.py).
#include "ht_fp64.cuh"

namespace {

__global__ void op_kernel(int op, long long n, const double* a, const double* b, double* out) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double x = a[i], y = b[i];
    out[i] = op == 0 ? recip(y) : op == 1 ? root(x) : op == 2 ? quot(x, y, recip(y))
           : op == 3 ? ratio(x, y) : quot_any(x, y, 1.0 / y);
}

// sets (x, y, z) and (x2, y2, z2), the second one read from the first's arrays reversed
__global__ void rd_kernel(long long n, const double* x, const double* y, const double* z,
                          double* out) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x, j = n - 1 - i;
    if (i >= n) return;
    elliptic_rd2(x[i], y[i], z[i], x[j], y[j], z[j], out + i, out + n + j);
}

}  // namespace

extern "C" int fp64_op(int op, long long n, const double* a, const double* b, double* out) {
    op_kernel<<<(unsigned)((n + 255) / 256), 256>>>(op, n, a, b, out);
    return (int)cudaGetLastError();
}

extern "C" int fp64_rd(long long n, const double* x, const double* y, const double* z,
                       double* out) {
    rd_kernel<<<(unsigned)((n + 255) / 256), 256>>>(n, x, y, z, out);
    return (int)cudaGetLastError();
}

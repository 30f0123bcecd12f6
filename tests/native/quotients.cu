// quot() of rb_quot.cuh over arrays, on the host and on the device, beside the plain division there.
#include "rb_quot.cuh"

template <typename R>
__global__ void quotients(const R *q, const R *s, R *got, R *want, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    got[i] = rb::quot(q[i], s[i]);
    want[i] = q[i] / s[i];
}

template <typename R>
static int run(const R *q, const R *s, R *got, R *want, int n, int device) {
    if (!device) {
        for (int i = 0; i < n; i++) {
            got[i] = rb::quot(q[i], s[i]);
            want[i] = q[i] / s[i];
        }
        return 0;
    }
    R *d = nullptr;
    const size_t b = sizeof(R) * (size_t)n;
    cudaError_t e = cudaMalloc(&d, 4 * b);
    if (e == cudaSuccess) e = cudaMemcpy(d, q, b, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(d + n, s, b, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) {
        quotients<R><<<(n + 255) / 256, 256>>>(d, d + n, d + 2 * (size_t)n, d + 3 * (size_t)n, n);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpy(got, d + 2 * (size_t)n, b, cudaMemcpyDeviceToHost);
    if (e == cudaSuccess) e = cudaMemcpy(want, d + 3 * (size_t)n, b, cudaMemcpyDeviceToHost);
    cudaFree(d);
    return (int)e;
}

extern "C" int quotients_f64(const double *q, const double *s, double *got, double *want, int n, int device) {
    return run(q, s, got, want, n, device);
}
extern "C" int quotients_f32(const float *q, const float *s, float *got, float *want, int n, int device) {
    return run(q, s, got, want, n, device);
}

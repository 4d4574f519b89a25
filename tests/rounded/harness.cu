/*
 * harness.cu -- TEST INFRASTRUCTURE ONLY.
 *
 * The device functions of fn_rounded.cuh, one element per thread, for
 * tests/test_gpu_rounded.py, which compares them with the host's IEEE
 * operations.
 */
#include <cuda_runtime.h>

#include "../../fibrenet_b200/csrc/fn_rounded.cuh"

using namespace fn;

enum { OP_ROOT = 0, OP_INVERSE_ROOT = 1, OP_PRODUCT_INVERSE = 2, OP_SQUARE_INVERSE = 3, OP_QUOTIENT = 4, OP_QUOTIENT_ANY = 5,
       OP_SQUARE_QUOTIENT = 6 };

static __global__ void k_rounded(int op, const double* a, const double* b, double* out, long long n) {
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i >= n) return;
    double l, il, m, im, r = 0.0;
    switch (op) {
    case OP_ROOT: /* sqrt(a) */
        root_and_inverse(a[i], l, il);
        r = l;
        break;
    case OP_INVERSE_ROOT: /* 1 / sqrt(a) as two operations, 0 for a = 0 */
        root_and_inverse(a[i], l, il);
        r = il;
        break;
    case OP_PRODUCT_INVERSE: /* 1 / (sqrt(a) sqrt(b)), as the angle's arms have it */
        root_and_inverse(a[i], l, il);
        root_and_inverse(b[i], m, im);
        r = fn_fast_range(l * m) ? recip_from(l * m, il * im) : 1.0 / (l * m);
        break;
    case OP_SQUARE_INVERSE: /* 1 / a from the seed of its root, as a contact's squared distance has it */
        m = rsqrt_seeded(a[i]);
        r = recip_from(a[i], m * m);
        break;
    case OP_QUOTIENT: /* a / b */
        r = quotient(a[i], b[i], 1.0 / b[i]);
        break;
    case OP_QUOTIENT_ANY: /* a / b for any a, b a finite root above 0 */
        r = quotient_any(a[i], b[i], 1.0 / b[i]);
        break;
    case OP_SQUARE_QUOTIENT: /* a / b from the seed of b's root, as a contact's quotients by its squared distance */
        m = rsqrt_seeded(b[i]);
        r = quotient(a[i], b[i], recip_near(b[i], m * m));
        break;
    }
    out[i] = r;
}

extern "C" __attribute__((visibility("default"))) int fr_run(int op, const double* a, const double* b, double* out,
                                                             long long n) {
    double *d[3] = {};
    const size_t bytes = sizeof(double) * (size_t)n;
    cudaError_t e = cudaSuccess;
    for (int k = 0; k < 3 && e == cudaSuccess; ++k) e = cudaMalloc(&d[k], bytes);
    if (e == cudaSuccess) e = cudaMemcpy(d[0], a, bytes, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(d[1], b, bytes, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) {
        k_rounded<<<(unsigned)((n + 255) / 256), 256>>>(op, d[0], d[1], d[2], n);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpy(out, d[2], bytes, cudaMemcpyDeviceToHost);
    for (double* p : d) cudaFree(p);
    return (int)e;
}

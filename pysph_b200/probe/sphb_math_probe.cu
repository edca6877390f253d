// sphb_math_probe.cu -- the pair loops' reciprocals, distances and quotients
// on arrays, for the test that compares them with 80-bit arithmetic.  Part
// of libsphb_probe.so, not of the particle path.

#include <cuda_runtime.h>

#include "sphb_kernels.cuh"

namespace sphb_probe {

// which 0: out = 1 / a.  1: out = sqrt(a), out2 = 1 / sqrt(a).  2: out = a / b
// by the reciprocal of b.
__global__ void k_math_probe(int which, int n, const double *a, const double *b, double *out,
                             double *out2)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    if (which == 0) {
        out[i] = sphb::rcp_pair(a[i]);
    } else if (which == 1) {
        double ir;
        out[i] = sphb::dist_pair(a[i], ir);
        out2[i] = ir;
    } else {
        out[i] = sphb::over_h(a[i], b[i], sphb::rcp_pair(b[i]));
    }
}

}  // namespace sphb_probe

// Device arrays of n doubles (b: which == 2; out2: which == 1).  Returns 0, -1
// for a bad argument, -3 when the launch failed.
extern "C" __attribute__((visibility("default"))) int sphb_math_probe(int which, int n,
                                                                      const double *a,
                                                                      const double *b, double *out,
                                                                      double *out2, void *stream)
{
    if (which < 0 || which > 2 || n < 1 || !a || !out || (which == 1 && !out2) ||
        (which == 2 && !b))
        return -1;
    sphb_probe::k_math_probe<<<(n + 255) / 256, 256, 0, (cudaStream_t)stream>>>(which, n, a, b,
                                                                              out, out2);
    return cudaGetLastError() == cudaSuccess ? 0 : -3;
}

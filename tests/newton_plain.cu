// Newton's method on a cubic as the three modules' computeFractal has it, one thread a pixel, its first sample: the
// step's expressions and the loops around it and nothing else, built with nvcc's default contraction
// (tests/test_gpu_newton_contracted.py compares the drop-in modules of the default build with it).
#include <thrust/complex.h>

template <class R> __device__ int root_of(thrust::complex<R> x, const double *roots)
{
    const R tolerance = 0.0001;
    for (int k = 0; k < 3; k++) {
        thrust::complex<R> d = x - thrust::complex<R>(roots[2 * k], roots[2 * k + 1]);
        if (abs(d.real()) < tolerance && abs(d.imag()) < tolerance) return k + 1;
    }
    return 0;
}

template <class R> __device__ thrust::complex<R> wired_step(thrust::complex<R> x)
{
    thrust::complex<R> x2 = x * x;
    thrust::complex<R> x3 = x2 * x;
    thrust::complex<R> f = x3 - 1;
    thrust::complex<R> df = 3 * x2;
    return x - (f / df);
}

template <class R> __device__ thrust::complex<R> generic_step(thrust::complex<R> x, const double *c)
{
    thrust::complex<R> x2 = x * x;
    thrust::complex<R> x3 = x2 * x;
    thrust::complex<R> f = c[0] + c[1] * x + c[2] * x2 + c[3] * x3;
    thrust::complex<R> df = c[1] + c[2] * 2 * x + c[3] * 3 * x2;
    return x - (f / df);
}

// kind: 2 wired, 3 generic (root of the state at steps 10, 10 + limit / 10, ... and at the limit), 4 iterations
template <class R, int KIND> __device__ int plain(thrust::complex<R> x, unsigned limit, const double *c, const double *roots)
{
    unsigned i = 0;
    if (KIND == 4) {
        while (i < limit) {
            x = generic_step<R>(x, c);
            ++i;
            if (root_of<R>(x, roots)) return i;
        }
        return i;
    }
    unsigned check = 10;
    while (i < limit) {
        x = KIND == 2 ? wired_step<R>(x) : generic_step<R>(x, c);
        ++i;
        if (i == check) {
            int r = root_of<R>(x, roots);
            if (r) return r;
            check += limit / 10;
        }
    }
    return root_of<R>(x, roots);
}

__device__ __forceinline__ float fused(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double fused(double a, double b, double c) { return __fma_rn(a, b, c); }

// out[y * w + x] for the rectangle (lbx, lby, rtx, rty) = r[0..3]
template <class R, int KIND>
__device__ void frame(float *out, int w, int h, const double *r, unsigned limit, const double *c, const double *roots)
{
    const int px = blockIdx.x * blockDim.x + threadIdx.x, py = blockIdx.y * blockDim.y + threadIdx.y;
    if (px >= w || py >= h) return;
    const R psx = ((R)r[2] - (R)r[0]) / (R)w, psy = ((R)r[3] - (R)r[1]) / (R)h;
    const R cx = fused((R)px, psx, (R)r[0]), cy = fused(-(R)py, psy, (R)r[3]);
    out[py * w + px] = (float)plain<R, KIND>(thrust::complex<R>(cx, cy), limit, c, roots);
}

#define ENTRY(name, R, KIND)                                                                                        \
    extern "C" __global__ void name(float *out, int w, int h, const double *r, unsigned limit, const double *c,     \
                                    const double *roots)                                                            \
    {                                                                                                               \
        frame<R, KIND>(out, w, h, r, limit, c, roots);                                                              \
    }
ENTRY(wired_f32, float, 2)
ENTRY(generic_f32, float, 3)
ENTRY(iterations_f32, float, 4)
ENTRY(wired_f64, double, 2)
ENTRY(generic_f64, double, 3)
ENTRY(iterations_f64, double, 4)

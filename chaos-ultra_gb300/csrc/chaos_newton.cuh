// chaos_newton.cuh -- the Newton-method fractals (newton wired / generic /
// colored by iterations): Newton's method on a cubic, coloured by the root a
// start point converges to, or by the iteration it converged at.
//
// Reference: src/main/cuda/fractals/newton_wired.cu:7-64,
// newton_generic.cu:11-72, newton_iterations.cu:12-67.  The complex arithmetic
// is thrust::complex, as in the reference, and the expressions keep the
// reference's operand types and order: with Real = float, a term like
// coefficients[1] * x is a double times a complex<float> and is evaluated as
// complex<double> before the assignment rounds it back, so the same
// expression forms are what reproduce the reference's results.  Built with
// --fmad=false it matches the reference built the same way; built with nvcc's
// default contraction (the default-build drop-in modules) nvcc fuses these
// expressions as it fuses the reference's own.
#pragma once

#include <thrust/complex.h>

#include "chaos_device.cuh"

namespace chaos {

// newton_wired.cu:18-41 (the roots of z^3 - 1 as literals)
__device__ __constant__ static const double kWiredRoots[6] = {1, 0, -0.5, 0.86602540378, -0.5, -0.86602540378};

template <class R> __device__ __forceinline__ thrust::complex<R> newton_step_wired(thrust::complex<R> x)
{
    thrust::complex<R> x_pow_2 = x * x;
    thrust::complex<R> x_pow_3 = x_pow_2 * x;
    thrust::complex<R> f_eval_x = x_pow_3 - 1;
    thrust::complex<R> f_derivative_eval_x = 3 * x_pow_2;
    return x - (f_eval_x / f_derivative_eval_x);
}

// newton_generic.cu:11-25: f = c0 + c1 x + c2 x^2 + c3 x^3
template <class R>
__device__ __forceinline__ thrust::complex<R> newton_step_generic(thrust::complex<R> x, const double *coefficients)
{
    thrust::complex<R> x_pow_2 = x * x;
    thrust::complex<R> x_pow_3 = x_pow_2 * x;
    thrust::complex<R> f_eval_x =
        coefficients[0] + coefficients[1] * x + coefficients[2] * x_pow_2 + coefficients[3] * x_pow_3;
    thrust::complex<R> f_derivative_eval_x = coefficients[1] + coefficients[2] * 2 * x + coefficients[3] * 3 * x_pow_2;
    return x - (f_eval_x / f_derivative_eval_x);
}

// x^3 + c0 (c0 != 0, c1 = c2 = 0, c3 = 1; the default polynomial): the generic
// step without its zero terms, which leave every sum as it is but for the
// sign of a zero, and without binary64 where Real = float: there the generic
// expression evaluates in complex<double> (28 of its operations run on the
// binary64 pipe, of which a warp's operation takes 76 cycles).
//   f:  c0 + x3 in binary64, rounded to binary32, is the binary32 sum (53 bits
//       are more than 2 x 24 + 2, so the second rounding changes nothing)
//   f': 3 x2 is exact in binary64, so it is rounded once, as here
// The sign of a zero changes no result: no quotient has a signed zero below
// it, and the root test takes absolute values.  A component that overflows to
// infinity makes the state NaN on both ways (infinite x2 gives f' with an
// infinite |f'|, so the quotient is infinity times zero).
// 960x540 pixels, 2 samples each, maxIter 200, with newton_compute's early
// answers: 824 -> 86 us a pass.
__device__ __forceinline__ bool newton_binomial(const double *c, bool single)
{
    return c[0] != 0.0 && c[1] == 0.0 && c[2] == 0.0 && c[3] == 1.0 && (!single || (double)(float)c[0] == c[0]);
}
__device__ __forceinline__ float newton_sum(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ double newton_sum(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ float newton_triple(float a) { return __fmul_rn(3.f, a); }
__device__ __forceinline__ double newton_triple(double a) { return __dmul_rn(3.0, a); }

template <class R> __device__ __forceinline__ thrust::complex<R> newton_step_binomial(thrust::complex<R> x, R c0)
{
    thrust::complex<R> x_pow_2 = x * x;
    thrust::complex<R> x_pow_3 = x_pow_2 * x;
    thrust::complex<R> f_eval_x(newton_sum(c0, x_pow_3.real()), x_pow_3.imag());
    thrust::complex<R> f_derivative_eval_x(newton_triple(x_pow_2.real()), newton_triple(x_pow_2.imag()));
    return x - (f_eval_x / f_derivative_eval_x);
}

// convergenceRoot: 1-based index of the root within 1e-4 on both axes, else 0
template <class R> __device__ __forceinline__ uint32_t newton_root(thrust::complex<R> x, const double *roots)
{
    const R tolerance = 0.0001;
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const thrust::complex<R> root(roots[2 * k], roots[2 * k + 1]);
        thrust::complex<R> difference = x - root;
        if (abs(difference.real()) < tolerance && abs(difference.imag()) < tolerance) return (uint32_t)(k + 1);
    }
    return 0;
}

// Whether four steps from step i end before step `end` (i <= end; i + 4 may wrap)
__host__ __device__ constexpr bool newton_group(uint32_t i, uint32_t end) { return end - i > 4u; }

// The modules' loops around a step.  A state that a step leaves as it was, or
// that has become NaN (which stays so), is the state at every later test: the
// answer is the test's on it, however many steps remain (looked at every fourth
// step).  Most start points settle bit for bit a few steps after they come near
// a root, well before the test of step 30 where the one of step 10 came too early.
// One copy of the step: a complex division is hundreds of instructions, and where
// a frame takes few samples (a zoom step) a warp meets them cold.  Wired,
// 7088x4663 zooming out, maxIter 300, 2 samples: 531 us with groups of four copies,
// 417 (491 with every step tested); 1920x1080 of the default polynomial, maxIter
// 200: 128 / 123.
template <class R, int F, class Step>
__device__ __forceinline__ uint32_t newton_run(uint32_t max_iterations, thrust::complex<R> x, const double *roots, Step step)
{
    auto settled = [](thrust::complex<R> z, thrust::complex<R> before) {
        return (z.real() == before.real() && z.imag() == before.imag()) || z.real() != z.real() || z.imag() != z.imag();
    };
    uint32_t i = 0;
    if (F == FRACTAL_NEWTON_ITERATIONS) {  // newton_iterations.cu:54-67
        while (i < max_iterations) {
            const thrust::complex<R> before = x;
            x = step(x);
            ++i;
            if (newton_root<R>(x, roots) != 0) return i;
            if ((i & 3u) == 0u && settled(x, before)) return max_iterations;
        }
        return i;
    }
    // newton_wired.cu:45-64, newton_generic.cu:53-72: test every maxIterations/10 steps after the 10th
    uint32_t check = 10;
    while (i < max_iterations) {
        const uint32_t end = min(check, max_iterations);
        while (i < end) {
            const uint32_t n = newton_group(i, end) ? 4u : end - i;
            thrust::complex<R> before = x;
#pragma unroll 1
            for (uint32_t k = 0; k < n; k++) {
                before = x;
                x = step(x);
            }
            i += n;
            if (n == 4u && settled(x, before)) return newton_root<R>(x, roots);
        }
        if (i == check) {
            uint32_t root = newton_root<R>(x, roots);
            if (root != 0) return root;
            const uint32_t gap = max_iterations / 10;
            check = check > 0xffffffffu - gap ? 0xffffffffu : check + gap;
        }
    }
    return newton_root<R>(x, roots);
}

// computeFractal of the three modules, as an unsigned value (the float the
// reference returns is an integer): the root index (wired, generic) or the
// iteration count (iterations).
//
// AS_WRITTEN: the reference's loops around its step, for code built with nvcc's
// contraction.  There the values are those of the products that nvcc fuses, and
// it fuses within a basic block: a choice between two forms of the step, or
// copies of it, moved some of them (640x360 pixels of the module's own
// polynomial in binary32 came out otherwise).
//
// Otherwise newton_run, with the step that the polynomial needs.
// (declared __forceinline__ in chaos_device.cuh; the attribute is not repeated here)
template <class R, int F, bool AS_WRITTEN>
__device__ uint32_t newton_compute(uint32_t max_iterations, R zx, R zy, const NewtonParams &p)
{
    thrust::complex<R> x(zx, zy);
    const double *roots = F == FRACTAL_NEWTON_WIRED ? kWiredRoots : p.roots;
    if constexpr (AS_WRITTEN) {
        uint32_t i = 0;
        if (F == FRACTAL_NEWTON_ITERATIONS) {  // newton_iterations.cu:54-67
            while (i < max_iterations) {
                x = newton_step_generic<R>(x, p.coefficients);
                ++i;
                if (newton_root<R>(x, roots) != 0) return i;
            }
            return i;
        }
        // newton_wired.cu:45-64, newton_generic.cu:53-72
        uint32_t check = 10;
        while (i < max_iterations) {
            x = F == FRACTAL_NEWTON_WIRED ? newton_step_wired<R>(x) : newton_step_generic<R>(x, p.coefficients);
            ++i;
            if (i == check) {
                uint32_t root = newton_root<R>(x, roots);
                if (root != 0) return root;
                check += max_iterations / 10;
            }
        }
        return newton_root<R>(x, roots);
    }
    if (F == FRACTAL_NEWTON_WIRED)
        return newton_run<R, F>(max_iterations, x, roots, [](thrust::complex<R> z) { return newton_step_wired<R>(z); });
    if (newton_binomial(p.coefficients, sizeof(R) == 4)) {
        const R c0 = (R)p.coefficients[0];
        return newton_run<R, F>(max_iterations, x, roots,
                                [=](thrust::complex<R> z) { return newton_step_binomial<R>(z, c0); });
    }
    return newton_run<R, F>(max_iterations, x, roots,
                            [&](thrust::complex<R> z) { return newton_step_generic<R>(z, p.coefficients); });
}

}  // namespace chaos

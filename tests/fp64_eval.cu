// Device evaluation of gbx::div and gbx::sqrt, host evaluation of their
// significand routines with a perturbed reciprocal approximation, and host
// evaluation of the fixed-point elementary functions.
#include "../celeritas_gb300/csrc/gbx/Fp64.hh"
#include "../celeritas_gb300/csrc/gbx/LibmInt.hh"

namespace
{
__global__ void evaluate(int op, double const* a, double const* b, double* y, int n)
{
    int const i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n)
        y[i] = op == 0 ? gbx::div(a[i], b[i]) : gbx::sqrt(a[i]);
}
}  // namespace

//! y = a / b (op 0) or sqrt(a) (op 1) on the device; returns the CUDA status
extern "C" int fp64_device(int op, double const* a, double const* b, double* y, int n)
{
    double* d = nullptr;
    std::size_t const bytes = sizeof(double) * n;
    if (int rc = cudaMalloc(&d, 3 * bytes))
        return rc;
    cudaMemcpy(d, a, bytes, cudaMemcpyHostToDevice);
    cudaMemcpy(d + n, b, bytes, cudaMemcpyHostToDevice);
    evaluate<<<(n + 255) / 256, 256>>>(op, d, d + n, d + 2 * n, n);
    int const rc = cudaMemcpy(y, d + 2 * n, bytes, cudaMemcpyDeviceToHost);
    cudaFree(d);
    return rc;
}

//! Significands [2^52, 2^53) of a / b (op 0) or of sqrt(a 2^-52) (op 1, a up
//! to 2^54), with the FP32 approximation moved by 'ulps'
extern "C" void fp64_host(int op,
                          std::uint64_t const* a,
                          std::uint64_t const* b,
                          std::uint64_t* y,
                          int n,
                          int ulps)
{
    using namespace gbx::fp64;
    for (int i = 0; i < n; ++i)
    {
        if (op == 0)
        {
            std::uint32_t const f
                = 0x3f800000u | (static_cast<std::uint32_t>(b[i] >> 29) & 0x7fffffu);
            y[i] = div_significand(a[i], b[i], approx_rcp(f) + ulps);
        }
        else
        {
            unsigned int const odd = (a[i] >> 53) & 1u;
            std::uint32_t const f = ((127u + odd) << 23)
                                    | (static_cast<std::uint32_t>(a[i] >> (29 + odd)) & 0x7fffffu);
            y[i] = sqrt_significand(a[i], approx_rsqrt(f) + ulps);
        }
    }
}

//! Bits of exp, log, sin, cos, expm1 or log1p (op 0-5) of x in fixed point;
//! decided[i] is 0 where the function leaves the argument to double-doubles
extern "C" void libm_fixed(int op,
                           std::uint64_t const* x,
                           std::uint64_t* y,
                           unsigned char* decided,
                           int n)
{
    namespace fixed = gbx::libm::fixed;
    for (int i = 0; i < n; ++i)
    {
        decided[i] = op == 0   ? fixed::exp(x[i], y + i)
                     : op == 1 ? fixed::log(x[i], y + i)
                     : op == 2 ? fixed::sin_cos(x[i], 0, y + i)
                     : op == 3 ? fixed::sin_cos(x[i], 1, y + i)
                     : op == 4 ? fixed::expm1(x[i], y + i)
                               : fixed::log1p(x[i], y + i);
    }
}

// Device evaluation of the mixed-precision field driver's shortcuts beside the
// operations whose results they must give.
#include "../celeritas_gb300/csrc/gbx/Field.hh"

namespace
{
using namespace gbx::mixed;

__device__ std::uint32_t bits(float x)
{
    return __float_as_uint(x);
}

//! inv_sqrt() of every fraction of the binades of exponents e and e + 1
__global__ void check_inv_sqrt(int e, unsigned int* bad)
{
    std::uint32_t const t = blockIdx.x * blockDim.x + threadIdx.x;
    for (int k = 0; k < 2; ++k)
    {
        float const x = __uint_as_float((static_cast<std::uint32_t>(127 + e + k) << 23) | t);
        if (!inv_sqrt_covers(x) || bits(inv_sqrt(x)) != bits(1.0f / sqrtf(x)))
            atomicAdd(bad, 1u);
    }
}

//! Acceptance and rounded error norm from the error estimates in 'in' (position
//! error, momentum error, momentum): shortcut and FP64 values
__global__ void evaluate_norm(gbx::FieldOptions opt, float const* in, float* out, int n)
{
    int const i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n)
        return;
    float const* v = in + 9 * i;
    StageResult r{};
    r.pos_error = {v[0], v[1], v[2]};
    r.mom_error = {v[3], v[4], v[5]};
    StartMomentum start{};
    start.value = {v[6], v[7], v[8]};
    start.square = square_pair(start.value);
    start.rounded = true;
    ErrorNorm const err = error_norm(r, start.square, opt);
    double const exact = error_norm_fp64(r, start, opt.epsilon_rel_max);
    out[4 * i] = above_one(err, r, start, opt);
    out[4 * i + 1] = exact > 1;
    out[4 * i + 2] = clamped_norm(err, r, start, opt);
    out[4 * i + 3] = float(gbx::min_of(gbx::max_of(exact, 1e-30), 1e30));
}

__global__ void convert(double const* d, float const* f, float* to, double* from, int n)
{
    int const i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n)
    {
        to[i] = gbx::fp64::narrow(d[i]);
        from[i] = gbx::fp64::widen(f[i]);
    }
}

template<class T>
T* to_device(T const* src, std::size_t n)
{
    T* p = nullptr;
    cudaMalloc(&p, n * sizeof(T));
    if (src)
        cudaMemcpy(p, src, n * sizeof(T), cudaMemcpyHostToDevice);
    return p;
}
}  // namespace

//! Fractions of two binades for which inv_sqrt() differs from 1 / sqrtf()
extern "C" int inv_sqrt_mismatches(int exponent, unsigned int* bad)
{
    unsigned int const zero = 0;
    unsigned int* d = to_device(&zero, 1);
    check_inv_sqrt<<<1 << 15, 256>>>(exponent, d);
    int const rc = cudaMemcpy(bad, d, sizeof(zero), cudaMemcpyDeviceToHost);
    cudaFree(d);
    return rc;
}

extern "C" int error_norms(double epsilon, float const* in, float* out, int n)
{
    gbx::FieldOptions opt;
    opt.epsilon_rel_max = epsilon;
    opt.derive();
    float* di = to_device(in, 9 * std::size_t(n));
    float* d_out = to_device<float>(nullptr, 4 * std::size_t(n));
    evaluate_norm<<<(n + 127) / 128, 128>>>(opt, di, d_out, n);
    int const rc = cudaMemcpy(out, d_out, 16 * std::size_t(n), cudaMemcpyDeviceToHost);
    cudaFree(di);
    cudaFree(d_out);
    return rc;
}

extern "C" int conversions(double const* d, float const* f, float* to, double* from, int n)
{
    double* dd = to_device(d, n);
    float* df = to_device(f, n);
    float* dt = to_device<float>(nullptr, n);
    double* dw = to_device<double>(nullptr, n);
    convert<<<(n + 255) / 256, 256>>>(dd, df, dt, dw, n);
    cudaMemcpy(to, dt, 4 * std::size_t(n), cudaMemcpyDeviceToHost);
    int const rc = cudaMemcpy(from, dw, 8 * std::size_t(n), cudaMemcpyDeviceToHost);
    for (void* p : {(void*)dd, (void*)df, (void*)dt, (void*)dw})
        cudaFree(p);
    return rc;
}

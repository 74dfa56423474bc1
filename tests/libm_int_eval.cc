// Host evaluation of the fixed-point elementary functions: the 128-bit result before it is
// rounded, and the error that its rounding allows.
#define GBX_LIBM_RECORD
#include "../celeritas_gb300/csrc/gbx/LibmInt.hh"

//! exp, log, sin, cos, expm1 or log1p (op 0-5) of x: |result| is (hi 2^64 + lo) 2^(e - 127)
//! with an error below 2^(e - bits); bits is 0 where the argument is not covered
extern "C" void libm_unrounded(int op,
                               std::uint64_t const* x,
                               std::uint64_t* hi,
                               std::uint64_t* lo,
                               int* e,
                               int* bits,
                               int n)
{
    namespace fixed = gbx::libm::fixed;
    for (int i = 0; i < n; ++i)
    {
        std::uint64_t y;
        fixed::last_rounded = {};
        op == 0   ? fixed::exp(x[i], &y)
        : op == 1 ? fixed::log(x[i], &y)
        : op == 2 ? fixed::sin_cos(x[i], 0, &y)
        : op == 3 ? fixed::sin_cos(x[i], 1, &y)
        : op == 4 ? fixed::expm1(x[i], &y)
                  : fixed::log1p(x[i], &y);
        hi[i] = static_cast<std::uint64_t>(fixed::last_rounded.v >> 64);
        lo[i] = static_cast<std::uint64_t>(fixed::last_rounded.v);
        e[i] = fixed::last_rounded.e;
        bits[i] = fixed::last_rounded.bits;
    }
}

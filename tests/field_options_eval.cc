// Host evaluation of the mixed-precision field driver's error norm for a tolerance.
#include "../celeritas_gb300/csrc/gbx/FieldMixed.hh"

//! Acceptance and rounded error norm from the error estimates in 'in' (position error,
//! momentum error, momentum): shortcut and FP64 values
extern "C" void error_norms(double epsilon, float const* in, float* out, int n)
{
    using namespace gbx::mixed;
    gbx::FieldOptions opt;
    opt.epsilon_rel_max = epsilon;
    opt.derive();
    for (int i = 0; i < n; ++i)
    {
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
}

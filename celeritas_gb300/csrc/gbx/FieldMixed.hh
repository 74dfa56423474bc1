// Field integration of the mixed-precision build: Dormand-Prince steps with
// FP32 stages under the reference's field driver (FieldDriver.hh:182-429).
//
// In a transport most steps of the loop wait for a few tracks that curl up in
// the field, each of which runs hundreds of Runge-Kutta steps one after the other,
// so the time that counts is one thread's. On GB300 an FP64 instruction (a
// conversion and a comparison too) takes its warp 45-64 cycles and overlaps with
// no other; an FP32 one 4-6. The driver therefore keeps the stages, the error
// estimate and the momentum in FP32 from one Runge-Kutta step to the next, and
// touches FP64 where FP64 is kept: the position, once per accepted step, and the
// step lengths.
// - The error norm (FP64 by definition: the larger of the squared position and
//   relative momentum errors over the squared tolerance) decides an acceptance
//   (is it above 1?) and gives an FP32 step-size factor. Both are taken from an
//   evaluation in pairs of FP32 numbers, accurate to 2^-40, wherever that decides
//   them, and from FP64 in the few cases left, so that both are what FP64 gives.
// - A chord far too long halves the step without the division and square root
//   that would give a factor below one half.
// - 1 / sqrt(|p|^2) of the stages takes 55 cycles instead of 109 (inv_sqrt).
// - FP32 arithmetic is spelled out (fma or not), so that no change around it
//   changes its contraction; where the compiler had contracted the copies of the
//   step in two ways both are kept (round_x).
// A step's stages, error estimate and chord take one track 780 cycles, most of them the
// seven stages' dependent chain. A 13-event c3 batch went from 500 to 386
// ms with this, four events in the field map from 555 to 403 ms, every track's
// state the same after every step.
#pragma once

#include "FieldState.hh"

namespace gbx
{
namespace mixed
{
using F3 = Vec3<float>;

// FP32 operations rounded one by one: the compiler contracts none of them
GBX_FORCEINLINE float fma(float a, float b, float c)
{
    return ::fmaf(a, b, c);
}
GBX_FORCEINLINE float mul(float a, float b)
{
#if defined(__CUDA_ARCH__)
    return __fmul_rn(a, b);
#else
    return a * b;
#endif
}
GBX_FORCEINLINE float add(float a, float b)
{
#if defined(__CUDA_ARCH__)
    return __fadd_rn(a, b);
#else
    return a + b;
#endif
}
GBX_FORCEINLINE float sub(float a, float b)
{
    return add(a, -b);
}

//! x^2 + y^2 + z^2, the square that is rounded by itself y's or ('round_x') x's
GBX_FORCEINLINE float square(F3 const& v, bool round_x = false)
{
    float const a = round_x ? v.y : v.x;
    float const b = round_x ? v.x : v.y;
    return fma(v.z, v.z, fma(a, a, mul(b, b)));
}

//! Whether inv_sqrt() covers x: neither x r nor the residuals below leave the
//! range of normal numbers
GBX_FORCEINLINE bool inv_sqrt_covers(float x)
{
    return x >= 0x1p-75f && x < 0x1p120f;
}

//! 1 / sqrt(x) as two operations rounded to nearest, where inv_sqrt_covers(x).
//! From the hardware's reciprocal square root r: the root by one Newton step of
//! x r, its reciprocal by two of r. For every float of two binades (hence of
//! even and of odd exponents) this is the result of the two IEEE operations,
//! without their branches on special values.
GBX_FORCEINLINE float inv_sqrt(float x)
{
#if defined(__CUDA_ARCH__)
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    float s = mul(x, r);
    s = fma(fma(-s, s, x), mul(0.5f, r), s);
    r = fma(r, fma(-s, r, 1.0f), r);
    r = fma(r, fma(-s, r, 1.0f), r);
    // Just below a power of two the second step stays an ulp short
    std::uint32_t const u = __float_as_uint(r);
    return __uint_as_float(u + ((__float_as_uint(s) & 0x7fffffu) == 0x7fffffu ? 1 : 0));
#else
    return 1.0f / std::sqrt(x);
#endif
}

//---------------------------------------------------------------------------//
//! Sum of two FP32 numbers, |lo| about half an ulp of hi or less
struct Pair
{
    float hi;
    float lo;
};

//! Exact sum (Knuth's)
GBX_FORCEINLINE Pair two_sum(float a, float b)
{
    float const s = add(a, b);
    float const t = sub(s, a);
    return {s, add(sub(a, sub(s, t)), sub(b, t))};
}
//! Exact sum for |a| >= |b| (Dekker's)
GBX_FORCEINLINE Pair fast_two_sum(float a, float b)
{
    float const s = add(a, b);
    return {s, sub(b, sub(s, a))};
}
//! x^2 + y^2 + z^2 to about 2^-45
GBX_FORCEINLINE Pair square_pair(F3 const& v)
{
    float const x = mul(v.x, v.x);
    float const y = mul(v.y, v.y);
    float const z = mul(v.z, v.z);
    float low = add(add(fma(v.x, v.x, -x), fma(v.y, v.y, -y)), fma(v.z, v.z, -z));
    Pair const a = two_sum(x, y);
    Pair const b = two_sum(a.hi, z);
    return fast_two_sum(b.hi, add(add(a.lo, b.lo), low));
}
GBX_FORCEINLINE Pair mul_pair(Pair a, Pair b)
{
    float const p = mul(a.hi, b.hi);
    float const e = fma(a.hi, b.lo, fma(a.lo, b.hi, fma(a.hi, b.hi, -p)));
    return fast_two_sum(p, e);
}
//! a / b to about 2^-44, for b in the range of normal numbers
GBX_FORCEINLINE Pair div_pair(Pair a, Pair b)
{
#if defined(__CUDA_ARCH__)
    float inv;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(inv) : "f"(b.hi));
#else
    float const inv = 1.0f / b.hi;
#endif
    float const q = mul(a.hi, inv);
    // a - q b, then one correction
    float r = fma(-q, b.hi, a.hi);
    r = add(r, fma(-q, b.lo, a.lo));
    return fast_two_sum(q, mul(r, inv));
}

//---------------------------------------------------------------------------//
//! FP32 field source of the stages: a uniform field, or an R-Z map
struct StageField
{
    F3 field;
    float coeffi;  //!< q / (p c) factor of the momentum derivative
    RZMapData const* map;
};

//! The R-Z map's field at an FP32 position (RZMapField): bilinear in (r, z)
GBX_NOINLINE F3 rzmap_field(RZMapData const& m, F3 pos)
{
    F3 value{0, 0, 0};
    float const r = std::sqrt(fma(pos.x, pos.x, mul(pos.y, pos.y)));
    if (!(pos.z >= m.z.front_f && pos.z <= m.z.back_f && r >= m.r.front_f
          && r <= m.r.back_f))
        return value;
    auto locate = [](FieldMapGrid const& g, float v, size_type* index) {
        float const u = sub(v, g.front_f) / g.delta_f;
        size_type const i = min_of(static_cast<size_type>(u), g.size - 2);
        *index = i;
        return sub(u, float(i));
    };
    size_type ir, iz;
    float const fr = locate(m.r, r, &ir);
    float const fz = locate(m.z, pos.z, &iz);
    size_type const nr = m.r.size;
    FieldMapElementF const* v = m.values_f;
    float low = v[iz * nr + ir].value_z;
    float high = v[(iz + 1) * nr + ir].value_z;
    value.z = fma(sub(high, low), fz, low);
    low = v[iz * nr + ir].value_r;
    high = v[iz * nr + ir + 1].value_r;
    float const tmp = (r != 0) ? fma(sub(high, low), fr, low) / r : low;
    value.x = mul(tmp, pos.x);
    value.y = mul(tmp, pos.y);
    return value;
}

//! One Dormand-Prince step from (p0, m0) over h, relative to its start
struct StageResult
{
    F3 increment;  //!< To the end position
    F3 momentum;  //!< At the end
    F3 pos_error;  //!< Error estimate of the position over the step
    F3 mom_error;  //!< Error estimate of the momentum
    float chord;  //!< Distance of Shampine's midpoint from the chord
};

//! Dormand-Prince 5(4) step with FP32 stages. The stages carry momenta,
//! derivatives and, for a field map, position increments from the start at
//! which the map is read. 'p0' is used with a map only. 'round_x' selects the
//! square that the stages after the first round by itself (see square()).
//! Without a map the step is one basic block, so that FP64 work beside it
//! overlaps; 'covered' tells whether the result holds, or (Generic) the IEEE
//! square root and division have to be taken.
template<bool UseMap, bool Generic>
GBX_FORCEINLINE StageResult dormand_prince_stages(StageField const& f,
                                                  float h,
                                                  F3 const& p0,
                                                  F3 const& m0,
                                                  bool round_x,
                                                  bool* covered)
{
    using F = float;
    // Butcher tableau, rounded to FP32
    constexpr F a[6][5] = {
        {0, 0, 0, 0, 0},
        {0.2f, 0, 0, 0, 0},
        {0.075f, 0.225f, 0, 0, 0},
        {F(44. / 45), F(-56. / 15), F(32. / 9), 0, 0},
        {F(19372. / 6561), F(-25360. / 2187), F(64448. / 6561), F(-212. / 729), 0},
        {F(9017. / 3168), F(-355. / 33), F(46732. / 5247), F(49. / 176), F(-5103. / 18656)}};
    constexpr double b1 = 35. / 384, b3 = 500. / 1113, b4 = 125. / 192,
                     b5 = -2187. / 6784, b6 = 11. / 84;
    constexpr double d1 = b1 - 5179. / 57600, d3 = b3 - 7571. / 16695,
                     d4 = b4 - 393. / 640, d5 = b5 + 92097. / 339200,
                     d6 = b6 - 187. / 2100, d7 = -1. / 40;
    constexpr F b[6] = {F(b1), 0, F(b3), F(b4), F(b5), F(b6)};
    constexpr F d[7] = {F(d1), 0, F(d3), F(d4), F(d5), F(d6), F(d7)};
    constexpr F c[7] = {F(6025192743. / 30085553152.), 0, F(51252292925. / 65400821598.),
                        F(-2691868925. / 45128329728.), F(187940372067. / 1594534317056.),
                        F(-1776094331. / 19743644256.), F(11237099. / 235043384.)};

    // d(pos)/ds = p/|p|, d(mom)/ds = (q/|p|) p x B(pos)
    F3 kp[7], km[7];
    bool all_covered = true;
    auto eval = [&](int i, F3 const& dp, F3 const& m) {
        F3 field = f.field;
        if constexpr (UseMap)
            field = rzmap_field(*f.map, F3{add(p0.x, dp.x), add(p0.y, dp.y), add(p0.z, dp.z)});
        F const sq = square(m, i > 0 && round_x);
        F inv;
        if constexpr (Generic)
            inv = 1.0f / std::sqrt(sq);
        else
            inv = inv_sqrt(sq);
        all_covered = all_covered && inv_sqrt_covers(sq);
        kp[i] = {mul(m.x, inv), mul(m.y, inv), mul(m.z, inv)};
        F const scale = mul(f.coeffi, inv);
        km[i] = {mul(scale, fma(m.y, field.z, -mul(m.z, field.y))),
                 mul(scale, fma(m.z, field.x, -mul(m.x, field.z))),
                 mul(scale, fma(m.x, field.y, -mul(m.y, field.x)))};
    };
    // v + sum_j w_j k_j
    auto accumulate = [](F3* v, F w, F3 const& k) {
        v->x = fma(w, k.x, v->x);
        v->y = fma(w, k.y, v->y);
        v->z = fma(w, k.z, v->z);
    };
    F3 const zero{0, 0, 0};
    eval(0, zero, m0);
#pragma unroll
    for (int i = 1; i < 6; ++i)
    {
        F3 m = m0;
        F3 dp = zero;
#pragma unroll
        for (int j = 0; j < i; ++j)
        {
            accumulate(&m, mul(h, a[i][j]), km[j]);
            if constexpr (UseMap)
                accumulate(&dp, mul(h, a[i][j]), kp[j]);
        }
        eval(i, dp, m);
    }
    // Fifth-order solution
    F3 dpos = zero;
    StageResult result;
    result.momentum = m0;
#pragma unroll
    for (int i = 0; i < 6; ++i)
    {
        accumulate(&dpos, b[i], kp[i]);
        accumulate(&result.momentum, mul(h, b[i]), km[i]);
    }
    F3 const inc{mul(h, dpos.x), mul(h, dpos.y), mul(h, dpos.z)};
    result.increment = inc;
    eval(6, inc, result.momentum);

    // Embedded error estimate: difference of the fifth- and fourth-order
    // solutions, for the position as a rate; Shampine's midpoint
    F3 epos = zero, emom = zero, mid = zero;
#pragma unroll
    for (int i = 0; i < 7; ++i)
    {
        if (i == 1)
            continue;
        accumulate(&epos, d[i], kp[i]);
        accumulate(&emom, d[i], km[i]);
        accumulate(&mid, c[i], kp[i]);
    }
    result.pos_error = epos;
    result.mom_error = {mul(h, emom.x), mul(h, emom.y), mul(h, emom.z)};
    F const half = mul(0.5f, h);
    mid = {mul(half, mid.x), mul(half, mid.y), mul(half, mid.z)};
    F3 const cross{fma(inc.y, mid.z, -mul(inc.z, mid.y)),
                   fma(inc.z, mid.x, -mul(inc.x, mid.z)),
                   fma(inc.x, mid.y, -mul(inc.y, mid.x))};
    result.chord = std::sqrt(square(cross) / square(inc));
    *covered = all_covered;
    return result;
}

//! The step with IEEE square roots and divisions (rarely taken)
template<bool UseMap>
GBX_NOINLINE StageResult
dormand_prince_generic(StageField f, float h, F3 p0, F3 m0, bool round_x)
{
    bool covered;
    return dormand_prince_stages<UseMap, true>(f, h, p0, m0, round_x, &covered);
}

//---------------------------------------------------------------------------//
//! Momentum at the start of a Runge-Kutta step, its square as an FP32 pair,
//! and the FP64 momentum where it is not the FP32 one ('rounded' false)
struct StartMomentum
{
    F3 value;
    Pair square;
    Real3 exact;
    bool rounded;
};

//! Squared error over squared tolerance of a step, evaluated in FP32 pairs
struct ErrorNorm
{
    Pair ratio;
    bool usable;  //!< Within the range where the pairs hold 2^-40
};

//! The error norm in FP64
GBX_NOINLINE double
error_norm_fp64(F3 pos_error, F3 mom_error, Real3 mom, double epsilon_rel_max)
{
    Real3 const ep{double(pos_error.x), double(pos_error.y), double(pos_error.z)};
    Real3 const em{double(mom_error.x), double(mom_error.y), double(mom_error.z)};
    double const errpos2 = dot_product(ep, ep);
    double const errvel2 = div(dot_product(em, em), dot_product(mom, mom));
    return div(max_of(errpos2, errvel2), ipow<2>(epsilon_rel_max));
}
GBX_FORCEINLINE double
error_norm_fp64(StageResult const& r, StartMomentum const& start, double epsilon_rel_max)
{
    Real3 mom = start.exact;
    if (start.rounded)
    {
        mom = {double(start.value.x), double(start.value.y), double(start.value.z)};
    }
    return error_norm_fp64(r.pos_error, r.mom_error, mom, epsilon_rel_max);
}
GBX_FORCEINLINE ErrorNorm error_norm(StageResult const& r, Pair msq, FieldOptions const& opt)
{
    Pair const pos = square_pair(r.pos_error);
    Pair const mom = square_pair(r.mom_error);
    Pair const vel = div_pair(mom, msq);
    Pair const larger
        = (pos.hi > vel.hi || (pos.hi == vel.hi && pos.lo > vel.lo)) ? pos : vel;
    ErrorNorm err;
    err.ratio = mul_pair(larger, Pair{opt.inv_tolerance[0], opt.inv_tolerance[1]});
    // Large enough that no low part of a square underflows, small enough that
    // nothing overflows (false for NaN)
    err.usable = msq.hi > 0x1p-20f && msq.hi < 0x1p60f && larger.hi > 0x1p-60f
                 && pos.hi < 0x1p60f && mom.hi < 0x1p60f;
    return err;
}

//! Whether the error norm is above 1: the step is rejected
GBX_FORCEINLINE bool above_one(ErrorNorm const& err,
                               StageResult const& r,
                               StartMomentum const& start,
                               FieldOptions const& opt)
{
    if (err.usable && std::fabs(err.ratio.hi - 1) > 0x1p-20f)
        return err.ratio.hi > 1;
    return error_norm_fp64(r, start, opt.epsilon_rel_max) > 1;
}

//! The error norm clamped to 1e-30..1e30 and rounded to FP32
GBX_FORCEINLINE float clamped_norm(ErrorNorm const& err,
                                   StageResult const& r,
                                   StartMomentum const& start,
                                   FieldOptions const& opt)
{
    float const e = err.ratio.hi;
    float const margin = mul(e, 0x1p-38f);
    if (err.usable && e < 1e25f && e > 1e-25f && add(e, add(err.ratio.lo, margin)) == e
        && add(e, sub(err.ratio.lo, margin)) == e)
    {
        return e;
    }
    double const err_sq = error_norm_fp64(r, start, opt.epsilon_rel_max);
    return float(min_of(max_of(err_sq, 1e-30), 1e30));
}

//! Step-size factor safety * norm^(power / 2); 'above' is above_one()
GBX_FORCEINLINE double new_step_scale(bool above,
                                      ErrorNorm const& err,
                                      StageResult const& r,
                                      StartMomentum const& start,
                                      FieldOptions const& opt)
{
    float const e = clamped_norm(err, r, start, opt);
    double const power = 0.5 * (above ? opt.pshrink : opt.pgrow);
    return opt.safety * fp64::widen(libm::exp(float(power) * libm::log(e)));
}
}  // namespace mixed

//! Field driver over the mixed-precision stepper.
//!
//! advance() is one loop around one Runge-Kutta step, whether the step looks for
//! a chord (find_next_chord), is one of an accurate advance (accurate_advance,
//! integrate_step, one_good_step) or is too short for either: a track that waits
//! for nothing but its own steps then runs through a small piece of code again
//! and again. The FP64 addition of an accepted step to the position is left
//! to the next turn, beside that step's FP32 work.
//!
//! RoundX: which square steps of at most the minimum length round by itself. The
//! one-thread-per-track kernel (true) and the persistent one (false) differ in it, as the
//! compiler had contracted them, so that either keeps its results; a track with such
//! a step may differ in the last bits between the two.
template<bool RoundX>
class MixedFieldDriver
{
  public:
    GBX_FORCEINLINE MixedFieldDriver(FieldOptions const& options,
                                     UniformFieldEquation const& rhs)
        : opt_(options)
    {
        this->set_rhs(rhs);
    }

    GBX_FORCEINLINE DriverResult advance(double step, OdeState const& state)
    {
        return stage_.map ? this->advance_in<true>(step, state)
                          : this->advance_in<false>(step, state);
    }

    //! Forget the chord limit of the previous propagation
    GBX_FORCEINLINE void reset() { max_chord_ = INFINITY; }
    GBX_FORCEINLINE void set_rhs(UniformFieldEquation const& rhs)
    {
        stage_.field = {float(rhs.field.x), float(rhs.field.y), float(rhs.field.z)};
        stage_.coeffi = float(rhs.coeffi);
        stage_.map = rhs.map;
    }

    GBX_FORCEINLINE double minimum_step() const { return opt_.minimum_step; }
    GBX_FORCEINLINE double delta_intersection() const { return opt_.delta_intersection; }
    GBX_FORCEINLINE short max_substeps() const { return opt_.max_substeps; }

  private:
    FieldOptions const& opt_;
    mixed::StageField stage_;
    double max_chord_{INFINITY};

    //! What the next Runge-Kutta step is for
    enum class Turn
    {
        minimum,  //!< The whole advance is at most the minimum step
        chord,  //!< Look for a chord close to the curve
        controlled,  //!< Accurate advance, with error control
        uncontrolled,  //!< Accurate advance, at most the minimum step
    };

    template<bool UseMap>
    GBX_FORCEINLINE DriverResult advance_in(double const step, OdeState const& state)
    {
        using namespace mixed;
        DriverResult result;
        Real3 pos = state.pos;
        // Increment of the last accepted step (a zero that adds nothing)
        F3 pending{-0.0f, -0.0f, -0.0f};
        StartMomentum start;
        start.exact = state.mom;
        start.value = {float(state.mom.x), float(state.mom.y), float(state.mom.z)};
        start.rounded = false;
        Turn turn = Turn::minimum;
        double h = step;
        if (step > opt_.minimum_step)
        {
            turn = Turn::chord;
            h = min_of(step, max_chord_);
            double const msq = dot_product(state.mom, state.mom);
            float const hi = float(msq);
            start.square = {hi, float(msq - double(hi))};
        }
        // Length of this Runge-Kutta step; of an accurate advance: the step it
        // began with, its length so far and to go, and its limits
        double taken = h;
        double curve_length = 0;
        double end_curve_length = 0;
        double h_threshold = 0;
        auto remaining_steps = opt_.max_nsteps;
        size_type tries = 0;
        for (;;)
        {
            bool const round_x = RoundX && turn == Turn::minimum;
            float const hf = fp64::narrow(taken);
            if constexpr (UseMap)
                add_to(&pos, &pending);
            F3 p0{0, 0, 0};
            if constexpr (UseMap)
                p0 = {float(pos.x), float(pos.y), float(pos.z)};
            bool covered;
            StageResult r = dormand_prince_stages<UseMap, false>(
                stage_, hf, p0, start.value, round_x, &covered);
            if constexpr (!UseMap)
                add_to(&pos, &pending);
            if (!covered)
                r = dormand_prince_generic<UseMap>(stage_, hf, p0, start.value, round_x);
            if (turn == Turn::minimum)
            {
                result.step = step;
                pending = r.increment;
                start.value = r.momentum;
                break;
            }
            if (turn == Turn::chord && r.chord > opt_.chord_limit)
            {
                // From chord_far on the factor is the smallest one
                double scale = FieldOptions::min_chord_shrink;
                if (!(r.chord > opt_.chord_far))
                {
                    scale = max_of(
                        fp64::sqrt_inline(fp64::div_inline(opt_.delta_chord, fp64::widen(r.chord))),
                        FieldOptions::min_chord_shrink);
                }
                taken *= scale;
                if (--remaining_steps > 0)
                    continue;
            }
            ErrorNorm const err = error_norm(r, start.square, opt_);
            bool const above = above_one(err, r, start, opt_);
            if (turn == Turn::chord)
            {
                if (taken < step)
                {
                    max_chord_ = taken * (1 / FieldOptions::min_chord_shrink);
                }
                if (!above)
                {
                    result.step = taken;
                    pending = r.increment;
                    start.value = r.momentum;
                    break;
                }
                // Cover the chord's length with steps under error control
                end_curve_length = taken;
                h = step * new_step_scale(true, err, r, start, opt_);
                if (!(h > FieldOptions::initial_step_tol * end_curve_length
                      && h < end_curve_length))
                {
                    h = end_curve_length;
                }
                h_threshold = opt_.epsilon_step * end_curve_length;
                remaining_steps = opt_.max_nsteps;
            }
            else
            {
                if (turn == Turn::controlled && above)
                {
                    taken *= max_of(new_step_scale(true, err, r, start, opt_),
                                    opt_.max_stepping_decrease);
                    if (--tries > 0)
                        continue;
                }
                curve_length += taken;
                bool const done = h < h_threshold || curve_length >= end_curve_length;
                if (!done)
                {
                    double scale = new_step_scale(above, err, r, start, opt_);
                    if (turn == Turn::controlled)
                        scale = min_of(scale, opt_.max_stepping_increase);
                    h = min_of(max_of(taken * scale, opt_.minimum_step),
                               end_curve_length - curve_length);
                }
                pending = r.increment;
                start.value = r.momentum;
                start.square = square_pair(r.momentum);
                start.rounded = true;
                if (done || --remaining_steps <= 0)
                {
                    result.step = min_of(curve_length, end_curve_length);
                    break;
                }
            }
            turn = h > opt_.minimum_step ? Turn::controlled : Turn::uncontrolled;
            taken = h;
            tries = opt_.max_nsteps;
        }
        add_to(&pos, &pending);
        result.state.pos = pos;
        result.state.mom = {
            double(start.value.x), double(start.value.y), double(start.value.z)};
        return result;
    }

    //! Add the pending increment to the position
    static GBX_FORCEINLINE void add_to(Real3* pos, mixed::F3* pending)
    {
        pos->x += double(pending->x);
        pos->y += double(pending->y);
        pos->z += double(pending->z);
        *pending = {-0.0f, -0.0f, -0.0f};
    }
};
}  // namespace gbx

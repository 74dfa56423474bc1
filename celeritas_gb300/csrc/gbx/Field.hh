// Charged-particle propagation in a uniform magnetic field: Dormand-Prince
// RK5(4) integration with an adaptive driver and a chord-based boundary
// search through the geometry.
//
// Follows src/celeritas/field/FieldPropagator.hh:150-333,
// FieldDriver.hh:182-429, DormandPrinceStepper.hh:102-222,
// MagFieldEquation.hh, detail/FieldUtils.hh and the defaults of
// FieldDriverOptions.hh:26-77.
//
// This file holds the FP64 build's driver, FP64 throughout, operation for
// operation as in the reference, and the propagator of both builds; the
// mixed-precision build's driver is in FieldMixed.hh.
#pragma once

#include <type_traits>

#include "FieldMixed.hh"
#include "FieldState.hh"
#include "Geometry.hh"

namespace gbx
{
GBX_FORCEINLINE void axpy(double a, OdeState const& x, OdeState* y)
{
    axpy(a, x.pos, &y->pos);
    axpy(a, x.mom, &y->mom);
}

GBX_FORCEINLINE Real3 cross_product(Real3 const& x, Real3 const& y)
{
    return {x.y * y.z - x.z * y.y, x.z * y.x - x.x * y.z, x.x * y.y - x.y * y.x};
}

GBX_FORCEINLINE double fastpow(double a, double b)
{
    return libm::exp(b * libm::log(a));
}

//! Field of an R-Z map at a position (RZMapField::operator(),
//! src/celeritas/field/RZMapField.hh:70-108): bilinear in (r, z) on the
//! uniform grids, zero outside the map, the radial component along (x, y)
GBX_FUNCTION Real3 rzmap_field(RZMapData const& m, Real3 const& pos)
{
    Real3 value{0, 0, 0};
    double const r = gbx::sqrt(ipow<2>(pos.x) + ipow<2>(pos.y));
    if (!(pos.z >= m.z.front && pos.z <= m.z.back && r >= m.r.front && r <= m.r.back))
        return value;
    // find_interp on a uniform grid (UniformGrid::find, operator[]); a value
    // on the last node takes the last interval
    auto locate = [](FieldMapGrid const& g, double v, size_type* index) {
        size_type i = static_cast<size_type>(div(v - g.front, g.delta));
        i = min_of(i, g.size - 2);
        double const lower = g.front + g.delta * i;
        double const upper = g.front + g.delta * (i + 1);
        *index = i;
        return div(v - lower, upper - lower);
    };
    size_type ir, iz;
    double const fr = locate(m.r, r, &ir);
    double const fz = locate(m.z, pos.z, &iz);
    size_type const nr = m.r.size;
    double low = m.values[iz * nr + ir].value_z;
    double high = m.values[(iz + 1) * nr + ir].value_z;
    value.z = low + (high - low) * fz;
    low = m.values[iz * nr + ir].value_r;
    high = m.values[iz * nr + ir + 1].value_r;
    double const tmp = (r != 0) ? div(low + (high - low) * fr, r) : low;
    value.x = tmp * pos.x;
    value.y = tmp * pos.y;
    return value;
}

//! The field equation with its field source fixed at compile time, so that
//! each FP64 Runge-Kutta step branches once on the source, not per stage
template<bool UseMap>
struct FixedFieldEquation
{
    UniformFieldEquation const& eq;

    GBX_FORCEINLINE OdeState operator()(OdeState const& y) const
    {
        double momentum_inv
            = fp64::div_inline(1.0, fp64::sqrt_inline(dot_product(y.mom, y.mom)));
        OdeState result;
        result.pos = {momentum_inv * y.mom.x,
                      momentum_inv * y.mom.y,
                      momentum_inv * y.mom.z};
        double const scale = eq.coeffi * momentum_inv;
        Real3 c = cross_product(y.mom, UseMap ? rzmap_field(*eq.map, y.pos) : eq.field);
        result.mom = {scale * c.x, scale * c.y, scale * c.z};
        return result;
    }
};

//! Dormand-Prince 5(4) step: the stages and the end state when taken; the error
//! estimate and Shampine's midpoint where the driver asks for them
template<class Equation>
class DormandPrinceStep
{
  public:
    GBX_FORCEINLINE void take(Equation const& rhs, double step, OdeState const& beg_state)
    {
        step_ = step;
        using R = double;
        constexpr R a11 = 0.2;
        constexpr R a21 = 0.075;
        constexpr R a22 = 0.225;
        constexpr R a31 = 44 / R(45);
        constexpr R a32 = -56 / R(15);
        constexpr R a33 = 32 / R(9);
        constexpr R a41 = 19372 / R(6561);
        constexpr R a42 = -25360 / R(2187);
        constexpr R a43 = 64448 / R(6561);
        constexpr R a44 = -212 / R(729);
        constexpr R a51 = 9017 / R(3168);
        constexpr R a52 = -355 / R(33);
        constexpr R a53 = 46732 / R(5247);
        constexpr R a54 = 49 / R(176);
        constexpr R a55 = -5103 / R(18656);

        k1_ = rhs(beg_state);
        OdeState state = beg_state;
        axpy(a11 * step, k1_, &state);
        OdeState const k2 = rhs(state);
        state = beg_state;
        axpy(a21 * step, k1_, &state);
        axpy(a22 * step, k2, &state);
        k3_ = rhs(state);
        state = beg_state;
        axpy(a31 * step, k1_, &state);
        axpy(a32 * step, k2, &state);
        axpy(a33 * step, k3_, &state);
        k4_ = rhs(state);
        state = beg_state;
        axpy(a41 * step, k1_, &state);
        axpy(a42 * step, k2, &state);
        axpy(a43 * step, k3_, &state);
        axpy(a44 * step, k4_, &state);
        k5_ = rhs(state);
        state = beg_state;
        axpy(a51 * step, k1_, &state);
        axpy(a52 * step, k2, &state);
        axpy(a53 * step, k3_, &state);
        axpy(a54 * step, k4_, &state);
        axpy(a55 * step, k5_, &state);
        k6_ = rhs(state);
        end_ = beg_state;
        axpy(a61 * step, k1_, &end_);
        axpy(a63 * step, k3_, &end_);
        axpy(a64 * step, k4_, &end_);
        axpy(a65 * step, k5_, &end_);
        axpy(a66 * step, k6_, &end_);
        k7_ = rhs(end_);
    }

    GBX_FORCEINLINE OdeState const& end_state() const { return end_; }

    //! Difference of the fifth- and fourth-order solutions
    GBX_FORCEINLINE OdeState error() const
    {
        using R = double;
        constexpr R d71 = a61 - 5179 / R(57600);
        constexpr R d73 = a63 - 7571 / R(16695);
        constexpr R d74 = a64 - 393 / R(640);
        constexpr R d75 = a65 + 92097 / R(339200);
        constexpr R d76 = a66 - 187 / R(2100);
        constexpr R d77 = -1 / R(40);
        OdeState result{{0, 0, 0}, {0, 0, 0}};
        axpy(d71 * step_, k1_, &result);
        axpy(d73 * step_, k3_, &result);
        axpy(d74 * step_, k4_, &result);
        axpy(d75 * step_, k5_, &result);
        axpy(d76 * step_, k6_, &result);
        axpy(d77 * step_, k7_, &result);
        return result;
    }

    //! Position in the middle of the step
    GBX_FORCEINLINE Real3 mid_pos(Real3 const& beg_pos) const
    {
        using R = double;
        constexpr R c71 = R(6025192743.) / R(30085553152.);
        constexpr R c73 = R(51252292925.) / R(65400821598.);
        constexpr R c74 = R(-2691868925.) / R(45128329728.);
        constexpr R c75 = R(187940372067.) / R(1594534317056.);
        constexpr R c76 = R(-1776094331.) / R(19743644256.);
        constexpr R c77 = R(11237099.) / R(235043384.);
        R const half_step = step_ / R(2);
        Real3 result = beg_pos;
        axpy(c71 * half_step, k1_.pos, &result);
        axpy(c73 * half_step, k3_.pos, &result);
        axpy(c74 * half_step, k4_.pos, &result);
        axpy(c75 * half_step, k5_.pos, &result);
        axpy(c76 * half_step, k6_.pos, &result);
        axpy(c77 * half_step, k7_.pos, &result);
        return result;
    }

  private:
    static constexpr double a61 = 35 / double(384);
    static constexpr double a63 = 500 / double(1113);
    static constexpr double a64 = 125 / double(192);
    static constexpr double a65 = -2187 / double(6784);
    static constexpr double a66 = 11 / double(84);

    double step_;
    OdeState k1_, k3_, k4_, k5_, k6_, k7_;
    OdeState end_;
};

//! What a warp is to take, and what the length that goes with it is
enum class WarpTask
{
    none,  //!< No step: the helpers are done
    chord,  //!< A step and its chord; its error unless that is above the length
    error,  //!< A step and its error, its position's relative to the length
};

//! A step taken by a warp: its end, and the two numbers by which the driver
//! accepts it
struct WarpStep
{
    OdeState end;
    double dchord;  //!< Distance of the midpoint from the chord (WarpTask::chord)
    double rel_err_sq;  //!< Relative squared error (not of a chord too far)
    bool active;  //!< A step was taken
};

#if defined(__CUDACC__)
//! Coefficients of the step: a11, a21 a22, a31..a33, a41..a44, a51..a55, a61 a63..a66;
//! d71 d73..d77; c71 c73..c77 (names of DormandPrinceStep)
static __device__ double const warp_step_coefficients[32] = {
    0.2,
    0.075,
    0.225,
    44 / double(45),
    -56 / double(15),
    32 / double(9),
    19372 / double(6561),
    -25360 / double(2187),
    64448 / double(6561),
    -212 / double(729),
    9017 / double(3168),
    -355 / double(33),
    46732 / double(5247),
    49 / double(176),
    -5103 / double(18656),
    35 / double(384),
    500 / double(1113),
    125 / double(192),
    -2187 / double(6784),
    11 / double(84),
    35 / double(384) - 5179 / double(57600),
    500 / double(1113) - 7571 / double(16695),
    125 / double(192) - 393 / double(640),
    -2187 / double(6784) + 92097 / double(339200),
    11 / double(84) - 187 / double(2100),
    -1 / double(40),
    double(6025192743.) / double(30085553152.),
    double(51252292925.) / double(65400821598.),
    double(-2691868925.) / double(45128329728.),
    double(187940372067.) / double(1594534317056.),
    double(-1776094331.) / double(19743644256.),
    double(11237099.) / double(235043384.)};

//! One Dormand-Prince step of one track by the 32 lanes of its warp, which all call
//! this; only lane 0's arguments count.
//!
//! On GB300 an FP64 instruction takes its warp 64 cycles whatever its lanes do, and
//! none overlaps another. With few tracks, each in a warp of its own, three lanes
//! hold the position, three the momentum and three the midpoint's position, so
//! that each of the 26 + 6 accumulations is one instruction instead of six, each
//! evaluation 8 instead of 19, and the 32 products of the step and a coefficient
//! one. Every lane does the operations of DormandPrinceStep, rel_err_sq and
//! distance_chord for its component, so the results are theirs bit for bit. An event
//! of 20 particles in the CMS-like detector 458 -> 363 ms, 7 with detector hits 77 -> 65
//! ms, 300 electrons in the calorimeter 230 -> 224.5 ms.
__device__ __noinline__ WarpStep warp_step(
    WarpTask task, UniformFieldEquation rhs, double step, OdeState beg, double length)
{
    auto from = [](double v, int lane) { return __shfl_sync(0xffffffffu, v, lane); };
    WarpStep result;
    __syncwarp();
    task = static_cast<WarpTask>(__shfl_sync(0xffffffffu, int(task), 0));
    result.active = task != WarpTask::none;
    if (!result.active)
        return result;
    step = from(step, 0);
    length = from(length, 0);
    rhs.coeffi = from(rhs.coeffi, 0);
    rhs.field = {from(rhs.field.x, 0), from(rhs.field.y, 0), from(rhs.field.z, 0)};
    rhs.map = reinterpret_cast<RZMapData const*>(
        __shfl_sync(0xffffffffu, reinterpret_cast<unsigned long long>(rhs.map), 0));
    beg.pos = {from(beg.pos.x, 0), from(beg.pos.y, 0), from(beg.pos.z, 0)};
    beg.mom = {from(beg.mom.x, 0), from(beg.mom.y, 0), from(beg.mom.z, 0)};

    // Lanes 0-2: position, 3-5: momentum, 6-8: position, for the midpoint (the
    // rest repeat lanes 0-8)
    int const lane = threadIdx.x & 31;
    int const group = (lane / 3) % 3;
    int const c = lane % 3;
    bool const is_mom = group == 1;
    // Component i % 3 without an indexed (local) array
    auto pick = [](Real3 const& v, int i) {
        i = i >= 3 ? i - 3 : i;
        return i == 0 ? v.x : (i == 1 ? v.y : v.z);
    };
    auto cross = [&](Real3 const& a, Real3 const& b) {
        return pick(a, c + 1) * pick(b, c + 2) - pick(a, c + 2) * pick(b, c + 1);
    };
    double const start = is_mom ? pick(beg.mom, c) : pick(beg.pos, c);
    double const product = warp_step_coefficients[lane] * (lane >= 26 ? step / 2 : step);
    double mom_sq;
    auto eval = [&](double y) {
        Real3 const mom{from(y, 3), from(y, 4), from(y, 5)};
        if (rhs.map)
            rhs.field = rzmap_field(*rhs.map, Real3{from(y, 0), from(y, 1), from(y, 2)});
        mom_sq = dot_product(mom, mom);
        double const inv = fp64::div_inline(1.0, fp64::sqrt_inline(mom_sq));
        double const scale = rhs.coeffi * inv;
        double const direction = is_mom ? cross(mom, rhs.field) : pick(mom, c);
        return (is_mom ? scale : inv) * direction;
    };
    auto add = [&](double* y, int i, double k) { *y = gbx_fma(from(product, i), k, *y); };
    double const k1 = eval(start);
    double const beg_mom_sq = mom_sq;
    double y = start;
    add(&y, 0, k1);
    double const k2 = eval(y);
    y = start;
    add(&y, 1, k1);
    add(&y, 2, k2);
    double const k3 = eval(y);
    y = start;
    add(&y, 3, k1);
    add(&y, 4, k2);
    add(&y, 5, k3);
    double const k4 = eval(y);
    y = start;
    add(&y, 6, k1);
    add(&y, 7, k2);
    add(&y, 8, k3);
    add(&y, 9, k4);
    double const k5 = eval(y);
    y = start;
    add(&y, 10, k1);
    add(&y, 11, k2);
    add(&y, 12, k3);
    add(&y, 13, k4);
    add(&y, 14, k5);
    double const k6 = eval(y);
    y = start;
    add(&y, 15, k1);
    add(&y, 16, k3);
    add(&y, 17, k4);
    add(&y, 18, k5);
    add(&y, 19, k6);
    double const k7 = eval(y);
    result.end = {{from(y, 0), from(y, 1), from(y, 2)}, {from(y, 3), from(y, 4), from(y, 5)}};
    // Error estimate, and the midpoint in lanes 6-8
    int const first = group == 2 ? 26 : 20;
    double z = group == 2 ? start : 0;
    add(&z, first, k1);
    add(&z, first + 1, k3);
    add(&z, first + 2, k4);
    add(&z, first + 3, k5);
    add(&z, first + 4, k6);
    add(&z, first + 5, k7);
    // Two dot products at a time: even lanes' and odd lanes'
    bool const odd = lane & 1;
    if (task == WarpTask::chord)
    {
        double const to_mid = z - start;
        double const to_end = y - start;
        Real3 const beg_mid{from(to_mid, 6), from(to_mid, 7), from(to_mid, 8)};
        Real3 const beg_end{from(to_end, 6), from(to_end, 7), from(to_end, 8)};
        double const component = cross(beg_end, beg_mid);
        Real3 v{from(component, 0), from(component, 1), from(component, 2)};
        if (odd)
            v = beg_end;
        double const square = dot_product(v, v);
        result.dchord = gbx::sqrt(div(from(square, 0), from(square, 1)));
        if (result.dchord > length)
            return result;
        length = step;
    }
    int const part = odd ? 3 : 0;
    Real3 const err{from(z, part), from(z, part + 1), from(z, part + 2)};
    double const ratio = div(dot_product(err, err), odd ? beg_mom_sq : ipow<2>(length));
    result.rel_err_sq = max_of(from(ratio, 0), from(ratio, 1));
    return result;
}

//! A value that the compiler does not know (there is one warp_step for all lanes)
__device__ __forceinline__ WarpTask opaque(WarpTask task)
{
    int value = static_cast<int>(task);
    asm volatile("" : "+r"(value));
    return static_cast<WarpTask>(value);
}

//! Steps of lane 0's track until it is through
__device__ __forceinline__ void help_field_warp()
{
    bool active = false;
    UniformFieldEquation rhs{};
    OdeState beg{};
    do
    {
        active = warp_step(opaque(WarpTask::none), rhs, 0, beg, 0).active;
    } while (active);
}

//! Lane 0, after its track: let the helpers go
__device__ __forceinline__ void end_field_warp()
{
    warp_step(opaque(WarpTask::none), UniformFieldEquation{}, 0, OdeState{}, 0);
}
#endif

//---------------------------------------------------------------------------//
// Field driver
//---------------------------------------------------------------------------//
//! Field driver of the FP64 build (FieldDriver.hh:182-429).
//!
//! advance() is one loop around one Runge-Kutta step, whether the step looks for
//! a chord (find_next_chord), is one of an accurate advance (accurate_advance,
//! integrate_step, one_good_step) or is too short for either. A step of one track
//! takes some 300 FP64 instructions of 64 cycles each, and a track that curls up in
//! the field hundreds of steps one after the other: the error estimate is formed
//! only for steps whose chord holds, the midpoint only while a chord is looked
//! for, and the loop's code is small enough to stay in the instruction cache.
//! One c3-like event of 20 particles 516 -> 478 ms, 7 with detector hits 84 -> 80
//! ms, against the estimate and midpoint of every step and a copy of the step for
//! each use.
template<bool Warp>
class FieldDriver
{
  public:
    GBX_FORCEINLINE FieldDriver(FieldOptions const& options,
                                UniformFieldEquation const& rhs)
        : opt_(options), rhs_(rhs)
    {
    }

    GBX_FORCEINLINE DriverResult advance(double step, OdeState const& state)
    {
        return rhs_.map ? this->advance_in(FixedFieldEquation<true>{rhs_}, step, state)
                        : this->advance_in(FixedFieldEquation<false>{rhs_}, step, state);
    }

    //! Forget the chord limit of the previous propagation
    GBX_FORCEINLINE void reset() { max_chord_ = INFINITY; }
    GBX_FORCEINLINE void set_rhs(UniformFieldEquation const& rhs) { rhs_ = rhs; }

    GBX_FORCEINLINE double minimum_step() const { return opt_.minimum_step; }
    GBX_FORCEINLINE double delta_intersection() const
    {
        return opt_.delta_intersection;
    }
    GBX_FORCEINLINE short max_substeps() const { return opt_.max_substeps; }

  private:
    FieldOptions const& opt_;
    UniformFieldEquation rhs_;
    double max_chord_{INFINITY};

    //! What the next Runge-Kutta step is for
    enum class Turn
    {
        minimum,  //!< The whole advance is at most the minimum step
        chord,  //!< Look for a chord close to the curve
        controlled,  //!< Accurate advance, with error control
        uncontrolled,  //!< Accurate advance, at most the minimum step
    };

    template<class Equation>
    GBX_FORCEINLINE DriverResult advance_in(Equation const& rhs,
                                            double const step,
                                            OdeState const& state)
    {
        DriverResult result;
        result.state = state;
        Turn turn = Turn::minimum;
        double h = step;
        if (step > opt_.minimum_step)
        {
            turn = Turn::chord;
            h = min_of(step, max_chord_);
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
            DormandPrinceStep<Equation> rk;
            WarpStep warp;
            double const chord_limit = opt_.delta_chord + FieldOptions::dchord_tol;
            if constexpr (Warp)
            {
#if defined(__CUDA_ARCH__)
                bool const chord = turn == Turn::chord;
                warp = warp_step(opaque(chord ? WarpTask::chord : WarpTask::error),
                                 rhs_,
                                 taken,
                                 result.state,
                                 chord ? chord_limit : taken);
#endif
            }
            else
            {
                rk.take(rhs, taken, result.state);
                warp.end = rk.end_state();
            }
            OdeState const& end_state = warp.end;
            if (turn == Turn::minimum)
            {
                result.state = end_state;
                result.step = step;
                return result;
            }
            if (turn == Turn::chord)
            {
                Real3 const& beg_pos = result.state.pos;
                double const dchord
                    = Warp ? warp.dchord
                           : distance_chord(beg_pos, rk.mid_pos(beg_pos), end_state.pos);
                if (dchord > chord_limit)
                {
                    // From chord_far on the factor is the smallest one
                    double scale = FieldOptions::min_chord_shrink;
                    if (!(dchord > opt_.chord_far))
                    {
                        scale = max_of(gbx::sqrt(div(opt_.delta_chord, dchord)),
                                       FieldOptions::min_chord_shrink);
                    }
                    double const tried = taken;
                    taken *= scale;
                    if (--remaining_steps > 0)
                        continue;
                    // The last trial stands whatever its chord: by its error over
                    // the length that would have been next
                    if constexpr (Warp)
                    {
#if defined(__CUDA_ARCH__)
                        warp = last_warp_step(rhs_, tried, result.state, taken);
#endif
                    }
                }
            }
            double const rel_err
                = Warp ? warp.rel_err_sq : rel_err_sq(rk.error(), taken, result.state.mom);
            // Scaled error of a step: above 1 the step is rejected
            double const err_sq = div(rel_err, ipow<2>(opt_.epsilon_rel_max));
            if (turn == Turn::chord)
            {
                if (taken < step)
                {
                    max_chord_ = taken * (1 / FieldOptions::min_chord_shrink);
                }
                if (!(err_sq > 1))
                {
                    result.state = end_state;
                    result.step = taken;
                    return result;
                }
                // Cover the chord's length with steps under error control
                end_curve_length = taken;
                h = step * this->new_step_scale(err_sq);
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
                if (turn == Turn::controlled && err_sq > 1)
                {
                    taken *= max_of(this->new_step_scale(err_sq), opt_.max_stepping_decrease);
                    if (--tries > 0)
                        continue;
                }
                curve_length += taken;
                bool const done = h < h_threshold || curve_length >= end_curve_length;
                if (!done)
                {
                    double scale = this->new_step_scale(err_sq);
                    if (turn == Turn::controlled)
                        scale = min_of(scale, opt_.max_stepping_increase);
                    h = min_of(max_of(taken * scale, opt_.minimum_step),
                               end_curve_length - curve_length);
                }
                result.state = end_state;
                if (done || --remaining_steps <= 0)
                {
                    result.step = min_of(curve_length, end_curve_length);
                    return result;
                }
            }
            turn = h > opt_.minimum_step ? Turn::controlled : Turn::uncontrolled;
            taken = h;
            tries = opt_.max_nsteps;
        }
    }

#if defined(__CUDACC__)
    //! A used-up search's last trial with its error over another length (out of line:
    //! beside the loop's own step it takes an event of 20 particles 0.3% longer)
    static __device__ __noinline__ WarpStep
    last_warp_step(UniformFieldEquation rhs, double step, OdeState beg, double length)
    {
        return warp_step(opaque(WarpTask::error), rhs, step, beg, length);
    }
#endif

    static GBX_FORCEINLINE double rel_err_sq(OdeState const& err_state,
                                             double step,
                                             Real3 const& mom)
    {
        double errpos2 = dot_product(err_state.pos, err_state.pos);
        double errvel2 = dot_product(err_state.mom, err_state.mom);
        errpos2 = div(errpos2, ipow<2>(step));
        errvel2 = div(errvel2, dot_product(mom, mom));
        return max_of(errpos2, errvel2);
    }

    static GBX_FORCEINLINE double distance_chord(Real3 const& beg_pos,
                                                 Real3 const& mid_pos,
                                                 Real3 const& end_pos)
    {
        Real3 beg_mid{mid_pos.x - beg_pos.x, mid_pos.y - beg_pos.y, mid_pos.z - beg_pos.z};
        Real3 beg_end{end_pos.x - beg_pos.x, end_pos.y - beg_pos.y, end_pos.z - beg_pos.z};
        Real3 cross = cross_product(beg_end, beg_mid);
        return gbx::sqrt(div(dot_product(cross, cross), dot_product(beg_end, beg_end)));
    }

    GBX_FORCEINLINE double new_step_scale(double err_sq) const
    {
        double const power = 0.5 * (err_sq > 1 ? opt_.pshrink : opt_.pgrow);
        return opt_.safety * fastpow(err_sq, power);
    }
};

//---------------------------------------------------------------------------//
// Field propagator
//---------------------------------------------------------------------------//
#ifdef GBX_CHECK_SAFE_BALL
//! Chord queries the surface-free ball answered, and those the full query
//! contradicted (CPU oracle check build only, single-threaded runs)
inline unsigned long long safe_ball_uses = 0;
inline unsigned long long safe_ball_mismatches = 0;
#endif

//! Propagation of a charged track up to 'step' along its curved trajectory,
//! stopping at the first boundary crossing (FieldPropagator::operator()),
//! split into its set-up, one substep of its loop and its completion so that
//! a kernel can interleave the substeps of different tracks. Running
//! init(), then substep() until done(), then finish() is the reference's
//! sequence of operations. RoundX is the mixed-precision driver's. Warp: this is
//! lane 0 of a warp whose lanes take the FP64 driver's steps together, the others
//! in help_field_warp().
template<bool RoundX = true, bool Warp = false>
class FieldPropagation
{
    static_assert(!Warp || sizeof(real_type) == sizeof(double),
                  "only the FP64 driver takes steps with its warp's lanes");

  public:
    GBX_FORCEINLINE FieldPropagation(FieldOptions const& opt,
                                     UniformFieldEquation const& rhs)
        : driver_(opt, rhs)
    {
    }

    //! Start a propagation; 'start_safety' is a safety distance already
    //! known at the track's position (0 if none)
    GBX_FORCEINLINE void
    init(GeoTrackView& geo, double momentum, double step, double start_safety = 0)
    {
        driver_.reset();
        state_.pos = geo.pos();
        Real3 const dir0 = geo.dir();
        state_.mom = {momentum * dir0.x, momentum * dir0.y, momentum * dir0.z};
        result_ = {0, geo.is_on_boundary(), false};
        safe_radius_ = 0;
        if (start_safety > 0 && off_axis(state_.pos))
        {
            double const radius = start_safety * (1 - 1e-6) - 1e-6;
            if (radius > 0)
            {
                safe_radius_ = radius;
                center_ = state_.pos;
            }
        }
        step_ = step;
        remaining_ = step;
        remaining_substeps_ = driver_.max_substeps();
    }

    //! Whether the substep loop has ended (checked after each substep)
    GBX_FORCEINLINE bool done() const
    {
        return !(remaining_ > driver_.minimum_step() && remaining_substeps_ > 0);
    }

    //! One iteration of the substep loop
    GBX_FORCEINLINE void substep(GeoTrackView& geo)
    {
        double const delta_intersection = driver_.delta_intersection();
        double const minimum_substep = driver_.minimum_step();
        double const bump_distance = delta_intersection * double(0.1);

        DriverResult substep = driver_.advance(remaining_, state_);
        // Chord from the current position to the substep end
        Real3 cdir{substep.state.pos.x - state_.pos.x,
                   substep.state.pos.y - state_.pos.y,
                   substep.state.pos.z - state_.pos.z};
        double const clen = norm(cdir);
        if constexpr (sizeof(real_type) == sizeof(double))
        {
            cdir.x = div(cdir.x, clen);
            cdir.y = div(cdir.y, clen);
            cdir.z = div(cdir.z, clen);
        }
        else
        {
            // One FP64 division instead of three
            double const inv_clen = div(1, clen);
            cdir.x *= inv_clen;
            cdir.y *= inv_clen;
            cdir.z *= inv_clen;
        }
        // The geometry's direction is always the last chord's (a query of a
        // later substep with a chord shorter than the minimum uses it)
        if (clen >= minimum_substep)
        {
            geo.set_dir(cdir);
        }
        double const max_dist = clen + delta_intersection;
#ifdef GBX_CHECK_SAFE_BALL
        // CPU oracle check build: always run the full query, and count the
        // queries the ball would have answered and any it would have got
        // wrong
        bool const ball = this->inside_safe_ball(geo, max_dist);
        Propagation linear_step = geo.find_next_step<false>(max_dist);
        if (ball)
        {
            ++safe_ball_uses;
            if (linear_step.boundary || linear_step.distance != max_dist)
                ++safe_ball_mismatches;
        }
#else
        Propagation linear_step = this->inside_safe_ball(geo, max_dist)
                                      ? geo.no_crossing(max_dist)
                                      : geo.find_next_step<false>(max_dist);
#endif
        if (!linear_step.boundary)
        {
            state_ = substep.state;
            result_.boundary = false;
            result_.distance += substep.step;
            remaining_ = step_ - result_.distance;
            geo.move_internal_to(state_.pos);
            --remaining_substeps_;
            return;
        }
        // Scaled length of the chord up to the crossing (only with one)
        double const update_length = div(substep.step * linear_step.distance, clen);
        auto is_intercept_close = [&]() {
            double delta_sq = 0;
            for (int i = 0; i < 3; ++i)
            {
                delta_sq += ipow<2>(state_.pos[i] - substep.state.pos[i]
                                    + linear_step.distance * cdir[i]);
            }
            return delta_sq <= ipow<2>(delta_intersection);
        };
        if (result_.boundary && (linear_step.distance) < bump_distance)
        {
            remaining_ = substep.step / 2;
        }
        else if (update_length <= minimum_substep || is_intercept_close()
                 || clen == 0)
        {
            result_.boundary = (linear_step.distance <= clen
                                || result_.distance + update_length <= step_
                                || clen == 0);
            if (!result_.boundary)
            {
                state_.pos = substep.state.pos;
                geo.move_internal_to(substep.state.pos);
            }
            result_.distance += min_of(update_length, substep.step);
            state_.mom = substep.state.mom;
            remaining_ = 0;
        }
        else
        {
            remaining_ = update_length;
        }
    }

    //! Complete the propagation after the loop
    GBX_FORCEINLINE Propagation finish(GeoTrackView& geo)
    {
        double const bump_distance = driver_.delta_intersection() * double(0.1);
        if (remaining_substeps_ == 0 && result_.distance < step_)
        {
            result_.looping = true;
        }
        else if (result_.distance > 0)
        {
            if (result_.boundary)
            {
                geo.move_to_boundary();
                state_.pos = geo.pos();
            }
            else if (result_.distance < step_)
            {
                result_.distance = step_;
            }
        }
        Real3 dir = make_unit_vector(state_.mom);
        geo.set_dir(dir);
        if (result_.distance == 0)
        {
            result_.distance = min_of(bump_distance, step_);
            result_.boundary = false;
            axpy(result_.distance, dir, &state_.pos);
            geo.move_internal_to(state_.pos);
        }
        return result_;
    }

    GBX_FORCEINLINE void set_rhs(UniformFieldEquation const& rhs)
    {
        driver_.set_rhs(rhs);
    }

  private:
    //! Whether the safety distance at a point bounds the distance to every
    //! surface: on (or within 1e-150 of) the z axis a z cylinder's safety is
    //! taken as infinite (its normal is undefined there, as in the
    //! reference's CalcSafetyDistance), so no ball is centred there
    static GBX_FORCEINLINE bool off_axis(Real3 const& pos)
    {
        return ipow<2>(pos.x) + ipow<2>(pos.y) > 1e-300;
    }

    //! Whether the chord query from the current position reaches no
    //! surface within max_dist, because the segment lies inside a ball that
    //! holds no surface of the current volume: then find_next_step would
    //! return max_dist without a crossing, and no_crossing() leaves the
    //! same result and state without solving the surfaces. Without a known
    //! safety the ball is centred where the track stands after its first
    //! substep of the step (a step of one substep never pays for it), with
    //! the safety distance
    //! there as radius, shrunk by 1e-6 relative and 1e-6 cm so that FP64
    //! rounding of the safety and of the distances cannot admit a crossing
    //! the full query would find. Any point of a plane or z cylinder is at
    //! least the safety distance (|x - v|, |r - R|) from the centre. A
    //! safety the multiple-scattering step limit measured at the start
    //! gives the ball from the first substep on.
    GBX_FORCEINLINE bool inside_safe_ball(GeoTrackView& geo, double max_dist)
    {
        if (safe_radius_ < 0 || !geo.is_clear_of_boundary())
            return false;
        if (safe_radius_ == 0)
        {
            if (result_.distance == 0 || !off_axis(state_.pos))
                return false;
            double const radius = geo.find_safety() * (1 - 1e-6) - 1e-6;
            if (!(radius > 0))
            {
                safe_radius_ = -1;
                return false;
            }
            safe_radius_ = radius;
            center_ = state_.pos;
        }
        double const room = safe_radius_ - max_dist;
        if (!(room > 0))
            return false;
        double dsq = 0;
        for (int i = 0; i < 3; ++i)
            dsq += ipow<2>(state_.pos[i] - center_[i]);
        return dsq < room * room;
    }

    std::conditional_t<sizeof(real_type) == sizeof(double), FieldDriver<Warp>, MixedFieldDriver<RoundX>>
        driver_;
    OdeState state_;
    Propagation result_;
    //! Ball free of surfaces: its center and radius (0: not yet measured,
    //! negative: too small to use)
    Real3 center_;
    double safe_radius_;
    double step_;
    double remaining_;
    short remaining_substeps_;
};

}  // namespace gbx

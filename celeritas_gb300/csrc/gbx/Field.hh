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

struct FieldStepperResult
{
    OdeState mid_state;
    OdeState end_state;
    OdeState err_state;
};

//! The field equation with its field source fixed at compile time, so that
//! each FP64 Runge-Kutta step branches once on the source, not per stage
template<bool UseMap>
struct FixedFieldEquation
{
    UniformFieldEquation const& eq;

    GBX_FORCEINLINE OdeState operator()(OdeState const& y) const
    {
        double momentum_inv = div(1.0, gbx::sqrt(dot_product(y.mom, y.mom)));
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

//! Dormand-Prince 5(4) step with Shampine's midpoint interpolation
template<class Equation>
GBX_FUNCTION FieldStepperResult dormand_prince_step_fp64(Equation const& rhs,
                                                         double step,
                                                         OdeState const& beg_state)
{
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
    constexpr R a61 = 35 / R(384);
    constexpr R a63 = 500 / R(1113);
    constexpr R a64 = 125 / R(192);
    constexpr R a65 = -2187 / R(6784);
    constexpr R a66 = 11 / R(84);
    constexpr R d71 = a61 - 5179 / R(57600);
    constexpr R d73 = a63 - 7571 / R(16695);
    constexpr R d74 = a64 - 393 / R(640);
    constexpr R d75 = a65 + 92097 / R(339200);
    constexpr R d76 = a66 - 187 / R(2100);
    constexpr R d77 = -1 / R(40);
    constexpr R c71 = R(6025192743.) / R(30085553152.);
    constexpr R c73 = R(51252292925.) / R(65400821598.);
    constexpr R c74 = R(-2691868925.) / R(45128329728.);
    constexpr R c75 = R(187940372067.) / R(1594534317056.);
    constexpr R c76 = R(-1776094331.) / R(19743644256.);
    constexpr R c77 = R(11237099.) / R(235043384.);

    FieldStepperResult result;
    OdeState k1 = rhs(beg_state);
    OdeState state = beg_state;
    axpy(a11 * step, k1, &state);
    OdeState k2 = rhs(state);
    state = beg_state;
    axpy(a21 * step, k1, &state);
    axpy(a22 * step, k2, &state);
    OdeState k3 = rhs(state);
    state = beg_state;
    axpy(a31 * step, k1, &state);
    axpy(a32 * step, k2, &state);
    axpy(a33 * step, k3, &state);
    OdeState k4 = rhs(state);
    state = beg_state;
    axpy(a41 * step, k1, &state);
    axpy(a42 * step, k2, &state);
    axpy(a43 * step, k3, &state);
    axpy(a44 * step, k4, &state);
    OdeState k5 = rhs(state);
    state = beg_state;
    axpy(a51 * step, k1, &state);
    axpy(a52 * step, k2, &state);
    axpy(a53 * step, k3, &state);
    axpy(a54 * step, k4, &state);
    axpy(a55 * step, k5, &state);
    OdeState k6 = rhs(state);
    result.end_state = beg_state;
    axpy(a61 * step, k1, &result.end_state);
    axpy(a63 * step, k3, &result.end_state);
    axpy(a64 * step, k4, &result.end_state);
    axpy(a65 * step, k5, &result.end_state);
    axpy(a66 * step, k6, &result.end_state);
    OdeState k7 = rhs(result.end_state);
    result.err_state = {{0, 0, 0}, {0, 0, 0}};
    axpy(d71 * step, k1, &result.err_state);
    axpy(d73 * step, k3, &result.err_state);
    axpy(d74 * step, k4, &result.err_state);
    axpy(d75 * step, k5, &result.err_state);
    axpy(d76 * step, k6, &result.err_state);
    axpy(d77 * step, k7, &result.err_state);
    double half_step = step / double(2);
    result.mid_state = beg_state;
    axpy(c71 * half_step, k1, &result.mid_state);
    axpy(c73 * half_step, k3, &result.mid_state);
    axpy(c74 * half_step, k4, &result.mid_state);
    axpy(c75 * half_step, k5, &result.mid_state);
    axpy(c76 * half_step, k6, &result.mid_state);
    axpy(c77 * half_step, k7, &result.mid_state);
    return result;
}

//! Dormand-Prince step with the problem's field source
GBX_FORCEINLINE FieldStepperResult dormand_prince_step(UniformFieldEquation const& rhs,
                                                       double step,
                                                       OdeState const& beg_state)
{
    if (rhs.map)
        return dormand_prince_step_fp64(FixedFieldEquation<true>{rhs}, step, beg_state);
    return dormand_prince_step_fp64(FixedFieldEquation<false>{rhs}, step, beg_state);
}

//---------------------------------------------------------------------------//
// Field driver
//---------------------------------------------------------------------------//
class FieldDriver
{
  public:
    GBX_FORCEINLINE FieldDriver(FieldOptions const& options,
                                UniformFieldEquation const& rhs)
        : opt_(options), rhs_(rhs)
    {
    }

    GBX_FUNCTION DriverResult advance(double step, OdeState const& state)
    {
        if (step <= opt_.minimum_step)
        {
            DriverResult result;
            result.state = dormand_prince_step(rhs_, step, state).end_state;
            result.step = step;
            return result;
        }
        ChordSearch output = this->find_next_chord(min_of(step, max_chord_), state);
        if (output.end.step < step)
        {
            max_chord_ = output.end.step * (1 / FieldOptions::min_chord_shrink);
        }
        if (output.err_sq > 1)
        {
            double next_step = step * this->new_step_scale(output.err_sq);
            output.end = this->accurate_advance(output.end.step, state, next_step);
        }
        return output.end;
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
    struct ChordSearch
    {
        DriverResult end;
        double err_sq;
    };
    struct Integration
    {
        DriverResult end;
        double proposed_step;
    };

    FieldOptions const& opt_;
    UniformFieldEquation rhs_;
    double max_chord_{INFINITY};

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

    //! Scaled error of a stepper result: above 1 the step is rejected
    GBX_FORCEINLINE double step_err_sq(FieldStepperResult const& result,
                                       double step,
                                       Real3 const& mom) const
    {
        return div(rel_err_sq(result.err_state, step, mom), ipow<2>(opt_.epsilon_rel_max));
    }

    //! Distance of the stepper's midpoint from the chord
    GBX_FORCEINLINE double chord_distance(FieldStepperResult const& result,
                                          OdeState const& state) const
    {
        return distance_chord(state.pos, result.mid_state.pos, result.end_state.pos);
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

    GBX_FUNCTION ChordSearch find_next_chord(double step, OdeState const& state) const
    {
        ChordSearch output;
        bool succeeded = false;
        auto remaining_steps = opt_.max_nsteps;
        FieldStepperResult result;
        do
        {
            result = dormand_prince_step(rhs_, step, state);
            double dchord = this->chord_distance(result, state);
            if (dchord > opt_.delta_chord + FieldOptions::dchord_tol)
            {
                double scale_step = max_of(gbx::sqrt(div(opt_.delta_chord, dchord)),
                                           FieldOptions::min_chord_shrink);
                step *= scale_step;
            }
            else
            {
                succeeded = true;
            }
        } while (!succeeded && --remaining_steps > 0);
        output.end.step = step;
        output.end.state = result.end_state;
        output.err_sq = this->step_err_sq(result, step, state.mom);
        return output;
    }

    GBX_FUNCTION Integration one_good_step(double step, OdeState const& state) const
    {
        Integration output;
        bool succeeded = false;
        size_type remaining_steps = opt_.max_nsteps;
        double err_sq;
        FieldStepperResult result;
        do
        {
            result = dormand_prince_step(rhs_, step, state);
            err_sq = this->step_err_sq(result, step, state.mom);
            if (err_sq > 1)
            {
                step *= max_of(this->new_step_scale(err_sq),
                               opt_.max_stepping_decrease);
            }
            else
            {
                succeeded = true;
            }
        } while (!succeeded && --remaining_steps > 0);
        output.end.state = result.end_state;
        output.end.step = step;
        output.proposed_step
            = step * min_of(this->new_step_scale(err_sq), opt_.max_stepping_increase);
        return output;
    }

    GBX_FUNCTION Integration integrate_step(double step, OdeState const& state) const
    {
        Integration output;
        if (step > opt_.minimum_step)
        {
            output = this->one_good_step(step, state);
        }
        else
        {
            FieldStepperResult result = dormand_prince_step(rhs_, step, state);
            output.end.state = result.end_state;
            output.end.step = step;
            double err_sq = this->step_err_sq(result, step, state.mom);
            output.proposed_step = step * this->new_step_scale(err_sq);
        }
        return output;
    }

    GBX_FUNCTION DriverResult accurate_advance(double step,
                                               OdeState const& state,
                                               double hinitial) const
    {
        double end_curve_length = step;
        double h = ((hinitial > FieldOptions::initial_step_tol * step)
                    && (hinitial < step))
                       ? hinitial
                       : step;
        double h_threshold = opt_.epsilon_step * step;
        Integration output;
        output.end.state = state;
        bool succeeded = false;
        double curve_length = 0;
        auto remaining_steps = opt_.max_nsteps;
        do
        {
            output = this->integrate_step(h, output.end.state);
            curve_length += output.end.step;
            if (h < h_threshold || curve_length >= end_curve_length)
            {
                succeeded = true;
            }
            else
            {
                h = min_of(max_of(output.proposed_step, opt_.minimum_step),
                           end_curve_length - curve_length);
            }
        } while (!succeeded && --remaining_steps > 0);
        output.end.step = min_of(curve_length, step);
        return output.end;
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
//! sequence of operations. RoundX is the mixed-precision driver's.
template<bool RoundX = true>
class FieldPropagation
{
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

  public:

  private:
    std::conditional_t<sizeof(real_type) == sizeof(double), FieldDriver, MixedFieldDriver<RoundX>>
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

//! Propagate a charged track up to 'step' along its curved trajectory,
//! stopping at the first boundary crossing (FieldPropagator::operator())
GBX_FUNCTION Propagation propagate_in_field(FieldOptions const& opt,
                                            UniformFieldEquation const& rhs,
                                            double momentum,
                                            GeoTrackView& geo,
                                            double step)
{
    FieldPropagation<> fp(opt, rhs);
    fp.init(geo, momentum, step);
    do
    {
        fp.substep(geo);
    } while (!fp.done());
    return fp.finish(geo);
}

}  // namespace gbx

// State and equation of motion shared by the field drivers of both builds.
#pragma once

#include "Data.hh"

namespace gbx
{
struct OdeState
{
    Real3 pos;
    Real3 mom;
};

//! Equation of motion in a magnetic field: d(pos)/ds = p/|p|,
//! d(mom)/ds = (q/|p|) p x B(pos) (MagFieldEquation). The field is uniform,
//! or an R-Z map evaluated at the state's position when 'map' is set.
struct UniformFieldEquation
{
    Real3 field;
    double coeffi;
    RZMapData const* map{nullptr};
};

//! End of a field driver's advance
struct DriverResult
{
    OdeState state;
    double step;
};
}  // namespace gbx

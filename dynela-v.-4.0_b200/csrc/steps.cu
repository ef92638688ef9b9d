// steps.cu - the builds of k_steps (dnl_steps.cuh), compiled once for each
// precision, nodes per element and time step method (STEPS_REAL, STEPS_NPE,
// STEPS_PI: __graft_entry__.py lists the eight).
#include "dnl_steps.cuh"

namespace dnl
{
template <> StepsBuild steps_build<STEPS_REAL, STEPS_NPE, STEPS_PI>(bool one, int budget)
{
  return one ? steps_build_budget<STEPS_REAL, STEPS_NPE, true, STEPS_PI>(budget)
             : steps_build_budget<STEPS_REAL, STEPS_NPE, false, STEPS_PI>(budget);
}
} // namespace dnl

// The step's layers for one weight format.
#include "step_layers.cuh"

namespace cq {

int launch_step_layers_i4(const StepArgs& a, const LaunchCfg& cfg) { return launch_step_layers_q<Q_I4>(a, cfg); }

}  // namespace cq

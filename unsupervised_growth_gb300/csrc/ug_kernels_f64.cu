// Double-precision kernels (the parity build).  Compiled with -fmad=false.
#define UG_DOUBLE_UNIT   // the double-precision launchers and their kernels belong to this unit alone
#include "ug_kernels_inst.cuh"

namespace ug {
template cudaError_t launch_trial_init<double>(const NetDev<double>&, const BatchDev<double>&, const LaunchCtx&);
template cudaError_t launch_interval<double>(const NetDev<double>&, const BatchDev<double>&, int, int, int,
                                             const RAStep<double>&, const IStep<double>&, const LaunchCtx&);
template cudaError_t launch_growth_reset<double>(const GrowthDev&, const LaunchCtx&);
template cudaError_t launch_growth_sync<double>(const GrowthDev&, const NetDev<double>&, const BatchDev<double>&, int, int, int,
                                             const LaunchCtx&, bool&);
template cudaError_t launch_growth_epilogue<double>(const GrowthDev&, const LaunchCtx&);
template cudaError_t launch_growth_remove<double>(const GrowthDev&, const int*, int, cudaStream_t);
template cudaError_t launch_check_bad<double>(const NetDev<double>&, const BatchDev<double>&, int*, cudaStream_t);
template cudaError_t epilogue_bulk_grid<double>(int, int, int*);
template cudaError_t growth_trial_plan<double>(int, int, int, int, GrowthPlan*);
template cudaError_t launch_growth_trial<double>(const GrowthDev&, const NetDev<double>&, BatchDev<double>, const RAStep<double>&,
                                              const IStep<double>&, const GrowthPlan&, const int*, int,
                                              unsigned long long*, int2*, cudaStream_t);
template cudaError_t launch_growth_head<double>(const TailDev<double>&, int*, cudaStream_t);
template cudaError_t launch_growth_tail<double>(const TailDev<double>&, cudaStream_t);
template cudaError_t group_grids<double>(GroupDev&, int, int);
template cudaError_t launch_group_trial<double>(const GroupDev&, const std::vector<int>&, int, bool, const LaunchCtx&,
                                                int64_t*);
template cudaError_t launch_state_init<double>(const NetDev<double>&, const BatchDev<double>&, cudaStream_t);
template cudaError_t launch_noise_segment<double>(const NetDev<double>&, const BatchDev<double>&, int, int, int, cudaStream_t);
template cudaError_t test_trial_plan<double>(int, int, int, TestPlan*);
template cudaError_t launch_test_trial<double>(const NetDev<double>&, const BatchDev<double>&, const RAStep<double>&,
                                            const IStep<double>&, const TestPlan&, const int*, int, int, int, unsigned*,
                                            cudaStream_t);

}  // namespace ug

// eval_f32.cu — the per-evaluation kernels in FP32.
#include "eval_kernels.cuh"

namespace llg {

template void fast_occupancy<float>(int, int, int, int, int*, int*, int*, int*, int*);
template FastCfg fast_config<float>(int, int);
template cudaError_t build_pass_tables<float>(void*, int, int, cudaStream_t);
template bool can_fuse<float>(const EvalSpec&, const EvalSpec&, const LaunchGeom&);
template cudaError_t launch_one<float>(int, const EvalSpec&, const LaunchGeom&, cudaStream_t, int*);
template cudaError_t launch_fused<float>(const EvalSpec&, const EvalSpec&, const LaunchGeom&, cudaStream_t, int*);
template cudaError_t prepare_eval_kernels<float>(size_t, size_t);

}  // namespace llg

// eval_f64.cu — the per-evaluation kernels in FP64.
#include "eval_kernels.cuh"

namespace llg {

template void fast_occupancy<double>(int, int, int, int, int*, int*, int*, int*, int*);
template FastCfg fast_config<double>(int, int);
template cudaError_t build_pass_tables<double>(void*, int, int, cudaStream_t);
template bool can_fuse<double>(const EvalSpec&, const EvalSpec&, const LaunchGeom&);
template cudaError_t launch_one<double>(int, const EvalSpec&, const LaunchGeom&, cudaStream_t, int*);
template cudaError_t launch_fused<double>(const EvalSpec&, const EvalSpec&, const LaunchGeom&, cudaStream_t, int*);
template cudaError_t prepare_eval_kernels<double>(size_t, size_t);

}  // namespace llg

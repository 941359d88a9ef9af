// mixture_simt_f64.cu — FP64 instantiation of the SIMT kernels (mixture_simt.cuh).
#include "mixture_simt.cuh"

namespace issm {

template int dispatch_simt<double>(const MixParams<double> &, cudaStream_t);

}  // namespace issm

// Explicit instantiation: register-blocked float32 inviscid Navier-Stokes stage kernels, COORD_CART.
#include "launch.cuh"
namespace fvm {
template cudaError_t launch_ns_strip_coord<COORD_CART>(int, int, NsStripSource&, int, int, cudaStream_t, int);
}

// k_ip012.cu -- single-instance kernels of the InnerProduct start that runs
// rounds 0-3 in two passes (bodies in ip012.cuh).
#include "ip012.cuh"

namespace effsc {

template <bool LSB>
__global__ void __launch_bounds__(TPB, 2) k_ip_r012(RoundArgs a) {
    chain_enter();
    ip012_body<LSB>(a, blockIdx.x, gridDim.x);
}
template <bool LSB>
__global__ void __launch_bounds__(TPB, 2) k_ip_r012m(RoundArgs a) {
    chain_enter();
    ip012_body<LSB, true>(a, blockIdx.x, gridDim.x);
}
template <bool LSB>
__global__ void __launch_bounds__(TPB, 2) k_ip_r3x(RoundArgs a) {
    chain_enter();
    ip3x_body<LSB>(a, blockIdx.x, gridDim.x);
}

bool launch_ip012_mirror(bool lsb, const RoundArgs& a, int grid, cudaStream_t s) {
    return lsb ? launch_chain(k_ip_r012m<true>, grid, TPB, 0, s, a) : launch_chain(k_ip_r012m<false>, grid, TPB, 0, s, a);
}
bool launch_ip012(bool lsb, const RoundArgs& a, int grid, cudaStream_t s) {
    return lsb ? launch_chain(k_ip_r012<true>, grid, TPB, 0, s, a) : launch_chain(k_ip_r012<false>, grid, TPB, 0, s, a);
}
bool launch_ip3x(bool lsb, bool copied, const RoundArgs& a, int grid, cudaStream_t s) {
    const bool dep = pdl_on(false) && !copied;
    return lsb ? launch_with(dep, k_ip_r3x<true>, grid, TPB, 0, s, a) : launch_with(dep, k_ip_r3x<false>, grid, TPB, 0, s, a);
}

}  // namespace effsc

// pp_ff_box10.cu -- force-field grids by boxes with 10 nodes per axis.
#include "pp_ff_box_kern.cuh"

namespace ppgpu {

int launch_ff_box10(const FFParams &prm, const BoxPrm &B, int mode, bool with_e, bool ortho, cudaStream_t st) {
    return launch_box_nodes<10>(prm, B, mode, with_e, ortho, st);
}

}  // namespace ppgpu

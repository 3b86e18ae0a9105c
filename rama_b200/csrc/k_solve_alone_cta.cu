// k_solve_alone_cta.cu -- one instance on one CTA, with the registers of a
// whole SM (see kernels.cuh).
#include "kernels.cuh"

using namespace rama;

__global__ void __launch_bounds__(THREADS, 1) k_solve_cta_alone(Instance *io)
{
    extern __shared__ __align__(16) char sm[];
    BlockTeam t;
    solve_instance(t, sm, make_scratch(io->ws, io->ws_bytes), io);
}

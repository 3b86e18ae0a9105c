// k_solve_alone_grid.cu -- one instance on a cooperative grid of one CTA per
// SM (see kernels.cuh).
#include "kernels.cuh"

using namespace rama;

__global__ void __launch_bounds__(THREADS, 1) k_solve_grid_alone(GridLaunch L)
{
    extern __shared__ __align__(16) char sm[];
    GridTeam t;
    solve_instance(t, sm, make_scratch(L.ws, L.ws_bytes), L.inst);
}

// mplb_table.cu -- instantiations of the fused steps on neighbour tables
// (fused_table.cuh), compiled without multiply-add contraction.
#include <cuda_runtime.h>

#include "fused_table.cuh"

using namespace mplb;

template <class L, int GM>
static void step(bool emit, bool st, const Params& P, const TableArgs& A, cudaStream_t s) {
    const unsigned nb = (P.n + 127) / 128;
    if (emit) {
        launch_step(k_table_finish<L, GM, true, false>, nb, 128, 0, s, P, A);
        return;
    }
    launch_step(k_table_sum<L, GM>, nb, 128, 0, s, P, A);
    if constexpr (GM == TABLE_MY) launch_step(k_table_heat<L>, nb, 128, 0, s, P, A);
    if (st) launch_step(k_table_finish<L, GM, false, true>, nb, 128, 0, s, P, A);
    else launch_step(k_table_finish<L, GM, false, false>, nb, 128, 0, s, P, A);
}

// One step (emit: the reference state after the last one); returns the launches made.
int mplb_table_step(int lat, int heat, bool emit, bool st, const Params& P, const TableArgs& A, cudaStream_t s) {
    if (lat == MPLB_D2Q9) {
        if (heat == TABLE_NONE) step<D2Q9T, TABLE_NONE>(emit, st, P, A, s);
        else if (heat == TABLE_LITEMP) step<D2Q9T, TABLE_LITEMP>(emit, st, P, A, s);
        else step<D2Q9T, TABLE_MY>(emit, st, P, A, s);
    } else {
        if (heat == TABLE_NONE) step<D3Q15T, TABLE_NONE>(emit, st, P, A, s);
        else step<D3Q15T, TABLE_MY>(emit, st, P, A, s);
    }
    return emit ? 1 : (heat == TABLE_MY ? 3 : 2);
}

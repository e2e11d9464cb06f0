// cg_plan_host.cu -- TEST HARNESS: the choice of the CG kernel by size
// (ucla_cmg_b200/csrc/cg_plan.cuh), compiled for the host.  Not part of the library.
#include "../../ucla_cmg_b200/csrc/cg_plan.cuh"

using namespace ep;

// 1: k_cn_smem with *ring_cols and *smem, 0: k_cn_half with *block threads, 2: k_cn_two;
// *grid 0: another plan of *per_sm CTAs per SM
extern "C" int cg_plan(int fp32, int ns, long long cols, int nslices, int ninst, int largest, int block, int grid, int per_sm,
                       int *out_block, int *ring_cols, int *smem, double *keep, int *out_grid, int *out_per_sm) {
    CgShape s{kSmemBatch, block, grid, per_sm, 0, 0, 1.0f};
    const bool yes = fp32 ? cg_fit<float>(ns, cols, nslices, ninst, largest, &s)
                          : cg_fit<double>(ns, cols, nslices, ninst, largest, &s);
    *out_block = s.block;
    *ring_cols = s.ring_cols;
    *smem = s.smem;
    *keep = s.keep;
    *out_grid = s.grid;
    *out_per_sm = s.per_sm;
    return yes ? (s.batch == kSmemBatch ? 1 : -1) : s.batch == 4 ? 0 : s.batch == kTwo + 4 ? 2 : -1;
}

// 1: a launch shape that the caller set runs k_cn_two
extern "C" int cg_named(int fp32, int batch, int block, int warps, int ninst, double mb) {
    return fp32 ? cg_named_two<float>(batch, block, warps, ninst, mb) : cg_named_two<double>(batch, block, warps, ninst, mb);
}

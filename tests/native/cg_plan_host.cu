// cg_plan_host.cu -- TEST HARNESS: the choice of the CG kernel by size
// (ucla_cmg_b200/csrc/cg_plan.cuh), compiled for the host.  Not part of the library.
#include "../../ucla_cmg_b200/csrc/cg_plan.cuh"

using namespace ep;

// 1: k_cn_smem with *ring_cols and *smem, 0: k_cn_half with *block threads
extern "C" int cg_plan(int fp32, int ns, long long cols, int nslices, int block, int grid, int per_sm, int *out_block,
                       int *ring_cols, int *smem, double *keep) {
    CgShape s{kSmemBatch, block, grid, per_sm, 0, 0, 1.0f};
    const bool yes = fp32 ? cg_fit<float>(ns, cols, nslices, &s) : cg_fit<double>(ns, cols, nslices, &s);
    *out_block = s.block;
    *ring_cols = s.ring_cols;
    *smem = s.smem;
    *keep = s.keep;
    return yes ? (s.batch == kSmemBatch ? 1 : -1) : (s.batch == 4 ? 0 : -1);
}

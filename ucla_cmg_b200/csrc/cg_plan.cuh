// cg_plan.cuh -- which CG kernel a planned launch runs, and k_cn_smem's shared
// memory: host arithmetic only.
#pragma once
#include <algorithm>

#include "common.cuh"

namespace ep {

// cg_batch value of the staged kernel (asynchronous copies of each warp's
// next units of SELL columns into shared memory)
constexpr int kStagedBatch = 32;
// the library's own choice (k_cn_smem; not a cg_batch value) and its shared memory at most
constexpr int kSmemBatch = 64;
// and of k_cn_one, the solve on one CTA
constexpr int kOneBatch = 65;
constexpr int kOneMax = 208 * 1024;
constexpr int kSmemMax = 216 * 1024;
constexpr int kUnit = 8, kUnitMax = 9;        // slice columns of a unit; a single left-over column joins the last
constexpr int kMaxUnits = 32;                 // units in a warp's ring, at most

// a launch whose shape is left to the library: kernel (batch), threads, CTAs
// and k_cn_smem's sizes (block: the asked size in, the launch's out)
struct CgShape { int batch, block, grid, per_sm, ring_cols, smem; float keep; };

// k_cn_smem: shared memory of a CTA with `cols` matrix columns per warp and ns
// slices at most
inline size_t smem_bytes(int block, int cols, int ns, int rsize) {
    return (size_t)(block / 32) * ((size_t)cols * kSlice * (4 + rsize) + kMaxUnits * 8) + ((size_t)ns + 1) * 4;
}

// The kernel for a matrix of `cols` columns in nslices slices, at most ns of them
// a CTA's, by the rule above cg_auto_shape: true with k_cn_smem's sizes, or
// k_cn_half in *out.  A CTA's slice bounds take shared memory too: where they
// leave a warp no ring of two units (from some 11000 slices a CTA in FP32, 1000
// in an FP64 batch's, whose large instance got few CTAs), k_cn_half, which needs
// none of it.
template <typename R>
bool cg_fit(int ns, long long cols, int nslices, CgShape *out) {
    const int warps = out->block / 32, spw = (ns + warps - 1) / warps, wide = (int)((cols + nslices - 1) / nslices);
    auto fit = [&](int kb) {
        const long long budget = (long long)kb * 1024 / out->per_sm - ((long long)ns + 1) * 4;
        return (int)((budget / warps - kMaxUnits * 8) / (kSlice * (4 + (int)sizeof(R))));
    };
    const int most = sizeof(R) == 4 ? 200 : 140;
    const bool stays = (long long)spw * wide <= fit(most);
    const double mb = (double)cols * kSlice * (4 + sizeof(R)) / 1e6;      // the matrix
    // a share that stays gets room for slices half as wide again
    out->ring_cols = (int)std::min<long long>(std::max<long long>((long long)spw * (wide + wide / 2), 2 * kUnitMax),
                                              fit(stays ? most : 120));
    // (a slice's gathers take up to two units of the ring at once)
    if ((!stays && mb <= (sizeof(R) == 8 && out->per_sm == 1 ? 27.0 : 60.0)) || out->ring_cols < 2 * kUnitMax) {
        out->batch = 4;
        out->block = 1024 / out->per_sm;
        out->ring_cols = 0;
        return false;
    }
    out->keep = mb <= 60.0 ? 1.0f : (float)(36.0 / mb);
    out->smem = (int)smem_bytes(out->block, out->ring_cols, ns, (int)sizeof(R));
    return true;
}

}  // namespace ep

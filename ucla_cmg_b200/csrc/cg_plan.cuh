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
// added to a gather width: k_cn_two, two passes an iteration
constexpr int kTwo = 128;
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

// Whether a launch shape that the caller set (gather width `batch`, threads a
// CTA, warps an SM) runs k_cn_two: a matrix of `mb` MB that streams from DRAM, and a
// shape that had more warps or wider gathers in flight before the one-pass sweep
// (CG us a step, k_cn_two / k_cn_half: FP32 2.2M nodes width 8 1917 / 2459, staged
// 1832 / 2445, 768 threads 2162 / 2672, but 0.8M 940 / 934 and width 4 with 32
// warps 2979 / 2357; FP64 2.2M width 8 3994 / 4627, staged 3545 / 4144, 768 threads
// 3640 / 4564, width 16 5158 / 4530; 100 instances of 1.8M nodes, width 4, 32 warps
// 2.0 / 2.0 ms in FP32, 3.0 / 3.2 in FP64).
template <typename R>
bool cg_named_two(int batch, int block, int warps, int ninst, double mb) {
    const bool one = ninst == 1;
    if (sizeof(R) == 4) return mb > (batch != 4 || block == 768 ? 85.0 : warps > 32 ? (one ? 300.0 : 200.0) : 1e30);
    if (batch != 4) return mb > (batch == 8 ? 140.0 : batch == kStagedBatch ? 180.0 : one ? 1e30 : 140.0);
    return mb > (block == 768 ? 130.0 : warps > 32 ? (one ? 150.0 : 130.0) : one ? 450.0 : 300.0);
}

// The kernel for a matrix of `cols` columns in nslices slices, `largest` of them
// the largest of ninst instances', at most ns a CTA's, by the rule above
// cg_auto_shape: true with k_cn_smem's sizes, or another kernel in *out (grid 0:
// as many CTAs as its per_sm, another plan).
//   A matrix that streams from DRAM on every sweep runs k_cn_two, with two CTAs of
// 768 threads an SM, or six of 256 where instances are many: CG us a step, one
// tissue FP32 2.2M nodes 2162 against 2018 from the ring, 3.2M 2979 / 3077, 5.5M
// 4910 / 5564; FP64 1.25M 2340 / 2006, 2.2M 3640 / 3763, 5.5M 8900 / 10020.  In
// batches sooner (4 slabs, 1.6M FP64 2455 / 2608; 10, 2.1M 3189 / 3725; 64, 1.2M
// 1702 / 1980, FP32 1195 / 1096; 100, 1.8M 2542 / 3410, FP32 1710 / 1826): the
// instances' CTAs are few then and their shares uneven, so with two CTAs per SM the
// size counts by the largest share.
//   A batch whose CTAs are fewer than four an instance, with an instance twice the
// mean, gets twice the CTAs of k_cn_half (250 slabs of 500 nodes and one of 98K,
// FP32 / FP64: 277 / 440 us against 577 / 984; and one of 5K: 189 / 287, 278 / 438).
//   A CTA's slice bounds take shared memory too: where they leave a warp no ring of
// two units (from some 11000 slices a CTA in FP32), k_cn_half, which needs none.
template <typename R>
bool cg_fit(int ns, long long cols, int nslices, int ninst, int largest, CgShape *out) {
    const int warps = out->block / 32, spw = (ns + warps - 1) / warps, wide = (int)((cols + nslices - 1) / nslices);
    auto fit = [&](int kb) {
        const long long budget = (long long)kb * 1024 / out->per_sm - ((long long)ns + 1) * 4;
        return (int)((budget / warps - kMaxUnits * 8) / (kSlice * (4 + (int)sizeof(R))));
    };
    const int most = sizeof(R) == 4 ? 200 : 140;
    const bool stays = (long long)spw * wide <= fit(most);
    const double mb = (double)cols * kSlice * (4 + sizeof(R)) / 1e6;      // the matrix
    if (mb <= 60.0 && out->grid < 4 * ninst && (long long)largest * ninst > 2ll * nslices) {
        out->batch = 4;
        out->block = 256;
        out->per_sm = 4;
        out->grid = 0;
        return false;
    }
    const double even = out->per_sm == 1 ? 1.0 : (double)ns * out->grid / nslices;         // 1: all shares alike
    const double stream = sizeof(R) == 4 ? (out->per_sm == 1 ? 390.0 : 260.0)
                                         : (ninst == 1 ? 350.0 : out->per_sm == 1 ? 250.0 : 150.0);
    if (mb * even > stream) {
        out->batch = kTwo + 4;
        out->per_sm = ninst <= 36 ? 2 : 6;
        out->block = 1536 / out->per_sm;
        out->grid = 0;
        return false;
    }
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

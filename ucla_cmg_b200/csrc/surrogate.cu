// surrogate.cu -- BF16 tensor-core (tcgen05) inference of the learned ionic
// step.
//
// Per tile of 128 nodes (one node = one TMEM lane):
//   1. features of the node (V, 18 states, I_stim, G_Ks, G_to, s-gate) ->
//      normalised -> BF16 row of the A operand in shared memory;
//   2. four layers: one elected thread issues tcgen05.mma (kind::f16, BF16 x
//      BF16 -> FP32 in TMEM, M = 128, N = 128 or 32, K = 16 per instruction)
//      with A = activations and B = the layer's weights, both resident in
//      shared memory as no-swizzle K-major core matrices, then
//      tcgen05.commit arrives on an mbarrier;
//   3. every warp reads its 32 TMEM lanes back (tcgen05.ld 32x32b), adds the
//      bias, applies tanh.approx and writes the next BF16 A operand;
//   4. the output layer's 19 values are de-normalised and added to the
//      node's state; nodes outside the training envelope (input box, fast
//      Na-gate product m^3 h, an active stimulus) are appended to a fallback
//      list that the plain FP32 kernel then runs.
// The weights (80 KB) are loaded once per CTA.  Every mbarrier wait is bounded;
// on timeout the CTA records the error, frees its TMEM and leaves.
//
// What bounds it: 384 tanh a node, 16 a clock and SM (66 us for 765K nodes), and
// the chain of a tile (row, four times barrier + MMA + commit + TMEM load, output),
// which several tiles in flight hide.  Biases, means and ranges are kernel
// parameters, so that they cost no load; one barrier a layer (each thread sees
// the commit itself); a layer's descriptors step by a constant; the next rows'
// loads go out under the output layer's MMA.  263K nodes: 92 us to 58 us.
#include <cuda_bf16.h>

#include "surrogate.cuh"
#include "tt_step.cuh"

namespace ep {

constexpr int OFF_W1 = 0;
constexpr int OFF_W2 = OFF_W1 + SG_W1 * 2;
constexpr int OFF_W3 = OFF_W2 + SG_W2 * 2;
constexpr int OFF_W4 = OFF_W3 + SG_W3 * 2;
constexpr int OFF_A = OFF_W4 + SG_W4 * 2;                 // 128 x 128 bf16
constexpr int OFF_MISC = OFF_A + SG_M * SG_H * 2;
constexpr int SG_SMEM = OFF_MISC + 64;
constexpr uint32_t SG_TMEM_COLS = 256;

__device__ __forceinline__ uint32_t smem_u32(const void *p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}

// UMMA shared-memory descriptor: no swizzle, K-major; lbo/sbo in bytes
__device__ __forceinline__ uint64_t umma_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
    return (uint64_t)((saddr >> 4) & 0x3FFFu) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
           ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46);
}

// instruction descriptor: BF16 x BF16 -> F32, both K-major
__host__ __device__ constexpr uint32_t idesc_bf16(int M, int N) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t *bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred P;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 P, [%1], %2;\n\t"
        "selp.b32 %0, 1, 0, P;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}

__device__ __forceinline__ void fence_proxy_async() {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_before() {
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}

__device__ __forceinline__ void tmem_alloc(uint32_t *holder, uint32_t ncols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(holder)),
                 "r"(ncols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}

__device__ __forceinline__ void umma_bf16(uint32_t d, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                          uint32_t accumulate) {
    const uint32_t z = 0;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n\t}"
        ::"r"(d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(z), "r"(z), "r"(z), "r"(z));
}

__device__ __forceinline__ void umma_commit(uint64_t *bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
                 : "memory");
}

// 32 consecutive FP32 columns of this thread's TMEM lane; the values are there
// after tmem_wait
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
          "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]),
          "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]),
          "=r"(r[30]), "=r"(r[31])
        : "r"(taddr));
}

// the loads issued so far have landed: r passes through, so that no use of it
// moves above the wait
__device__ __forceinline__ void tmem_wait(uint32_t (&r)[32]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int j = 0; j < 32; j++) asm volatile("" : "+r"(r[j]));
}

__device__ __forceinline__ float tanh_fast(float x) {
    float y;
    asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

__device__ __forceinline__ uint32_t pack_bf16(float a, float b) {
    __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<uint32_t *>(&v);
}

// one layer of K inputs and N outputs: D[128 x N] = A[128 x K] W^T, W = [N x K];
// one thread issues.  The descriptors' address fields count 16 bytes: 16 further
// is the next two 128-byte core matrices along K.
template <int K, int N>
__device__ __forceinline__ void issue_layer(uint32_t d, uint32_t sA, uint32_t sW, uint64_t *bar) {
    constexpr uint32_t sbo = (uint32_t)(K / 8) * 128u;
    const uint64_t da = umma_desc(sA, 128u, sbo), dw = umma_desc(sW, 128u, sbo);
#pragma unroll
    for (int kk = 0; kk < K / 16; kk++) umma_bf16(d, da + 16u * kk, dw + 16u * kk, idesc_bf16(SG_M, N), kk > 0 ? 1u : 0u);
    umma_commit(bar);
}

// hidden layer l's MMAs; the weights' images lie one behind the other
__device__ __forceinline__ void issue_hidden(int l, uint32_t d, uint32_t sA, uint32_t sW, uint64_t *bar) {
    tc_fence_after();
    if (l == 0) issue_layer<SG_KIN, SG_H>(d, sA, sW + OFF_W1, bar);
    else issue_layer<SG_H, SG_H>(d, sA, sW + (l == 1 ? OFF_W2 : OFF_W3), bar);
}

__device__ __forceinline__ void issue_output(uint32_t d, uint32_t sA, uint32_t sW, uint64_t *bar) {
    tc_fence_after();
    issue_layer<SG_H, SG_NOUT>(d, sA, sW + OFF_W4, bar);
}

// Each thread's bounded wait for the next commit, at most `polls` try-waits
// (0: kMbarPolls).  A thread that gives up sets the error, lets the MMAs in
// flight end (again bounded) and reports false; the caller carries that to its
// next barrier, where the whole group leaves.  A thread sees the commit itself,
// so no barrier follows the wait.
constexpr unsigned int kMbarPolls = 1u << 22;
__device__ __forceinline__ bool wait_commit(uint64_t *bar, uint32_t &phase, unsigned int *err, unsigned int polls) {
    bool ok = false;
    const unsigned int lim = polls ? polls : kMbarPolls;
    for (unsigned int it = 0; it < lim && !ok; it++) ok = mbar_try_wait(bar, phase);
    if (!ok) {
        atomicExch(err, 1u);
        for (unsigned int it = 0; it < kMbarPolls; it++)
            if (mbar_try_wait(bar, phase)) break;
    }
    phase ^= 1u;
    __syncwarp();
    tc_fence_after();
    return __all_sync(0xffffffffu, ok);
}

// Hidden layer l's epilogue: TMEM -> +bias -> tanh -> BF16 A row (K = 128
// layout) for columns [64 h, 64 h + 64) of row r.  Both 32-column loads go out
// before the first is used; the biases are kernel parameters, which an add
// reads as its constant operand.
__device__ __forceinline__ void hidden_epilogue(const SurrogateAux &x, int l, int h, uint32_t tmem_row,
                                                unsigned char *A, int r) {
    uint32_t v[2][32];
    tmem_ld32(tmem_row + 64u * h, v[0]);
    tmem_ld32(tmem_row + 64u * h + 32u, v[1]);
    const float *b = x.b[l] + 64 * h;
    tmem_wait(v[0]);
    tmem_wait(v[1]);
#pragma unroll
    for (int c = 0; c < 8; c++) {
        uint32_t w[4];
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int k = 8 * c + 2 * j;
            w[j] = pack_bf16(tanh_fast(__uint_as_float(v[k >> 5][k & 31]) + b[k]),
                             tanh_fast(__uint_as_float(v[k >> 5][(k & 31) + 1]) + b[k + 1]));
        }
        uint4 *dst = (uint4 *)(A + ((r >> 3) * (SG_H / 8) + 8 * h + c) * 128 + (r & 7) * 16);
        *dst = make_uint4(w[0], w[1], w[2], w[3]);
    }
}

// One node's input features (V, 18 states, I_stim, G_Ks, G_to, s-gate), or its
// 32 raw inputs: the loads alone, so that they can be in flight before they
// are used.  x[19] is the stimulus.
__device__ __forceinline__ void load_row(const SurrogateArgs &a, long long step, bool raw, int i, bool valid,
                                         float (&x)[SG_KIN]) {
#pragma unroll
    for (int k = 0; k < SG_KIN; k++) x[k] = 0.f;
    if (valid && raw) {
#pragma unroll
        for (int k = 0; k < SG_KIN; k++) x[k] = a.rawX[(size_t)i * SG_KIN + k];
    } else if (valid) {
        const int ty = a.type ? a.type[i] : 0;
        int q = a.stim_head ? a.stim_head[i] : -1;
        const float gks = a.gks ? a.gks[i] : 1.f;
        x[0] = a.V[i];
#pragma unroll
        for (int k = 0; k < 18; k++) x[k + 1] = a.S[(size_t)k * a.pitch + i];
        const float *c = a.consts + (size_t)ty * a.nconst;
        x[20] = c[15] * gks;
        x[21] = c[20];
        x[22] = c[53];
        long long best = -1;
        while (q >= 0) {
            const long long on = a.stim_on[q], off = a.stim_off[q];
            if (step >= on && step < off && on > best) { best = on; x[19] = a.stim_amp[q]; }
            q = a.stim_next[q];
        }
    }
}

// The row's BF16 form in A (K = 32 layout): logarithms of the wide-range
// features, normalisation; returns whether the node is inside the training
// envelope.
__device__ __forceinline__ bool store_row(const SurrogateArgs &a, bool raw, bool valid, float (&x)[SG_KIN], int row,
                                          unsigned char *A) {
    bool inside = false;
    if (valid && !raw) {
        inside = (x[19] == 0.f);
        x[19] = x[19] / (a.Cm * a.Xi);
        const float m = x[7], h = x[8];
        inside = inside && (m * m * m * h <= a.aux.nah_max);
        const unsigned int lm = a.aux.log_mask;
#pragma unroll
        for (int k = 0; k < SG_NF; k++) {
            // quantities spanning decades enter as logarithms
            const float xt = ((lm >> k) & 1u) ? __logf(fmaxf(x[k], 1e-30f)) : x[k];
            inside = inside && (xt >= a.aux.env_lo[k]) && (xt <= a.aux.env_hi[k]);
            x[k] = (xt - a.aux.in_mean[k]) * a.aux.in_rstd[k];
        }
    }
#pragma unroll
    for (int c = 0; c < 4; c++) {
        uint4 *dst = (uint4 *)(A + ((row >> 3) * (SG_KIN / 8) + c) * 128 + (row & 7) * 16);
        *dst = make_uint4(pack_bf16(x[8 * c], x[8 * c + 1]), pack_bf16(x[8 * c + 2], x[8 * c + 3]),
                          pack_bf16(x[8 * c + 4], x[8 * c + 5]), pack_bf16(x[8 * c + 6], x[8 * c + 7]));
    }
    return inside;
}

// One node's share of the output stage: the network's de-normalised
// changes applied (or, in the hybrid form, its six concentrations handed to
// k_hybrid), and the nodes outside the envelope or with an output outside
// its training range appended to the fallback list.  yv: the node's 32
// output-layer accumulators (bias not yet added).
__device__ __forceinline__ void output_node(const SurrogateArgs &a, int i, bool valid,
                                            bool raw, bool inside, const uint32_t (&yv)[32], double t0,
                                            unsigned int &my_fb) {
    const SurrogateAux &x = a.aux;
    if (valid && raw) {
#pragma unroll
        for (int j = 0; j < SG_NOUT; j++) a.rawY[(size_t)i * SG_NOUT + j] = __uint_as_float(yv[j]) + x.b[3][j];
    } else if (valid) {
        // the six concentrations the hybrid form replaces, loaded before
        // any store of this node (the stores below could alias them for
        // the compiler, which would otherwise serialise load and store)
        const int cslot[6] = {0, 1, 2, 9, 16, 17};
        float xs[6];
        if (x.v_update == 2) {
#pragma unroll
            for (int j = 0; j < 6; j++) xs[j] = a.S[(size_t)cslot[j] * a.pitch + i];
        }
        // de-normalise; a used output outside the range seen in training
        // sends the node to the plain model as well
        float d[SG_NY];
        bool out_ok = inside;
#pragma unroll
        for (int j = 0; j < SG_NY; j++) {
            // only the outputs the update reads (out_mask: the six concentrations
            // in the hybrid form, every output otherwise) are range-checked and
            // mapped back; the others are never read
            d[j] = 0.f;
            if ((x.out_mask >> j) & 1u) {
                const float u = (__uint_as_float(yv[j]) + x.b[3][j]) * x.out_std[j] + x.out_mean[j];
                out_ok = out_ok && (u >= x.out_lo[j]) && (u <= x.out_hi[j]);
                const float sc = x.out_scale[j];
                d[j] = sc > 0.f ? sc * sinhf(fminf(fmaxf(u, -80.f), 80.f)) : u;
            }
        }
        const unsigned int lm = x.log_mask;
        if (x.v_update == 2) a.take[i] = out_ok ? 1 : 0;
        if (!out_ok) {
            const int slot = atomicAdd(a.fallback_count, 1);
            a.fallback_list[slot] = i;
            my_fb++;
        } else if (x.v_update == 2) {
            // the new concentrations; k_hybrid advances gates and V
#pragma unroll
            for (int j = 0; j < 6; j++) {
                const int q = cslot[j];
                a.pred[(size_t)j * a.pitch + i] =
                    ((lm >> (q + 1)) & 1u) ? xs[j] * __expf(d[q + 1]) : xs[j] + d[q + 1];
            }
        } else {
            // every quantity from the network (all loads before the stores)
            float xk[18];
#pragma unroll
            for (int k = 0; k < 18; k++) xk[k] = a.S[(size_t)k * a.pitch + i];
#pragma unroll
            for (int k = 0; k < 18; k++) {
                // log-scaled states are updated multiplicatively: x' = x exp(d)
                a.S[(size_t)k * a.pitch + i] = ((lm >> (k + 1)) & 1u) ? xk[k] * __expf(d[k + 1]) : xk[k] + d[k + 1];
            }
            const float V0 = a.V[i], V1 = V0 + d[0];
            a.V[i] = V1;
            if (a.track) {
                Track tr = a.track[i];
                if (tr.t_rep < 0.f) {
                    bool dirty = false;
                    track_interval(tr, dirty, V0, V1, t0, (float)a.t_per_step, a.act_thr);
                    if (dirty) a.track[i] = tr;
                }
            }
        }
    }
}

// the weights' global image -> shared memory (already in core-matrix order)
__device__ __forceinline__ void load_weights(const SurrogateArgs &a, unsigned char *smem) {
    const uint4 *src = (const uint4 *)a.wimg;
    uint4 *dst = (uint4 *)smem;
    for (int k = threadIdx.x; k < SG_WTOT * 2 / 16; k += blockDim.x) dst[k] = __ldg(src + k);
}

// One tile of 128 nodes per CTA, for the sizes where a tile's chain is all there
// is: its eight warps share the hidden epilogues (warp w reads TMEM lane quarter
// w % 4, column half w / 4); threads 0..127 own one node each (features, the
// output layer, the envelope decision).
__global__ void __launch_bounds__(SG_THREADS, 1) k_surrogate(const __grid_constant__ SurrogateArgs a) {
    extern __shared__ __align__(1024) unsigned char smem[];
    const int tid = threadIdx.x, warp = tid >> 5;
    const int row = tid & (SG_M - 1), half = tid >> 7;
    const bool owner = half == 0;                 // warp-uniform
    uint64_t *bar = (uint64_t *)(smem + OFF_MISC);
    uint32_t *holder = (uint32_t *)(smem + OFF_MISC + 16);
    unsigned char *A = smem + OFF_A;
    const bool raw = a.rawX != nullptr;
    const long long step = raw ? 0 : *a.step_ptr;
    const double t0 = (double)step * a.t_per_step;
    const int i = (int)blockIdx.x * SG_M + row;
    const bool valid = owner && i < a.n;

    float x[SG_KIN];
    if (owner) load_row(a, step, raw, i, valid, x);
    load_weights(a, smem);
    if (tid == 0) mbar_init(bar, 1);
    if (warp == 0) tmem_alloc(holder, SG_TMEM_COLS);
    const bool inside = owner && store_row(a, raw, valid, x, row, A);
    fence_proxy_async();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *holder;
    const uint32_t lane_off = (uint32_t)(32 * (warp & 3)) << 16;
    const uint32_t d_hid = tmem, d_out = tmem + 128u;
    const uint32_t sW = smem_u32(smem), sA = smem_u32(A);
    uint32_t phase = 0;
    unsigned int my_fb = 0;
    bool ok = true;
    // A is complete: the next layer's MMAs may go out (false: a wait gave up)
    auto ready = [&]() -> bool {
        fence_proxy_async();
        tc_fence_before();
        return !__syncthreads_or(!ok);
    };
#pragma unroll 1
    for (int l = 0; l < 3 && ready(); l++) {
        if (tid == 0) issue_hidden(l, d_hid, sA, sW, bar);
        ok = wait_commit(bar, phase, a.err, a.mbar_polls);
        if (ok) hidden_epilogue(a.aux, l, half, d_hid + lane_off, A, row);
    }
    if (ready()) {
        if (tid == 0) issue_output(d_out, sA, sW, bar);
        ok = wait_commit(bar, phase, a.err, a.mbar_polls);
        if (ok && owner) {
            uint32_t yv[32];
            tmem_ld32(d_out + lane_off, yv);
            tmem_wait(yv);
            output_node(a, i, valid, raw, inside, yv, t0, my_fb);
        }
    }
    // count fallback node-steps
    for (int o = 16; o > 0; o >>= 1) my_fb += __shfl_xor_sync(0xffffffffu, my_fb, o);
    if ((tid & 31) == 0 && my_fb && a.status) atomicAdd(&a.status->fallback, (unsigned long long)my_fb);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 0) tmem_dealloc(tmem, SG_TMEM_COLS);
}

// ---------------------------------------------------------------------------
// The same network with four tile pipelines in one CTA per SM (512 threads =
// four warpgroups).  Warpgroup g owns slot g: an A buffer of its own, TMEM
// columns [128 g, 128 g + 128) (the output layer reuses the first 32 once the
// last hidden epilogue has read them), an mbarrier and a named barrier; it
// runs its tiles start to end -- row build, four MMA layers, output --
// while the other three do the same, so four tiles' chains are in flight per
// SM with one copy of the weights (80 KB).  Each thread owns one node of its slot's tile and its whole row in
// the hidden epilogues.  Same instructions per tile, same results.
constexpr int SG4_SLOTS = 4;
constexpr int SG4_THREADS = SG4_SLOTS * SG_M;
constexpr int OFF4_A = OFF_W4 + SG_W4 * 2;
constexpr int OFF4_MISC = OFF4_A + SG4_SLOTS * SG_M * SG_H * 2;
constexpr int SG4_SMEM = OFF4_MISC + 128;
constexpr uint32_t SG4_TMEM_COLS = 512;

// whether any of a warpgroup's 128 threads says so: a barrier (named `id`) too
__device__ __forceinline__ bool wg_any(bool pred, int id) {
    uint32_t r;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.u32 p, %1, 0;\n\t"
        "bar.red.or.pred q, %2, 128, p;\n\t"
        "selp.u32 %0, 1, 0, q;\n\t}"
        : "=r"(r)
        : "r"((uint32_t)pred), "r"(id)
        : "memory");
    return r != 0;
}

__global__ void __launch_bounds__(SG4_THREADS, 1) k_surrogate4(const __grid_constant__ SurrogateArgs a) {
    extern __shared__ __align__(1024) unsigned char smem[];
    const int tid = threadIdx.x, warp = tid >> 5;
    const int g = tid >> 7, row = tid & (SG_M - 1);
    const int bid = 1 + g;                        // named barrier of this warpgroup
    uint64_t *bars = (uint64_t *)(smem + OFF4_MISC);
    uint32_t *holder = (uint32_t *)(smem + OFF4_MISC + 64);
    unsigned char *A = smem + OFF4_A + (size_t)g * SG_M * SG_H * 2;
    const bool raw = a.rawX != nullptr;
    const long long step = raw ? 0 : *a.step_ptr;
    const double t0 = (double)step * a.t_per_step;
    const int ntiles = (a.n + SG_M - 1) / SG_M;
    // a CTA's slots take tiles a grid apart, so that the last tiles spread over
    // the SMs instead of filling the slots of a few
    const int first = (int)blockIdx.x + (int)gridDim.x * g, stride = (int)gridDim.x * SG4_SLOTS;
    float x[SG_KIN];
    bool inside = false;
    load_row(a, step, raw, first * SG_M + row, first * SG_M + row < a.n, x);
    load_weights(a, smem);
    if (tid == 0)
        for (int k = 0; k < SG4_SLOTS; k++) mbar_init(bars + k, 1);
    if (warp == 0) tmem_alloc(holder, SG4_TMEM_COLS);
    inside = store_row(a, raw, first * SG_M + row < a.n, x, row, A);
    fence_proxy_async();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *holder;
    const uint32_t lane_off = (uint32_t)(32 * (warp & 3)) << 16;
    const uint32_t d_acc = tmem + 128u * (uint32_t)g;
    const uint32_t sW = smem_u32(smem);
    const uint32_t sA = smem_u32(A);
    uint64_t *bar = bars + g;
    uint32_t phase = 0;
    unsigned int my_fb = 0;
    bool ok = true;
    auto ready = [&]() -> bool {
        fence_proxy_async();
        tc_fence_before();
        return !wg_any(!ok, bid);
    };
    for (int tile = first; tile < ntiles; tile += stride) {
        const int i = tile * SG_M + row, i1 = (tile + stride) * SG_M + row;
#pragma unroll 1
        for (int l = 0; l < 3 && ready(); l++) {
            if (row == 0) issue_hidden(l, d_acc, sA, sW, bar);
            ok = wait_commit(bar, phase, a.err, a.mbar_polls);
#pragma unroll 1
            for (int h = 0; h < 2 && ok; h++) hidden_epilogue(a.aux, l, h, d_acc + lane_off, A, row);
        }
        if (!ready()) break;
        if (row == 0) issue_output(d_acc, sA, sW, bar);
        // the next tile's rows are loaded under the output layer's MMA
        load_row(a, step, raw, i1, i1 < a.n, x);
        ok = wait_commit(bar, phase, a.err, a.mbar_polls);
        if (!ok) continue;
        uint32_t yv[32];
        tmem_ld32(d_acc + lane_off, yv);
        tmem_wait(yv);
        tc_fence_before();
        output_node(a, i, i < a.n, raw, inside, yv, t0, my_fb);
        // the output layer's MMA has read A; the next MMA overwrites the
        // accumulator after the barrier in front of it
        inside = store_row(a, raw, i1 < a.n, x, row, A);
    }
    for (int o = 16; o > 0; o >>= 1) my_fb += __shfl_xor_sync(0xffffffffu, my_fb, o);
    if ((tid & 31) == 0 && my_fb && a.status) atomicAdd(&a.status->fallback, (unsigned long long)my_fb);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 0) tmem_dealloc(tmem, SG4_TMEM_COLS);
}

// The hybrid form's physics for the nodes the network took: the reference's
// gate update and current balance over the sub-steps, with the six
// concentrations moving from their start to the network's end values
// (geometrically for the log-scaled Cai and Cass).  One thread per node.
__global__ void __launch_bounds__(128, 4) k_hybrid(const __grid_constant__ SurrogateArgs a) {
    const SurrogateAux &x = a.aux;
    const long long step = *a.step_ptr;
    const double t0 = (double)step * a.t_per_step;
    const unsigned int lm = x.log_mask;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < a.n; i += gridDim.x * blockDim.x) {
        if (!a.take[i]) continue;
        float s[18], c0[6], c1[6];
#pragma unroll
        for (int k = 0; k < 18; k++) s[k] = a.S[(size_t)k * a.pitch + i];
        const int cslot[6] = {0, 1, 2, 9, 16, 17};
#pragma unroll
        for (int j = 0; j < 6; j++) {
            c0[j] = s[cslot[j]];
            c1[j] = a.pred[(size_t)j * a.pitch + i];
        }
        const int ty = a.type ? a.type[i] : 0;
        const float *c = a.consts + (size_t)ty * a.nconst;
        const float gks_i = a.gks ? a.gks[i] : 1.f;
        Track tr = {-1.f, -1.f, -1.f, 1e30f};
        bool dirty = false;
        const bool trk = a.track != nullptr;
        if (trk) tr = a.track[i];
        const int ns = x.hyb_sub > 0 ? x.hyb_sub : a.nsub;
        const float hu = (float)a.t_per_step / (float)ns;
        const float rdt = 1.f / (float)a.t_per_step;
        float V = a.V[i], tsum = 0.f;
        double tsub = t0;
        for (int k = 0; k < ns; k++) {
            const float h = x.hyb_sub > 0 ? hu : a.sub_dt[k];
            tts::tt_gate_step(s, V, h, c);
            tsum += h;
            const float w = fminf(tsum * rdt, 1.f);
#pragma unroll
            for (int j = 0; j < 6; j++) {
                const int q = cslot[j];
                s[q] = ((lm >> (q + 1)) & 1u) ? c0[j] * __powf(c1[j] / c0[j], w) : c0[j] + w * (c1[j] - c0[j]);
            }
            const float v1 = V + h * tts::tt_dvdt<float>(V, s, c, 0.f, gks_i);
            if (trk && tr.t_rep < 0.f) track_interval(tr, dirty, V, v1, tsub, h, a.act_thr);
            V = v1;
            tsub += (double)h;
        }
#pragma unroll
        for (int k = 0; k < 18; k++) a.S[(size_t)k * a.pitch + i] = s[k];
        a.V[i] = V;
        if (dirty) a.track[i] = tr;
    }
}

// variant 0: the faster kernel for the size.  Up to one tile an SM a tile's
// chain is all there is, and it is shorter in k_surrogate, where eight warps
// share an epilogue (1.5 us of 40 a step at 1.5K-10K nodes, equal at 19K);
// beyond, chains in flight count: against two CTAs an SM of one chain each, four
// chains took the ionic phase of 46K nodes from 51.8 to 47.6 us, of 263K from
// 106 to 91, of 765K from 222 to 193.  1: k_surrogate4 at every size.
int launch_surrogate(const SurrogateArgs &a, cudaStream_t s, int variant) {
    int dev = 0, nsm = 148;
    EP_CUDA(cudaGetDevice(&dev));
    EP_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
    const int ntiles = (a.n + SG_M - 1) / SG_M;
    if (ntiles <= 0) return EP_OK;
    // the shared-memory limit is per kernel and per device; setting it again
    // is cheap and keeps a second device right
    if (variant == 1 || ntiles > nsm) {
        EP_CUDA(cudaFuncSetAttribute(k_surrogate4, cudaFuncAttributeMaxDynamicSharedMemorySize, SG4_SMEM));
        k_surrogate4<<<ntiles < nsm ? ntiles : nsm, SG4_THREADS, SG4_SMEM, s>>>(a);
    } else {
        EP_CUDA(cudaFuncSetAttribute(k_surrogate, cudaFuncAttributeMaxDynamicSharedMemorySize, SG_SMEM));
        k_surrogate<<<ntiles, SG_THREADS, SG_SMEM, s>>>(a);
    }
    EP_CUDA(cudaGetLastError());
    return EP_OK;
}

int launch_hybrid(const SurrogateArgs &a, cudaStream_t s) {
    if (a.n <= 0) return EP_OK;
    k_hybrid<<<(a.n + 127) / 128, 128, 0, s>>>(a);
    EP_CUDA(cudaGetLastError());
    return EP_OK;
}

}  // namespace ep

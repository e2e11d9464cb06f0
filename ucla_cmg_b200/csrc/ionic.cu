// ionic.cu -- the ionic phase of one split step, one thread per node.
//
// Each thread loads its node's state once (SoA, coalesced), runs all ionic
// sub-steps of the global step in registers -- Compute_Ion followed by the
// lumped-capacitance update V <- V + h dV/dt of EP_CrankNicholson.cc:124-133
// -- applies its stimulus window, tracks activation/repolarisation, and
// writes the state back once.
#include <algorithm>

#include "kernels.cuh"

namespace ep {

template <typename R>
__device__ __forceinline__ R node_istim(const IonicArgs<R> &a, int i, long long step) {
    if (a.istim) return a.istim[i];
    if (a.stim_head == nullptr) return R(0);
    int k = a.stim_head[i];
    long long best_on = -1;
    R amp = R(0);
    while (k >= 0) {
        const long long on = a.stim_on[k], off = a.stim_off[k];
        if (step >= on && step < off && on > best_on) { best_on = on; amp = a.stim_amp[k]; }
        k = a.stim_next[k];
    }
    return amp;
}

template <typename R>
__device__ __forceinline__ void track_update(Track &tr, bool &dirty, R v0, R v1, double t0, R h, R thr) {
    track_interval(tr, dirty, (float)v0, (float)v1, t0, (float)h, (float)thr);
}

template <int P> struct Part {
    static constexpr int value = P;
};

// the ten Tusscher kernel in the reference's order of operations (tt.cuh),
// apart from EP_TUSSCHER's own (tt_step.cuh), so that neither carries the
// other's registers
constexpr int kTusscherRef = 100 + EP_TUSSCHER;

// The sub-step lengths of one global step: the fixed sequence sub_dt, or
// (stride) the per-node sequence of CardiacBody::getVoltageFromIonicCurrent
// (Body/CardiacBody.cc:819-904): one sub-step of stride_dt; when its rate
// truncates to the integer 0 the stride grows fivefold; sub-steps then
// fill the global step, the last one shortened to end on it.
template <typename R> struct SubSteps {
    R dT, h, totT = R(0), hs;
    bool multi, more = true;
    int k = 0, kmax;
    __device__ __forceinline__ explicit SubSteps(const IonicArgs<R> &a) {
        dT = (R)a.t_per_step;
        multi = a.stride && dT / a.stride_dt > R(1);
        kmax = a.stride ? (multi ? (int)(dT / a.stride_dt) + 3 : 1) : a.nsub;
        h = a.stride ? a.stride_dt : a.sub_dt[0];
        hs = a.stride_dt;
    }
    // sets h to the next sub-step's length; false: the step is done
    __device__ __forceinline__ bool next(const IonicArgs<R> &a) {
        if (k >= kmax || !more) return false;
        if (!a.stride) {
            h = a.sub_dt[k];
            more = k + 1 < a.nsub;
        } else if (k == 0) {
            h = a.stride_dt;
            more = multi;
        } else {
            more = !(totT + hs > dT);
            h = more ? hs : dT - totT;
        }
        return true;
    }
    __device__ __forceinline__ void took(const IonicArgs<R> &a, R dvdt) {
        if (a.stride) {
            totT += h;
            if (k == 0) {
                const int slope = (fabs((double)dvdt) < 2.0e9) ? (int)dvdt : 1;
                if (!slope) hs *= R(5);
            }
        }
        k++;
    }
};

// one node's ionic phase (all sub-steps), counters accumulated by the caller.
// False (Mahajan without TEN only): a sub-step wants to be redone in ten, which is
// left to a second pass; nothing of the node is changed.
template <typename R, int MODEL, int NS, bool TEN = false>
__device__ __forceinline__ bool ionic_node(const IonicArgs<R> &a, const int i, unsigned int &my_newton,
                                           unsigned int &my_caps, unsigned int &my_bad) {
    const long long step = *a.step_ptr;
    const double t_start = (double)step * a.t_per_step;
    R V = a.V[i];
    R s[NS + 1];
#pragma unroll
    for (int k = 0; k < NS; k++) s[k + 1] = a.S[(size_t)k * a.pitch + i];
    const int ty = a.type ? a.type[i] : 0;
    const R istim = node_istim(a, i, step);
    Track tr = {-1.f, -1.f, -1.f, 1e30f};
    bool dirty = false;
    if (a.track) tr = a.track[i];
    const bool do_track = a.track != nullptr && tr.t_rep < 0.f;
    double tsub = t_start;
    R last = R(0);
    // one loop with one Compute_Ion call site, so the model code is inlined once
    SubSteps<R> sub(a);
    while (sub.next(a)) {
        const R h = sub.h;
        R dvdt;
        if constexpr (MODEL == EP_TUSSCHER || MODEL == kTusscherRef) {
            const R *__restrict__ c = a.consts + (size_t)ty * a.nconst;
            const R gks = a.gks ? a.gks[i] : R(1);
            const R ist = -istim / (a.Cm * a.Xi);
            int it = 0;
            if constexpr (MODEL == EP_TUSSCHER) dvdt = tts::tt_compute_ion<R>(s + 1, V, ist, h, c, gks, a.tt, it);
            else dvdt = tt_compute_ion<R>(s + 1, V, ist, h, c, gks, a.tt, it);
            my_newton += it;
            if (it >= a.tt.newton_cap) my_caps++;
        } else if constexpr (MODEL == EP_MAHAJAN || MODEL == EP_MAHAJAN_FAIL) {
            const R *__restrict__ c = a.consts + (size_t)ty * a.nconst;
            R r[26];
            s[0] = V;
            // TEN: one call site for all evaluations; a single sub-step is known to
            // want ten, its first one is skipped
            bool ten = TEN && !a.stride && a.nsub == 1;
            R he = ten ? h / R(10) : h;
            if (ten) my_newton++;
#pragma unroll 1
            for (int e = ten ? 1 : 0; e <= (TEN ? 10 : 0); e++) {
                mh_rhs(s, c, he, istim / (a.Cm * a.Xi), r);
                dvdt = r[0];
                if (e == 0 && mh_wants_substeps(dvdt, a.mh_abs)) {
                    if (!TEN) return false;
                    my_newton++;
                    ten = true;
                    he = h / R(10);
                    continue;
                }
#pragma unroll
                for (int j = 0; j < 26; j++) s[j] += r[j] * he;
                if (!ten) break;
            }
        } else if constexpr (MODEL == EP_PURKINJE) {
            // the stimulus in uA/cm^3 and the model's (or the user's) Xi;
            // C_m does not enter (Purkinje.cc:183-213)
            const R *__restrict__ c = a.consts + (size_t)ty * a.nconst;
            int ten = 0;
            dvdt = pk_compute_ion<R>(s, V, istim, a.Xi, h, c, ten);
            my_newton += ten;
        } else {
            dvdt = lr_compute_ion<R>(s + 1, V, istim, a.Cm, h, a.lr_table);
        }
        last = dvdt;
        const R v1 = V + h * dvdt;
        if (do_track) track_update(tr, dirty, V, v1, tsub, h, a.act_thr);
        V = v1;
        tsub += (double)h;
        sub.took(a, dvdt);
    }
    if (!isfinite((double)V)) my_bad = 1;
    if (a.dvdt_out) a.dvdt_out[i] = last;
    else a.V[i] = V;
#pragma unroll
    for (int k = 0; k < NS; k++) a.S[(size_t)k * a.pitch + i] = s[k + 1];
    if (dirty) a.track[i] = tr;
    return true;
}

// counters: one atomic per block
__device__ __forceinline__ void ionic_status(DevStatus *status, unsigned int my_newton, unsigned int my_caps,
                                             unsigned int my_bad, unsigned long long &s_newton, unsigned int &s_caps,
                                             unsigned int &s_bad) {
    for (int o = 16; o > 0; o >>= 1) {
        my_newton += __shfl_xor_sync(0xffffffffu, my_newton, o);
        my_caps += __shfl_xor_sync(0xffffffffu, my_caps, o);
        my_bad += __shfl_xor_sync(0xffffffffu, my_bad, o);
    }
    if ((threadIdx.x & 31) == 0) {
        if (my_newton) atomicAdd(&s_newton, (unsigned long long)my_newton);
        if (my_caps) atomicAdd(&s_caps, my_caps);
        if (my_bad) atomicAdd(&s_bad, my_bad);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        if (s_newton) atomicAdd(&status->newton_iters, s_newton);
        if (s_caps) atomicAdd(&status->newton_cap_hits, s_caps);
        if (s_bad) atomicAdd(&status->nonfinite, s_bad);
    }
}

// Mahajan.  The steep nodes (|dV/dt| > 20: an upstroke's, 2 % of the nodes in a
// wave but in a third of its warps) redo the sub-step in ten, eleven evaluations
// of the rates one behind the other.  A CTA therefore runs several chunks of 128
// nodes and puts their steep nodes aside, then takes these in groups of 32, one
// lane a node and each of the four warps one part of the rates (mh_part).
// 214K nodes: 123 us a step to 41.  Bound by the latency of one evaluation's chain
// for every chunk of the CTA, then ten parts' chains (some 20 us).
// FP64 takes a list of more than two groups one thread a node: 128 nodes cost 105 us
// (140 with two CTAs an SM), a group 45 (87), since its four parts are uneven and each
// forms the logarithms and reciprocals that they share.  (A front along the node order,
// 2 / 25 % of 67K nodes: 197 / 341 us a step in groups, 137 / 139 so; of 529K: 511 /
// 1465, 338 / 745; in FP32 groups are never the slower ones: 128 nodes 55 us either way.)
// The whole list by its length, so that a run repeats to the bit; the two ways differ
// in the rounding of the compiler's fused products.
constexpr int kMhChunks = 8;                     // chunks put aside together, at most
constexpr int kMhMany = 65;
template <typename R> struct MhShared {
    int list[kMhChunks * 128], count;
    R s[26][32];                                 // the group's states ([0] and [19] are registers)
    R ex[9][32];                                 // MhExchange
};

// `node`'s whole ionic phase by lane `lane` of all four warps (off: no node,
// the lane only keeps the others company)
template <typename R>
__device__ __forceinline__ void mh_group(const IonicArgs<R> &a, MhShared<R> &sh, const int i, const bool on,
                                         unsigned int &my_newton, unsigned int &my_bad) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const long long step = *a.step_ptr;
    const R *__restrict__ c = a.consts + (size_t)(a.type ? a.type[i] : 0) * a.nconst;
    R V = a.V[i], nai = a.S[(size_t)18 * a.pitch + i];
    for (int k = warp; k < MH_NS; k += 4) sh.s[k + 1][lane] = a.S[(size_t)k * a.pitch + i];
    const R ist = node_istim(a, i, step) / (a.Cm * a.Xi);
    Track tr = {-1.f, -1.f, -1.f, 1e30f};
    bool dirty = false;
    if (a.track) tr = a.track[i];
    const bool do_track = a.track != nullptr && tr.t_rep < 0.f;
    double tsub = (double)step * a.t_per_step;
    R last = R(0);
    // a single sub-step is known to want ten: its first evaluation is skipped
    const bool single = !a.stride && a.nsub == 1;
    SubSteps<R> sub(a);
    __syncthreads();
    for (;;) {
        const bool act = sub.next(a) && on;
        if (!__syncthreads_or(act)) break;
        const R h = sub.h, h10 = h / R(10);
        R sv = V;
        bool ten = act;
#pragma unroll 1
        for (int e = single ? 1 : 0; e <= 10; e++) {
            const R he = e ? h10 : h;
            R s[26], r[26];
            MhExchange<R> x;
            MhOwn<R> own;
            s[0] = sv;
#pragma unroll
            for (int k = 1; k < 26; k++) s[k] = sh.s[k][lane];
            s[19] = nai;
            if (warp == 0) {
                mh_part<0>(s, c, he, r, x, own);
                sh.ex[0][lane] = x.xina;
            } else if (warp == 1) {
                mh_part<1>(s, c, he, r, x, own);
                sh.ex[1][lane] = x.po; sh.ex[2][lane] = x.rxa; sh.ex[3][lane] = x.xikr;
            } else if (warp == 2) {
                mh_part<2>(s, c, he, r, x, own);
                sh.ex[4][lane] = x.xik1; sh.ex[5][lane] = x.xito; sh.ex[6][lane] = x.xinak;
            } else {
                mh_part<3>(s, c, he, r, x, own);
                sh.ex[7][lane] = x.xiks; sh.ex[8][lane] = x.jnaca;
            }
            __syncthreads();
            x.xina = sh.ex[0][lane]; x.po = sh.ex[1][lane]; x.rxa = sh.ex[2][lane]; x.xikr = sh.ex[3][lane];
            x.xik1 = sh.ex[4][lane]; x.xito = sh.ex[5][lane]; x.xinak = sh.ex[6][lane];
            x.xiks = sh.ex[7][lane]; x.jnaca = sh.ex[8][lane];
            R r0, r19;
            mh_totals(c, ist, x, r0, r19);
            if (e == 0) ten = act && mh_wants_substeps(r0, a.mh_abs);
            if (act && (e > 0) == ten) {
                auto own_states = [&](auto P) {
#pragma unroll
                    for (int k = 1; k < 26; k++)
                        if ((mh_part_states(P.value) >> k) & 1u) sh.s[k][lane] = s[k] + r[k] * he;
                };
                if (warp == 0) own_states(Part<0>{});
                else if (warp == 1) own_states(Part<1>{});
                else if (warp == 2) own_states(Part<2>{});
                else { mh_finish(s, c, x, own, r); own_states(Part<3>{}); }
                sv += r0 * he;
                nai += r19 * he;
                last = r0;
            }
            if (!__syncthreads_or(ten)) break;
        }
        if (act) {
            if (ten && warp == 0) my_newton++;
            const R v1 = V + h * last;
            if (do_track) track_update(tr, dirty, V, v1, tsub, h, a.act_thr);
            V = v1;
            tsub += (double)h;
            sub.took(a, last);
        }
    }
    if (on) {
        for (int k = warp; k < MH_NS; k += 4)
            if (k != 18) a.S[(size_t)k * a.pitch + i] = sh.s[k + 1][lane];
        if (warp == 0) {
            if (!isfinite((double)V)) my_bad = 1;
            if (a.dvdt_out) a.dvdt_out[i] = last;
            else a.V[i] = V;
            a.S[(size_t)18 * a.pitch + i] = nai;
            if (dirty) a.track[i] = tr;
        }
    }
    __syncthreads();                             // the next group's states overwrite these
}

template <typename R, int MINB>
__global__ void __launch_bounds__(128, MINB) k_mahajan(const IonicArgs<R> a, int chunks) {
    __shared__ unsigned long long s_newton;
    __shared__ unsigned int s_caps, s_bad;
    __shared__ MhShared<R> sh;
    if (threadIdx.x == 0) { s_newton = 0; s_caps = 0; s_bad = 0; sh.count = 0; }
    __syncthreads();
    unsigned int my_newton = 0, my_bad = 0;
    for (int m = 0; m < chunks; m++) {           // chunks <= kMhChunks
        const int i = (m * gridDim.x + blockIdx.x) * 128 + threadIdx.x;
        unsigned int none = 0;
        if (i < a.n && !(a.skip && a.skip[i]) && !ionic_node<R, EP_MAHAJAN, MH_NS>(a, i, none, none, my_bad))
            sh.list[atomicAdd(&sh.count, 1)] = i;
    }
    __syncthreads();
    const int count = sh.count;
    if (sizeof(R) == 8 && count >= kMhMany) {
        unsigned int none = 0;
        for (int k = threadIdx.x; k < count; k += 128)
            ionic_node<R, EP_MAHAJAN, MH_NS, sizeof(R) == 8>(a, sh.list[k], my_newton, none, my_bad);
    } else {
        for (int g = 0; g < count; g += 32) {
            const int k = g + (threadIdx.x & 31);
            mh_group(a, sh, sh.list[k < count ? k : g], k < count, my_newton, my_bad);
        }
    }
    ionic_status(a.status, my_newton, 0, my_bad, s_newton, s_caps, s_bad);
}

// MINB > 1 asks the compiler for MINB resident CTAs of 128 threads per SM
// (fewer registers, some spilled to L1)
template <typename R, int MODEL, int NS, int MINB>
__global__ void __launch_bounds__(128, MINB) k_ionic(const IonicArgs<R> a) {
    __shared__ unsigned long long s_newton;
    __shared__ unsigned int s_caps, s_bad;
    if (threadIdx.x == 0) { s_newton = 0; s_caps = 0; s_bad = 0; }
    __syncthreads();
    unsigned int my_newton = 0, my_caps = 0, my_bad = 0;
    // every node or the fallback list of the learned step (the nodes it
    // could not take).  One call site, so both modes run the same machine
    // code and a node's result does not depend on which mode advanced it.
    const int cnt = a.node_list ? *a.list_count : a.n;
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < cnt; k += gridDim.x * blockDim.x) {
        const int node = a.node_list ? a.node_list[k] : k;
        if (a.skip && a.skip[node]) continue;
        ionic_node<R, MODEL, NS>(a, node, my_newton, my_caps, my_bad);
    }
    ionic_status(a.status, my_newton, my_caps, my_bad, s_newton, s_caps, s_bad);
}

template <typename R, int MINB>
static void dispatch_ionic(int model, const IonicArgs<R> &a, int grid, int block, int nsm, cudaStream_t st) {
    switch (model) {
    case EP_TUSSCHER:
        if (a.tt.jac_true && !a.ref_order) k_ionic<R, EP_TUSSCHER, TT_NS, MINB><<<grid, block, 0, st>>>(a);
        else k_ionic<R, kTusscherRef, TT_NS, MINB><<<grid, block, 0, st>>>(a);
        break;
    case EP_MAHAJAN:
    case EP_MAHAJAN_FAIL:
        {
            // one wave of CTAs, as evenly filled as whole chunks allow
            const int n128 = div_up(a.n, 128);
            const int chunks = std::min(kMhChunks, std::max(1, div_up(n128, nsm * (MINB > 1 ? MINB : 2))));
            k_mahajan<R, MINB><<<div_up(n128, chunks), 128, 0, st>>>(a, chunks);
        }
        break;
    case EP_PURKINJE:
        k_ionic<R, EP_PURKINJE, PK_NS, MINB><<<grid, block, 0, st>>>(a);
        break;
    default:
        k_ionic<R, EP_LUORUDY, LR_NS, 1><<<grid, block, 0, st>>>(a);
        break;
    }
}

template <typename R>
int launch_ionic(int model, const IonicArgs<R> &a, cudaStream_t st, int block, int min_ctas) {
    if (block != 64 && block != 128) { set_error("ionic block must be 64 or 128"); return EP_ERR_ARG; }
    if (min_ctas != 0 && min_ctas != 3 && min_ctas != 4) { set_error("ionic min_ctas must be 0, 3 or 4"); return EP_ERR_ARG; }
    if (model != EP_TUSSCHER && model != EP_MAHAJAN && model != EP_MAHAJAN_FAIL && model != EP_LUORUDY &&
        model != EP_LUORUDYWITHGATE && model != EP_PURKINJE) {
        set_error("unknown model %d", model);
        return EP_ERR_ARG;
    }
    int grid = div_up(a.n, block);
    if (a.n == 0) return EP_OK;
    int dev = 0, nsm = 148;
    EP_CUDA(cudaGetDevice(&dev));
    EP_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
    // a list's length is only known on the device: a fixed grid strides over it,
    // no larger than what is resident at once (ten Tusscher and Purkinje)
    if (a.node_list) grid = std::min(grid, 4 * nsm);
    if constexpr (sizeof(R) == 8) {
        dispatch_ionic<R, 1>(model, a, grid, block, nsm, st);       // FP64: the compiler's register choice
    } else {
        // the library's choice: four resident CTAs for ten Tusscher (128
        // registers; 24-slab batch 58 us a step against 62 with three and 77
        // unbounded), three for the others (Mahajan, 214K nodes: 41 us against
        // 43; four spill)
        // unbounded, without spills, for the reference's order of operations where
        // two CTAs an SM take all nodes at once (28.6K nodes: 42.6 us against 44.9
        // with four; 214K, two waves of two: 241 against 139)
        const bool wave = model == EP_TUSSCHER && (!a.tt.jac_true || a.ref_order) && a.n <= 2 * 128 * nsm;
        if (min_ctas == 0 && wave) {
            k_ionic<R, kTusscherRef, TT_NS, 1><<<grid, block, 0, st>>>(a);
            EP_CUDA(cudaGetLastError());
            return EP_OK;
        }
        if (min_ctas == 0) min_ctas = model == EP_TUSSCHER ? 4 : 3;
        if (min_ctas == 3) dispatch_ionic<R, 3>(model, a, grid, block, nsm, st);
        else dispatch_ionic<R, 4>(model, a, grid, block, nsm, st);
    }
    EP_CUDA(cudaGetLastError());
    return EP_OK;
}

template int launch_ionic<float>(int, const IonicArgs<float> &, cudaStream_t, int, int);
template int launch_ionic<double>(int, const IonicArgs<double> &, cudaStream_t, int, int);

}  // namespace ep
